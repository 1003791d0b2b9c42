// Role-masked chunked flash-attention prefill for sm_100a: TMA-fed tcgen05.mma with TMEM accumulators.
//
// A work item = one 128-row query tile x one kv-head x up to two query heads of that kv-head's group.  The two heads
// share every K/V tile that is loaded.  S = Q.K^T of a step (tile, head) is read into registers at once, P has TMEM columns of its
// own: the tensor core computes the next scores and O += P.V of earlier steps while the softmax warps of both heads work.
// The kernel is persistent: one CTA per SM takes items from a global counter (heaviest query tiles first).
//
//   warp 0      TMA producer: K and V of every kept KV tile, item after item, through one ring of tile-sized slots, and what the
//               softmax warps need to know about a tile (which one it is, which masks it needs, the row limits of its columns)
//   warp 3      scheduler: fetches the next item, builds its kept-tile bitmap while the current item runs, loads its Q tiles
//   warp 1      MMA issuer (one lane) of S = Q_h.K^T (SS, N = 128), warp 2 of O_h += P_h.V (TS, P from TMEM)
//   warps 4-7   softmax of head slot 0: one thread per query row, the 128-entry score row read with tcgen05.ld, online
//   warps 8-11  softmax of head slot 1  softmax in registers, P written to TMEM as packed bf16
//
// Chunks finer than a tile: far behind the queries only the global chunks are still visible, a few in every tile.  Those
// are not computed in place but gathered: the keys of 128 / C listed chunks (FarLists) make a full tile.  Chunks of 8 rows and
// more are copied chunk by chunk (boxes of C rows); finer ones come from a copy of the listed rows in the workspace, made once
// per call (far_rows_kernel), since single rows arrive at ~8 cycles each from tile::gather4, 4000 for a K / V tile pair.  The
// bitmap then only holds the tiles from the first one on in which some other chunk is still visible, and dense ones in front of
// it: a tile nearly all of whose chunks are listed is cheaper in place (see far_dense_min).  The work of a query
// tile falls from the tiles that hold a visible key towards the keys that are visible: prompt of 8192 tokens with one role
// per token, 10 % global, 0.91 -> 0.21 ms (0.29 with tile::gather4); forward of 8 x 4096 tokens with chunks of 16, 0.51 -> 0.26 ms.
// Which KV tiles are visited comes from the role bitmap: a bitmap of kept tiles is built in shared memory from the
// per-tile max / min row limits (nats_b200_role_prep); tiles without a visible entry are never loaded.  Only tiles
// whose min limit does not cover the whole query tile (and the diagonal) pay for per-element masking.
//
// TMEM (512 columns): see PrefillTmem.  Every mbarrier wait is bounded: on a time-out the CTA raises the caller's status
// word, drains and exits.
#include <cuda.h>

#include "common.cuh"

namespace nats {

constexpr int kPrefillThreads = 384;
#ifndef NATS_REGS_LOW
#define NATS_REGS_LOW 72
#endif
#ifndef NATS_REGS_HIGH
#define NATS_REGS_HIGH 216
#endif
// setmaxnreg split: 128 * low + 256 * high must not exceed the 384 * 168 registers of the launch
constexpr int kRegsLow = NATS_REGS_LOW, kRegsHigh = NATS_REGS_HIGH;
static_assert(128 * kRegsLow + 256 * kRegsHigh <= 384 * 168, "setmaxnreg budget");
constexpr uint32_t kBoxBytes = 128 * 64 * 2;            // one TMA box: 128 rows x 64 bf16, 128-byte swizzled
#ifndef NATS_RELAX_NS
#define NATS_RELAX_NS 200
#endif
constexpr int kRelaxNs = NATS_RELAX_NS;
#ifndef NATS_RELAX_PROD_NS
#define NATS_RELAX_PROD_NS 0
#endif
constexpr int kRelaxProdNs = NATS_RELAX_PROD_NS;
constexpr float kRescaleThreshold = 8.0f;               // log2 units: O is rescaled only when the row max grows by more
#ifndef NATS_WAIT_LIMIT_NS
#define NATS_WAIT_LIMIT_NS (400ull * 1000ull * 1000ull)
#endif
constexpr unsigned long long kWaitLimitNs = NATS_WAIT_LIMIT_NS;

enum : int { kErrQ = 1, kErrKvFull, kErrKvEmpty, kErrSFull, kErrPFull, kErrOFull, kErrList, kErrOEmpty, kErrSmemAlign, kErrPipeLock, kErrSEmpty };

struct PrefillParams {
    void* o;                          // [B,Hq,N,D], or with the heads inside the tokens [B,N,Hq,D]: strides in elements
    long long o_batch, o_head, o_row;
    int o_f32;                        // 0: bf16, 1: fp32
    float* lse;                       // [B,Hq,N] or nullptr: log2 of the row's sum of exp2(score * scale * log2 e)
    const int32_t* lim;               // [B,Hkv,Nc]: last query POSITION that may see KV chunk c
    const int32_t* tile_max;          // [B,Hkv,Ntk]: max / min of lim over the chunks of a 128-row KV tile
    const int32_t* tile_min;
    // chunks visible for good (see FarLists), or all nullptr: the tiles in front of the first tile with another visible chunk
    // are not walked (but for the dense ones), their listed chunks are gathered into full tiles instead
    const int32_t* far_list;
    const int32_t* far_before;
    const int32_t* far_open;
    int far_cap, far_rows;            // chunks below 8 rows: rows of the copy in front of its tails, and with them; else 0
    int32_t* status;
    int32_t* work_counter;            // next work item; zero at launch (the role metadata kernel in front clears it)
    int total_items;                  // B * Hkv * n_groups * Nt
    // N query rows; query row i sits at position q_off + i of the KV sequence of Nkv rows (a first call has q_off = 0 and
    // Nkv = N; a call over an existing cache attends to the cache rows in front of its own tokens).
    // Nc / Ntk: chunks / 128-row tiles of the KV sequence, Nt: query tiles.
    int Hq, Hkv, N, Nkv, q_off, C, Nc, Nt, Ntk, nrep, n_groups;   // n_groups = ceil(nrep / heads per item)
    int c_shift;                      // log2(C), -1 if C is no power of two

    float scale_log2;
};

// ---- PTX wrappers -------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t sm_cycles() {         // wraps every 2.2 s at 1965 MHz
    uint32_t t;
    asm volatile("mov.u32 %0, %clock;" : "=r"(t));
    return t;
}
// Bounded wait.  Returns false when the wait was given up (by this thread or, earlier, by another one of the CTA).
// With abort_flag == nullptr only the time limit ends the wait (used to drain copies after the CTA has given up).
// RELAX > 0: sleep that many nanoseconds between polls (roles that run ahead of the critical path and should not take
// issue slots from the softmax warps of their scheduler).  Every lane of a waiting warp polls: letting one lane poll and
// broadcast the result was measured 25 % slower for the whole kernel.
template <int RELAX = 0>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int32_t* status, int code) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
#pragma unroll 1
    for (uint32_t it = 0;; ++it) {
        if (RELAX > 0) __nanosleep(RELAX);
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 63u) {
            if (abort_flag != nullptr && *abort_flag) return false;
            if (global_ns() - t0 > kWaitLimitNs) {
                if (abort_flag != nullptr) *abort_flag = 1;
                atomicCAS(status, 0, code);
                return false;
            }
        }
    }
}

// L2 eviction priority of a TMA load: K / V tiles are read again by the CTAs that work on neighbouring query tiles and
// should stay, Q tiles are read once
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "l"(policy) : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc], and the above, with the descriptors given as (low word, shared high word): within one kernel only
// the start address and the leading byte offset (low word) differ between operands, so the issuing thread adds small constants to 32-bit
// registers instead of carrying 64-bit descriptors around.  ACC is a compile-time flag so that no predicate has to be computed per MMA.
template <int ACC>
__device__ __forceinline__ void mma_ss_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "n"(ACC) : "memory");
}
template <int ACC>
__device__ __forceinline__ void mma_ts_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(desc_hi), "r"(idesc), "n"(ACC) : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp gets its lane's columns
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr),
          "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr),
          "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// 32-byte store (one sector) to a 32-byte aligned global address
__device__ __forceinline__ void st32(void* p, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// ---- descriptors ----------------------------------------------------------------------------------
// Shared-memory matrix descriptor of a 128-byte swizzled tile whose rows are 128 bytes (what one TMA box leaves):
// start address >> 4 in [0,14), leading byte offset >> 4 in [16,30), stride byte offset >> 4 in [32,46),
// descriptor version 1 in [46,48), swizzle mode 2 (128 B) in [61,64).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) | ((uint64_t)(sbo_bytes >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
// Instruction descriptor, kind::f16: fp32 accumulate, bf16 A and B, A K-major, B K-major or MN-major, M = 128.
__host__ __device__ constexpr uint32_t instr_desc(int n, bool b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// packed fp32 pairs: one instruction for two lanes of a multiply-add or add
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// ---- shared memory --------------------------------------------------------------------------------
struct ItemHeader {
    int valid;      // 0: no more work; else 1 + the KV tile in front of which the keys are gathered
    int t;          // query tile
    int b, bh;      // batch index, b * Hkv + kv-head
    int head0;      // query head of slot 0
    int nslots;     // 1 or 2 query heads in this item
    int n_kept;     // 128-column KV tiles: gathered ones first, then the kept tiles of the bitmap
    int far_keys;   // keys of the gathered tiles (the last one may be part empty)
};

constexpr int kBitWords = kMaxTiles / 32;
constexpr int kTailRows = 8;    // rows of the smallest box: 128 bytes each, one swizzle atom

// K/V ring: slots of one 128-row tile each, filled in the order K_0 V_0 K_1 V_1 ... of the kept tiles (all items in
// one sequence).  A K slot is free again when both heads' Q.K^T of that tile have completed, a V slot after both P.V.
template <int D>
struct PrefillSmem {
    static constexpr int kHeads = D <= 128 ? 2 : 1;      // query heads of an item (head_dim 256: O fills the TMEM of one head pair)
    static constexpr int kSlots = D == 256 ? 2 : D == 128 ? 5 : 8;
    static constexpr uint32_t kTileBytes = 128 * D * 2;
    uint8_t q[kHeads][kTileBytes];             // one Q tile per head slot; D/64 boxes of 16 KB each
    uint8_t ring[kSlots][kTileBytes];          // K or V tile; D/64 boxes of 16 KB each
    uint32_t keep[2][kBitWords];               // bit kt: KV tile kt of the item has a visible entry (double buffered)
    // what the softmax warps need to know about a tile, from the producer: (tile << 2) | kLimits | kCausal (a gathered tile: tile -1),
    // and with kLimits the row limit of each of its columns
    // A softmax warp reads an entry behind its arrival at bar_s_empty, so that a finished Q.K^T does not show that the entry has been read; a
    // finished P.V does, since it needed the P of both heads.  When the producer writes the entry of tile T it has waited for the slots of
    // K_T and of V_(T-1), one of which held V_(T - kSlots/2 - 1): entries of tiles up to that one are free.
    static constexpr int kMetas = D == 128 ? 3 : 8;
    static_assert(kMetas >= kSlots / 2 + 1, "an entry could be overwritten before the softmax warps have read it");
    alignas(16) int32_t limits[kMetas][kTile];
    int32_t tile[kMetas];
    ItemHeader item[2];
    unsigned long long bar_q_full[2], bar_q_empty[2];          // per head slot: its Q tile has landed / its last Q.K^T of the item is done
    unsigned long long bar_full[kSlots], bar_empty[kSlots];
    unsigned long long bar_s_full[2], bar_s_empty[2];          // per head slot / per score buffer
    unsigned long long bar_p_full[2], bar_o_full[2], bar_o_empty[2];
    unsigned long long bar_list_full[2], bar_list_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(ItemHeader) == 32, "a ninth word, loaded by every warp per item, made the kernel 1 to 1.5 % slower");
static_assert(sizeof(PrefillSmem<128>) <= 232448 && sizeof(PrefillSmem<256>) <= 232448, "shared memory of the widest kernels");

// TMEM columns: O of each head slot, one score buffer for all steps (what 512 columns hold at head_dim 128; at 256 there is one head)
// or one per head slot, P (bf16) of each head slot
template <int D>
struct PrefillTmem {
    static constexpr uint32_t kScoreBufs = D == 64 ? 2 : 1;
    static constexpr uint32_t kHeads = D <= 128 ? 2 : 1;
    static __device__ __forceinline__ uint32_t o(uint32_t h) { return h * D; }
    static __device__ __forceinline__ uint32_t s(uint32_t b) { return kHeads * D + b * 128; }
    static __device__ __forceinline__ uint32_t p(uint32_t h) { return kHeads * D + kScoreBufs * 128 + h * 64; }
};

constexpr int kListConsumers = 1 + 2 + 8;     // producer, two issuers, one lane of each of the eight softmax warps

enum : int { kCausal = 1, kLimits = 2 };      // some column of the tile lies behind some row / a chunk's row limit cuts through the tile

// Walks the set bits of an item's kept-tile bitmap in ascending order.
struct TileWalk {
    const uint32_t* keep;
    int w;
    uint32_t cur;
    __device__ __forceinline__ void init(const uint32_t* k) { keep = k; w = 0; cur = k[0]; }
    // next kept tile; the caller asks for no more tiles than the item has
    __device__ __forceinline__ int next() {
        while (cur == 0u) cur = keep[++w];
        const int b = __ffs(cur) - 1;
        cur &= cur - 1u;
        return w * 32 + b;
    }
};

// A bounded wait whose outcome is the same for every lane of the warp (all 32 lanes call it): lanes may see a time-out
// or the CTA's abort flag at different polls, and what follows (.sync.aligned instructions, __syncwarp) needs the
// whole warp on one path.
template <int RELAX = 0>
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int32_t* status, int code) {
    const bool ok = mbar_wait<RELAX>(bar, parity, abort_flag, status, code);
    return __all_sync(0xffffffffu, ok);
}
// The same for the softmax warps, whose code has to stay short: a loop around the look, the SM's cycle counter as the clock, and what
// follows a time-out in a function of its own.  They wait about twice as long as the other warps (0.8 s at 1965 MHz): where a softmax
// warp waits for an issuer that waits in turn, the status names the issuer's wait.  Behind the last item of a CTA nobody else is left to
// give up: the epilogue's wait for the last P.V ends by this limit only.  A look in front of the loop saves the others reading the clock;
// with FINE the shorter code is worth more: us per call, a limit on the number of looks (none in time) / this with / this without the look in
// front, forward of 8 x 4096 tokens with chunks of 16 187.8 / 189.9 / 182.4, 32k tokens with chunks of 128 1053 / 1048 / 1061, 8 x 15001
// 3211 / 3200 / 3240, 2 x 131k 19270 / 19260 / 19290.
constexpr uint32_t kSoftmaxWaitCycles = (uint32_t)(4 * kWaitLimitNs);
static_assert(4 * kWaitLimitNs < (1ull << 32), "the cycle counter is read with 32 bits");
__device__ __noinline__ bool give_up(volatile int* abort_flag, int32_t* status, int code) {
    if (*abort_flag == 0) {
        *abort_flag = 1;
        atomicCAS(status, 0, code);
    }
    return false;
}
template <bool FINE>
__device__ __forceinline__ bool warp_wait_short(uint32_t bar, uint32_t parity, volatile int* abort_flag, int32_t* status, int code) {
    if (!FINE && __builtin_expect(__all_sync(0xffffffffu, mbar_try_wait(bar, parity)), 1)) return true;
    const uint32_t t0 = sm_cycles();
#pragma unroll 1
    do {
        if (__builtin_expect(__all_sync(0xffffffffu, mbar_try_wait(bar, parity)), 1)) return true;
    } while (__all_sync(0xffffffffu, sm_cycles() - t0 < kSoftmaxWaitCycles && *abort_flag == 0));
    return give_up(abort_flag, status, code);
}

// Waits of the producer, the issuers and the scheduler: a look and a branch in their code, the loop is a function of its own.
__device__ __noinline__ bool util_wait_loop(uint32_t bar, uint32_t parity, volatile int* abort_flag, int32_t* status, int code, bool relax) {
    return __all_sync(0xffffffffu, relax ? mbar_wait<kRelaxNs>(bar, parity, abort_flag, status, code) : mbar_wait(bar, parity, abort_flag, status, code));
}
template <int RELAX = 0>
__device__ __forceinline__ bool util_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int32_t* status, int code) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return util_wait_loop(bar, parity, abort_flag, status, code, RELAX > 0);
}

// Persistent kernel: every CTA takes work items (query tile x kv-head x head pair) from a global counter until none is
// left.  Per-item set-up (kept-tile bitmap, Q load) and tear-down (O -> global) overlap the main loops of the
// neighbouring items: warp 3 prepares the bitmap of the next item while the current one runs, the producer streams the
// next item's K/V through the same ring without a bubble, Q of the next item is loaded as soon as the last Q.K^T of the
// current one has completed, and a head's epilogue only delays that head's own chain.
//
// Per step (kept tile j, head):  S = Q.K_j^T (D / 16 MMAs of N = 128)  ->  the 128-entry score row in registers, S free for the next
// step's scores  ->  softmax  ->  P (bf16) in columns of its own, free since P.V_{j-1}  ->  O += P.V_j.  Q.K^T needs only free scores,
// P.V only P: two issuers, each in step order, nothing else orders the MMAs.  (With P over S and a head's P.V_j and Q.K_{j+1}^T queued
// as one batch a head's chain was softmax, then batch, 4317 cycles a tile for 2048 of MMAs; now 2873.)
//
// What binds it now is the pipes and what stands between them: MUFU 70 % and tensor pipe 69 % busy on a small case with chunks of 128, 50 % and 25 %
// with chunks of 16, where masks take as long as a third of the softmax.  Instruction fetch bound it before: the warps of both heads stream
// through a tile's straight-line code at different places, next to the issuer of their scheduler, and spent 1.5 to 2.4 warps per issue in
// stalls for instructions (now 0.3).  So the code is kept short: the heads of an issuer in a rolled loop and waits as a look and a branch,
// rows masked by one compare per column with limits that the producer leaves in shared memory, the epilogue in pieces of 32 columns.
// us per launch, P over S / the above without the short code / with it: 32k tokens 1258 / 1185 / 1075, 2 x 131k 23394 / 21175 / 19370,
// 8 x 15001 3804 / 3684 / 3257, 8192 tokens with one role per token 179 / 195 / 144, 8 x 4096 with chunks of 16 237 / 288 / 195.  Then
// one compare per column for limits and diagonal together where 32 columns lie in one chunk (1065 -> 1053, 19600 -> 19130, 3260 -> 3215),
// MMAs in a loop with FINE (144 -> 142, 195 -> 187), waits without a look in front of their loop with FINE (142 -> 141, 188 -> 182).
//
// FINE: chunks that are not a multiple of 32 keys, or gathered tiles.  Without it the loops carry neither the masks column by column
// nor the gathered tiles.
template <int D, bool FINE>
__global__ void __launch_bounds__(kPrefillThreads, 1)
prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
               const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_k_far,
               const __grid_constant__ CUtensorMap map_v_far, const __grid_constant__ CUtensorMap map_k_copy,
               const __grid_constant__ CUtensorMap map_v_copy, const PrefillParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    using Smem = PrefillSmem<D>;
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    constexpr int NBOX = D / 64;                       // TMA boxes per tile
    constexpr int NS = Smem::kSlots;
    using TM = PrefillTmem<D>;
    constexpr uint32_t SB = TM::kScoreBufs;
    constexpr uint32_t TILE_BYTES = Smem::kTileBytes;  // one Q, K or V tile (128 rows)
    constexpr uint32_t IDESC_QK = instr_desc(kTile, false);
    constexpr uint32_t IDESC_PV = instr_desc(D, true);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    volatile int* abort_flag = &sm.abort_flag;

    if (tid == 0) {
        int bad = (*reinterpret_cast<volatile int32_t*>(p.status) != 0);
        if ((smem_u32(smem_raw) & 1023u) != 0u) {      // the swizzled tiles need a 1024-byte aligned base
            atomicCAS(p.status, 0, kErrSmemAlign);
            bad = 1;
        }
        sm.abort_flag = bad;
    }
    __syncthreads();
    if (sm.abort_flag) return;                         // an earlier CTA gave up: do not start (uniform for the CTA)

    // ---- set-up: barriers, TMEM ----
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(smem_u32(&sm.bar_full[s]), 1);
            mbar_init(smem_u32(&sm.bar_empty[s]), 1);
        }
        for (int h = 0; h < 2; ++h) {
            mbar_init(smem_u32(&sm.bar_q_full[h]), 1);
            mbar_init(smem_u32(&sm.bar_q_empty[h]), 1);              // one arrival per item that uses the head slot
            mbar_init(smem_u32(&sm.bar_s_full[h]), 1);
            mbar_init(smem_u32(&sm.bar_s_empty[h]), 4);            // one arrival per softmax warp
            mbar_init(smem_u32(&sm.bar_p_full[h]), 4);
            mbar_init(smem_u32(&sm.bar_o_full[h]), 1);
            mbar_init(smem_u32(&sm.bar_o_empty[h]), 4);
            mbar_init(smem_u32(&sm.bar_list_full[h]), 1);
            mbar_init(smem_u32(&sm.bar_list_empty[h]), kListConsumers);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        prefetch_tmap(&map_q);
        prefetch_tmap(&map_k);
        prefetch_tmap(&map_v);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&sm.tmem_base), 512);
        tmem_relinquish();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem_base;

    // Register budget: the softmax warpgroups get more registers (setmaxnreg.inc at the top of their branch), the
    // producer / issuer / scheduler warpgroup needs little and gives registers back.
    if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsLow));      // one site for the whole warpgroup

    if (warp == 3) {
        // =============================== scheduler: next work item and its kept-tile bitmap ===============================
        const int per_z = p.Nt * p.Hkv * p.n_groups;
        bool ok = true;
        int q_loads[2] = {0, 0};
        const uint64_t pol_q = l2_policy_evict_first();
        for (int ic = 0; ok; ++ic) {
            const int slot = ic & 1, use = ic >> 1;
            if (use > 0) ok = util_wait<kRelaxNs>(smem_u32(&sm.bar_list_empty[slot]), (use - 1) & 1, abort_flag, p.status, kErrList);
            if (!ok) break;
            int w = 0;
            if (lane == 0) w = atomicAdd(p.work_counter, 1);
            w = __shfl_sync(0xffffffffu, w, 0);
            const bool have = w < p.total_items;
            int n_kept = 0;
            if (have) {
                const int z = w / per_z, rem = w - z * per_z;
                const int y = rem / p.Nt, x = rem - y * p.Nt;
                const int t = p.Nt - 1 - x;                        // heavy (late) query tiles first
                const int grp = y % p.n_groups, hkv = y / p.n_groups;
                const int bh = z * p.Hkv + hkv;
                // positions of the first and last query row of the tile; KV tiles up to the one holding the last row
                const int q_lo = p.q_off + t * kTile, q_hi = p.q_off + min(t * kTile + kTile, p.N) - 1;
                const int kt_last = q_hi / kTile;
                const int32_t* tmax = p.tile_max + (size_t)bh * p.Ntk;
                // The tiles in front of near_first hold no visible chunk but listed ones: only the dense ones among them, whose chunks
                // are not gathered, stay in the bitmap.  near_first <= the tile of the first query row, so every listed key in
                // front of it is in that row's past.
                const int32_t* open = FINE && p.far_open != nullptr ? p.far_open + (size_t)bh * p.Ntk : nullptr;
                const int near_cap = q_lo / kTile;
                int near_first = open != nullptr ? -1 : 0;
                for (int s0 = 0; s0 <= kt_last; s0 += 32) {        // tiles 0..kt_last with a visible entry
                    const int kt = s0 + lane;
                    const bool keep = kt <= kt_last && tmax[kt] >= q_lo;
                    unsigned m = __ballot_sync(0xffffffffu, keep);
                    if (near_first < 0) {
                        const int o = kt <= near_cap ? open[kt] : 0;
                        const unsigned om = __ballot_sync(0xffffffffu, kt <= near_cap && (kt == near_cap || (o >> 1) >= q_lo));
                        if (om != 0u) near_first = s0 + __ffs(om) - 1;
                        const unsigned in_place = __ballot_sync(0xffffffffu, o & 1) | (om != 0u ? 0xffffffffu << (near_first - s0) : 0u);
                        m &= in_place;
                    }
                    if (lane == 0) sm.keep[slot][s0 >> 5] = m;
                    n_kept += __popc(m);
                }
                int far_keys = 0;
                if (open != nullptr) {
                    far_keys = p.far_before[(size_t)bh * (p.Ntk + 1) + near_first] * p.C;
                    n_kept += (far_keys + kTile - 1) / kTile;
                }
                if (lane == 0) {
                    ItemHeader hd;
                    hd.valid = 1 + max(near_first, 0); hd.t = t; hd.b = z; hd.bh = bh; hd.head0 = hkv * p.nrep + grp * Smem::kHeads;
                    hd.nslots = min(Smem::kHeads, p.nrep - grp * Smem::kHeads); hd.n_kept = n_kept; hd.far_keys = far_keys;
                    sm.item[slot] = hd;
                }
            } else if (lane == 0) {
                sm.item[slot].valid = 0;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sm.bar_list_full[slot]));
            if (!have) break;
            // Q of this item, head slot by head slot: a slot is reloaded as soon as that head's last Q.K^T of the previous
            // item has completed (the K/V producer is not held up by it, and one head does not wait for the other)
            const ItemHeader hd = sm.item[slot];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!ok) break;
                // only a slot that held a query head before is waited for, and an empty one never arrives: the issuer of an
                // empty slot may run a whole item ahead of the other one, so that an arrival per item would complete the
                // barrier twice before this warp looks at it, and the wait for the older phase would not end
                if (h < hd.nslots) {
                    if (q_loads[h] > 0) ok = util_wait<kRelaxNs>(smem_u32(&sm.bar_q_empty[h]), (q_loads[h] - 1) & 1, abort_flag, p.status, kErrQ);
                    if (!ok) break;
                    if (lane == 0) {
                        mbar_expect_tx(smem_u32(&sm.bar_q_full[h]), TILE_BYTES);
                        for (int x = 0; x < NBOX; ++x)
                            tma_load_3d(smem_u32(&sm.q[h][x * kBoxBytes]), &map_q, smem_u32(&sm.bar_q_full[h]), x * 64, hd.t * kTile,
                                        hd.b * p.Hq + hd.head0 + h, pol_q);
                    }
                    ++q_loads[h];
                }
                __syncwarp();
            }
        }
        if (!ok) {
            // given up: let Q copies that are still in flight land before the shared memory is released
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (q_loads[h] > 0) mbar_wait(smem_u32(&sm.bar_q_full[h]), (q_loads[h] - 1) & 1, nullptr, p.status, kErrQ);
        }
    } else if (warp == 0) {
        // =============================== TMA producer ===============================
        uint32_t g = 0;                                 // ring slots filled so far (all items): two per kept tile
        int meta = 0;                                   // entry of the next tile
        const uint64_t pol_kv = l2_policy_evict_last();
        bool ok = true;
        for (int ic = 0; ok; ++ic) {
            const int slot = ic & 1;
            ok = util_wait(smem_u32(&sm.bar_list_full[slot]), (ic >> 1) & 1, abort_flag, p.status, kErrList);
            if (!ok) break;
            const ItemHeader hd = sm.item[slot];
            if (!hd.valid) break;
            TileWalk walk;
            walk.init(sm.keep[slot]);
            const int n_far = (hd.far_keys + kTile - 1) / kTile;
            // Looked up a tile ahead, while the producer waits for a ring slot: which tile comes next, whether its rows need masks,
            // and the row limits of its columns lane, 32 + lane, ...
            const int q_lo = p.q_off + hd.t * kTile, q_hi = p.q_off + min(hd.t * kTile + kTile, p.N) - 1;
            const int32_t* lim = p.lim + (size_t)hd.bh * p.Nc;
            const int32_t* tmin = p.tile_min + (size_t)hd.bh * p.Ntk;
            int next_tile = 0, next_min = 0;
            int32_t next_lim[4];
            auto look_up = [&](int j) {
                if (FINE && j < n_far) return;
                next_tile = walk.next();
                next_min = tmin[next_tile];
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const int col = next_tile * kTile + 32 * w + lane;
                    next_lim[w] = col < p.Nkv ? lim[!FINE || p.c_shift >= 0 ? col >> p.c_shift : col / p.C] : -1;
                }
            };
            look_up(0);
            const int32_t* far_list = p.far_list + (size_t)hd.bh * p.Nc;       // read only while n_far > 0
            for (int j = 0; j < hd.n_kept && ok; ++j) {
                const bool far = FINE && j < n_far;
                const int row0 = far ? j * kTile : next_tile * kTile;
                // Rows of a gathered tile: a box of 128 rows of the copy of the listed rows, or boxes of box_rows rows, the i-th
                // from lane i: a listed chunk where it lies, or (chunks below 8 rows, only for the part empty tile) eight rows
                // of the copy or its tail.  What lies behind the last listed key of the item is read as zero, from rows
                // behind the array: P is zero there, and 0 * V is zero only for a finite V, so no later key may stand there.
                const int far_left = hd.far_keys - j * kTile;
                const bool boxes = far && (p.far_cap == 0 || far_left < kTile);
                const int box_shift = far ? max(p.c_shift, 3) : 3, box_rows = 1 << box_shift, n_boxes = kTile >> box_shift;
                int box_row = 0;
                if (boxes) {
                    const int key = j * kTile + ((lane & (n_boxes - 1)) << box_shift);
                    if (p.far_cap == 0) box_row = key < hd.far_keys ? far_list[key >> box_shift] * box_rows : p.Nkv;
                    else box_row = key + box_rows <= hd.far_keys ? key : key < hd.far_keys ? p.far_cap + kTailRows * (hd.valid - 1) : p.far_rows;
                }
#pragma unroll 1
                for (int kv = 0; kv < 2 && ok; ++kv, ++g) {
                    const int s = g % NS;
                    if (g >= (uint32_t)NS) ok = util_wait<kRelaxProdNs>(smem_u32(&sm.bar_empty[s]), ((g / NS) & 1) ^ 1, abort_flag, p.status, kErrKvEmpty);
                    if (!ok) break;
                    if (kv == 0) {
                        // the ring slots of this K and of the V in front are free: so is the entry (see kMetas)
                        const int flags = far ? (far_left < kTile ? kCausal : 0)
                                              : (row0 + kTile - 1 > q_lo ? kCausal : 0) | (next_min < q_hi ? kLimits : 0);
                        if (flags & kLimits) {
#pragma unroll
                            for (int w = 0; w < 4; ++w) sm.limits[meta][32 * w + lane] = next_lim[w];
                        }
                        if (lane == 0) sm.tile[meta] = far ? -4 | flags : next_tile << 2 | flags;
                        meta = meta + 1 == Smem::kMetas ? 0 : meta + 1;
                        __syncwarp();
                    }
#ifdef NATS_TEST_WITHHOLD_FIRST_V
                    // test builds only: the V tile of a CTA's first kept tile is never loaded, so that a bounded wait runs out
                    const bool withhold = g == 1;
#else
                    const bool withhold = false;
#endif
                    if (lane == 0 && !withhold) {
                        mbar_expect_tx(smem_u32(&sm.bar_full[s]), TILE_BYTES);
                        if (!boxes) {
                            const CUtensorMap* map = kv == 0 ? (far ? &map_k_copy : &map_k) : (far ? &map_v_copy : &map_v);
                            for (int x = 0; x < NBOX; ++x)
                                tma_load_3d(smem_u32(&sm.ring[s][x * kBoxBytes]), map, smem_u32(&sm.bar_full[s]), x * 64, row0, hd.bh, pol_kv);
                        }
                    }
                    __syncwarp();
                    if (boxes && !withhold) {
                        const CUtensorMap* map = kv == 0 ? &map_k_far : &map_v_far;
                        const uint32_t dst = smem_u32(&sm.ring[s][0]), bar = smem_u32(&sm.bar_full[s]);
                        // n_boxes <= 16 divides 32: the lanes of a box share its parts of 64 columns
                        for (int x = lane / n_boxes; x < NBOX; x += 32 / n_boxes)
                            tma_load_3d(dst + x * kBoxBytes + (lane & (n_boxes - 1)) * box_rows * 128, map, bar, x * 64, box_row, hd.bh, pol_kv);
                        __syncwarp();
                    }
                }
                if (j + 1 < hd.n_kept) look_up(j + 1);
            }
            if (ok && lane == 0) mbar_arrive(smem_u32(&sm.bar_list_empty[slot]));
        }
        if (!ok) {
            // given up: let copies that are still in flight land before the shared memory is released
            for (uint32_t x = g > (uint32_t)NS ? g - NS : 0; x < g; ++x)
                mbar_wait(smem_u32(&sm.bar_full[x % NS]), (x / NS) & 1, nullptr, p.status, kErrKvFull);
        }
    } else if (warp == 1 || warp == 2) {
        // =============================== MMA issuers: warp 1 for S = Q.K^T, warp 2 for O += P.V ===============================
        // Each walks the steps (item, KV tile, head slot) in the same order and waits only for what its own MMAs read or
        // overwrite, so that Q.K^T of later steps runs beside the softmax and the P.V of earlier ones.
        // descriptors as (low word, high word): the high word (stride byte offset 1024, version, 128-byte swizzle) is the
        // same for Q, K and V; the low word holds the start address >> 4 and the leading byte offset >> 4
        constexpr uint32_t T16 = TILE_BYTES >> 4;
        const bool qk = warp == 1;
        const uint64_t q_desc = smem_desc(smem_u32(&sm.q[0][0]), 16, 1024);
        const uint64_t r_desc = smem_desc(smem_u32(&sm.ring[0][0]), qk ? 16 : kBoxBytes, 1024);
        const uint32_t desc_hi = (uint32_t)(q_desc >> 32);
        const uint32_t q_lo0 = (uint32_t)q_desc, r_lo0 = (uint32_t)r_desc;
        uint32_t g = 0;               // ring slots of the items so far
        uint32_t k = 0;               // steps so far (one score buffer)
        // tiles and items of head slot 0 / 1 so far: slot 1 has been empty in `gap` tiles and `skip` items
        uint32_t gt = 0, na = 0, gap = 0, skip = 0;
        bool ok = true;
        for (int ic = 0; ok; ++ic) {
            const int slot = ic & 1;
            ok = util_wait(smem_u32(&sm.bar_list_full[slot]), (ic >> 1) & 1, abort_flag, p.status, kErrList);
            if (!ok) break;
            const ItemHeader hd = sm.item[slot];
            if (!hd.valid) break;
            const int n = hd.n_kept, nslots = hd.nslots;
            if (qk) {
                for (int j = 0; j < n && ok; ++j) {
                    const uint32_t gk = g + 2 * j;                 // ring index of K_j
                    ok = util_wait(smem_u32(&sm.bar_full[gk % NS]), (gk / NS) & 1, abort_flag, p.status, kErrKvFull);
                    const uint32_t kl = r_lo0 + (gk % NS) * T16;
#pragma unroll 1
                    for (int h = 0; h < nslots && ok; ++h) {
                        const uint32_t items = na - (h ? skip : 0), tiles = gt + j - (h ? gap : 0);
                        if (j == 0) ok = util_wait(smem_u32(&sm.bar_q_full[h]), items & 1, abort_flag, p.status, kErrQ);
                        // the scores this step overwrites are in the registers of their softmax warps
                        const uint32_t sb = SB == 2 ? h : 0, use = SB == 2 ? tiles : k++;
                        if (ok && use > 0) ok = util_wait(smem_u32(&sm.bar_s_empty[sb]), (use - 1) & 1, abort_flag, p.status, kErrSEmpty);
                        if (!ok) break;
                        tc_fence_after();
                        if (lane == 0) {
                            // S[128 x 128] = Q_h[128 x D] . K_j[128 x D]^T : D/16 MMAs of K = 16
                            const uint32_t tS = tmem + TM::s(sb), ql = q_lo0 + (uint32_t)h * T16;
                            mma_ss_lo<0>(tS, ql, kl, desc_hi, IDESC_QK);
#pragma unroll
                            for (int ks = 1; ks < 4; ++ks) mma_ss_lo<1>(tS, ql + 2 * ks, kl + 2 * ks, desc_hi, IDESC_QK);
#pragma unroll(FINE ? 1 : 3)
                            for (int x = 1; x < NBOX; ++x) {
                                const uint32_t off = (uint32_t)x * (kBoxBytes >> 4);
#pragma unroll
                                for (int ks = 0; ks < 4; ++ks) mma_ss_lo<1>(tS, ql + off + 2 * ks, kl + off + 2 * ks, desc_hi, IDESC_QK);
                            }
                            tc_commit(smem_u32(&sm.bar_s_full[h]));
                            if (h == nslots - 1) tc_commit(smem_u32(&sm.bar_empty[gk % NS]));
                            if (j == n - 1) tc_commit(smem_u32(&sm.bar_q_empty[h]));
                        }
                        __syncwarp();
                    }
                }
            } else {
                for (int j = 0; j < n && ok; ++j) {
                    const uint32_t gv = g + 2 * j + 1;             // ring index of V_j
                    ok = util_wait(smem_u32(&sm.bar_full[gv % NS]), (gv / NS) & 1, abort_flag, p.status, kErrKvFull);
                    const uint32_t vl = r_lo0 + (gv % NS) * T16;
#pragma unroll 1
                    for (int h = 0; h < nslots && ok; ++h) {
                        const uint32_t items = na - (h ? skip : 0), tiles = gt + j - (h ? gap : 0);
                        // the first P.V of an item overwrites O_h: the previous item's epilogue must have read it
                        if (j == 0 && items > 0) ok = util_wait(smem_u32(&sm.bar_o_empty[h]), (items - 1) & 1, abort_flag, p.status, kErrOEmpty);
                        if (ok) ok = util_wait(smem_u32(&sm.bar_p_full[h]), tiles & 1, abort_flag, p.status, kErrPFull);
                        if (!ok) break;
                        tc_fence_after();
                        if (lane == 0) {
                            // O_h[128 x D] (+)= P_j[128 x 128 keys] . V_j[128 x D] : 8 MMAs of K = 16; V is MN-major (D contiguous)
                            const uint32_t tO = tmem + TM::o(h), tP = tmem + TM::p(h);
                            if (FINE) {
                                // two at a time: 8 x 4096 tokens, head_dim 64, chunks of 16 195 -> 187 us; with the larger tiles in place
                                // that are the rule without FINE all eight in a row are faster (32k tokens 1075 against 1107)
#pragma unroll 2
                                for (int ks = 0; ks < 8; ++ks)
                                    mma_ts(tO, tP + ks * 8, ((uint64_t)desc_hi << 32) | (vl + (uint32_t)(ks * (2048 >> 4))), IDESC_PV, j > 0 || ks > 0);
                            } else {
                                if (j == 0) mma_ts_lo<0>(tO, tP, vl, desc_hi, IDESC_PV);
                                else mma_ts_lo<1>(tO, tP, vl, desc_hi, IDESC_PV);
#pragma unroll
                                for (int ks = 1; ks < 8; ++ks) mma_ts_lo<1>(tO, tP + ks * 8, vl + (uint32_t)(ks * (2048 >> 4)), desc_hi, IDESC_PV);
                            }
#ifdef NATS_TEST_WITHHOLD_LAST_O
                            // test builds only: the end of an item's last P.V is never told, so that the epilogue's wait runs out
                            if (j < n - 1)
#endif
                            tc_commit(smem_u32(&sm.bar_o_full[h]));
                            if (h == nslots - 1) tc_commit(smem_u32(&sm.bar_empty[gv % NS]));
                        }
                        __syncwarp();
                    }
                }
            }
            g += 2 * n;
            gt += n;
            ++na;
            if (nslots == 1) { gap += n; ++skip; }
            if (ok && lane == 0) mbar_arrive(smem_u32(&sm.bar_list_empty[slot]));
        }
    } else if (warp >= 4) {
        // =============================== softmax + epilogue ===============================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsHigh));
        const int h = (warp - 4) / 4;                    // head slot
        const int row = (warp & 3) * 32 + lane;          // query row inside the tile == TMEM lane
        const uint32_t lane_addr = ((uint32_t)((warp & 3) * 32)) << 16;
        const uint32_t sb = SB == 2 ? h : 0;             // score buffer
        const uint32_t tS = tmem + lane_addr + TM::s(sb);
        const uint32_t tP = tmem + lane_addr + TM::p(h);
        const uint32_t tO = tmem + lane_addr + TM::o(h);
        const float scale = p.scale_log2;
        const bool o_wide = (reinterpret_cast<uintptr_t>(p.o) & 31u) == 0;     // 32-byte stores need a 32-byte aligned output
        uint32_t gt = 0;                                 // tiles of this head so far
        int metas = 0;                                   // tiles of all items so far, modulo kMetas
        bool ok = true;
        for (int ic = 0; ok; ++ic) {
            const int slot = ic & 1;
            ok = warp_wait_short<FINE>(smem_u32(&sm.bar_list_full[slot]), (ic >> 1) & 1, abort_flag, p.status, kErrList);
            if (!ok) break;
            const ItemHeader hd = sm.item[slot];
            if (!hd.valid) break;
            if (h < hd.nslots) {
                const int n = hd.n_kept;
                const int qpos = p.q_off + hd.t * kTile + row;   // position of this thread's query row in the KV sequence
                float m_ref = -INFINITY, l_sum = 0.f;
                int meta = metas;
                for (int j = 0; j < n; ++j, ++gt) {
                    ok = warp_wait_short<FINE>(smem_u32(&sm.bar_s_full[h]), gt & 1, abort_flag, p.status, kErrSFull);
                    if (!ok) break;
                    tc_fence_after();
                    // the score row of this thread in registers: four loads in flight, one wait; the buffer is then free
                    uint32_t sreg[kTile];
#pragma unroll
                    for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&sreg[c * 32]));
                    tc_wait_ld();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&sm.bar_s_empty[sb]));
                    // masks: -inf, of which exp2 makes an exact 0
                    const int tile = sm.tile[meta];
                    if (FINE && (tile & kLimits)) {
                        const int32_t* limits = sm.limits[meta];
#pragma unroll
                        for (int i = 0; i < kTile; i += 4) {
                            const int4 l = *reinterpret_cast<const int4*>(limits + i);
                            if (qpos > l.x) sreg[i] = 0xff800000u;
                            if (qpos > l.y) sreg[i + 1] = 0xff800000u;
                            if (qpos > l.z) sreg[i + 2] = 0xff800000u;
                            if (qpos > l.w) sreg[i + 3] = 0xff800000u;
                        }
                    }
                    if (FINE ? tile & kCausal : tile & (kCausal | kLimits)) {
                        // the last column this row may see; the last gathered tile ends with the listed keys
                        const int last = FINE && tile < 0 ? hd.far_keys - j * kTile - 1 : qpos - (tile >> 2) * kTile;
#pragma unroll
                        for (int w = 0; w < 4; ++w) {
                            // without FINE 32 columns lie in one chunk
                            const int last_w = !FINE && (tile & kLimits) && qpos > sm.limits[meta][32 * w] ? -1 : last;
#pragma unroll
                            for (int i = 32 * w; i < 32 * w + 32; ++i) sreg[i] = i > last_w ? 0xff800000u : sreg[i];
                        }
                    }
                    meta = meta + 1 == Smem::kMetas ? 0 : meta + 1;
                    float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
                    for (int i = 0; i < kTile; i += 8) {
                        mx0 = max3(mx0, __uint_as_float(sreg[i]), __uint_as_float(sreg[i + 1]));
                        mx1 = max3(mx1, __uint_as_float(sreg[i + 2]), __uint_as_float(sreg[i + 3]));
                        mx2 = max3(mx2, __uint_as_float(sreg[i + 4]), __uint_as_float(sreg[i + 5]));
                        mx3 = max3(mx3, __uint_as_float(sreg[i + 6]), __uint_as_float(sreg[i + 7]));
                    }
                    const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * scale;       // scale > 0
                    // online softmax with lazy rescaling: the reference maximum only moves when the row max grew by > threshold
                    float alpha = 1.f;
                    bool need = false;
                    if (mx > m_ref + kRescaleThreshold) {           // also true for the first visible tile (m_ref = -inf)
                        if (m_ref != -INFINITY) {                   // a row without visible entries so far has O = 0, l = 0
                            alpha = ex2(m_ref - mx);
                            l_sum *= alpha;
                            need = true;
                        }
                        m_ref = mx;
                    }
                    if (j > 0 && __any_sync(0xffffffffu, need)) {
                        // O_h is rescaled in place, behind the P.V of the previous tile
                        ok = warp_wait_short<FINE>(smem_u32(&sm.bar_o_full[h]), (gt - 1) & 1, abort_flag, p.status, kErrOFull);
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll 1
                        for (int c = 0; c < D / 32; ++c) {
                            uint32_t r[32];
                            tmem_ld32(tO + c * 32, r);
                            tc_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
                            tmem_st32(tO + c * 32, r);
                        }
                    }
                    const float m_neg = (m_ref == -INFINITY) ? 0.f : -m_ref;
                    // P = exp2(S * scale - m), row sum in fp32, P packed to bf16
                    const uint64_t scale2 = pack2(scale, scale), mneg2 = pack2(m_neg, m_neg);
                    uint64_t ls2 = pack2(0.f, 0.f);
                    // the P.V of this head's previous tile must have read what is overwritten below: asked now, it has long ended
                    const bool pv_done = mbar_try_wait(smem_u32(&sm.bar_o_full[h]), (gt - 1) & 1);
                    uint32_t pk[kTile / 2];
#pragma unroll
                    for (int i = 0; i < kTile; i += 2) {
                        const uint64_t x2 = fma2(pack2(__uint_as_float(sreg[i]), __uint_as_float(sreg[i + 1])), scale2, mneg2);
                        float x0, x1;
                        unpack2(x2, x0, x1);
                        const float p0 = ex2(x0), p1 = ex2(x1);
                        ls2 = add2(ls2, pack2(p0, p1));
                        pk[i / 2] = pack_bf16(p0, p1);
                    }
                    if (__builtin_expect(!__all_sync(0xffffffffu, pv_done), 0)) {
                        ok = warp_wait_short<FINE>(smem_u32(&sm.bar_o_full[h]), (gt - 1) & 1, abort_flag, p.status, kErrOFull);
                        if (!ok) break;
                    }
                    tc_fence_after();
                    tmem_st32(tP, *reinterpret_cast<const uint32_t(*)[32]>(&pk[0]));
                    tmem_st32(tP + 32, *reinterpret_cast<const uint32_t(*)[32]>(&pk[32]));
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();                         // every lane's row of P is in TMEM and fenced
                    if (lane == 0) mbar_arrive(smem_u32(&sm.bar_p_full[h]));
                    {
                        float a, b;
                        unpack2(ls2, a, b);
                        l_sum += a + b;
                    }
                }
                // epilogue: O / l -> bf16 -> global; O_h is handed back to the issuer as soon as it sits in registers
                if (ok) ok = warp_wait_short<FINE>(smem_u32(&sm.bar_o_full[h]), (gt - 1) & 1, abort_flag, p.status, kErrOFull);
                if (ok) {
                    tc_fence_after();
                    const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
                    const int qi = hd.t * kTile + row;           // query row
                    const long long o_at = hd.b * p.o_batch + (hd.head0 + h) * p.o_head + qi * p.o_row;
                    __nv_bfloat16* orow = (__nv_bfloat16*)p.o + o_at;
                    constexpr int OW = 32;                         // columns of O held in registers at a time
                    if (p.lse != nullptr && qi < p.N)
                        p.lse[((size_t)hd.b * p.Hq + hd.head0 + h) * p.N + qi] = l_sum > 0.f ? m_ref + log2f(l_sum) : -INFINITY;
#pragma unroll 1
                    for (int c0 = 0; c0 < D; c0 += OW) {
                        uint32_t oreg[OW];
#pragma unroll
                        for (int c = 0; c < OW / 32; ++c) tmem_ld32(tO + c0 + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&oreg[c * 32]));
                        tc_wait_ld();
                        if (c0 + OW >= D) {                          // O_h is in registers: hand it back to the issuer
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(smem_u32(&sm.bar_o_empty[h]));
                        }
                        if (p.o_f32) {
                            if (qi < p.N) {
                                float* frow = (float*)p.o + o_at + c0;
#pragma unroll
                                for (int i = 0; i < OW; i += 8) {
                                    uint32_t w[8];
#pragma unroll
                                    for (int x = 0; x < 8; ++x) w[x] = __float_as_uint(__uint_as_float(oreg[i + x]) * inv);
                                    if (o_wide) {
                                        st32(frow + i, w);
                                    } else {
                                        st16(frow + i, make_uint4(w[0], w[1], w[2], w[3]));
                                        st16(frow + i + 4, make_uint4(w[4], w[5], w[6], w[7]));
                                    }
                                }
                            }
                        } else if (qi < p.N) {
                            // a thread owns a whole output row (D * 2 bytes): 32-byte stores, one full sector each
#pragma unroll
                            for (int i = 0; i < OW; i += 16) {
                                uint32_t w[8];
#pragma unroll
                                for (int x = 0; x < 8; ++x)
                                    w[x] = pack_bf16(__uint_as_float(oreg[i + 2 * x]) * inv, __uint_as_float(oreg[i + 2 * x + 1]) * inv);
                                if (o_wide) {
                                    st32(orow + c0 + i, w);
                                } else {
                                    st16(orow + c0 + i, make_uint4(w[0], w[1], w[2], w[3]));
                                    st16(orow + c0 + i + 8, make_uint4(w[4], w[5], w[6], w[7]));
                                }
                            }
                        }
                    }
                }
            }
            metas = (metas + hd.n_kept) % Smem::kMetas;
            __syncwarp();
            if (ok && lane == 0) mbar_arrive(smem_u32(&sm.bar_list_empty[slot]));
        }
    }
    // ---- teardown ----
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (sm.abort_flag) {
            // MMAs may still be running: give them time before the accumulator columns are released
            const unsigned long long t0 = global_ns();
            while (global_ns() - t0 < 200000ull) {}
        }
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace nats

#include "prefill_pair.cuh"

namespace nats {

// ---- host side ------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn) return fn;
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    fn = (EncodeTiledFn)ptr;
    return fn;
}

// [heads, N, D] bf16 viewed as a 3-D tensor (D innermost); box = 64 x box_rows x 1 with 128-byte swizzle; rows past N read zero
// 3-D map over [heads, rows, D] bf16; consecutive heads are head_stride_rows rows apart (>= rows: a cache buffer is
// longer than the part of it that is valid; rows behind `rows` read as zero).
static int make_map(CUtensorMap* map, const void* base, long long heads, long long N, int D, int box_rows, long long head_stride_rows = 0) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return fail(NATS_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    if (head_stride_rows <= 0) head_stride_rows = N;
    cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)N, (cuuint64_t)heads};
    cuuint64_t strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)head_stride_rows * D * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(NATS_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return NATS_OK;
}

struct PrefillWs { size_t lim, tmax, tmin, counter, total, list, before, open, rows_k, rows_v, total_far; int row_cap, copy_rows; };
// N = rows of the KV sequence.  `total` bytes are enough for any call; with `total_far` bytes there is room for what the
// gathered tiles need (0: this chunk size has none): the lists of the chunks that stay visible and, for chunks below 8 rows,
// copies of their K and V rows, up to row_cap (a quarter of the sequence) per head, and tails of kTailRows per tile (see
// far_rows_kernel), copy_rows in all.  The line of a quarter is one of memory: a prompt of 8192 tokens with one role per token, 32 / 8
// heads of 128, takes with room for an eighth / a quarter / a half 138 / 138 / 138 us at 10 % global, 251 / 180 / 181 at 20 %, 430 / 324 /
// 267 at 40 %.  From 8 rows on boxes of K and V themselves need no copy and no room; at head_dim 128 and 256 they are the slower
// way: 8192 tokens, chunks of 8, 32 / 8 heads, boxes / copies, 10, 20 and 40 % global, us: head_dim 64 116 / 119, 167 / 162, 278 / 317; 128
// 154 / 129, 234 / 170, 392 / 321; 256 401 / 307, 630 / 405, 1034 / 795.  D = 0: the head_dim is not known, so that there is no room for rows.
static PrefillWs prefill_ws(int B, int Hkv, int N, int C, int D) {
    PrefillWs w = {};
    const size_t BH = (size_t)B * Hkv, Nc = cdiv(N, C), Nt = cdiv(N, kTile);
    const size_t per_tile = align_up(BH * Nt * 4, 256), per_chunk = align_up(BH * Nc * 4, 256);
    w.lim = 0;
    w.tmax = per_chunk;
    w.tmin = w.tmax + per_tile;
    w.counter = w.tmin + per_tile;
    w.total = w.counter + 256;
    if (C < kTile && kTile % C == 0 && (C >= 8 || D > 0)) {
        w.list = w.total;
        w.before = w.list + per_chunk;
        w.open = w.before + align_up(BH * (Nt + 1) * 4, 256);
        w.rows_k = w.rows_v = w.total_far = w.open + per_tile;
        if (C < 8) {
            w.row_cap = (N / 4 + kTile - 1) / kTile * kTile;
            w.copy_rows = w.row_cap + kTailRows * (int)Nt;
            w.rows_v = w.rows_k + BH * w.copy_rows * D * 2;
            w.total_far = w.rows_v + BH * w.copy_rows * D * 2;
        }
    }
    return w;
}

// Whether a call gathers the far chunks: where there is room and the sequence is long enough.  Eight sequences, 16 / 8 heads,
// window 256, 10 % global, in place / gathered, us: chunks of 1 (head_dim 64) 512 tokens 29 / 34, 1024 62 / 52, 1536 106 / 71, 2000 159 / 92;
// chunks of 16 (128) 512 29 / 31, 1024 58 / 52, 1536 92 / 70, 2000 134 / 92; chunks of 32 (128) 512 28 / 30, 1024 55 / 52, 1536 86 / 77, 2000
// 122 / 101, 3000 201 / 144; chunks of 64 (64) 512 29 / 30, 1024 53 / 49, 1536 80 / 72, 2000 106 / 93, 3000 173 / 141.  (For chunks above
// 16 the line was drawn where an earlier form of the kernel broke even; the present one would gather from 1024 on.)
static int far_min_rows(int C) { return C <= 16 ? 1024 : 2048; }
static bool use_far(const PrefillWs& w, size_t workspace_bytes, int C, int q_end, bool pair) {
    return w.total_far != 0 && workspace_bytes >= w.total_far && q_end >= far_min_rows(C) && !pair;
}
// How many listed chunks make a tile dense, so that it stays in place.  A gathered tile costs more than one in place where its
// boxes are many (all chunks global, 12288 tokens, time over the same in place: 64 boxes a tile (chunks of 8, head_dim 256) 2.20, 32
// (16 / 256, 8 / 128) 1.25 and 1.59, 16 (32 / 256, 16 / 128, 8 / 64) 1.04, 1.16 and 1.25, fewer 1.00 to 1.04), the masks of a tile
// in place make it up to 1/12 dearer; a full tile needs neither masks nor gathering.  With 100, 90 and 70 % of the chunks global the rule
// takes at most 4 % longer than the better of gathering all and nothing (eleven pairs of chunk size and head_dim), and is up to 7 %
// faster than both.  Chunks below 8 have no dense tiles: their copies are loaded in boxes of 128 rows, and the test would cost them time.
static int far_dense_min(int C, int D) {
    if (C < 8) return 0x7fffffff;
    const int cpt = kTile / C, boxes = cpt * (D / 64);
    const int cost = boxes >= 64 ? 39 : boxes >= 32 ? 25 : 16;             // of a gathered tile, in 16ths of a full one
    return min(cpt, cdiv(cpt * 18, cost));
}
static FarLists far_lists(const PrefillWs& w, uint8_t* ws, int C, int D) {
    FarLists far;
    far.list = (int32_t*)(ws + w.list); far.before_tile = (int32_t*)(ws + w.before); far.open_max = (int32_t*)(ws + w.open);
    if (w.row_cap) far.max_listed = w.row_cap / C;
    far.dense_min = far_dense_min(C, D);
    return far;
}

// Copies the listed rows of K and V (see PrefillWs), 64 per block.  Behind them stand kTailRows rows for every 128-row tile: the
// last of the rows listed in front of the tile that do not make a whole group of eight, then zeros (the part empty tile of an
// item is loaded in groups of eight and must not hold rows of later keys).  Moves 4 D bytes per row and tensor: 3 MB for 8192
// tokens with 10 % global.
constexpr int kFarThreads = 256, kFarRowsPerBlock = 64;
struct FarRowsParams {
    const uint8_t* k; const uint8_t* v;              // [BH, head_rows, D] bf16
    uint8_t* rows_k; uint8_t* rows_v;                // [BH, rows, D]
    const int32_t* list; const int32_t* before_tile;
    long long head_rows;
    int Nc, Ntk, Nkv, C, D, cap, rows;
};
__global__ void __launch_bounds__(kFarThreads) far_rows_kernel(const FarRowsParams p) {
    const int bh = blockIdx.y;
    const int32_t* before = p.before_tile + (size_t)bh * (p.Ntk + 1);
    const int32_t* list = p.list + (size_t)bh * p.Nc;
    const int count = min((long long)before[p.Ntk] * p.C, (long long)p.cap);
    const int r0 = blockIdx.x * kFarRowsPerBlock, r1 = min(r0 + kFarRowsPerBlock, p.rows);
    const int vpt = p.D / 8;
    for (int i = threadIdx.x; i < (r1 - r0) * vpt; i += kFarThreads) {
        const int r = r0 + i / vpt, vec = i % vpt;
        int n = count, key = r;                      // copied: the key-th of n listed rows
        if (r >= p.cap) {
            n = before[(r - p.cap) / kTailRows] * p.C;
            if (n > p.cap) continue;
            key = n / kTailRows * kTailRows + r % kTailRows;
        } else if (r >= count) {
            continue;
        }
        uint4 a = make_uint4(0, 0, 0, 0), b = a;
        if (key < n) {
            const int row = list[key / p.C] * p.C + key % p.C;
            if (row < p.Nkv) {                       // the last chunk of the sequence may be part empty
                const size_t src = (((size_t)bh * p.head_rows + row) * vpt + vec) * 16;
                a = ld16(p.k + src);
                b = ld16(p.v + src);
            }
        }
        const size_t dst = (((size_t)bh * p.rows + r) * vpt + vec) * 16;
        st16(p.rows_k + dst, a);
        st16(p.rows_v + dst, b);
    }
}

constexpr int kMaxDevices = 64;

template <int D, bool FINE>
static int launch_prefill(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mkf,
                          const CUtensorMap& mvf, const CUtensorMap& mkc, const CUtensorMap& mvc, const PrefillParams& p,
                          cudaStream_t st) {
    const size_t smem = sizeof(PrefillSmem<D>);
    int dev = 0, sms = 0;
    NATS_CHECK_CUDA(cudaGetDevice(&dev));
    // the opt-in to more than 48 KB of dynamic shared memory is a per-device attribute of the kernel
    static bool attr_set[kMaxDevices] = {};
    if (dev < 0 || dev >= kMaxDevices || !attr_set[dev]) {
        NATS_CHECK_CUDA(cudaFuncSetAttribute(prefill_kernel<D, FINE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (dev >= 0 && dev < kMaxDevices) attr_set[dev] = true;
    }
    NATS_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int grid = p.total_items < sms ? p.total_items : sms;      // one persistent CTA per SM
    prefill_kernel<D, FINE><<<grid, kPrefillThreads, smem, st>>>(mq, mk, mv, mkf, mvf, mkc, mvc, p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

static int launch_prefill_pair(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const PrefillParams& p, cudaStream_t st) {
    const size_t smem = sizeof(PairSmem);
    int dev = 0, sms = 0;
    NATS_CHECK_CUDA(cudaGetDevice(&dev));
    static bool attr_set[kMaxDevices] = {};
    if (dev < 0 || dev >= kMaxDevices || !attr_set[dev]) {
        NATS_CHECK_CUDA(cudaFuncSetAttribute(prefill_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (dev >= 0 && dev < kMaxDevices) attr_set[dev] = true;
    }
    NATS_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int grid = 2 * p.total_items < sms ? 2 * p.total_items : sms;        // one persistent CTA pair per SM pair
    grid &= ~1;
    prefill_pair_kernel<<<grid, kPrefillThreads, smem, st>>>(mq, mk, mv, p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

// CTA pairs (cta_group::2) for head_dim 128 and group sizes that are a multiple of four; NATS_B200_PAIR=0 turns them off
static bool use_pair_kernel(int D, int nrep) {
    static int mode = -1;
    if (mode < 0) {
        const char* e = getenv("NATS_B200_PAIR");
        mode = (e != nullptr && e[0] == '1') ? 1 : 0;
    }
    return mode == 1 && D == 128 && nrep % 4 == 0;
}

// Tensor maps, parameters and launch shared by the entry points.  N query rows at positions q_off .. q_off + N - 1 of a
// KV sequence of Nkv rows whose heads are kv_head_stride rows apart (0: contiguous).
static int run_prefill(const void* d_q, const void* d_k, const void* d_v, void* d_o, int B, int Hq, int Hkv, int N, int Nkv,
                       int q_off, long long kv_head_stride, int D, int C, float sm_scale, const int32_t* lim,
                       const int32_t* tmax, const int32_t* tmin, int32_t* counter, int32_t* d_status, cudaStream_t st,
                       const FarLists& far, uint8_t* far_k, uint8_t* far_v, int far_cap, int far_rows, float* d_lse = nullptr, bool o_tokens = false, bool o_f32 = false) {
    const bool pair = use_pair_kernel(D, Hq / Hkv) && !o_f32;
    CUtensorMap mq, mk, mv, mkf, mvf, mkc, mvc;
    if (int rc = make_map(&mq, d_q, B * Hq, N, D, 128)) return rc;
    if (int rc = make_map(&mk, d_k, B * Hkv, Nkv, D, pair ? 64 : 128, kv_head_stride)) return rc;     // a pair's CTA loads half the rows of a K tile
    if (int rc = make_map(&mv, d_v, B * Hkv, Nkv, D, 128, kv_head_stride)) return rc;
    mkf = mkc = mk;
    mvf = mvc = mv;
    if (far.list != nullptr && far_cap > 0) {
        FarRowsParams f;
        f.k = (const uint8_t*)d_k; f.v = (const uint8_t*)d_v; f.rows_k = far_k; f.rows_v = far_v; f.list = far.list; f.before_tile = far.before_tile;
        f.head_rows = kv_head_stride > 0 ? kv_head_stride : Nkv;
        f.Nc = cdiv(Nkv, C); f.Ntk = cdiv(Nkv, kTile); f.Nkv = Nkv; f.C = C; f.D = D; f.cap = far_cap; f.rows = far_rows;
        far_rows_kernel<<<dim3(cdiv(far_rows, kFarRowsPerBlock), B * Hkv), kFarThreads, 0, st>>>(f);
        NATS_CHECK_CUDA(cudaGetLastError());
        if (int rc = make_map(&mkc, far_k, B * Hkv, far_rows, D, 128)) return rc;
        if (int rc = make_map(&mvc, far_v, B * Hkv, far_rows, D, 128)) return rc;
        if (int rc = make_map(&mkf, far_k, B * Hkv, far_rows, D, kTailRows)) return rc;
        if (int rc = make_map(&mvf, far_v, B * Hkv, far_rows, D, kTailRows)) return rc;
    } else if (far.list != nullptr) {
        if (int rc = make_map(&mkf, d_k, B * Hkv, Nkv, D, C, kv_head_stride)) return rc;       // boxes of one chunk
        if (int rc = make_map(&mvf, d_v, B * Hkv, Nkv, D, C, kv_head_stride)) return rc;
    }
    PrefillParams p;
    p.far_list = far.list; p.far_before = far.before_tile; p.far_open = far.open_max;
    p.far_cap = far.list != nullptr ? far_cap : 0;
    p.far_rows = far_rows;
    p.o_batch = (long long)N * Hq * D;
    p.o_head = o_tokens ? D : (long long)N * D;
    p.o_row = o_tokens ? (long long)Hq * D : D;
    p.o_f32 = o_f32;
    p.o = d_o; p.lse = d_lse; p.lim = lim; p.tile_max = tmax; p.tile_min = tmin; p.status = d_status;
    p.Hq = Hq; p.Hkv = Hkv; p.N = N; p.Nkv = Nkv; p.q_off = q_off; p.C = C;
    p.c_shift = (C & (C - 1)) ? -1 : __builtin_ctz((unsigned)C);
    p.Nc = cdiv(Nkv, C); p.Nt = cdiv(N, kTile); p.Ntk = cdiv(Nkv, kTile);
    const int heads_per_item = D <= 128 ? 2 : 1;
    p.nrep = Hq / Hkv; p.n_groups = (p.nrep + heads_per_item - 1) / heads_per_item;
    p.work_counter = counter;
    const long long items = (long long)B * Hkv * p.n_groups * p.Nt;
    NATS_CHECK_ARG(items <= 0x7fffffffLL - 65536, "too many work items (%lld)", items);
    p.total_items = (int)items;
    p.scale_log2 = sm_scale * 1.4426950408889634f;
    if (pair) {
        p.n_groups = p.nrep / 4;
        p.total_items = B * Hkv * p.n_groups * p.Nt;
        return launch_prefill_pair(mq, mk, mv, p, st);
    }
    if (p.c_shift >= 5 && far.list == nullptr) {
        if (D == 64) return launch_prefill<64, false>(mq, mk, mv, mkf, mvf, mkc, mvc, p, st);
        if (D == 256) return launch_prefill<256, false>(mq, mk, mv, mkf, mvf, mkc, mvc, p, st);
        return launch_prefill<128, false>(mq, mk, mv, mkf, mvf, mkc, mvc, p, st);
    }
    if (D == 64) return launch_prefill<64, true>(mq, mk, mv, mkf, mvf, mkc, mvc, p, st);
    if (D == 256) return launch_prefill<256, true>(mq, mk, mv, mkf, mvf, mkc, mvc, p, st);
    return launch_prefill<128, true>(mq, mk, mv, mkf, mvf, mkc, mvc, p, st);
}

}  // namespace nats

using namespace nats;

extern "C" __attribute__((visibility("default"))) size_t nats_b200_prefill_workspace_bytes(int B, int Hkv, int N, int C) {
    if (B <= 0 || Hkv <= 0 || N <= 0 || C <= 0) return 0;
    const PrefillWs w = prefill_ws(B, Hkv, N, C, 0);
    return w.total_far ? w.total_far : w.total;
}

extern "C" __attribute__((visibility("default"))) size_t nats_b200_prefill_workspace_bytes_for(int B, int Hkv, int N, int D, int C) {
    if (B <= 0 || Hkv <= 0 || N <= 0 || D <= 0 || C <= 0) return 0;
    const PrefillWs w = prefill_ws(B, Hkv, N, C, D);
    return w.total_far ? w.total_far : w.total;
}

static int prefill_first_call(const void* d_q, const void* d_k, const void* d_v, void* d_o, const uint8_t* d_roles,
                              int B, int Hq, int Hkv, int N, int D, int C, int SW, float sm_scale,
                              void* d_workspace, size_t workspace_bytes, int64_t* d_kept_tiles, int32_t* d_status,
                              void* stream, float* d_lse, int32_t* d_n_visible, bool o_tokens = false,
                              bool o_f32 = false) {
    NATS_CHECK_ARG(B > 0 && Hq > 0 && Hkv > 0 && N > 0 && Hq % Hkv == 0, "bad shape B=%d Hq=%d Hkv=%d N=%d", B, Hq, Hkv, N);
    NATS_CHECK_ARG(C > 0 && SW > 0 && SW % C == 0, "sliding window %d must be a positive multiple of the chunk size %d", SW, C);
    NATS_CHECK_ARG(d_q && d_k && d_v && d_o && d_roles && d_workspace && d_status, "null pointer");
    NATS_CHECK_ARG(((uintptr_t)d_q | (uintptr_t)d_k | (uintptr_t)d_v | (uintptr_t)d_o | (uintptr_t)d_workspace) % 16 == 0,
                   "q, k, v, o and the workspace must be 16-byte aligned");
    NATS_CHECK_ARG(sm_scale > 0.f, "sm_scale must be positive");
    if (D != 64 && D != 128 && D != 256) return fail(NATS_ERR_UNSUPPORTED, "prefill supports head_dim 64, 128 and 256, got %d", D);
    NATS_CHECK_ARG(N <= kMaxTiles * kTile, "N = %d exceeds the prefill limit %d", N, kMaxTiles * kTile);
    NATS_CHECK_ARG((long long)B <= 65535 && (long long)Hkv * ((Hq / Hkv + 1) / 2) <= 65535, "grid too large");
    const PrefillWs w = prefill_ws(B, Hkv, N, C, D);
    if (workspace_bytes < w.total)
        return fail(NATS_ERR_WORKSPACE, "prefill workspace: %zu bytes given, %zu needed", workspace_bytes, w.total);
    uint8_t* ws = (uint8_t*)d_workspace;
    int32_t* lim = (int32_t*)(ws + w.lim);
    int32_t* tmax = (int32_t*)(ws + w.tmax);
    int32_t* tmin = (int32_t*)(ws + w.tmin);
    FarLists far;
    if (use_far(w, workspace_bytes, C, N, use_pair_kernel(D, Hq / Hkv) && !o_f32)) far = far_lists(w, ws, C, D);
    if (int rc = role_prep(d_roles, B, Hkv, N, C, SW, lim, tmax, tmin, d_kept_tiles, far, (int32_t*)(ws + w.counter), stream)) return rc;
    if (d_n_visible != nullptr)
        if (int rc = nats_b200_visible_counts(lim, B, Hq, Hkv, N, C, d_n_visible, stream)) return rc;
    return run_prefill(d_q, d_k, d_v, d_o, B, Hq, Hkv, N, N, 0, 0, D, C, sm_scale, lim, tmax, tmin,
                       (int32_t*)(ws + w.counter), d_status, (cudaStream_t)stream, far, ws + w.rows_k, ws + w.rows_v, w.row_cap, w.copy_rows, d_lse, o_tokens, o_f32);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_prefill_fwd(const void* d_q, const void* d_k, const void* d_v, void* d_o, const uint8_t* d_roles,
                                     int B, int Hq, int Hkv, int N, int D, int C, int SW, float sm_scale,
                                     void* d_workspace, size_t workspace_bytes, int64_t* d_kept_tiles, int32_t* d_status,
                                     void* stream) {
    return prefill_first_call(d_q, d_k, d_v, d_o, d_roles, B, Hq, Hkv, N, D, C, SW, sm_scale, d_workspace, workspace_bytes,
                              d_kept_tiles, d_status, stream, nullptr, nullptr);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_prefill_fwd_out(
    const void* d_q, const void* d_k, const void* d_v, void* d_o, int o_tokens, int o_f32, const uint8_t* d_roles,
    int B, int Hq, int Hkv, int N, int D, int C, int SW, float sm_scale, void* d_workspace, size_t workspace_bytes,
    int64_t* d_kept_tiles, int32_t* d_status, void* stream) {
    return prefill_first_call(d_q, d_k, d_v, d_o, d_roles, B, Hq, Hkv, N, D, C, SW, sm_scale, d_workspace, workspace_bytes,
                              d_kept_tiles, d_status, stream, nullptr, nullptr, o_tokens != 0, o_f32 != 0);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_prefill_fwd_stats(
    const void* d_q, const void* d_k, const void* d_v, void* d_o, const uint8_t* d_roles,
    int B, int Hq, int Hkv, int N, int D, int C, int SW, float sm_scale, void* d_workspace, size_t workspace_bytes,
    int64_t* d_kept_tiles, float* d_lse, int32_t* d_n_visible, int32_t* d_status, void* stream) {
    NATS_CHECK_ARG(d_lse != nullptr && d_n_visible != nullptr, "null pointer");
    return prefill_first_call(d_q, d_k, d_v, d_o, d_roles, B, Hq, Hkv, N, D, C, SW, sm_scale, d_workspace, workspace_bytes,
                              d_kept_tiles, d_status, stream, d_lse, d_n_visible);
}

extern "C" __attribute__((visibility("default"))) size_t nats_b200_prefill_past_workspace_bytes(int B, int Hkv, int n_kv, int C) {
    if (B <= 0 || Hkv <= 0 || n_kv <= 0 || C <= 0) return 0;
    return nats_b200_prefill_workspace_bytes(B, Hkv, n_kv, C);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_prefill_past_fwd(
    const void* d_q, const void* d_cache_k, const void* d_cache_v, void* d_o, const uint8_t* d_roles_new,
    const uint8_t* d_valid, int valid_stride, const int64_t* d_size_global, const int64_t* d_size_local,
    int B, int Hq, int Hkv, int x_len, int D, int C, int SW, int cache_capacity, int t0, int fill, int tail,
    float sm_scale, void* d_workspace, size_t workspace_bytes, int64_t* d_kept_tiles, int32_t* d_status, void* stream) {
    NATS_CHECK_ARG(B > 0 && Hq > 0 && Hkv > 0 && x_len > 0 && Hq % Hkv == 0, "bad shape B=%d Hq=%d Hkv=%d x_len=%d", B, Hq, Hkv, x_len);
    NATS_CHECK_ARG(C > 0 && SW > 0 && SW % C == 0, "sliding window %d must be a positive multiple of the chunk size %d", SW, C);
    NATS_CHECK_ARG(d_q && d_cache_k && d_cache_v && d_o && d_roles_new && d_valid && d_size_global && d_size_local &&
                   d_workspace && d_status, "null pointer");
    NATS_CHECK_ARG(((uintptr_t)d_q | (uintptr_t)d_cache_k | (uintptr_t)d_cache_v | (uintptr_t)d_o | (uintptr_t)d_workspace) % 16 == 0,
                   "q, the cache, o and the workspace must be 16-byte aligned");
    NATS_CHECK_ARG(sm_scale > 0.f, "sm_scale must be positive");
    NATS_CHECK_ARG(t0 >= SW && t0 % C == 0 && fill >= 0 && fill < C, "tail offset %d must be a multiple of the chunk size >= the window, fill %d in [0, chunk)", t0, fill);
    NATS_CHECK_ARG(tail >= 0 && tail < SW && tail % C == 0, "ring tail %d must be a multiple of the chunk size inside the window", tail);
    if (D != 64 && D != 128 && D != 256) return fail(NATS_ERR_UNSUPPORTED, "prefill supports head_dim 64, 128 and 256, got %d", D);
    const long long n_kv = (long long)t0 + fill + x_len;
    NATS_CHECK_ARG(n_kv <= cache_capacity, "the cache holds %d rows, %lld are needed (the new tokens must have been appended)", cache_capacity, n_kv);
    NATS_CHECK_ARG(n_kv <= (long long)kMaxTiles * kTile, "cache + new tokens = %lld rows exceed the prefill limit %d", n_kv, kMaxTiles * kTile);
    const PrefillWs w = prefill_ws(B, Hkv, (int)n_kv, C, D);
    if (workspace_bytes < w.total)
        return fail(NATS_ERR_WORKSPACE, "prefill workspace: %zu bytes given, %zu needed", workspace_bytes, w.total);
    uint8_t* ws = (uint8_t*)d_workspace;
    int32_t* lim = (int32_t*)(ws + w.lim);
    int32_t* tmax = (int32_t*)(ws + w.tmax);
    int32_t* tmin = (int32_t*)(ws + w.tmin);
    FarLists far;
    if (use_far(w, workspace_bytes, C, (int)n_kv, use_pair_kernel(D, Hq / Hkv))) far = far_lists(w, ws, C, D);
    if (int rc = role_prep_past(d_roles_new, d_valid, d_size_global, d_size_local, B, Hkv, x_len, C, SW,
                                          valid_stride, t0, fill, tail, lim, tmax, tmin, d_kept_tiles, far, (int32_t*)(ws + w.counter), stream)) return rc;
    return run_prefill(d_q, d_cache_k, d_cache_v, d_o, B, Hq, Hkv, x_len, (int)n_kv, t0 + fill, cache_capacity, D, C, sm_scale,
                       lim, tmax, tmin, (int32_t*)(ws + w.counter), d_status, (cudaStream_t)stream, far,
                       ws + w.rows_k, ws + w.rows_v, w.row_cap, w.copy_rows);
}

// =================================================================================================
// Prefill without any allocation by the caller or by this library
// =================================================================================================
namespace nats {

constexpr size_t kStaticScratchBytes = 1u << 20;   // 1 MiB per GPU that loads the library, held until the process exits

// Scratch for the role metadata (row limits and per-tile max / min limits) of nats_b200_prefill_fwd_static.
// In host code this name is only a stand-in for the symbol: the device address is obtained once per device below.
static __device__ __align__(256) uint8_t g_prefill_scratch[kStaticScratchBytes];
static void* g_prefill_scratch_addr[kMaxDevices] = {};

// Device address of the scratch array on the current device; looked up on the first call per device.
static int static_scratch(void** out) {
    int dev = -1;
    NATS_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(NATS_ERR_UNSUPPORTED, "device index %d is outside [0, %d)", dev, kMaxDevices);
    if (g_prefill_scratch_addr[dev] == nullptr) {
        void* ptr = nullptr;
        NATS_CHECK_CUDA(cudaGetSymbolAddress(&ptr, g_prefill_scratch));
        if (ptr == nullptr) return fail(NATS_ERR_CUDA, "no address of g_prefill_scratch on device %d", dev);
        g_prefill_scratch_addr[dev] = ptr;
    }
    *out = g_prefill_scratch_addr[dev];
    return NATS_OK;
}

}  // namespace nats

extern "C" __attribute__((visibility("default"))) size_t nats_b200_prefill_static_scratch_bytes(void) {
    return nats::kStaticScratchBytes;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_prefill_fwd_static(
    const void* d_q, const void* d_k, const void* d_v, void* d_o, const uint8_t* d_roles,
    int B, int Hq, int Hkv, int N, int D, int C, int SW, float sm_scale,
    int64_t* d_kept_tiles, int32_t* d_status, void* stream) {
    if (B <= 0 || Hkv <= 0 || N <= 0 || C <= 0) return fail(NATS_ERR_INVALID_ARG, "bad shape B=%d Hkv=%d N=%d C=%d", B, Hkv, N, C);
    const size_t need = nats::prefill_ws(B, Hkv, N, C, D).total;
    if (need > nats::kStaticScratchBytes)
        return fail(NATS_ERR_WORKSPACE,
                    "this shape needs %zu bytes of role metadata, the built-in scratch holds %zu: use nats_b200_prefill_fwd "
                    "with a caller-provided workspace", need, (size_t)nats::kStaticScratchBytes);
    void* scratch = nullptr;
    if (int rc = nats::static_scratch(&scratch)) return rc;
    return nats_b200_prefill_fwd(d_q, d_k, d_v, d_o, d_roles, B, Hq, Hkv, N, D, C, SW, sm_scale, scratch,
                                 nats::kStaticScratchBytes, d_kept_tiles, d_status, stream);
}

