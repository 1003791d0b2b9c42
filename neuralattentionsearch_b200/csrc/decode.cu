// Decode attention over the compacted ragged cache: split-KV, GQA-aware, HBM-bound.
//
// One block owns kSeg consecutive tokens of the *logical* sequence of one (batch, kv-head):
//     [ valid ring slots | kept tokens [SW,len) | tokens of the unfinished chunk [T0,T0+fill) | the new token ]
// and its four warps take 16-token tiles of it in turn.  A tile's K and V rows travel global -> shared memory with
// cp.async (16 bytes per lane, bypassing L1) through a per-warp ring of kDecStages tiles, so two tiles are in flight
// while one is consumed and the bytes in flight cost no registers.  All query heads of the group are served by the one
// read: S = Q.K^T runs as mma.sync m16n8k16 with the (up to 8) query heads as the M rows and 8 tokens as N; the
// score fragments are exactly the A fragments of O += P.V, so P never leaves registers.  The instruction count per byte
// is then small enough that the kernel is limited by HBM, not by issue slots.
// Blocks of a (batch, kv-head) leave partial (max, sum, acc) in the workspace; the block that arrives last combines
// them (an atomic ticket, nobody waits).  The block owning the last logical token also appends it to the cache.
#include "place.cuh"

namespace nats {

#ifndef NATS_DEC_SEG
#define NATS_DEC_SEG 1024
#endif
#ifndef NATS_DEC_STAGES
#define NATS_DEC_STAGES 3
#endif
constexpr int kSeg = NATS_DEC_SEG;          // logical tokens per block
constexpr int kDecStages = NATS_DEC_STAGES; // ring depth per warp
constexpr int kDecThreads = 128;
constexpr int kDecWarps = kDecThreads / 32;
constexpr int kTileTok = 16;                // tokens per warp tile
constexpr int kMaxRep = 8;                  // query heads per kv-head the fragment rows cover (rows 8..15 stay zero)

struct DecodeParams {
    const __nv_bfloat16* q;        // [B,Hq,1,D]
    const __nv_bfloat16* k_new;    // [B,Hkv,1,D]
    const __nv_bfloat16* v_new;
    __nv_bfloat16* o;              // [B,Hq,1,D]
    __nv_bfloat16* ck;             // [B,Hkv,Lcap,D]
    __nv_bfloat16* cv;
    uint8_t* valid;                // [B,Hkv,Lcap]
    const long long* size_global;  // [B,Hkv]
    const long long* size_local;
    const int32_t* state;          // [0] = T0
    int32_t* counters;             // [B*Hkv]   (workspace)
    float* partials;               // [B*Hkv, max_splits, nrep, D+2] or [B*Hkv, splits of the launch, strands, nrep, D+4]   (workspace)
    int Hq, Hkv, nrep, Lcap, SW, fill, max_splits;
    int fill_from_state;           // 1: the number of tokens in the unfinished chunk is read from state[4] (static launches)
    float scale_log2;              // sm_scale * log2(e)
    PlaceParams place;             // STEP kernels only
};

// Decode kernels that follow one another in a stream may overlap (programmatic dependent launch; where they do: overlaps): a kernel is
// then scheduled once every block of the one in front has started, and looks at memory only behind this wait, that is when that
// kernel has ended.
__device__ __forceinline__ void wait_for_previous_launch() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Ticket of a block that has left its results: true for the last of n blocks of the (batch, kv-head).
// STEP, no chunk completed: every block of the launch has read the step counters by now, the last one to come here advances
// them.  Another warp does that beside the ticket, so that no step waits for it: a recorded step of 16 heads of 128 (four query heads each,
// 2400 rows) 13.0 -> 12.0 us against counters advanced behind the output; 512 heads of 4400 rows 174.4 -> 173.4.  (One arrival per
// block or per head makes no difference: 64 sequences of 8 heads, 7000 rows, 208.7 us either way.)
template <bool STEP>
__device__ __forceinline__ bool last_arrival(const DecodeParams& p, int bh, int n, int fill) {
    __shared__ int s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();                             // orders what the block wrote before the barrier
        const int ticket = atomicAdd(&p.counters[bh], 1);
        s_last = (ticket == n - 1);
        if (s_last) p.counters[bh] = 0;
        __threadfence();
    } else if (STEP && threadIdx.x == 32 && fill + 1 != p.place.C) {
        int32_t* state = p.place.state;
        if (atomicAdd(&state[2], 1) == (int)(gridDim.x * gridDim.y * gridDim.z) - 1) {
            state[2] = 0;
            state[4] = fill + 1;
        }
    }
    __syncthreads();
    return s_last;
}

// The end of a step that has completed a chunk, run by the last block of every (batch, kv-head): nobody reads that head's cache
// any more.  The chunk is placed; the last head to come here advances the step counters (every block of the launch has read
// them by then: each of them, those without a segment included, took a ticket first).
__device__ __forceinline__ void finish_chunk(const DecodeParams& p, int bh, int n_heads, int T0) {
    const PlaceParams& pl = p.place;
    const int tail = pl.state[5];
    const int new_len = place_chunk<kDecThreads>(pl, bh, T0, tail);
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(&pl.state[1], new_len);
        __threadfence();
        if (atomicAdd(&pl.state[2], 1) == n_heads - 1) {
            __threadfence();
            pl.state[2] = 0;
            pl.state[0] = atomicExch(&pl.state[1], 0);
            pl.state[4] = 0;
            pl.state[5] = (tail + pl.C) % pl.SW;
        }
    }
}

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 16-byte asynchronous global -> shared copy that bypasses L1; with valid == false nothing is read and zeros are written
__device__ __forceinline__ void cp_async16(uint32_t smem_dst, const void* gsrc, bool valid) {
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_dst), "l"(gsrc), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// D (16x8, fp32) += A (16x16, bf16, row) * B (16x8, bf16, col)
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// STEP: the placement of a completed chunk and the step counters in the same launch (see last_arrival, finish_chunk)
template <int D, bool STEP>
__global__ void __launch_bounds__(kDecThreads) decode_kernel(const DecodeParams p) {
    constexpr int ROWB = D * 2;                      // bytes of a K or V row
    constexpr int CHUNKS = ROWB / 16;                // 16-byte chunks per row: 16 (D = 128) or 8 (D = 64)
    constexpr int TILE_BYTES = kTileTok * ROWB;      // one tile of K (and as much again of V)
    constexpr int STAGE_BYTES = 2 * TILE_BYTES;
    constexpr int CP_PER_LANE = kTileTok * CHUNKS / 32;   // cp.async per lane for one of K / V
    constexpr int ROWS_PER_CP = 32 / CHUNKS;         // rows one warp-wide cp.async covers
    constexpr int PSTRIDE = D + 2;                   // floats of a partial result per query head
    constexpr unsigned FULL = 0xffffffffu;
    const float NEG_INF = -INFINITY;

    const int seg = blockIdx.x, hkv = blockIdx.y, b = blockIdx.z;
    const int bh = b * p.Hkv + hkv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrep = p.nrep;
    wait_for_previous_launch();
    const int len = (int)(p.size_global[bh] + p.size_local[bh]);
    const int T0 = p.state[0];
    const int fill = p.fill_from_state ? p.state[4] : p.fill;
    const int Ltot = len + fill + 1;
    const int nsplit = (Ltot + kSeg - 1) / kSeg;
    if (!STEP && seg >= nsplit) return;
    if (seg < nsplit) {
    const int r0 = seg * kSeg, r1 = min(Ltot, r0 + kSeg);

    extern __shared__ __align__(128) uint8_t dsm[];
    __shared__ __align__(16) uint8_t s_ring_ok[kSeg];
    // after the main loop the ring memory holds the per-warp partial results
    float (*s_acc)[kMaxRep][D] = reinterpret_cast<float (*)[kMaxRep][D]>(dsm);
    float (*s_m)[kMaxRep] = reinterpret_cast<float (*)[kMaxRep]>(dsm + kDecWarps * kMaxRep * D * 4);
    float (*s_l)[kMaxRep] = reinterpret_cast<float (*)[kMaxRep]>(dsm + kDecWarps * kMaxRep * (D + 1) * 4);
    static_assert(kDecWarps * kMaxRep * (D + 2) * 4 <= kDecWarps * kDecStages * STAGE_BYTES, "combine scratch must fit into the ring");

    const __nv_bfloat16* ck = p.ck + (size_t)bh * p.Lcap * D;
    const __nv_bfloat16* cv = p.cv + (size_t)bh * p.Lcap * D;
    const uint8_t* valid = p.valid + (size_t)bh * p.Lcap;
    const __nv_bfloat16* kn = p.k_new + (size_t)bh * D;
    const __nv_bfloat16* vn = p.v_new + (size_t)bh * D;

    if (r0 < p.SW) {
        for (int i = tid; i < kSeg; i += kDecThreads) s_ring_ok[i] = (r0 + i < p.SW) ? valid[r0 + i] : 1;
    }
    // the block that owns the last logical token appends it (nobody reads that cache row in this launch)
    if (r1 == Ltot && warp == 0 && lane < CHUNKS) {
        const size_t dst = ((size_t)bh * p.Lcap + T0 + fill) * D + lane * 8;
        st16(p.ck + dst, ld16(kn + lane * 8));
        st16(p.cv + dst, ld16(vn + lane * 8));
        if (lane == 0) p.valid[(size_t)bh * p.Lcap + T0 + fill] = 1;
    }
    // Q as A fragments (rows = query heads of the group, 16 dims per k-step); rows >= nrep and rows 8..15 are zero
    const int hrow = lane >> 2, quad = lane & 3;
    uint32_t qa[D / 16][2];
    {
        const __nv_bfloat16* qrow = p.q + ((size_t)b * p.Hq + (size_t)hkv * nrep + hrow) * D;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            qa[ks][0] = hrow < nrep ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + quad * 2) : 0u;
            qa[ks][1] = hrow < nrep ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 8 + quad * 2) : 0u;
        }
    }
    if (r0 < p.SW) __syncthreads();

    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(dsm) + warp * kDecStages * STAGE_BYTES;
    const int n_tiles = (r1 - r0 + kTileTok - 1) / kTileTok;            // tiles of this block
    const int my_tiles = (n_tiles - warp + kDecWarps - 1) / kDecWarps;   // tiles warp, warp + 4, ... are this warp's

    // issue the copies of this warp's it-th tile: row r of the tile, chunk c goes to r*ROWB + ((c ^ (r & 7)) * 16)
    auto issue = [&](int it) {
        const int i0 = r0 + (it * kDecWarps + warp) * kTileTok;
        const uint32_t dst = ring + (it % kDecStages) * STAGE_BYTES;
        const int c = lane % CHUNKS, rsub = lane / CHUNKS;
        if (i0 + kTileTok <= p.SW) {
            // a ring tile none of whose slots is valid (a whole chunk that was not a sliding one) is not read at all
            const uint4 f = *reinterpret_cast<const uint4*>(&s_ring_ok[i0 - r0]);
            if ((f.x | f.y | f.z | f.w) == 0u) return;
        }
        if (i0 + kTileTok <= len) {                      // whole tile inside ring + kept tokens: logical == physical
            const __nv_bfloat16* kp = ck + (size_t)i0 * D + c * 8;
            const __nv_bfloat16* vp = cv + (size_t)i0 * D + c * 8;
#pragma unroll
            for (int x = 0; x < CP_PER_LANE; ++x) {
                const int r = x * ROWS_PER_CP + rsub;
                const uint32_t off = r * ROWB + ((c ^ (r & 7)) << 4);
                cp_async16(dst + off, kp + (size_t)r * D, true);
                cp_async16(dst + TILE_BYTES + off, vp + (size_t)r * D, true);
            }
        } else {
#pragma unroll
            for (int x = 0; x < CP_PER_LANE; ++x) {
                const int r = x * ROWS_PER_CP + rsub;
                const int i = i0 + r;
                const bool ok = i < r1;
                const __nv_bfloat16 *kp = ck, *vp = cv;
                if (ok) {
                    if (i < len) { kp = ck + (size_t)i * D; vp = cv + (size_t)i * D; }
                    else if (i < len + fill) { const size_t ph = (size_t)(T0 + (i - len)); kp = ck + ph * D; vp = cv + ph * D; }
                    else { kp = kn; vp = vn; }
                }
                const uint32_t off = r * ROWB + ((c ^ (r & 7)) << 4);
                cp_async16(dst + off, kp + c * 8, ok);
                cp_async16(dst + TILE_BYTES + off, vp + c * 8, ok);
            }
        }
    };

    float oacc[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; ++n) { oacc[n][0] = oacc[n][1] = oacc[n][2] = oacc[n][3] = 0.f; }
    float m_run = NEG_INF, l_run = 0.f;              // of query head `hrow`; l is this lane's share until the end

#pragma unroll
    for (int it = 0; it < kDecStages - 1; ++it) {
        if (it < my_tiles) issue(it);
        cp_async_commit();
    }
    for (int it = 0; it < my_tiles; ++it) {
        __syncwarp();                                // every lane is done reading the stage that is refilled now
        if (it + kDecStages - 1 < my_tiles) issue(it + kDecStages - 1);
        cp_async_commit();
        cp_async_wait<kDecStages - 1>();
        __syncwarp();                                // ... and sees the other lanes' copies of the stage consumed now
        const int i0 = r0 + (it * kDecWarps + warp) * kTileTok;
        const uint32_t sk = ring + (it % kDecStages) * STAGE_BYTES, sv = sk + TILE_BYTES;
        unsigned vmask = 0xffffu;                    // which of the 16 tokens exist and are valid
        if (i0 < p.SW || i0 + kTileTok > r1) {
            bool ok = false;
            if (lane < kTileTok) {
                const int i = i0 + lane;
                ok = i < r1 && (i >= p.SW || s_ring_ok[i - r0] != 0);
            }
            vmask = __ballot_sync(FULL, ok) & 0xffffu;
            if (vmask == 0u) continue;               // nothing visible in this tile (its copies were skipped as well)
        }
        // ---- S[heads x 16 tokens] = Q . K^T ----
        float sc[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
            const int r = nt * 8 + (lane & 7);
#pragma unroll
            for (int kp = 0; kp < D / 32; ++kp) {
                uint32_t kb[4];
                const int chunk = kp * 4 + (lane >> 3);
                ldmatrix_x4(sk + r * ROWB + ((chunk ^ (r & 7)) << 4), kb);
                mma_bf16(sc[nt], qa[2 * kp][0], 0u, qa[2 * kp][1], 0u, kb[0], kb[1]);
                mma_bf16(sc[nt], qa[2 * kp + 1][0], 0u, qa[2 * kp + 1][1], 0u, kb[2], kb[3]);
            }
        }
        // ---- online softmax of head `hrow` over the 4 scores this lane holds (tokens nt*8 + quad*2 + {0,1}) ----
        float s[4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = nt * 8 + quad * 2 + e;
                s[nt * 2 + e] = ((vmask >> t) & 1u) ? sc[nt][e] * p.scale_log2 : NEG_INF;
            }
        float mt = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
        mt = fmaxf(mt, __shfl_xor_sync(FULL, mt, 1));
        mt = fmaxf(mt, __shfl_xor_sync(FULL, mt, 2));
        const float m_new = fmaxf(m_run, mt);
        const float mu = (m_new == NEG_INF) ? 0.f : m_new;
        const float alpha = fast_exp2(m_run - mu);
        const float p0 = fast_exp2(s[0] - mu), p1 = fast_exp2(s[1] - mu), p2 = fast_exp2(s[2] - mu), p3 = fast_exp2(s[3] - mu);
        l_run = l_run * alpha + (p0 + p1) + (p2 + p3);
        m_run = m_new;
        if (__any_sync(FULL, alpha != 1.f)) {
#pragma unroll
            for (int n = 0; n < D / 8; ++n) { oacc[n][0] *= alpha; oacc[n][1] *= alpha; }
        }
        const uint32_t pa0 = pack2_bf16(p0, p1), pa2 = pack2_bf16(p2, p3);
        // ---- O[heads x D] += P . V ----
#pragma unroll
        for (int np = 0; np < D / 16; ++np) {
            uint32_t vb[4];
            const int r = ((lane >> 3) & 1) * 8 + (lane & 7);
            const int chunk = np * 2 + (lane >> 4);
            ldmatrix_x4_trans(sv + r * ROWB + ((chunk ^ (r & 7)) << 4), vb);
            mma_bf16(oacc[2 * np], pa0, 0u, pa2, 0u, vb[0], vb[1]);
            mma_bf16(oacc[2 * np + 1], pa0, 0u, pa2, 0u, vb[2], vb[3]);
        }
    }

    // ---- combine the warps of this block (the ring is drained first: its memory is reused) ----
    cp_async_wait<0>();
    __syncthreads();
    l_run += __shfl_xor_sync(FULL, l_run, 1);
    l_run += __shfl_xor_sync(FULL, l_run, 2);
    if (hrow < nrep) {
        if (quad == 0) { s_m[warp][hrow] = m_run; s_l[warp][hrow] = l_run; }
#pragma unroll
        for (int n = 0; n < D / 8; ++n)
            *reinterpret_cast<float2*>(&s_acc[warp][hrow][n * 8 + quad * 2]) = make_float2(oacc[n][0], oacc[n][1]);
    }
    __syncthreads();
    float* part_out = p.partials + ((size_t)bh * p.max_splits + seg) * nrep * PSTRIDE;
    for (int idx = tid; idx < nrep * D; idx += kDecThreads) {
        const int h = idx / D, d = idx % D;
        float mf = NEG_INF;
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) mf = fmaxf(mf, s_m[w][h]);
        const float mu = (mf == NEG_INF) ? 0.f : mf;
        float a = 0.f, l = 0.f;
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) {
            const float wgt = fast_exp2(s_m[w][h] - mu);
            a = fmaf(s_acc[w][h][d], wgt, a);
            l = fmaf(s_l[w][h], wgt, l);
        }
        if (nsplit == 1) {
            const float inv = l > 0.f ? 1.f / l : 0.f;
            p.o[((size_t)b * p.Hq + (size_t)hkv * nrep + h) * D + d] = __float2bfloat16_rn(a * inv);
        } else {
            part_out[h * PSTRIDE + d] = a;
            if (d == 0) { part_out[h * PSTRIDE + D] = mf; part_out[h * PSTRIDE + D + 1] = l; }
        }
    }
    }
    if (!STEP && nsplit == 1) return;
    // ---- the last block of this (batch, kv-head) combines the splits ----
    if (!last_arrival<STEP>(p, bh, STEP ? (int)gridDim.x : nsplit, fill)) return;
    const float* parts = p.partials + (size_t)bh * p.max_splits * nrep * PSTRIDE;
    if (nsplit > 1)
    for (int idx = tid; idx < nrep * D; idx += kDecThreads) {
        const int h = idx / D, d = idx % D;
        float mf = NEG_INF;
        for (int s = 0; s < nsplit; ++s) mf = fmaxf(mf, __ldcg(parts + ((size_t)s * nrep + h) * PSTRIDE + D));
        const float mu = (mf == NEG_INF) ? 0.f : mf;
        float a = 0.f, l = 0.f;
        for (int s = 0; s < nsplit; ++s) {
            const float* ps = parts + ((size_t)s * nrep + h) * PSTRIDE;
            const float wgt = fast_exp2(__ldcg(ps + D) - mu);
            a = fmaf(__ldcg(ps + d), wgt, a);
            l = fmaf(__ldcg(ps + D + 1), wgt, l);
        }
        const float inv = l > 0.f ? 1.f / l : 0.f;
        p.o[((size_t)b * p.Hq + (size_t)hkv * nrep + h) * D + d] = __float2bfloat16_rn(a * inv);
    }
    if (STEP && fill + 1 == p.place.C) finish_chunk(p, bh, gridDim.y * gridDim.z, T0);
}

// =================================================================================================
// The same step for launches that would leave most of the chip idle (few sequences, short caches)
// =================================================================================================
// decode_kernel gives a segment's 64 tiles to the four warps of one block, two tiles of each in flight: with fewer blocks
// than SMs a step then lasts as long as 16 tiles one after the other.  Here every one of those warps gets a block of its own
// (a "strand": tiles s, s + 4, ... of the segment), which issues the copies of all its (at most 16) tiles at once.  The four
// warps of the block compute the scores of four tiles each; after one block barrier each of them walks over all tiles for
// a quarter of the columns of O.  The arithmetic on every value is the one of decode_kernel in the same order -- the running
// maximum, the row sum and each accumulator see the strand's tiles in sequence, strands and segments are combined in the same
// two steps -- so that a head's output does not depend on which of the two kernels the size of the batch selects.
// One launch in a graph of 20, us, decode_kernel / strands, four query heads per kv-head, 2800 rows per head, head_dim 128: 24
// segments 18.9 / 10.8, 96 19.3 / 13.1; head_dim 64: 24 segments 16.1 / 8.6, 144 16.5 / 11.7 (lines: use_strands).  What is left of a
// short launch (10 us) is a chain of latencies: sizes, copies, scores, partial results, ticket, combination.
constexpr int kStrandTiles = kSeg / kTileTok / kDecWarps;
constexpr int kStrandTilesPerWarp = kStrandTiles / kDecWarps;
static_assert(kStrandTiles % kDecWarps == 0, "tiles of a strand are dealt to the warps in equal numbers");

template <int D, bool BOTH>
constexpr int strand_smem() { return kStrandTiles * ((BOTH ? 2 : 1) * kTileTok * D * 2 + 32 * 16 + kMaxRep * 4); }

// BOTH: V has slots of its own and its copies start together with those of K.  Otherwise a warp puts V where it has just read
// K, half the shared memory: three blocks instead of one on an SM at head_dim 128, for launches of more blocks than SMs.
template <int D, bool STEP, bool BOTH>
__global__ void __launch_bounds__(kDecThreads) decode_strand_kernel(const DecodeParams p) {
    constexpr int ROWB = D * 2, CHUNKS = ROWB / 16, TILE_BYTES = kTileTok * ROWB;
    constexpr int V_SLOTS = BOTH ? kStrandTiles * TILE_BYTES : 0, TILES_BYTES = kStrandTiles * TILE_BYTES + V_SLOTS;
    constexpr int CP_PER_LANE = kTileTok * CHUNKS / 32, ROWS_PER_CP = 32 / CHUNKS;
    constexpr int TPW = kStrandTilesPerWarp, PSTRIDE = D + 4;      // a partial result: D columns, maximum, row sum (16-byte rows)
    constexpr int NP = D / 16 / kDecWarps;           // 16-column blocks of O per warp
    constexpr unsigned FULL = 0xffffffffu;
    const float NEG_INF = -INFINITY;

    const int seg = blockIdx.x / kDecWarps, strand = blockIdx.x % kDecWarps, hkv = blockIdx.y, b = blockIdx.z;
    const int bh = b * p.Hkv + hkv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrep = p.nrep;
    wait_for_previous_launch();
    const int len = (int)(p.size_global[bh] + p.size_local[bh]);
    const int T0 = p.state[0];
    const int fill = p.fill_from_state ? p.state[4] : p.fill;
    const int Ltot = len + fill + 1;
    const int nsplit = (Ltot + kSeg - 1) / kSeg;
    if (!STEP && seg >= nsplit) return;
    extern __shared__ __align__(128) uint8_t dsm[];
    float* parts = p.partials + (size_t)bh * gridDim.x * nrep * PSTRIDE;      // gridDim.x: strands of the launch's splits
    if (seg < nsplit) {
    const int r0 = seg * kSeg, r1 = min(Ltot, r0 + kSeg);

    float4* s_score = reinterpret_cast<float4*>(dsm + TILES_BYTES);             // [tile][lane]
    float (*s_tmax)[kMaxRep] = reinterpret_cast<float (*)[kMaxRep]>(dsm + TILES_BYTES + kStrandTiles * 32 * 16);
    __shared__ unsigned s_vmask[kStrandTiles];

    const __nv_bfloat16* ck = p.ck + (size_t)bh * p.Lcap * D;
    const __nv_bfloat16* cv = p.cv + (size_t)bh * p.Lcap * D;
    const uint8_t* valid = p.valid + (size_t)bh * p.Lcap;
    const __nv_bfloat16* kn = p.k_new + (size_t)bh * D;
    const __nv_bfloat16* vn = p.v_new + (size_t)bh * D;

    // the block that owns the last logical token appends it (nobody reads that cache row in this launch)
    if (strand == 0 && r1 == Ltot && warp == 0 && lane < CHUNKS) {
        const size_t dst = ((size_t)bh * p.Lcap + T0 + fill) * D + lane * 8;
        st16(p.ck + dst, ld16(kn + lane * 8));
        st16(p.cv + dst, ld16(vn + lane * 8));
        if (lane == 0) p.valid[(size_t)bh * p.Lcap + T0 + fill] = 1;
    }

    // ---- copies of this warp's tiles, one group each; which of their tokens exist and are valid is read meanwhile (ring tiles
    // without a valid slot are copied here too: their bytes cost less than waiting for the flags) ----
    const uint32_t tiles = (uint32_t)__cvta_generic_to_shared(dsm);
    auto issue = [&](int x, const __nv_bfloat16* cache, const __nv_bfloat16* fresh, int slots) {
        const int t = x * kDecWarps + warp;                                   // tile of the strand
        const int i0 = r0 + (t * kDecWarps + strand) * kTileTok;
        if (i0 < r1) {
            const uint32_t dst = tiles + slots + t * TILE_BYTES;
            const int c = lane % CHUNKS, rsub = lane / CHUNKS;
            const bool plain = i0 + kTileTok <= len;                          // whole tile inside ring + kept tokens: logical == physical
#pragma unroll
            for (int y = 0; y < CP_PER_LANE; ++y) {
                const int r = y * ROWS_PER_CP + rsub;
                const int i = i0 + r;
                const bool ok = plain || i < r1;
                const __nv_bfloat16* src = cache;
                if (plain || i < len) src = cache + (size_t)i * D;
                else if (i < len + fill) src = cache + (size_t)(T0 + (i - len)) * D;
                else if (ok) src = fresh;
                cp_async16(dst + r * ROWB + ((c ^ (r & 7)) << 4), src + c * 8, ok);
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int x = 0; x < TPW; ++x) issue(x, ck, kn, 0);
    if (BOTH) {
#pragma unroll
        for (int x = 0; x < TPW; ++x) issue(x, cv, vn, V_SLOTS);
    }
    unsigned vmask[TPW];
    {
        bool ok[TPW];
#pragma unroll
        for (int x = 0; x < TPW; ++x) {
            const int i = r0 + ((x * kDecWarps + warp) * kDecWarps + strand) * kTileTok + lane;
            ok[x] = lane < kTileTok && i < r1;
            if (ok[x] && i < p.SW) ok[x] = valid[i] != 0;
        }
#pragma unroll
        for (int x = 0; x < TPW; ++x) vmask[x] = __ballot_sync(FULL, ok[x]) & 0xffffu;
    }
    const int hrow = lane >> 2, quad = lane & 3;
    uint32_t qa[D / 16][2];
    {
        const __nv_bfloat16* qrow = p.q + ((size_t)b * p.Hq + (size_t)hkv * nrep + hrow) * D;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            qa[ks][0] = hrow < nrep ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + quad * 2) : 0u;
            qa[ks][1] = hrow < nrep ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 8 + quad * 2) : 0u;
        }
    }
    // ---- scores of this warp's tiles ----
#pragma unroll
    for (int x = 0; x < TPW; ++x) {
        const int t = x * kDecWarps + warp;
        // groups in flight behind K of this tile: K of the later ones, and V of all or of the earlier ones
        if (!BOTH) cp_async_wait<TPW - 1>();
        else if (x == 0) cp_async_wait<2 * TPW - 1>();
        else if (x == 1) cp_async_wait<2 * TPW - 2>();
        else if (x == 2) cp_async_wait<2 * TPW - 3>();
        else cp_async_wait<2 * TPW - 4>();
        __syncwarp();                                // every lane's copies of the tile are there
        if (lane == 0) s_vmask[t] = vmask[x];
        if (vmask[x] == 0u) {
            if (!BOTH) cp_async_commit();
            continue;
        }
        const uint32_t sk = tiles + t * TILE_BYTES;
        float sc[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
            const int r = nt * 8 + (lane & 7);
#pragma unroll
            for (int kp = 0; kp < D / 32; ++kp) {
                uint32_t kb[4];
                const int chunk = kp * 4 + (lane >> 3);
                ldmatrix_x4(sk + r * ROWB + ((chunk ^ (r & 7)) << 4), kb);
                mma_bf16(sc[nt], qa[2 * kp][0], 0u, qa[2 * kp][1], 0u, kb[0], kb[1]);
                mma_bf16(sc[nt], qa[2 * kp + 1][0], 0u, qa[2 * kp + 1][1], 0u, kb[2], kb[3]);
            }
        }
        if (!BOTH) {
            __syncwarp();                            // every lane is done with K: V takes its place
            issue(x, cv, vn, 0);
        }
        float s[4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                s[nt * 2 + e] = ((vmask[x] >> (nt * 8 + quad * 2 + e)) & 1u) ? sc[nt][e] * p.scale_log2 : NEG_INF;
        float mt = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
        mt = fmaxf(mt, __shfl_xor_sync(FULL, mt, 1));
        mt = fmaxf(mt, __shfl_xor_sync(FULL, mt, 2));
        s_score[t * 32 + lane] = make_float4(s[0], s[1], s[2], s[3]);
        if (quad == 0) s_tmax[t][hrow] = mt;
    }
    static_assert(TPW == 4, "wait counts above");
    cp_async_wait<0>();
    __syncthreads();
    // ---- online softmax over the strand's tiles; this warp's columns of O += P . V ----
    float oacc[2 * NP][4];
#pragma unroll
    for (int n = 0; n < 2 * NP; ++n) { oacc[n][0] = oacc[n][1] = oacc[n][2] = oacc[n][3] = 0.f; }
    float m_run = NEG_INF, l_run = 0.f;
    const int n_tiles = (r1 - r0 + kTileTok - 1) / kTileTok;
    const int my_tiles = (n_tiles - strand + kDecWarps - 1) / kDecWarps;
#pragma unroll 4
    for (int t = 0; t < my_tiles; ++t) {
        if (s_vmask[t] == 0u) continue;              // nothing visible in this tile (what was copied of it is not looked at)
        const float4 s = s_score[t * 32 + lane];
        const float m_new = fmaxf(m_run, s_tmax[t][hrow]);
        const float mu = (m_new == NEG_INF) ? 0.f : m_new;
        const float alpha = fast_exp2(m_run - mu);
        const float p0 = fast_exp2(s.x - mu), p1 = fast_exp2(s.y - mu), p2 = fast_exp2(s.z - mu), p3 = fast_exp2(s.w - mu);
        l_run = l_run * alpha + (p0 + p1) + (p2 + p3);
        m_run = m_new;
#pragma unroll
        for (int n = 0; n < 2 * NP; ++n) { oacc[n][0] *= alpha; oacc[n][1] *= alpha; }
        const uint32_t pa0 = pack2_bf16(p0, p1), pa2 = pack2_bf16(p2, p3);
        const uint32_t sv = tiles + V_SLOTS + t * TILE_BYTES;
#pragma unroll
        for (int np = 0; np < NP; ++np) {
            uint32_t vb[4];
            const int r = ((lane >> 3) & 1) * 8 + (lane & 7);
            const int chunk = (warp * NP + np) * 2 + (lane >> 4);
            ldmatrix_x4_trans(sv + r * ROWB + ((chunk ^ (r & 7)) << 4), vb);
            mma_bf16(oacc[2 * np], pa0, 0u, pa2, 0u, vb[0], vb[1]);
            mma_bf16(oacc[2 * np + 1], pa0, 0u, pa2, 0u, vb[2], vb[3]);
        }
    }
    l_run += __shfl_xor_sync(FULL, l_run, 1);
    l_run += __shfl_xor_sync(FULL, l_run, 2);
    // ---- partial result of the strand ----
    if (hrow < nrep) {
        float* out = parts + ((size_t)blockIdx.x * nrep + hrow) * PSTRIDE;
#pragma unroll
        for (int n = 0; n < 2 * NP; ++n)
            *reinterpret_cast<float2*>(out + warp * (D / kDecWarps) + n * 8 + quad * 2) = make_float2(oacc[n][0], oacc[n][1]);
        if (warp == 0 && quad == 0) { out[D] = m_run; out[D + 1] = l_run; }
    }
    }
    const int n_strands = nsplit * kDecWarps;
    if (!last_arrival<STEP>(p, bh, STEP ? (int)gridDim.x : n_strands, fill)) return;
    // ---- the last block of this (batch, kv-head): strands of a segment, then segments ----
    // weights first (they do not depend on the column): strand within its segment, segment within the head
    float* s_wgt = reinterpret_cast<float*>(dsm);                              // [n_strands][nrep]
    float* s_seg_m = s_wgt + n_strands * nrep;                                 // [nsplit][nrep] segment maximum, then its weight
    float* s_seg_l = s_seg_m + nsplit * nrep;                                  // [nsplit][nrep] segment row sum
    for (int idx = tid; idx < nsplit * nrep; idx += kDecThreads) {
        const int sgm = idx / nrep, h = idx % nrep;
        float mw[kDecWarps], lw[kDecWarps];
        float mf = NEG_INF;
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) {
            const float* ps = parts + ((size_t)(sgm * kDecWarps + w) * nrep + h) * PSTRIDE + D;
            mw[w] = __ldcg(ps);
            lw[w] = __ldcg(ps + 1);
            mf = fmaxf(mf, mw[w]);
        }
        const float mu = (mf == NEG_INF) ? 0.f : mf;
        float l = 0.f;
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) {
            const float wgt = fast_exp2(mw[w] - mu);
            s_wgt[(sgm * kDecWarps + w) * nrep + h] = wgt;
            l = fmaf(lw[w], wgt, l);
        }
        s_seg_m[idx] = mf;
        s_seg_l[idx] = l;
    }
    __syncthreads();
    // four columns per thread, 16-byte loads: with nrep * D = 512 every thread makes one pass over the strands
    for (int idx = tid; idx < nrep * (D / 4); idx += kDecThreads) {
        const int h = idx / (D / 4), d = (idx % (D / 4)) * 4;
        float mf = NEG_INF;
        for (int sgm = 0; sgm < nsplit; ++sgm) mf = fmaxf(mf, s_seg_m[sgm * nrep + h]);
        const float mu = (mf == NEG_INF) ? 0.f : mf;
        float a[4] = {0.f, 0.f, 0.f, 0.f}, l = 0.f;
#pragma unroll 4
        for (int sgm = 0; sgm < nsplit; ++sgm) {
            float as[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int w = 0; w < kDecWarps; ++w) {
                const int st = sgm * kDecWarps + w;
                const float4 x = __ldcg(reinterpret_cast<const float4*>(parts + ((size_t)st * nrep + h) * PSTRIDE + d));
                const float wgt = s_wgt[st * nrep + h];
                as[0] = fmaf(x.x, wgt, as[0]);
                as[1] = fmaf(x.y, wgt, as[1]);
                as[2] = fmaf(x.z, wgt, as[2]);
                as[3] = fmaf(x.w, wgt, as[3]);
            }
            const float wgt = fast_exp2(s_seg_m[sgm * nrep + h] - mu);
#pragma unroll
            for (int e = 0; e < 4; ++e) a[e] = fmaf(as[e], wgt, a[e]);
            l = fmaf(s_seg_l[sgm * nrep + h], wgt, l);
        }
        const float inv = l > 0.f ? 1.f / l : 0.f;
        uint2 w;
        w.x = pack2_bf16(a[0] * inv, a[1] * inv);
        w.y = pack2_bf16(a[2] * inv, a[3] * inv);
        *reinterpret_cast<uint2*>(p.o + ((size_t)b * p.Hq + (size_t)hkv * nrep + h) * D + d) = w;
    }
    if (STEP && fill + 1 == p.place.C) finish_chunk(p, bh, gridDim.y * gridDim.z, T0);
}

// Launches (segments in all, `splits` of them per (batch, kv-head)) in which every strand gets its own block.  Time of decode_kernel
// over that of strands in a graph of 20 (each of them overlapping where overlaps() says so), 1 / 2 / 4 / 8 query heads per kv-head, on both
// sides of the lines:
//   head_dim 64    1 split: 160 segments 1.19 / 1.18 / 1.19 / 1.19, 192 0.85 / 0.84 / 0.87 / 0.87;  8 splits: 160 1.10 / 1.14 / 1.23 / 1.31,
//                  192 0.92 / 0.92 / 0.98 / 1.10;  16 splits: 96 0.99 / 0.97 / 1.04 / 1.23, 112 1.01 / 0.96 / 1.00 / 1.09;
//                  24 splits, 72 segments: 0.89 / 0.83 / 0.98 / 1.21;  48 splits, 96: 0.65 / 0.63 / 0.76 / 1.07
//   head_dim 128   1 split: 72 segments 1.06 / 1.06 / 1.08 / 1.06, 96 1.03 / 1.04 / 1.05 / 1.02;  4 and 8 splits: 96 segments 1.08 to 1.39, 112
//                  0.83 to 1.14;  16 splits: 96 0.98 / 1.07 / 1.28 / 1.31;  24 splits: 96 0.93 / 1.04 / 1.36 / 1.38;  48 splits: 96 0.77 /
//                  0.94 / 1.32 / 1.31
// Recorded steps (4 query heads): the same lines but for head_dim 64 with 8 splits, where 112 and 144 segments are at 0.96 and 0.95.
// One split needs no combination in decode_kernel; with many splits the last block of a head combines four times as many
// partial results, which more query heads make up for (decode_kernel goes over them head by head).
constexpr int max_strand_segments(int D) { return D == 64 ? 160 : 96; }
static bool use_strands(int D, long long segments, int splits, int nrep) {
    if (D == 64) return segments <= (splits <= 12 ? max_strand_segments(64) : 96) && splits <= (nrep < 8 ? 16 : 48);
    return segments <= (splits == 1 ? 72 : max_strand_segments(128)) && splits <= (nrep == 1 ? 16 : nrep < 4 ? 24 : 96);
}
// V gets slots of its own while all strands fit on the chip at once (148 SMs, one block each at head_dim 128, three at 64).  Time of
// strands with V in the place of K over this, 8 to 36 segments: head_dim 64 1.02 to 1.04 with 2 and 3 splits, 0.99 to 1.00 with 1 and 4, 0.95 to
// 0.99 with 8, 48 to 96 segments 0.92 to 1.05; head_dim 128 up to 3 splits 0.98 to 1.00, recorded steps 1.00 to 1.03, with 4 splits 0.82 to 0.93.
static bool use_both(int D, long long segments, int splits) { return D == 64 ? segments <= 111 : segments <= 37 && splits <= 3; }

// Whether a launch of n blocks overlaps the end of one like it in front of it (see wait_for_previous_launch).  Blocks that find no place
// beside that launch's go where its blocks end first, so that some SMs hold more of them than others.  That costs more than it gives unless
// all find a place beside it, or the launch fills every SM's places as it is.  us per recorded step, behind one another / overlapped (rows
// per head without the window of 512, chunks of 128):
//   head_dim 64    strands: 8 heads x 1100 rows (96 of 444 places) 8.43 / 8.23, 16 x 1900 (256 of 444) 9.60 / 9.90, 16 x 3900 (384 of 444)
//                  11.68 / 11.21, 32 x 1900 (512 of 740) 10.74 / 11.52, 16 x 7800 (640 of 740) 16.64 / 15.94; segments: 64 x 1900 (256 of 592)
//                  16.27 / 15.90, 64 x 3900 (384 of 592) 17.72 / 19.11, 128 x 1900 (512 of 592) 17.97 / 17.45, 128 x 3900 (768) 31.97 / 31.48
//   head_dim 128   strands: 16 heads x 1100 rows (192 of 444) 11.29 / 10.91, 16 x 1900 (256 of 444) 11.97 / 12.58, 16 x 3900 (384 of 444) 14.74 /
//                  14.32; segments: 32 x 1900 (128 of 296) 16.72 / 16.53, 64 x 1100 (192 of 296) 22.24 / 21.74, 128 x 3900 (768) 52.28 / 51.71
struct Places { int sms, per_sm; };
static bool overlaps(long long n, const Places& at) {
    return 2 * n <= (long long)at.sms * at.per_sm || n > (long long)at.sms * (at.per_sm - 1);
}

// The opt-in to more than 48 KB of dynamic shared memory is a per-device attribute of a kernel; the blocks that fit beside one another are
// counted with it.
static cudaError_t prepare_kernel(void (*kernel)(const DecodeParams), int smem, Places (&known)[64], Places& at) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool kept = dev >= 0 && dev < 64;
    at = kept ? known[dev] : Places{};
    if (at.sms > 0 && at.per_sm > 0) return cudaSuccess;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&at.sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&at.per_sm, kernel, kDecThreads, (size_t)smem)) != cudaSuccess) return e;
    if (kept) known[dev] = at;
    return cudaSuccess;
}

static cudaError_t launch(void (*kernel)(const DecodeParams), const DecodeParams& p, dim3 grid, int smem, Places (&known)[64], cudaStream_t st) {
    Places at;
    if (const cudaError_t e = prepare_kernel(kernel, smem, known, at)) return e;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kDecThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = overlaps((long long)grid.x * grid.y * grid.z, at) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <int D, bool STEP, bool BOTH>
static cudaError_t launch_strands(const DecodeParams& p, dim3 grid, cudaStream_t st) {
    static Places known[64] = {};
    grid.x *= kDecWarps;
    return launch(decode_strand_kernel<D, STEP, BOTH>, p, grid, strand_smem<D, BOTH>(), known, st);
}

template <int D, bool STEP>
static cudaError_t launch_decode(const DecodeParams& p, dim3 grid, cudaStream_t st) {
    const long long segments = (long long)grid.x * grid.y * grid.z;
    if (use_strands(D, segments, grid.x, p.nrep))
        return use_both(D, segments, grid.x) ? launch_strands<D, STEP, true>(p, grid, st) : launch_strands<D, STEP, false>(p, grid, st);
    constexpr int smem = kDecWarps * kDecStages * 2 * kTileTok * D * 2;
    static Places known[64] = {};
    return launch(decode_kernel<D, STEP>, p, grid, smem, known, st);
}

static size_t decode_counter_bytes(int B, int Hkv) { return align_up((size_t)B * Hkv * sizeof(int32_t), 256); }
static int decode_max_splits(int max_len) { return cdiv(max_len + 1, kSeg); }
// floats of the partial results: one set per split of a (batch, kv-head) and query head, or, in launches of strands, four per segment
// of the launch and query head (such a launch has at most max_strand_segments of them, and at least one per (batch, kv-head))
static size_t decode_partial_floats(int B, int Hkv, int nrep, int D, int max_splits) {
    const long long heads = (long long)B * Hkv, limit = max_strand_segments(D);
    const size_t whole = (size_t)heads * max_splits * nrep * (D + 2);
    const size_t strands = heads > limit ? 0 : (size_t)min(heads * max_splits, limit) * kDecWarps * nrep * (D + 4);
    return whole > strands ? whole : strands;
}

}  // namespace nats

using namespace nats;

extern "C" __attribute__((visibility("default"))) size_t nats_b200_decode_workspace_bytes(int B, int Hq, int Hkv, int D, int max_len) {
    if (B <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0 || max_len < 0 || Hq % Hkv) return 0;
    const int nrep = Hq / Hkv;
    return decode_counter_bytes(B, Hkv) + decode_partial_floats(B, Hkv, nrep, D, decode_max_splits(max_len)) * sizeof(float);
}

static int decode_impl(const void* d_q, const void* d_k_new, const void* d_v_new, void* d_o,
                       void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap,
                       const int64_t* d_size_global, const int64_t* d_size_local, const int32_t* d_state,
                       int fill, int max_len_bound, int fill_from_state, const uint8_t* d_roles,
                       int B, int Hq, int Hkv, int D, int C, int SW, float sm_scale,
                       void* d_workspace, size_t workspace_bytes, void* stream) {
    NATS_CHECK_ARG(B > 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0, "bad head counts B=%d Hq=%d Hkv=%d", B, Hq, Hkv);
    NATS_CHECK_ARG(C > 0 && SW > 0 && SW % C == 0, "sliding window %d must be a positive multiple of the chunk size %d", SW, C);
    NATS_CHECK_ARG(d_q && d_k_new && d_v_new && d_o && d_cache_k && d_cache_v && d_valid && d_size_global && d_size_local &&
                   d_state && d_workspace, "null pointer");
    NATS_CHECK_ARG(((uintptr_t)d_q | (uintptr_t)d_k_new | (uintptr_t)d_v_new | (uintptr_t)d_o | (uintptr_t)d_cache_k |
                    (uintptr_t)d_cache_v | (uintptr_t)d_workspace) % 16 == 0, "pointers must be 16-byte aligned");
    NATS_CHECK_ARG(fill >= 0 && fill < C, "fill %d must lie in [0, chunk size %d)", fill, C);
    NATS_CHECK_ARG(max_len_bound >= SW && max_len_bound + fill < Lcap,
                   "length bound %d (+ fill %d) does not fit the cache capacity %d", max_len_bound, fill, Lcap);
    NATS_CHECK_ARG(B <= 65535 && Hkv <= 65535, "B and Hkv must not exceed 65535");
    const int nrep = Hq / Hkv;
    if (!(D == 64 || D == 128) || nrep > kMaxRep)
        return fail(NATS_ERR_UNSUPPORTED, "decode supports head_dim {64,128} and up to %d query heads per kv-head; got %d, %d",
                    kMaxRep, D, nrep);
    const int max_len = max_len_bound + C;
    const size_t need = nats_b200_decode_workspace_bytes(B, Hq, Hkv, D, max_len);
    if (workspace_bytes < need) return fail(NATS_ERR_WORKSPACE, "decode workspace: %zu bytes given, %zu needed", workspace_bytes, need);
    DecodeParams p;
    p.q = (const __nv_bfloat16*)d_q; p.k_new = (const __nv_bfloat16*)d_k_new; p.v_new = (const __nv_bfloat16*)d_v_new;
    p.o = (__nv_bfloat16*)d_o; p.ck = (__nv_bfloat16*)d_cache_k; p.cv = (__nv_bfloat16*)d_cache_v; p.valid = d_valid;
    p.size_global = (const long long*)d_size_global; p.size_local = (const long long*)d_size_local; p.state = d_state;
    p.counters = (int32_t*)d_workspace;
    p.partials = (float*)((uint8_t*)d_workspace + decode_counter_bytes(B, Hkv));
    p.Hq = Hq; p.Hkv = Hkv; p.nrep = nrep; p.Lcap = Lcap; p.SW = SW; p.fill = fill; p.fill_from_state = fill_from_state;
    p.max_splits = decode_max_splits(max_len);
    p.scale_log2 = sm_scale * 1.4426950408889634f;
    dim3 grid(cdiv(max_len_bound + fill + 1, kSeg), Hkv, B);
    const bool step = d_roles != nullptr;
    p.place = PlaceParams{};
    if (step) {
        p.place.roles = d_roles; p.place.ck = (uint8_t*)d_cache_k; p.place.cv = (uint8_t*)d_cache_v; p.place.valid = d_valid;
        p.place.size_global = (long long*)d_size_global; p.place.size_local = (long long*)d_size_local;
        p.place.state = const_cast<int32_t*>(d_state);
        p.place.C = C; p.place.SW = SW; p.place.Lcap = Lcap; p.place.rowB = D * 2;
    }
    const cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = (D == 64) ? (step ? launch_decode<64, true>(p, grid, st) : launch_decode<64, false>(p, grid, st))
                              : (step ? launch_decode<128, true>(p, grid, st) : launch_decode<128, false>(p, grid, st));
    NATS_CHECK_CUDA(e);
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_decode_fwd(const void* d_q, const void* d_k_new, const void* d_v_new, void* d_o,
                                    void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap,
                                    const int64_t* d_size_global, const int64_t* d_size_local, const int32_t* d_state,
                                    int fill, int max_len_bound,
                                    int B, int Hq, int Hkv, int D, int C, int SW, float sm_scale,
                                    void* d_workspace, size_t workspace_bytes, void* stream) {
    return decode_impl(d_q, d_k_new, d_v_new, d_o, d_cache_k, d_cache_v, d_valid, Lcap, d_size_global, d_size_local, d_state,
                       fill, max_len_bound, 0, nullptr, B, Hq, Hkv, D, C, SW, sm_scale, d_workspace, workspace_bytes, stream);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_decode_step_fwd(const void* d_q, const void* d_k_new, const void* d_v_new, void* d_o,
                                         void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap,
                                         const int64_t* d_size_global, const int64_t* d_size_local, const int32_t* d_state,
                                         int max_len_bound, int B, int Hq, int Hkv, int D, int C, int SW, float sm_scale,
                                         void* d_workspace, size_t workspace_bytes, void* stream) {
    // the fill is read on the device: size everything for the largest one
    return decode_impl(d_q, d_k_new, d_v_new, d_o, d_cache_k, d_cache_v, d_valid, Lcap, d_size_global, d_size_local, d_state,
                       C - 1, max_len_bound, 1, nullptr, B, Hq, Hkv, D, C, SW, sm_scale, d_workspace, workspace_bytes, stream);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_decode_step(const void* d_q, const void* d_k_new, const void* d_v_new, void* d_o,
                                         const uint8_t* d_roles, void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap,
                                         int64_t* d_size_global, int64_t* d_size_local, int32_t* d_state,
                                         int max_len_bound, int B, int Hq, int Hkv, int D, int C, int SW, float sm_scale,
                                         void* d_workspace, size_t workspace_bytes, void* stream) {
    NATS_CHECK_ARG(d_roles != nullptr, "null pointer");
    return decode_impl(d_q, d_k_new, d_v_new, d_o, d_cache_k, d_cache_v, d_valid, Lcap, d_size_global, d_size_local, d_state,
                       C - 1, max_len_bound, 1, d_roles, B, Hq, Hkv, D, C, SW, sm_scale, d_workspace, workspace_bytes, stream);
}
