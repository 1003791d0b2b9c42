// Role-mask metadata, eviction (keep-set ranks + stream compaction) and decode-step chunk placement.
// All of it is integer / byte work bounded by HBM traffic and launch latency: one block per (batch, kv-head)
// for the scans, 16-byte vectorised row copies for the data movement.
#include <stdarg.h>

#include "place.cuh"

namespace nats {

// ---- host-side error text ---------------------------------------------------------------------
static thread_local char g_err[512] = "";
char* last_error_buf() { return g_err; }
int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

constexpr int kScanThreads = 256;

// =================================================================================================
// role_prep: per-chunk row limit, per-tile max/min limit, kept-tile count
// =================================================================================================
constexpr int kPrepThreads = 1024, kPrepWarps = kPrepThreads / 32;

// Row limits of Nc chunks whose first token sits at position pos0: lim[c] = last query position that may see chunk c.
// The index of the next global chunk (the last chunk counts as global) is a reversed inclusive min-scan, kPrepThreads chunks
// at a time from the end of the sequence: a ballot per warp, the warps' results side by side in shared memory, one block
// barrier per step (the buffer alternates).  *first_gf receives the index of the first global (or last) chunk.  All threads
// of the block call; the limits are visible to the block on return.
__device__ void scan_role_limits(const uint8_t* __restrict__ roles, int Nc, int C, int SW, int pos0,
                                 int32_t* __restrict__ lim, int (*s)[kPrepWarps], int* first_gf) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int carry = Nc - 1, buf = 0;
    for (int hi = Nc; hi > 0; hi -= kPrepThreads, buf ^= 1) {
        const int c = hi - 1 - tid;
        const int role = (c >= 0) ? roles[c] : NATS_ROLE_LOCAL;
        const bool gf = c >= 0 && (role == NATS_ROLE_GLOBAL || c == Nc - 1);
        const unsigned m = __ballot_sync(0xffffffffu, gf);
        const int w_first = hi - 1 - warp * 32;                            // chunk of lane 0; chunks descend with the lane
        if (lane == 0) s[buf][warp] = m ? w_first - (31 - __clz(m)) : kNoLimit;       // the warp's smallest such chunk
        __syncthreads();
        const int all = s[buf][lane];
        const int before = __reduce_min_sync(0xffffffffu, lane < warp ? all : kNoLimit);
        const unsigned mine = m & (0xffffffffu >> (31 - lane));
        int fill = min(before, carry);
        if (mine) fill = min(fill, w_first - (31 - __clz(mine)));
        if (c >= 0) {
            long long l;
            if (role == NATS_ROLE_SLIDING) l = (long long)pos0 + (long long)c * C + SW + C - 1;
            else if (gf) l = kNoLimit;
            else l = (long long)pos0 + ((long long)fill + 1) * C - 1;
            lim[c] = (int)min(l, (long long)kNoLimit);
            if (c == 0) *first_gf = fill;
        }
        carry = min(carry, __reduce_min_sync(0xffffffffu, all));
    }
    __syncthreads();
}
static_assert(kPrepWarps == 32, "a warp holds one value per warp of the block");

// Per 128-row KV tile: max / min of the limits of the chunks it overlaps, and how many query tiles keep it.  Query row i
// sits at position q_off + i; there are Nt query tiles of 128 rows.  Fine chunks: a warp per tile (coalesced loads); others:
// a thread per tile.  open_max (may be null) and dense_min: see FarLists.  Returns this thread's share of the kept count.
__device__ unsigned long long tile_limits(const int32_t* __restrict__ lim, int Nkv, int C, int Ntk, int q_off, int Nt,
                                          int32_t* __restrict__ tmax, int32_t* __restrict__ tmin, int32_t* __restrict__ open_max, int dense_min) {
    unsigned long long mine = 0;
    const bool wide = C < 16;
    const int lane = threadIdx.x & 31;
    const int first_tile = wide ? threadIdx.x >> 5 : threadIdx.x, step = wide ? kPrepWarps : kPrepThreads;
    for (int kt = first_tile; kt < Ntk; kt += step) {
        const int c0 = (int)(((long long)kt * kTile) / C);
        const int c1 = (int)(min((long long)kt * kTile + kTile - 1, (long long)Nkv - 1) / C);
        int mx = -1, mn = kNoLimit, om = -1, listed = 0;
        for (int c = wide ? c0 + lane : c0; c <= c1; c += wide ? 32 : 1) {
            const int l = lim[c];
            mx = max(mx, l);
            mn = min(mn, l);
            if (l != kNoLimit) om = max(om, l);
            else ++listed;
        }
        if (wide) {
            mx = __reduce_max_sync(0xffffffffu, mx);
            mn = __reduce_min_sync(0xffffffffu, mn);
            om = __reduce_max_sync(0xffffffffu, om);
            listed = __reduce_add_sync(0xffffffffu, listed);
            if (lane != 0) continue;
        }
        tmax[kt] = mx;
        tmin[kt] = mn;
        if (open_max != nullptr) open_max[kt] = 2 * min(om, kOpenMax) + (listed >= dense_min ? 1 : 0);
        // query tiles t that keep the tile: last row position >= first tile row, first row position <= mx
        const long long first = (long long)kt * kTile - q_off - (kTile - 1);
        const int t_min = first <= 0 ? 0 : (int)((first + kTile - 1) / kTile);
        if (mx >= q_off) {
            const int t_max = min(Nt - 1, (mx - q_off) / kTile);
            if (t_max >= t_min) mine += (unsigned long long)(t_max - t_min + 1);
        }
    }
    return mine;
}

// The chunks that stay visible for good, in order, and how many of them lie in front of every 128-row tile (chunks divide a
// tile: cpt per tile), without those of dense tiles.  All threads of the block call, after scan_role_limits and tile_limits.
__device__ void list_far_chunks(const int32_t* __restrict__ lim, int Nc, int cpt, int Ntk, int32_t* __restrict__ list,
                                int32_t* __restrict__ before_tile, int32_t* __restrict__ open_max, int max_listed, int dense_min, int (*s)[kPrepWarps]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int base = 0, buf = 0;
    const bool any_dense = dense_min <= cpt;
    if (any_dense) __syncthreads();                       // open_max of every tile is there
    for (int c0 = 0; c0 < Nc; c0 += kPrepThreads, buf ^= 1) {
        const int c = c0 + tid;
        const bool dense = any_dense && c < Nc && (open_max[c / cpt] & 1);
        const bool keep = c < Nc && lim[c] == kNoLimit && !dense;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) s[buf][warp] = __popc(m);
        __syncthreads();
        const int all = s[buf][lane];
        const int rank = base + __reduce_add_sync(0xffffffffu, lane < warp ? all : 0) + __popc(m & ((1u << lane) - 1u));
        if (keep) list[rank] = c;
        if (c < Nc && c % cpt == 0) before_tile[c / cpt] = rank;
        base += __reduce_add_sync(0xffffffffu, all);
    }
    if (tid == 0) before_tile[Ntk] = base;
    if (base <= max_listed) return;
    __syncthreads();
    for (int kt = tid; kt < Ntk; kt += kPrepThreads)
        if (before_tile[kt + 1] > max_listed) open_max[kt] = 2 * kOpenMax;
}

__global__ void __launch_bounds__(kPrepThreads)
role_prep_kernel(const uint8_t* __restrict__ roles, int Nc, int N, int C, int SW, int Nt,
                 int32_t* __restrict__ lim, int32_t* __restrict__ tmax, int32_t* __restrict__ tmin,
                 long long* __restrict__ kept, FarLists far, int32_t* __restrict__ counter) {
    if (counter != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *counter = 0;
    const int bh = blockIdx.x, tid = threadIdx.x;
    roles += (size_t)bh * Nc;
    lim += (size_t)bh * Nc;
    tmax += (size_t)bh * Nt;
    tmin += (size_t)bh * Nt;
    __shared__ int s[2][kPrepWarps];
    __shared__ int first_gf;
    __shared__ unsigned long long kept_sm;
    if (tid == 0) kept_sm = 0;
    scan_role_limits(roles, Nc, C, SW, 0, lim, s, &first_gf);
    const unsigned long long mine = tile_limits(lim, N, C, Nt, 0, Nt, tmax, tmin, far.list ? far.open_max + (size_t)bh * Nt : nullptr, far.dense_min);
    if (far.list != nullptr)
        list_far_chunks(lim, Nc, kTile / C, Nt, far.list + (size_t)bh * Nc, far.before_tile + (size_t)bh * (Nt + 1), far.open_max + (size_t)bh * Nt,
                        far.max_listed, far.dense_min, s);
    if (kept != nullptr) {
        if (mine) atomicAdd(&kept_sm, mine);
        __syncthreads();
        if (tid == 0) kept[bh] = (long long)kept_sm;
    }
}

// The same metadata for a multi-token call over an existing cache.  The KV sequence is the physical cache layout
// [ring | kept global | kept local | gap | unfinished chunk + new tokens]; T0 = first position of the unfinished chunk.
struct PastPrepParams {
    const uint8_t* roles;                       // [BH, Ncn] roles of the chunks from the unfinished one on
    const uint8_t* valid;                       // [BH, Lcap]; only the ring flags [0, SW) of a head are read
    const long long* size_global; const long long* size_local;
    int32_t* lim; int32_t* tmax; int32_t* tmin; long long* kept;
    int Ncn, Lcap, T0, C, SW, tail, Nq, q_off, Nkv, Nc, Ntk, Nt;
    FarLists far;
    int32_t* counter;
};

__global__ void __launch_bounds__(kPrepThreads) role_prep_past_kernel(const PastPrepParams p) {
    if (p.counter != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *p.counter = 0;
    const int bh = blockIdx.x, tid = threadIdx.x;
    const uint8_t* roles = p.roles + (size_t)bh * p.Ncn;
    const uint8_t* valid = p.valid + (size_t)bh * p.Lcap;
    int32_t* lim = p.lim + (size_t)bh * p.Nc;
    __shared__ int s[2][kPrepWarps];
    __shared__ int first_gf;
    __shared__ unsigned long long kept_sm;
    if (tid == 0) kept_sm = 0;
    const int n_old = p.T0 / p.C, W = p.SW / p.C;
    // new chunks: the rule of a first call, positions counted from T0
    scan_role_limits(roles, p.Ncn, p.C, p.SW, p.T0, lim + n_old, s, &first_gf);
    // cached chunks
    const int sg = (int)(p.size_global[bh] / p.C), sl = (int)(p.size_local[bh] / p.C);
    const long long lim_local = (long long)p.T0 + ((long long)first_gf + 1) * p.C - 1;   // until the first new global chunk ends
    for (int j = tid; j < n_old; j += kPrepThreads) {
        int l;
        if (j < W) {
            // ring slot j was written `age` chunks before the newest one; a sliding chunk is seen by the SW/C chunks after it
            const int age = ((p.tail / p.C - 1 - j) % W + W) % W;
            l = valid[(size_t)j * p.C] ? p.T0 + (W - age) * p.C - 1 : -1;
        } else if (j < sg) {
            l = kNoLimit;
        } else if (j < sg + sl) {
            l = (int)min(lim_local, (long long)kNoLimit);
        } else {
            l = -1;                                   // between this head's length and the longest head's
        }
        lim[j] = l;
    }
    __syncthreads();
    const unsigned long long mine = tile_limits(lim, p.Nkv, p.C, p.Ntk, p.q_off, p.Nt, p.tmax + (size_t)bh * p.Ntk, p.tmin + (size_t)bh * p.Ntk,
                                                p.far.list ? p.far.open_max + (size_t)bh * p.Ntk : nullptr, p.far.dense_min);
    if (p.far.list != nullptr)
        list_far_chunks(lim, p.Nc, kTile / p.C, p.Ntk, p.far.list + (size_t)bh * p.Nc, p.far.before_tile + (size_t)bh * (p.Ntk + 1),
                        p.far.open_max + (size_t)bh * p.Ntk, p.far.max_listed, p.far.dense_min, s);
    if (p.kept != nullptr) {
        if (mine) atomicAdd(&kept_sm, mine);
        __syncthreads();
        if (tid == 0) p.kept[bh] = (long long)kept_sm;
    }
}

// Number of keys every query row may see (first call).  A chunk c ends being visible in front of chunk (lim[c] + 1) / C: limits
// are one short of a chunk boundary.  A row of chunk x sees the rows up to its own, less C for every chunk that has ended by
// x.  A block takes span chunks of a kv-head: one pass over the limits counts the chunks that have ended in front of its first
// chunk and, in a histogram, at each of its chunks; a scan turns it into the number per chunk, and the rows are written for
// each query head of the group.  A block reads all limits up to its last chunk, so that the reads still grow with the square of the
// length, by span rows at a time (a loop over the chunks in front of every row reads one chunk per row and chunk).
constexpr int kCountRows = 4096;                 // rows per block; 256 chunks (the histogram) where those are fewer

__global__ void __launch_bounds__(kScanThreads)
visible_count_kernel(const int32_t* __restrict__ lim, int Hq, int Hkv, int N, int C, int Nc, int span, int32_t* __restrict__ out) {
    const int bh = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    lim += (size_t)bh * Nc;
    const int x0 = blockIdx.x * span, x1 = min(x0 + span, Nc);
    __shared__ int ended[kScanThreads];          // [i]: chunks that end in front of chunk x0 + i, then the running total
    __shared__ int s_warp[kScanThreads / 32];
    __shared__ int s_before;
    ended[tid] = 0;
    if (tid == 0) s_before = 0;
    __syncthreads();
    int before = 0;
    for (int c = tid; c < x1; c += kScanThreads) {
        const int l = lim[c];
        if (l == kNoLimit) continue;
        const int e = (l + 1) / C;
        if (e < x0) ++before;
        else if (e < x1) atomicAdd(&ended[e - x0], 1);
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0 && before) atomicAdd(&s_before, before);
    __syncthreads();
    const int incl = warp_incl_scan(ended[tid], lane);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int total = s_before + incl;
    for (int w = 0; w < warp; ++w) total += s_warp[w];
    ended[tid] = total;
    __syncthreads();
    const int nrep = Hq / Hkv, b = bh / Hkv, hkv = bh % Hkv;
    const long long q1 = min((long long)x1 * C, (long long)N);
    for (long long q = (long long)x0 * C + tid; q < q1; q += kScanThreads) {
        const int n = (int)q + 1 - C * ended[(int)(q / C) - x0];
        for (int r = 0; r < nrep; ++r) out[((size_t)b * Hq + hkv * nrep + r) * N + q] = n;
    }
}

// =================================================================================================
// evict_plan: keep flags -> destination ranks (ballot + prefix sum), sizes, max length
// =================================================================================================
__device__ __forceinline__ void publish_max_len(int32_t* state, int len, int nblocks, const int32_t* status = nullptr, int32_t* report = nullptr) {
    // state[1] accumulates the maximum over blocks; the last block to arrive publishes it in state[0]
    // and leaves the scratch words zero for the next call.  No block ever waits for another.
    // report (host memory, may be null) gets the maximum and *status as well.
    __shared__ int last;
    if (threadIdx.x == 0) {
        atomicMax(&state[1], len);
        __threadfence();
        const int ticket = atomicAdd(&state[2], 1);
        last = (ticket == nblocks - 1);
        if (last) {
            __threadfence();
            const int m = atomicExch(&state[1], 0);
            state[0] = m;
            state[2] = 0;
            if (report != nullptr) {
                report[0] = m;
                report[1] = *reinterpret_cast<const volatile int32_t*>(status);
            }
        }
    }
}

// base == nullptr: first call (the cache is empty: sizes are outputs).  Otherwise the sizes are read and updated, and
// base[bh] receives the chunk slot (counted from position 0) the first kept chunk of this call goes to: behind the
// kept locals if the call brings no global chunk, else behind the kept globals (the locals in front of it are dropped).
__global__ void __launch_bounds__(kPrepThreads)
evict_plan_kernel(const uint8_t* __restrict__ roles, int Nc, int n_full, int C, int SW,
                  int32_t* __restrict__ rank, long long* __restrict__ size_global,
                  long long* __restrict__ size_local, int32_t* __restrict__ state, int32_t* __restrict__ base,
                  const int32_t* status, int32_t* report) {
    const int bh = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    roles += (size_t)bh * Nc;
    rank += (size_t)bh * Nc;
    __shared__ int s_last[kPrepWarps];
    __shared__ int s_count[2][kPrepWarps];
    // pass 1: last global chunk among the complete chunks
    int lg = -1;
    for (int c = tid; c < n_full; c += kPrepThreads)
        if (roles[c] == NATS_ROLE_GLOBAL) lg = c;
    lg = __reduce_max_sync(0xffffffffu, lg);
    if (lane == 0) s_last[warp] = lg;
    __syncthreads();
    const int last_g = __reduce_max_sync(0xffffffffu, s_last[lane]);
    // pass 2: ordered ranks of the kept chunks, kPrepThreads at a time: ballots, the warps' counts side by side in shared
    // memory (kept in the low half, global in the high half), one block barrier per step (the buffer alternates)
    int n_kept = 0, n_g = 0, buf = 0;
    for (int c0 = 0; c0 < Nc; c0 += kPrepThreads, buf ^= 1) {
        const int c = c0 + tid;
        const int role = (c < n_full) ? roles[c] : -1;
        const bool is_g = role == NATS_ROLE_GLOBAL;
        const bool keep = is_g || (role == NATS_ROLE_LOCAL && c > last_g);
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        const unsigned mg = __ballot_sync(0xffffffffu, is_g);
        if (lane == 0) s_count[buf][warp] = __popc(m) | (__popc(mg) << 16);
        __syncthreads();
        const int all = s_count[buf][lane];
        const int before = n_kept + __reduce_add_sync(0xffffffffu, lane < warp ? all & 0xffff : 0);
        // kept chunk: its rank; other chunks: -1 - (kept chunks in front of it), so that the number of kept chunks up to any
        // index can be read off without a scan (the compaction finds the chunk of a given rank by bisection)
        const int kept_before = before + __popc(m & ((1u << lane) - 1u));
        if (c < Nc) rank[c] = keep ? kept_before : -1 - kept_before;
        n_kept += __reduce_add_sync(0xffffffffu, all & 0xffff);
        n_g += __reduce_add_sync(0xffffffffu, all >> 16);
    }
    long long sg0 = SW, sl0 = 0;
    if (base != nullptr) { sg0 = size_global[bh]; sl0 = size_local[bh]; }
    const long long sg = sg0 + (long long)C * n_g;
    const long long sl = (last_g >= 0 ? 0 : sl0) + (long long)C * (n_kept - n_g);
    __syncthreads();                                      // every thread has read the sizes
    if (tid == 0) {
        size_global[bh] = sg;
        size_local[bh] = sl;
        if (base != nullptr) base[bh] = (int)((last_g >= 0 ? sg0 : sg0 + sl0) / C);
    }
    publish_max_len(state, (int)(sg + sl), gridDim.x, status, report);
}

// =================================================================================================
// evict_compact: ring fill + kept-chunk copies + pending tail + zero / valid bookkeeping
// =================================================================================================
constexpr int kCopyThreads = 256;
constexpr int kTokPerBlock = 64;

struct CompactParams {
    // source of the tokens of this call: [BH, src_stride, rowB] bytes; token t of the call sits at row src_off + t.
    // First call: the caller's K/V (src_off 0).  Call over an existing cache: the old cache buffer, to which the new
    // tokens were appended behind the unfinished chunk (src_off = old T0); it also holds the old ring and kept region.
    const uint8_t* k; const uint8_t* v; const uint8_t* old_valid;
    const uint8_t* roles; const int32_t* rank;   // [BH, Nc]
    const int32_t* base;                         // [BH] or nullptr (first call: SW / C)
    const long long* size_global; const long long* size_local; const int32_t* state;
    uint8_t* ck; uint8_t* cv; uint8_t* valid;    // [BH, Lcap, rowB], [BH, Lcap]
    long long src_stride;                        // rows per head of the source
    int src_off, tail, N, Nc, n_full, C, SW, Lcap, rowB;        // rowB = D * 2 bytes; N = tokens of the call
    int nB;                                      // blocks of the ring section
};

// eight bf16 of a source row: from bf16, or from fp32 rounded on the way (the source row is twice as long)
template <bool F32>
__device__ __forceinline__ uint4 load_row_vec(const uint8_t* base, size_t off) {
    if (!F32) return ld16_stream(base + off);
    return round8(ld16_stream(base + 2 * off), ld16_stream(base + 2 * off + 16));
}

template <bool F32>
__global__ void __launch_bounds__(kCopyThreads) evict_compact_kernel(const CompactParams p) {
    const int bh = blockIdx.y, tid = threadIdx.x;
    const int vpt = p.rowB >> 4;                          // 16-byte vectors per token row
    const int tpp = kCopyThreads / vpt;                   // tokens per pass
    const int trow = tid / vpt, tvec = (tid % vpt) << 4;
    const uint8_t* k = p.k + (size_t)bh * p.src_stride * p.rowB * (F32 ? 2 : 1);
    const uint8_t* v = p.v + (size_t)bh * p.src_stride * p.rowB * (F32 ? 2 : 1);
    uint8_t* ck = p.ck + (size_t)bh * p.Lcap * p.rowB;
    uint8_t* cv = p.cv + (size_t)bh * p.Lcap * p.rowB;
    uint8_t* valid = p.valid + (size_t)bh * p.Lcap;
    const uint8_t* roles = p.roles + (size_t)bh * p.Nc;
    const int32_t* rank = p.rank + (size_t)bh * p.Nc;
    const bool past = p.base != nullptr;
    const int base = past ? p.base[bh] : p.SW / p.C;      // chunk slot of the first kept chunk of this call
    const uint4 zero = make_uint4(0, 0, 0, 0);
    int blk = blockIdx.x;
    if (blk < p.nB) {
        if (trow >= tpp) return;                          // head dims whose vector count does not divide 256
        // section B: the last min(n_full, SW/C) complete chunks of the call go to the ring slots behind the tail (data if
        // the chunk is a sliding one, else zeros + invalid); slots the call does not reach keep what they held
        const int n_upd = min(p.n_full, p.SW / p.C);
        const int n_fills = n_upd * p.C;
        const int src0 = (p.n_full - n_upd) * p.C;
        const int s0 = blk * kTokPerBlock;
        for (int i = trow; i < kTokPerBlock; i += tpp) {
            const int slot = s0 + i;
            if (slot >= p.SW) break;
            const int j = (slot - p.tail + p.SW) % p.SW;          // position in the write order of this call
            const size_t dst = (size_t)slot * p.rowB + tvec;
            if (j < n_fills) {
                const bool sw = roles[(src0 + j) / p.C] == NATS_ROLE_SLIDING;
                const size_t src = (size_t)(p.src_off + src0 + j) * p.rowB + tvec;
                st16(ck + dst, sw ? load_row_vec<F32>(k, src) : zero);
                st16(cv + dst, sw ? load_row_vec<F32>(v, src) : zero);
                if (tvec == 0) valid[slot] = sw ? 1 : 0;
            } else if (past) {
                st16(ck + dst, ld16_stream(k + dst));
                st16(cv + dst, ld16_stream(v + dst));
                if (tvec == 0) valid[slot] = p.old_valid[(size_t)bh * p.src_stride + slot];
            } else {
                st16(ck + dst, zero);
                st16(cv + dst, zero);
                if (tvec == 0) valid[slot] = 0;
            }
        }
        return;
    }
    blk -= p.nB;
    // main region, destination-driven.  [SW, base*C) = what the cache kept from before this call; [base*C, len) = the kept
    // chunks of this call (slot r holds the chunk whose rank is r: ranks grow with the chunk index, so the chunk is found
    // by bisection); [len, Lcap) is zero except the tokens of the unfinished chunk at [T0, T0+rem).  Launching blocks per
    // destination instead of per source token matters: most source chunks are not kept.
    // Step 1: one thread per destination token of the block works out where its row comes from (source row in k / v,
    // -1: zeros, -2: leave alone), so that the bisection's chain of dependent loads is paid once per block and not in front
    // of every copy.  Step 2: every thread loads all of its 16-byte vectors, then stores them.
    __shared__ int s_src[kTokPerBlock];
    const int len = (int)(p.size_global[bh] + p.size_local[bh]);
    const int T0 = p.state[0];
    const int rem = p.N - p.n_full * p.C;
    const int d0 = p.SW + blk * kTokPerBlock;
    if (tid < kTokPerBlock) {
        const int d = d0 + tid;
        int src = -2;
        if (d < p.Lcap) {
            const bool in_tail = d >= T0 && d < T0 + rem;
            valid[d] = (d < len || in_tail) ? 1 : 0;
            if (d < len) {
                if (d < base * p.C) {
                    if (past) src = d;
                } else {
                    // the chunk of rank r: the smallest index up to which r + 1 chunks are kept
                    const int r = d / p.C - base;
                    int lo = r, hi = p.n_full - 1;                 // it cannot sit in front of index r
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        const int v = rank[mid];
                        const int kept_upto = v >= 0 ? v + 1 : -1 - v;         // kept chunks in [0, mid]
                        if (kept_upto >= r + 1) hi = mid; else lo = mid + 1;
                    }
                    src = p.src_off + lo * p.C + d % p.C;
                }
            } else if (in_tail) {
                src = p.src_off + p.n_full * p.C + (d - T0);
            } else {
                src = -1;
            }
        }
        s_src[tid] = src;
    }
    __syncthreads();
    if (trow >= tpp) return;                              // head dims whose vector count does not divide 256
    constexpr int kBatch = 4;
    for (int i0 = trow; i0 < kTokPerBlock; i0 += kBatch * tpp) {
        uint4 a[kBatch], b[kBatch];
        int sr[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int i = i0 + u * tpp;
            sr[u] = i < kTokPerBlock ? s_src[i] : -2;
            a[u] = b[u] = zero;
            if (sr[u] >= 0) {
                const size_t src = (size_t)sr[u] * p.rowB + tvec;
                a[u] = load_row_vec<F32>(k, src);
                b[u] = load_row_vec<F32>(v, src);
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            if (sr[u] == -2) continue;
            const size_t dst = (size_t)(d0 + i0 + u * tpp) * p.rowB + tvec;
            st16(ck + dst, a[u]);
            st16(cv + dst, b[u]);
        }
    }
}

// bf16 copies of up to three fp32 arrays: a caller's q, k and v in one launch.  Bound by HBM at sizes that matter and by the
// launch at small ones.
struct Bf16Params {
    const uint8_t* x[3]; uint8_t* y[3];
    long long n8[3];                             // groups of eight elements
};

__global__ void __launch_bounds__(kCopyThreads) to_bf16_kernel(const Bf16Params p) {
    const long long step = (long long)gridDim.x * kCopyThreads;
#pragma unroll
    for (int a = 0; a < 3; ++a)
        for (long long i = (long long)blockIdx.x * kCopyThreads + threadIdx.x; i < p.n8[a]; i += step)
            st16(p.y[a] + i * 16, round8(ld16_stream(p.x[a] + i * 32), ld16_stream(p.x[a] + i * 32 + 16)));
}

// Appends the K/V of new tokens to a cache buffer at row `pos` of every (b,h) and marks them valid.
struct AppendParams {
    const uint8_t* k; const uint8_t* v;          // [BH, x_len, rowB]
    uint8_t* ck; uint8_t* cv; uint8_t* valid;    // [BH, Lcap, rowB], [BH, Lcap]
    int x_len, pos, Lcap, rowB;
};

__global__ void __launch_bounds__(kCopyThreads) cache_append_kernel(const AppendParams p) {
    const int bh = blockIdx.y, tid = threadIdx.x;
    const int vpt = p.rowB >> 4, tpp = kCopyThreads / vpt;
    const int trow = tid / vpt, tvec = (tid % vpt) << 4;
    if (trow >= tpp) return;
    const uint8_t* k = p.k + (size_t)bh * p.x_len * p.rowB;
    const uint8_t* v = p.v + (size_t)bh * p.x_len * p.rowB;
    uint8_t* ck = p.ck + ((size_t)bh * p.Lcap + p.pos) * p.rowB;
    uint8_t* cv = p.cv + ((size_t)bh * p.Lcap + p.pos) * p.rowB;
    uint8_t* valid = p.valid + (size_t)bh * p.Lcap + p.pos;
    const int t0 = blockIdx.x * kTokPerBlock;
    for (int i = trow; i < kTokPerBlock; i += tpp) {
        const int t = t0 + i;
        if (t >= p.x_len) break;
        const size_t o = (size_t)t * p.rowB + tvec;
        st16(ck + o, ld16_stream(k + o));
        st16(cv + o, ld16_stream(v + o));
        if (tvec == 0) valid[t] = 1;
    }
}

// A larger buffer, written once: rows [0, pos) from the old one, the new tokens behind them, zeros and invalid flags to its end.
// Bound by HBM: a segment of 4 000 tokens over 14 000 rows (8 heads of 128, room for 21 000) takes one pass over what is read and
// written; fills of the new buffers, strided copies of the old ones and the append took three (a prompt of 24 576 tokens in four segments,
// 32 / 8 heads of 128: 1140 -> 1050 us in all).
struct GrowParams {
    AppendParams a;                              // the new buffers and the new tokens
    const uint8_t* k; const uint8_t* v; const uint8_t* valid;      // [BH, rows, rowB], [BH, rows]
    int rows;
};

__global__ void __launch_bounds__(kCopyThreads) cache_grow_append_kernel(const GrowParams p) {
    constexpr int kInFlight = 4;
    const AppendParams& a = p.a;
    const int bh = blockIdx.y, tid = threadIdx.x;
    const int vpt = a.rowB >> 4, tpp = kCopyThreads / vpt;
    const int trow = tid / vpt, tvec = (tid % vpt) << 4;
    if (trow >= tpp) return;
    const size_t old_row = (size_t)bh * p.rows, new_row = (size_t)bh * a.x_len, dst_row = (size_t)bh * a.Lcap;
    const int end = min(a.Lcap, (int)(blockIdx.x + 1) * kTokPerBlock);
    for (int r0 = blockIdx.x * kTokPerBlock + trow; r0 < end; r0 += tpp * kInFlight) {
        uint4 kk[kInFlight], vv[kInFlight];
#pragma unroll
        for (int x = 0; x < kInFlight; ++x) {
            const int r = r0 + x * tpp;
            kk[x] = vv[x] = make_uint4(0, 0, 0, 0);
            if (r < min(a.pos, end)) {
                const size_t o = (old_row + r) * a.rowB + tvec;
                kk[x] = ld16_stream(p.k + o);
                vv[x] = ld16_stream(p.v + o);
            } else if (r < min(a.pos + a.x_len, end)) {
                const size_t o = (new_row + r - a.pos) * a.rowB + tvec;
                kk[x] = ld16_stream(a.k + o);
                vv[x] = ld16_stream(a.v + o);
            }
        }
#pragma unroll
        for (int x = 0; x < kInFlight; ++x) {
            const int r = r0 + x * tpp;
            if (r >= end) break;
            const size_t o = (dst_row + r) * a.rowB + tvec;
            st16(a.ck + o, kk[x]);
            st16(a.cv + o, vv[x]);
            if (tvec == 0) a.valid[dst_row + r] = r < a.pos ? p.valid[old_row + r] : r < a.pos + a.x_len;
        }
    }
}

// =================================================================================================
// decode_place: a chunk completed by decode steps goes to the ring and, unless sliding, behind the kept chunks
// =================================================================================================
__global__ void __launch_bounds__(kCopyThreads) decode_place_kernel(const PlaceParams p) {
    int tail = p.tail;
    if (p.from_state) {
        if (p.state[4] + 1 != p.C) return;        // the step did not complete a chunk (uniform for the grid)
        tail = p.state[5];
    }
    const int new_len = place_chunk<kCopyThreads>(p, blockIdx.x, p.state[0], tail);
    publish_max_len(p.state, new_len, gridDim.x);
}

}  // namespace nats

// =================================================================================================
// C ABI
// =================================================================================================
using namespace nats;

extern "C" __attribute__((visibility("default"))) const char* nats_b200_last_error(void) { return last_error_buf(); }

extern "C" __attribute__((visibility("default"))) const char* nats_b200_build_info(void) {
    return "libnats_b200 sm_100a; prefill tile 128x128 (tcgen05/TMEM/TMA), head_dim {64,128}, N <= 524288; "
           "decode head_dim {64,128}, group size 1..8";
}

static int check_common(int B, int Hkv, int N, int C, int SW) {
    NATS_CHECK_ARG(B > 0 && Hkv > 0 && N > 0, "B, Hkv and N must be positive (got %d, %d, %d)", B, Hkv, N);
    NATS_CHECK_ARG(C > 0 && SW > 0 && SW % C == 0, "sliding window %d must be a positive multiple of the chunk size %d", SW, C);
    NATS_CHECK_ARG((long long)B * Hkv <= 65535, "B * Hkv = %lld exceeds the grid limit 65535", (long long)B * Hkv);
    return NATS_OK;
}

int nats::role_prep(const uint8_t* d_roles, int B, int Hkv, int N, int C, int SW, int32_t* d_lim, int32_t* d_tile_max,
                    int32_t* d_tile_min, int64_t* d_kept_tiles, const FarLists& far, int32_t* d_counter, void* stream) {
    if (int rc = check_common(B, Hkv, N, C, SW)) return rc;
    NATS_CHECK_ARG(d_roles && d_lim && d_tile_max && d_tile_min, "null pointer");
    const int Nc = cdiv(N, C), Nt = cdiv(N, kTile);
    role_prep_kernel<<<B * Hkv, kPrepThreads, 0, (cudaStream_t)stream>>>(
        d_roles, Nc, N, C, SW, Nt, d_lim, d_tile_max, d_tile_min, (long long*)d_kept_tiles, far, d_counter);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_role_prep(const uint8_t* d_roles, int B, int Hkv, int N, int C, int SW,
                                   int32_t* d_lim, int32_t* d_tile_max, int32_t* d_tile_min, int64_t* d_kept_tiles,
                                   void* stream) {
    return role_prep(d_roles, B, Hkv, N, C, SW, d_lim, d_tile_max, d_tile_min, d_kept_tiles, FarLists{}, nullptr, stream);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_visible_counts(const int32_t* d_lim, int B, int Hq, int Hkv, int N, int C,
                                                                    int32_t* d_n_visible, void* stream) {
    NATS_CHECK_ARG(B > 0 && Hq > 0 && Hkv > 0 && N > 0 && C > 0 && Hq % Hkv == 0 && (long long)B * Hkv <= 65535,
                   "bad shape B=%d Hq=%d Hkv=%d N=%d C=%d", B, Hq, Hkv, N, C);
    NATS_CHECK_ARG(d_lim && d_n_visible, "null pointer");
    const int Nc = cdiv(N, C);
    int span = kCountRows / C;
    span = span < 1 ? 1 : span > kScanThreads ? kScanThreads : span;
    dim3 grid(cdiv(Nc, span), B * Hkv);
    visible_count_kernel<<<grid, kScanThreads, 0, (cudaStream_t)stream>>>(d_lim, Hq, Hkv, N, C, Nc, span, d_n_visible);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_evict_plan(const uint8_t* d_roles, int B, int Hkv, int N, int C, int SW,
                                    int32_t* d_rank, int64_t* d_size_global, int64_t* d_size_local, int32_t* d_state,
                                    void* stream) {
    if (int rc = check_common(B, Hkv, N, C, SW)) return rc;
    NATS_CHECK_ARG(d_roles && d_rank && d_size_global && d_size_local && d_state, "null pointer");
    const int Nc = cdiv(N, C);
    evict_plan_kernel<<<B * Hkv, kPrepThreads, 0, (cudaStream_t)stream>>>(
        d_roles, Nc, N / C, C, SW, d_rank, (long long*)d_size_global, (long long*)d_size_local, d_state, nullptr, nullptr, nullptr);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

int nats::role_prep_past(
    const uint8_t* d_roles_new, const uint8_t* d_valid, const int64_t* d_size_global, const int64_t* d_size_local,
    int B, int Hkv, int x_len, int C, int SW, int valid_stride, int t0, int fill, int tail,
    int32_t* d_lim, int32_t* d_tile_max, int32_t* d_tile_min, int64_t* d_kept_tiles, const FarLists& far, int32_t* d_counter, void* stream) {
    if (int rc = check_common(B, Hkv, x_len, C, SW)) return rc;
    NATS_CHECK_ARG(d_roles_new && d_valid && d_size_global && d_size_local && d_lim && d_tile_max && d_tile_min, "null pointer");
    NATS_CHECK_ARG(t0 >= SW && t0 % C == 0 && fill >= 0 && fill < C, "tail offset %d must be a chunk multiple >= the window, fill %d in [0, chunk)", t0, fill);
    NATS_CHECK_ARG(tail >= 0 && tail < SW && tail % C == 0, "ring tail %d must be a chunk multiple inside the window %d", tail, SW);
    NATS_CHECK_ARG(valid_stride >= SW, "the flags of a head (%d) must cover the ring (%d)", valid_stride, SW);
    NATS_CHECK_ARG((long long)t0 + fill + x_len <= 0x7fffffffLL - 2 * (long long)(SW + C), "sequence too long");
    PastPrepParams p;
    p.roles = d_roles_new; p.valid = d_valid;
    p.size_global = (const long long*)d_size_global; p.size_local = (const long long*)d_size_local;
    p.lim = d_lim; p.tmax = d_tile_max; p.tmin = d_tile_min; p.kept = (long long*)d_kept_tiles;
    p.Ncn = cdiv(fill + x_len, C); p.Lcap = valid_stride; p.T0 = t0; p.C = C; p.SW = SW; p.tail = tail;
    p.Nq = x_len; p.q_off = t0 + fill; p.Nkv = t0 + fill + x_len;
    p.Nc = cdiv(p.Nkv, C); p.Ntk = cdiv(p.Nkv, kTile); p.Nt = cdiv(x_len, kTile);
    p.far = far;
    p.counter = d_counter;
    role_prep_past_kernel<<<B * Hkv, kPrepThreads, 0, (cudaStream_t)stream>>>(p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_role_prep_past(
    const uint8_t* d_roles_new, const uint8_t* d_valid, const int64_t* d_size_global, const int64_t* d_size_local,
    int B, int Hkv, int x_len, int C, int SW, int valid_stride, int t0, int fill, int tail,
    int32_t* d_lim, int32_t* d_tile_max, int32_t* d_tile_min, int64_t* d_kept_tiles, void* stream) {
    return role_prep_past(d_roles_new, d_valid, d_size_global, d_size_local, B, Hkv, x_len, C, SW, valid_stride, t0, fill, tail,
                          d_lim, d_tile_max, d_tile_min, d_kept_tiles, FarLists{}, nullptr, stream);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_evict_plan_past(
    const uint8_t* d_roles_new, int B, int Hkv, int n_tokens, int C, int SW, int32_t* d_rank, int32_t* d_base,
    int64_t* d_size_global, int64_t* d_size_local, int32_t* d_state, void* stream) {
    if (int rc = check_common(B, Hkv, n_tokens, C, SW)) return rc;
    NATS_CHECK_ARG(d_roles_new && d_rank && d_base && d_size_global && d_size_local && d_state, "null pointer");
    evict_plan_kernel<<<B * Hkv, kPrepThreads, 0, (cudaStream_t)stream>>>(
        d_roles_new, cdiv(n_tokens, C), n_tokens / C, C, SW, d_rank, (long long*)d_size_global, (long long*)d_size_local,
        d_state, d_base, nullptr, nullptr);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_evict_plan_report(
    const uint8_t* d_roles, int B, int Hkv, int n_tokens, int C, int SW, int32_t* d_rank, int32_t* d_base,
    int64_t* d_size_global, int64_t* d_size_local, int32_t* d_state, const int32_t* d_status, int32_t* h_report, void* stream) {
    if (int rc = check_common(B, Hkv, n_tokens, C, SW)) return rc;
    NATS_CHECK_ARG(d_roles && d_rank && d_size_global && d_size_local && d_state && d_status && h_report, "null pointer");
    void* report = nullptr;
    NATS_CHECK_CUDA(cudaHostGetDevicePointer(&report, h_report, 0));
    evict_plan_kernel<<<B * Hkv, kPrepThreads, 0, (cudaStream_t)stream>>>(
        d_roles, cdiv(n_tokens, C), n_tokens / C, C, SW, d_rank, (long long*)d_size_global, (long long*)d_size_local,
        d_state, d_base, d_status, (int32_t*)report);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

static int check_row(int D) {
    NATS_CHECK_ARG(D > 0 && (D * 2) % 16 == 0 && D <= 2048 && 256 % ((D * 2) / 16) == 0,
                   "head_dim %d: a bf16 row must be a whole number of 16-byte vectors that divides 256", D);
    return NATS_OK;
}

template <bool F32>
static int evict_compact_first(const void* d_k, const void* d_v, const uint8_t* d_roles, const int32_t* d_rank,
                                       const int64_t* d_size_global, const int64_t* d_size_local, const int32_t* d_state,
                                       int B, int Hkv, int N, int D, int C, int SW,
                                       void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap, void* stream) {
    if (int rc = check_common(B, Hkv, N, C, SW)) return rc;
    if (int rc = check_row(D)) return rc;
    NATS_CHECK_ARG(d_k && d_v && d_roles && d_rank && d_size_global && d_size_local && d_state && d_cache_k && d_cache_v && d_valid,
                   "null pointer");
    NATS_CHECK_ARG(((uintptr_t)d_k | (uintptr_t)d_v | (uintptr_t)d_cache_k | (uintptr_t)d_cache_v) % 16 == 0,
                   "K/V and cache pointers must be 16-byte aligned");
    NATS_CHECK_ARG(Lcap >= SW + C, "cache capacity %d is smaller than ring + one chunk (%d)", Lcap, SW + C);
    CompactParams p;
    p.k = (const uint8_t*)d_k; p.v = (const uint8_t*)d_v; p.roles = d_roles; p.rank = d_rank;
    p.old_valid = nullptr; p.base = nullptr; p.src_stride = N; p.src_off = 0; p.tail = 0;
    p.size_global = (const long long*)d_size_global; p.size_local = (const long long*)d_size_local; p.state = d_state;
    p.ck = (uint8_t*)d_cache_k; p.cv = (uint8_t*)d_cache_v; p.valid = d_valid;
    p.N = N; p.Nc = cdiv(N, C); p.n_full = N / C; p.C = C; p.SW = SW; p.Lcap = Lcap; p.rowB = D * 2;
    p.nB = cdiv(SW, kTokPerBlock);
    const int nC = cdiv(Lcap - SW, kTokPerBlock);
    dim3 grid(p.nB + nC, B * Hkv);
    evict_compact_kernel<F32><<<grid, kCopyThreads, 0, (cudaStream_t)stream>>>(p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_evict_compact(const void* d_k, const void* d_v, const uint8_t* d_roles, const int32_t* d_rank,
                                       const int64_t* d_size_global, const int64_t* d_size_local, const int32_t* d_state,
                                       int B, int Hkv, int N, int D, int C, int SW,
                                       void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap, void* stream) {
    return evict_compact_first<false>(d_k, d_v, d_roles, d_rank, d_size_global, d_size_local, d_state, B, Hkv, N, D, C, SW, d_cache_k, d_cache_v,
                                      d_valid, Lcap, stream);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_evict_compact_f32(const float* d_k, const float* d_v, const uint8_t* d_roles, const int32_t* d_rank,
                                       const int64_t* d_size_global, const int64_t* d_size_local, const int32_t* d_state,
                                       int B, int Hkv, int N, int D, int C, int SW,
                                       void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap, void* stream) {
    return evict_compact_first<true>(d_k, d_v, d_roles, d_rank, d_size_global, d_size_local, d_state, B, Hkv, N, D, C, SW, d_cache_k, d_cache_v,
                                      d_valid, Lcap, stream);
}

extern "C" __attribute__((visibility("default"))) int nats_b200_evict_compact_past(
    const void* d_old_k, const void* d_old_v, const uint8_t* d_old_valid, int old_capacity,
    const uint8_t* d_roles_new, const int32_t* d_rank, const int32_t* d_base,
    const int64_t* d_size_global, const int64_t* d_size_local, const int32_t* d_state,
    int B, int Hkv, int n_tokens, int D, int C, int SW, int t0_old, int tail_old,
    void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap, void* stream) {
    if (int rc = check_common(B, Hkv, n_tokens, C, SW)) return rc;
    if (int rc = check_row(D)) return rc;
    NATS_CHECK_ARG(d_old_k && d_old_v && d_old_valid && d_roles_new && d_rank && d_base && d_size_global && d_size_local &&
                   d_state && d_cache_k && d_cache_v && d_valid, "null pointer");
    NATS_CHECK_ARG(((uintptr_t)d_old_k | (uintptr_t)d_old_v | (uintptr_t)d_cache_k | (uintptr_t)d_cache_v) % 16 == 0,
                   "cache pointers must be 16-byte aligned");
    NATS_CHECK_ARG(d_old_k != d_cache_k && d_old_v != d_cache_v && d_old_valid != d_valid, "the compaction is out of place: old and new cache must differ");
    NATS_CHECK_ARG(t0_old >= SW && t0_old % C == 0 && (long long)t0_old + n_tokens <= old_capacity,
                   "old cache: tail offset %d (+ %d tokens) does not fit its capacity %d", t0_old, n_tokens, old_capacity);
    NATS_CHECK_ARG(tail_old >= 0 && tail_old < SW && tail_old % C == 0, "ring tail %d must be a chunk multiple inside the window %d", tail_old, SW);
    NATS_CHECK_ARG(Lcap >= SW + C, "cache capacity %d is smaller than ring + one chunk (%d)", Lcap, SW + C);
    CompactParams p;
    p.k = (const uint8_t*)d_old_k; p.v = (const uint8_t*)d_old_v; p.old_valid = d_old_valid; p.roles = d_roles_new; p.rank = d_rank;
    p.base = d_base; p.src_stride = old_capacity; p.src_off = t0_old; p.tail = tail_old;
    p.size_global = (const long long*)d_size_global; p.size_local = (const long long*)d_size_local; p.state = d_state;
    p.ck = (uint8_t*)d_cache_k; p.cv = (uint8_t*)d_cache_v; p.valid = d_valid;
    p.N = n_tokens; p.Nc = cdiv(n_tokens, C); p.n_full = n_tokens / C; p.C = C; p.SW = SW; p.Lcap = Lcap; p.rowB = D * 2;
    p.nB = cdiv(SW, kTokPerBlock);
    const int nC = cdiv(Lcap - SW, kTokPerBlock);
    dim3 grid(p.nB + nC, B * Hkv);
    evict_compact_kernel<false><<<grid, kCopyThreads, 0, (cudaStream_t)stream>>>(p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_to_bf16(
    const float* d_x0, void* d_y0, long long n0, const float* d_x1, void* d_y1, long long n1,
    const float* d_x2, void* d_y2, long long n2, void* stream) {
    const float* x[3] = {d_x0, d_x1, d_x2};
    void* y[3] = {d_y0, d_y1, d_y2};
    const long long n[3] = {n0, n1, n2};
    Bf16Params p;
    long long most = 0;
    for (int a = 0; a < 3; ++a) {
        NATS_CHECK_ARG(n[a] >= 0 && n[a] % 8 == 0, "element counts must be multiples of 8, got %lld", n[a]);
        NATS_CHECK_ARG(n[a] == 0 || (x[a] && y[a]), "null pointer");
        NATS_CHECK_ARG(((uintptr_t)x[a] | (uintptr_t)y[a]) % 16 == 0, "pointers must be 16-byte aligned");
        p.x[a] = (const uint8_t*)x[a]; p.y[a] = (uint8_t*)y[a]; p.n8[a] = n[a] / 8;
        most = p.n8[a] > most ? p.n8[a] : most;
    }
    if (most == 0) return NATS_OK;
    const long long blocks = (most + kCopyThreads - 1) / kCopyThreads;
    to_bf16_kernel<<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), kCopyThreads, 0, (cudaStream_t)stream>>>(p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_cache_append(
    const void* d_k_new, const void* d_v_new, void* d_cache_k, void* d_cache_v, uint8_t* d_valid,
    int B, int Hkv, int x_len, int D, int Lcap, int pos, void* stream) {
    NATS_CHECK_ARG(B > 0 && Hkv > 0 && x_len > 0 && (long long)B * Hkv <= 65535, "bad shape B=%d Hkv=%d x_len=%d", B, Hkv, x_len);
    if (int rc = check_row(D)) return rc;
    NATS_CHECK_ARG(d_k_new && d_v_new && d_cache_k && d_cache_v && d_valid, "null pointer");
    NATS_CHECK_ARG(((uintptr_t)d_k_new | (uintptr_t)d_v_new | (uintptr_t)d_cache_k | (uintptr_t)d_cache_v) % 16 == 0,
                   "K/V and cache pointers must be 16-byte aligned");
    NATS_CHECK_ARG(pos >= 0 && (long long)pos + x_len <= Lcap, "rows [%d, %d) do not fit the cache capacity %d", pos, pos + x_len, Lcap);
    AppendParams p;
    p.k = (const uint8_t*)d_k_new; p.v = (const uint8_t*)d_v_new;
    p.ck = (uint8_t*)d_cache_k; p.cv = (uint8_t*)d_cache_v; p.valid = d_valid;
    p.x_len = x_len; p.pos = pos; p.Lcap = Lcap; p.rowB = D * 2;
    dim3 grid(cdiv(x_len, kTokPerBlock), B * Hkv);
    cache_append_kernel<<<grid, kCopyThreads, 0, (cudaStream_t)stream>>>(p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_cache_grow_append(
    const void* d_old_k, const void* d_old_v, const uint8_t* d_old_valid, int old_rows, const void* d_k_new, const void* d_v_new,
    void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int B, int Hkv, int x_len, int D, int Lcap, int pos, void* stream) {
    NATS_CHECK_ARG(B > 0 && Hkv > 0 && x_len > 0 && pos >= 0, "bad sizes B=%d Hkv=%d x_len=%d pos=%d", B, Hkv, x_len, pos);
    NATS_CHECK_ARG(d_old_k && d_old_v && d_old_valid && d_k_new && d_v_new && d_cache_k && d_cache_v && d_valid, "null pointer");
    NATS_CHECK_ARG(d_old_k != d_cache_k && d_old_v != d_cache_v && d_old_valid != d_valid, "the larger buffers must not be the old ones");
    NATS_CHECK_ARG(((uintptr_t)d_old_k | (uintptr_t)d_old_v | (uintptr_t)d_k_new | (uintptr_t)d_v_new | (uintptr_t)d_cache_k |
                    (uintptr_t)d_cache_v) % 16 == 0, "K, V and the buffers must be 16-byte aligned");
    if (int rc = check_row(D)) return rc;
    NATS_CHECK_ARG(pos <= old_rows, "%d rows to keep, the old buffer has %d", pos, old_rows);
    NATS_CHECK_ARG((long long)pos + x_len <= Lcap, "rows [%d, %lld) do not fit the capacity %d", pos, (long long)pos + x_len, Lcap);
    NATS_CHECK_ARG((long long)B * Hkv <= 65535, "B * Hkv = %lld exceeds the grid limit 65535", (long long)B * Hkv);
    GrowParams p;
    p.a.k = (const uint8_t*)d_k_new; p.a.v = (const uint8_t*)d_v_new;
    p.a.ck = (uint8_t*)d_cache_k; p.a.cv = (uint8_t*)d_cache_v; p.a.valid = d_valid;
    p.a.x_len = x_len; p.a.pos = pos; p.a.Lcap = Lcap; p.a.rowB = D * 2;
    p.k = (const uint8_t*)d_old_k; p.v = (const uint8_t*)d_old_v; p.valid = d_old_valid; p.rows = old_rows;
    cache_grow_append_kernel<<<dim3(cdiv(Lcap, kTokPerBlock), B * Hkv), kCopyThreads, 0, (cudaStream_t)stream>>>(p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

// One thread: the step counters of the static decode step.  state[4] = tokens in the unfinished chunk, state[5] = ring
// write position.  Runs behind the (conditional) placement kernel of the same step.
__global__ void decode_step_advance_kernel(int32_t* state, int C, int SW) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int fill = state[4] + 1;
    if (fill == C) {
        state[4] = 0;
        state[5] = (state[5] + C) % SW;
    } else {
        state[4] = fill;
    }
}

extern "C" __attribute__((visibility("default"))) int nats_b200_decode_step_place(const uint8_t* d_roles, void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap,
                                                                       int64_t* d_size_global, int64_t* d_size_local, int32_t* d_state,
                                                                       int B, int Hkv, int D, int C, int SW, void* stream) {
    if (int rc = check_common(B, Hkv, 1, C, SW)) return rc;
    if (int rc = check_row(D)) return rc;
    NATS_CHECK_ARG(d_roles && d_cache_k && d_cache_v && d_valid && d_size_global && d_size_local && d_state, "null pointer");
    PlaceParams p;
    p.roles = d_roles; p.ck = (uint8_t*)d_cache_k; p.cv = (uint8_t*)d_cache_v; p.valid = d_valid;
    p.size_global = (long long*)d_size_global; p.size_local = (long long*)d_size_local; p.state = d_state;
    p.C = C; p.SW = SW; p.Lcap = Lcap; p.rowB = D * 2; p.tail = 0; p.from_state = 1;
    decode_place_kernel<<<B * Hkv, kCopyThreads, 0, (cudaStream_t)stream>>>(p);
    NATS_CHECK_CUDA(cudaGetLastError());
    decode_step_advance_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(d_state, C, SW);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}

extern "C" __attribute__((visibility("default"))) int nats_b200_decode_place(const uint8_t* d_roles, void* d_cache_k, void* d_cache_v, uint8_t* d_valid, int Lcap,
                                      int64_t* d_size_global, int64_t* d_size_local, int32_t* d_state,
                                      int tail, int B, int Hkv, int D, int C, int SW, void* stream) {
    if (int rc = check_common(B, Hkv, 1, C, SW)) return rc;
    if (int rc = check_row(D)) return rc;
    NATS_CHECK_ARG(d_roles && d_cache_k && d_cache_v && d_valid && d_size_global && d_size_local && d_state, "null pointer");
    NATS_CHECK_ARG(tail >= 0 && tail < SW && tail % C == 0, "ring tail %d must be a chunk multiple inside the window %d", tail, SW);
    PlaceParams p;
    p.roles = d_roles; p.ck = (uint8_t*)d_cache_k; p.cv = (uint8_t*)d_cache_v; p.valid = d_valid;
    p.size_global = (long long*)d_size_global; p.size_local = (long long*)d_size_local; p.state = d_state;
    p.C = C; p.SW = SW; p.Lcap = Lcap; p.rowB = D * 2; p.tail = tail; p.from_state = 0;
    decode_place_kernel<<<B * Hkv, kCopyThreads, 0, (cudaStream_t)stream>>>(p);
    NATS_CHECK_CUDA(cudaGetLastError());
    return NATS_OK;
}
