// Shared host/device helpers of libnats_b200 (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "../../include/nats_b200.h"

namespace nats {

constexpr int kTile = 128;           // query rows / key columns per MMA tile of the prefill
constexpr int kMaxTiles = 4096;      // prefill: N <= kMaxTiles * kTile
constexpr int32_t kNoLimit = 0x7fffffff;

// ---- host-side error text (thread local) ----------------------------------------------------
char* last_error_buf();
int fail(int code, const char* fmt, ...);

#define NATS_CHECK_ARG(cond, ...)                                   \
    do {                                                            \
        if (!(cond)) return ::nats::fail(NATS_ERR_INVALID_ARG, __VA_ARGS__); \
    } while (0)

// A call that has failed leaves its error behind in the runtime, too, where the check behind the next launch would find it and report a
// launch that was right: the error is taken from there as well.
#define NATS_CHECK_CUDA(expr)                                                                     \
    do {                                                                                          \
        cudaError_t e_ = (expr);                                                                  \
        if (e_ != cudaSuccess) {                                                                  \
            (void)cudaGetLastError();                                                             \
            return ::nats::fail(NATS_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_));   \
        }                                                                                         \
    } while (0)

// Chunks that stay visible for good, per (batch, kv-head), without those of dense tiles (dense_min of them or more in a 128-row KV
// tile): list [Nc] = their indices in order, before_tile [Ntk + 1] = how many of them lie in front of a tile (at the end: all),
// open_max [Ntk] = twice the largest row limit of the tile's other chunks (-1: it has none; kOpenMax: as large or larger, or more
// than max_listed lie in front of the next tile), plus one if the tile is dense.  list == nullptr: not wanted.  Only for
// chunk sizes that divide a tile.
constexpr int kOpenMax = 0x3fffffff;
struct FarLists {
    int32_t* list = nullptr;
    int32_t* before_tile = nullptr;
    int32_t* open_max = nullptr;
    int max_listed = 0x7fffffff;
    int dense_min = 0x7fffffff;
};

// the C entry points nats_b200_role_prep / _past with the lists beside the limits; *d_counter (may be null) is set to zero
int role_prep(const uint8_t* d_roles, int B, int Hkv, int N, int C, int SW, int32_t* d_lim, int32_t* d_tile_max,
              int32_t* d_tile_min, int64_t* d_kept_tiles, const FarLists& far, int32_t* d_counter, void* stream);
int role_prep_past(const uint8_t* d_roles_new, const uint8_t* d_valid, const int64_t* d_size_global, const int64_t* d_size_local,
                   int B, int Hkv, int x_len, int C, int SW, int valid_stride, int t0, int fill, int tail,
                   int32_t* d_lim, int32_t* d_tile_max, int32_t* d_tile_min, int64_t* d_kept_tiles, const FarLists& far, int32_t* d_counter, void* stream);

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
inline int cdiv(int a, int b) { return (a + b - 1) / b; }

// ---- device helpers --------------------------------------------------------------------------
__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// 16-byte global accesses
__device__ __forceinline__ uint4 ld16(const void* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void st16(void* p, uint4 v) { *reinterpret_cast<uint4*>(p) = v; }
// streaming variants: data that is touched once should not displace the L2 working set
__device__ __forceinline__ uint4 ld16_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// eight fp32 values (two vectors) rounded to bf16
__device__ __forceinline__ uint4 round8(uint4 lo, uint4 hi) {
    const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
        r[i] = *reinterpret_cast<const uint32_t*>(&b);
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}

}  // namespace nats
