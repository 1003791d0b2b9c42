// Placement of a chunk that decode steps have completed: the tail of the step kernels and a kernel of its own.
#pragma once
#include "common.cuh"

namespace nats {

struct PlaceParams {
    const uint8_t* roles;                         // [BH]
    uint8_t* ck; uint8_t* cv; uint8_t* valid;     // [BH, Lcap, rowB], [BH, Lcap]
    long long* size_global; long long* size_local; int32_t* state;
    int C, SW, Lcap, rowB, tail;
    int from_state;                               // 1: static launch -- act only if state[4] + 1 == C, ring position = state[5]
};

// The unfinished chunk of (batch, kv-head) bh, all C tokens of it, goes to the ring slots behind `tail` (data if it is a
// sliding chunk, zeros and invalid flags otherwise) and, unless it is sliding, behind the kept tokens.  All NT threads of the
// block call.  Returns the head's new length.
template <int NT>
__device__ __forceinline__ int place_chunk(const PlaceParams& p, int bh, int T0, int tail) {
    const int tid = threadIdx.x;
    const int vpt = p.rowB >> 4, tpp = NT / vpt;
    const int trow = tid / vpt, tvec = (tid % vpt) << 4;
    uint8_t* ck = p.ck + (size_t)bh * p.Lcap * p.rowB;
    uint8_t* cv = p.cv + (size_t)bh * p.Lcap * p.rowB;
    uint8_t* valid = p.valid + (size_t)bh * p.Lcap;
    const int role = p.roles[bh];
    const long long sg = p.size_global[bh], sl = p.size_local[bh];
    const int len = (int)(sg + sl);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    int dst, new_len;
    long long nsg = sg, nsl = sl;
    if (role == NATS_ROLE_GLOBAL) { dst = (int)sg; nsg = sg + p.C; nsl = 0; }
    else if (role == NATS_ROLE_LOCAL) { dst = len; nsl = sl + p.C; }
    else { dst = -1; }
    new_len = (int)(nsg + nsl);
    if (trow < tpp) {
        for (int i = trow; i < p.C; i += tpp) {
            const size_t src = (size_t)(T0 + i) * p.rowB + tvec;
            const uint4 kk = ld16(ck + src), vv = ld16(cv + src);
            const int slot = (tail + i) % p.SW;
            const size_t rdst = (size_t)slot * p.rowB + tvec;
            const bool sw = role == NATS_ROLE_SLIDING;
            st16(ck + rdst, sw ? kk : zero);
            st16(cv + rdst, sw ? vv : zero);
            if (tvec == 0) valid[slot] = sw ? 1 : 0;
            if (dst >= 0 && dst != T0) {
                const size_t mdst = (size_t)(dst + i) * p.rowB + tvec;
                st16(ck + mdst, kk);
                st16(cv + mdst, vv);
            }
        }
    }
    __syncthreads();   // every read of the pending chunk (and of the sizes) is done before what it replaces is cleared
    if (trow < tpp) {
        // cleared: the locals a global chunk has just dropped, [new_len, len), and the slot of the pending chunk unless the
        // chunk stayed there; everything else behind a head's length is zero already
        for (int d = new_len + trow; d < len; d += tpp) {
            const size_t o = (size_t)d * p.rowB + tvec;
            st16(ck + o, zero);
            st16(cv + o, zero);
            if (tvec == 0) valid[d] = 0;
        }
        const int end = min(T0 + p.C, p.Lcap);
        for (int d = max(T0, new_len) + trow; d < end; d += tpp) {
            const size_t o = (size_t)d * p.rowB + tvec;
            st16(ck + o, zero);
            st16(cv + o, zero);
            if (tvec == 0) valid[d] = 0;
        }
        if (dst >= 0)
            for (int i = trow; i < p.C; i += tpp)
                if (tvec == 0) valid[dst + i] = 1;
    }
    if (tid == 0) {
        p.size_global[bh] = nsg;
        p.size_local[bh] = nsl;
    }
    return new_len;
}

}  // namespace nats
