// route.cuh -- top-k routing of one row by one warp, shared by every kernel that routes.
#pragma once
#include "common.cuh"

namespace sl {

// One warp routes one row.  Restates swift/Sources/QwispCore/SeedlessFusedVerify.swift:180-214 including the ORDER of its
// 256-slot halving trees.  Softmax in f32, gates rounded to fp16, top-k by k rounds of arg-max on the raw logits (strict >
// keeps the lower slot), fp16 sequential sum of the chosen gates, fp16 divide.  In two parts, because the chosen experts
// are what a weight fetch is waiting for and the gates are needed only at the combine.
//
// Order of the reference's selection tree (256 slots halved to 128, 64, ... 1, the lower slot of
// each compared pair winning ties): larger logit first, then smaller bit-reversed slot number (the
// last level compares slots 0 and 1, so bit 0 of the slot decides first).  A 24-bit key
// (order-preserving fp16 bits, then 255 - bitreverse8(slot)) has the same order, so k hardware
// warp-max reductions select the same experts in the same sequence.  Every lane sorts its 8 keys first, so a round is
// one reduction and a shift of the winner's list (looking for the key to strike out in every lane took three times as long).
// SMEM: lrow points to shared memory (plain loads); otherwise to global memory written by other CTAs of a
// running kernel or by an earlier kernel (L1-bypassing loads).
template <bool SMEM>
__device__ __forceinline__ uint4 route_load(const __half* lrow, int E, int lane) {       // slots 8 * lane ..; -inf behind E
    uint4 raw = make_uint4(0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u);
    if ((E & 7) == 0) {                                                   // rows of E halves stay 16-byte aligned only then
        if (lane * 8 < E) raw = SMEM ? reinterpret_cast<const uint4*>(lrow)[lane] : __ldcg(reinterpret_cast<const uint4*>(lrow) + lane);
    } else {
        __half* rh = reinterpret_cast<__half*>(&raw);
        for (int i = 0; i < 8; ++i) if (lane * 8 + i < E) rh[i] = SMEM ? lrow[lane * 8 + i] : __ldcg(lrow + lane * 8 + i);
    }
    return raw;
}
// -> lane k: the k-th choice (k < topk)
__device__ __forceinline__ int route_select(uint4 raw, int E, int topk, int lane) {
    unsigned key[8];
    const __half* rh = reinterpret_cast<const __half*>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        unsigned hb = __half_as_ushort(rh[i]);
        if (hb == 0x8000u) hb = 0u;                                       // -0 compares equal to +0
        hb = (hb & 0x8000u) ? (~hb & 0xffffu) : (hb | 0x8000u);
        const int slot = lane * 8 + i;
        key[i] = (slot < E) ? ((hb << 8) | (255u - (__brev((unsigned)slot) >> 24))) : 0u;
    }
#define SL_CE(a, b) { const unsigned hi_ = max(key[a], key[b]), lo_ = min(key[a], key[b]); key[a] = hi_; key[b] = lo_; }
    SL_CE(0, 1) SL_CE(2, 3) SL_CE(4, 5) SL_CE(6, 7)                       // odd-even merge sort, descending
    SL_CE(0, 2) SL_CE(1, 3) SL_CE(4, 6) SL_CE(5, 7)
    SL_CE(1, 2) SL_CE(5, 6)
    SL_CE(0, 4) SL_CE(1, 5) SL_CE(2, 6) SL_CE(3, 7)
    SL_CE(2, 4) SL_CE(3, 5)
    SL_CE(1, 2) SL_CE(3, 4) SL_CE(5, 6)
#undef SL_CE
    int my_id = 0;
#pragma unroll 1
    for (int k = 0; k < topk; ++k) {
        const unsigned best = __reduce_max_sync(0xffffffffu, key[0]);
        if (lane == k) my_id = (int)(__brev(255u - (best & 0xffu)) >> 24);
        if (key[0] == best) {
#pragma unroll
            for (int i = 0; i < 7; ++i) key[i] = key[i + 1];
            key[7] = 0u;
        }
    }
    return my_id;
}
// -> lane k: the gate of the k-th choice.  buf: 256 floats of shared memory owned by this warp.
// Lane l looks at slots l, l+32, .., l+224, so the tree levels 128/64/32 are lane-local and the levels 16..1 are
// xor-shuffles whose results are meaningful in lanes < s -- the same pairs (i, i+s) the reference combines.
__device__ __forceinline__ __half route_gate(uint4 raw, int my_id, int E, int topk, float* buf, int lane) {
    const __half* rh = reinterpret_cast<const __half*>(&raw);
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < 8; ++i) { const float v = h2f(rh[i]); buf[lane * 8 + i] = v; mx = fmaxf(mx, v); }
    __syncwarp();
    mx = warp_max(mx);
    float ex[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { const int slot = j * 32 + lane; ex[j] = (slot < E) ? expf(buf[slot] - mx) : 0.0f; }
    float r0 = __fadd_rn(ex[0], ex[4]), r1 = __fadd_rn(ex[1], ex[5]), r2 = __fadd_rn(ex[2], ex[6]), r3 = __fadd_rn(ex[3], ex[7]);
    r0 = __fadd_rn(r0, r2); r1 = __fadd_rn(r1, r3);
    r0 = __fadd_rn(r0, r1);
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) r0 = __fadd_rn(r0, __shfl_xor_sync(0xffffffffu, r0, s));
    const float Z = __shfl_sync(0xffffffffu, r0, 0);
    const float my_ex = expf(buf[my_id] - mx);                            // the exp of the lane's own choice, formed as above
    // gate of the k-th choice = fp16(exp / Z); the sum runs in fp16 in ascending k, then each is divided by it
    const __half g = f2h(__fdiv_rn(my_ex, Z));
    __half ss = f2h(0.0f);
#pragma unroll 4
    for (int k = 0; k < topk; ++k) ss = hadd_rn(ss, __ushort_as_half((unsigned short)__shfl_sync(0xffffffffu, (unsigned)__half_as_ushort(g), k)));
    __syncwarp();
    return hdiv_rn(g, ss);
}
// early_flag (shared memory, may be null): set to early_value as soon as inds_out is complete, before the gates.
template <bool SMEM>
__device__ __noinline__ void route_row_impl(const __half* lrow, int E, int topk, int* inds_out, __half* scores_out, float* buf, int lane,
                                            volatile int* early_flag = nullptr, int early_value = 0) {
    const uint4 raw = route_load<SMEM>(lrow, E, lane);
    const int my_id = route_select(raw, E, topk, lane);
    if (lane < topk) inds_out[lane] = my_id;
    if (early_flag) {                                                      // publish the choices before the gate arithmetic
        __syncwarp();
        if (lane == 0) { __threadfence_block(); *early_flag = early_value; }
    }
    const __half g = route_gate(raw, my_id, E, topk, buf, lane);
    if (lane < topk) scores_out[lane] = g;
    __syncwarp();
}

__device__ __forceinline__ void route_row_warp(const __half* lrow, int E, int topk, int* inds_out, __half* scores_out, float* buf, int lane) {
    route_row_impl<false>(lrow, E, topk, inds_out, scores_out, buf, lane);
}
__device__ __forceinline__ void route_row_smem(const __half* lrow, int E, int topk, int* inds_out, __half* scores_out, float* buf, int lane,
                                               volatile int* early_flag = nullptr, int early_value = 0) {
    route_row_impl<true>(lrow, E, topk, inds_out, scores_out, buf, lane, early_flag, early_value);
}

}  // namespace sl
