// rows_kernels.cu -- the many-row forms of the 4-bit group-64 GEMV family: calls with more than one activation row
// (batched decode, verify rows, strict-mode prompt chunks).
//
// The pass kernels (kernels.cu) walk the rows in passes of 8 and pay one grid wave, one weight fetch and
// one dequantisation per pass.  Here the weights of a tile are fetched and dequantised ONCE per 8*RG rows and a row's
// arithmetic is kept exactly as in the pass kernels, so every output is bit-identical to what the same row gives
// alone (the batch-invariance rule of the reference, swift/Sources/QwispCore/SeedlessMetalForward.swift:160-185):
//   - per group of 64 inputs the same chain of four m16n8k16 MMAs (an MMA column never mixes with another column);
//   - scale * sum and bias * (sum of the group's activations) accumulated over the 4 groups of a 256-input slice;
//   - slice values added in ascending order starting from 0.
//
//   k_rows_prep      the prologue (plain / RMSNorm / gated RMSNorm) of every row, written once per call: the
//                    activations in the products' order (0,1,4,5,2,3,6,7 inside every 8) + the per-group sums.
//   k_gemv_rows      dense projection: a CTA holds a block of 8, 16 or 32 rows over the whole K, its warps stream tiles of 16
//                    weight rows through rings of their own (k_gemv_rows_split: short runs, shared out by slices).
//   k_head_rows      lm_head + argmax in the same form.
//   k_expert_rows    routed + shared experts grouped by expert: every warp walks tiles of its CTA's run on its own.
//   k_moe_combine    weighted sum of a row's top-k expert rows in ascending k + shared expert + residual.
#include "kernels.h"
#include "gemv.cuh"
#include "mixer_math.cuh"
#include "route.cuh"

namespace sl {

// ================================================================================ prologue rows
struct RowsPrepArgs {
    const __half* x; int ldx;            // rows (plain) / residual stream (rmsnorm) / mixer output (gated norm)
    const __half* nw; const float* nw32; // norm weight
    const __half* z; int ldz;            // gate input of the gated norm
    float eps; int K;
    __half* xq; float* sxq;              // out: [M][K] in the products' order, [M][K/64]
};
// grid (M), K/256 warps: warp = one 256-input chunk of the row (the unit of stage_finish())
template <int PRO>
__global__ void __launch_bounds__(512) k_rows_prep(RowsPrepArgs a) {
    __shared__ float part[16];
    const int row = blockIdx.x, ch = threadIdx.x >> 5, lane = threadIdx.x & 31, chunks = a.K >> 8;
    const int k0 = (ch << 8) + lane * 8;
    pdl_wait();
    pdl_launch_dependents();
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(a.x + (size_t)row * a.ldx + k0));
    uint4 o;
    if (PRO == PRO_PLAIN) {
        o = v;
    } else if (PRO == PRO_RMSNORM) {
        const float ss = warp_sum(sumsq8(v));
        if (lane == 0) part[ch] = ss;
        __syncthreads();
        float tot = 0.f;
        for (int c = 0; c < chunks; ++c) tot += part[c];
        const float inv = __frsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)a.K), a.eps));
        o = rms_apply8(v, *reinterpret_cast<const uint4*>(a.nw + k0), inv);
    } else {
        const uint4 zv = __ldcg(reinterpret_cast<const uint4*>(a.z + (size_t)row * a.ldz + k0));
        const uint4 wv = *reinterpret_cast<const uint4*>(a.nw + (k0 & 127));
        o = normgate8<PRO>(v, zv, wv, a.nw32, k0, a.eps);
    }
    rows_store(a.xq + (size_t)row * a.K, a.sxq + (size_t)row * (a.K >> 6), k0, o, lane);
}
static void launch_rows_prep_args(int pro, const RowsPrepArgs& a, int M, cudaStream_t st, bool pdl) {
    const unsigned threads = (unsigned)(a.K >> 8) * 32u;
    profile_launch("k_rows_prep", st, [&] {
        if (pro == PRO_PLAIN) return launch_pdl(pdl, k_rows_prep<PRO_PLAIN>, dim3((unsigned)M), threads, 0, st, a);
        if (pro == PRO_RMSNORM) return launch_pdl(pdl, k_rows_prep<PRO_RMSNORM>, dim3((unsigned)M), threads, 0, st, a);
        if (pro == PRO_NORMGATE) return launch_pdl(pdl, k_rows_prep<PRO_NORMGATE>, dim3((unsigned)M), threads, 0, st, a);
        return launch_pdl(pdl, k_rows_prep<PRO_NORMGATE32>, dim3((unsigned)M), threads, 0, st, a);
    });
}
void launch_rows_prep_plain(const __half* x, int ldx, int M, int K, __half* xq, float* sxq, cudaStream_t st, bool pdl) {
    RowsPrepArgs p{x, ldx, nullptr, nullptr, nullptr, 0, 0.f, K, xq, sxq};
    launch_rows_prep_args(PRO_PLAIN, p, M, st, pdl);
}

// ================================================================================ shared compute
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
// Wait of the expert kernel's ring, bounded in TIME (~50 ms): the first wait of a CTA that runs out raises the CTA's
// abort word, and every later wait of that CTA gives up at once, so a stall costs one timeout per CTA, not one per block.
// For whole warps: the lanes agree on the outcome, because what follows needs all of them.
constexpr long long XR_TIMEOUT = 100000000ll;                 // cycles
__device__ __forceinline__ bool xr_wait_lane(uint64_t* bar, uint32_t parity, volatile int* abort_word, long long timeout) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        for (int i = 0; i < 64; ++i) if (mbar_try_wait(bar, parity)) return true;
        if (*abort_word) return false;
        if (clock64() - t0 > timeout) { *abort_word = 1; return false; }
    }
}
template <bool STALL>
__device__ __forceinline__ bool xr_wait(uint64_t* bar, uint32_t parity, volatile int* abort_word) {
    return __all_sync(0xffffffffu, xr_wait_lane(bar, parity, abort_word, STALL ? XR_TIMEOUT / 32 : XR_TIMEOUT));
}

constexpr int XR_DEPTH = 2;                   // slices in a warp's ring
constexpr int XR_UNIT = 2048 + 256;           // bytes of a slice of a tile: nibbles, then scales and biases
// slice s of a tile (nibbles w, scales sc) into a ring slot of the calling warp
__device__ __forceinline__ void ring_request(unsigned char* slot, const uint4* w, const uint4* sc, int s, int lane) {
    uint4* d = reinterpret_cast<uint4*>(slot);
    const uint4* p = w + s * 128 + lane;
    cp_async16(d + lane, p); cp_async16(d + lane + 32, p + 32); cp_async16(d + lane + 64, p + 64); cp_async16(d + lane + 96, p + 96);
    if (lane < 16) cp_async16(d + 128 + lane, sc + s * 16 + lane);
}
// One slice (4 groups of 64 inputs) of a 16-row tile, in a ring slot, against 8*RG staged rows.
// xp: the slice's activations of this lane's row of group 0 (row r, + 16 t), rows xstride halves apart; sxp: the
// group sums [group][row] of the slice, at column 2t, groups sxstride floats apart.  acc[q]: (row A, col 2t), (A, 2t+1),
// (B, 2t), (B, 2t+1) of row group q.  The order of operations per column is that of compute_slice_x().
template <int RG>
__device__ __forceinline__ void compute_rows(const unsigned char* slot, const __half* xp, int xstride, const float* sxp, int sxstride,
                                             int lane, float accS[RG][4], float accB[RG][4]) {
    const uint4* w = reinterpret_cast<const uint4*>(slot);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const uint4 wv = w[g * 32 + lane];
        uint32_t a0[4], b0[4], a1[4], b1[4];
        dequant8(wv.x, a0); dequant8(wv.z, b0); dequant8(wv.y, a1); dequant8(wv.w, b1);
        const uint2 sv = *reinterpret_cast<const uint2*>(slot + 2048 + (g >> 1) * 128 + (lane >> 2) * 16 + (g & 1) * 8);
        const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&sv.x));
        const float2 fb = __half22float2(*reinterpret_cast<const __half2*>(&sv.y));
#pragma unroll
        for (int q = 0; q < RG; ++q) {
            const uint4 X0 = *reinterpret_cast<const uint4*>(xp + (size_t)q * 8 * xstride + 64 * g), X1 = *reinterpret_cast<const uint4*>(xp + (size_t)q * 8 * xstride + 64 * g + 8);
            const float2 sx = *reinterpret_cast<const float2*>(sxp + g * sxstride + q * 8);
            float c[4];
            mma_f16_z(c, a0[0], b0[0], a0[1], b0[1], X0.x, X0.y);
            mma_f16(c, a0[2], b0[2], a0[3], b0[3], X0.z, X0.w);
            mma_f16(c, a1[0], b1[0], a1[1], b1[1], X1.x, X1.y);
            mma_f16(c, a1[2], b1[2], a1[3], b1[3], X1.z, X1.w);
            accS[q][0] = fmaf(fa.x, c[0], accS[q][0]); accS[q][1] = fmaf(fa.x, c[1], accS[q][1]);
            accS[q][2] = fmaf(fb.x, c[2], accS[q][2]); accS[q][3] = fmaf(fb.x, c[3], accS[q][3]);
            accB[q][0] = fmaf(fa.y, sx.x, accB[q][0]); accB[q][1] = fmaf(fa.y, sx.y, accB[q][1]);
            accB[q][2] = fmaf(fb.y, sx.x, accB[q][2]); accB[q][3] = fmaf(fb.y, sx.y, accB[q][3]);
        }
    }
}
// slice value = scale part + bias part, added to the running total (which starts from 0, as reduce_tiles() does)
template <int RG>
__device__ __forceinline__ void add_slice(float tot[RG][4], const float accS[RG][4], const float accB[RG][4]) {
#pragma unroll
    for (int q = 0; q < RG; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) tot[q][i] = __fadd_rn(tot[q][i], __fadd_rn(accS[q][i], accB[q][i]));
}

// ================================================================================ dense projection
struct RowsDenseArgs {
    Q4R q; int N, K, M;
    const __half* xq; const float* sxq;  // prepared rows
    __half* y; int ldy;
    const __half* x; int ldx;            // or plain rows, which every CTA prepares for itself (x != nullptr)
};
// Bound by instruction issue, shared-memory reads and MMAs about equally (a slice of 16 weight rows against 32 rows: 485
// instructions of a warp, 150 cycles of shared-memory reads, 64 MMAs; it takes 235 cycles of a multiprocessor).  The form
// before had 8 warps a multiprocessor, weights in registers and two CTA barriers a slice.  By events (about 5 us of them
// the events'), in / out: 512 rows 134 -> 97, 60 -> 51 us; 64 rows 30 -> 23, 20 -> 19; 17 rows 16.6 -> 15.5, 18.7 -> 12.7.
// Two forms; in both a CTA has one block of rows in shared memory and an equal run of the tiles of 16 weight rows (grid: CTAs
// of a block, blocks), and every warp its own ring of weight slices, so that no barrier stands in the stream.
struct RdGeom { int row0, nrows, lo, hi; };                   // the CTA's rows and tiles
__device__ __forceinline__ RdGeom rd_geom(const RowsDenseArgs& a, int nr) {
    const int row0 = blockIdx.y * nr, ntiles = a.N >> 4;
    return {row0, min(nr, a.M - row0), (int)((long)ntiles * blockIdx.x / gridDim.x), (int)((long)ntiles * (blockIdx.x + 1) / gridDim.x)};
}
// inputs k0 .. k0 + kc - 1 of the rows into xs [row][kc + 8] (16 bytes of skew: conflict-free loads), their group sums into sxs [group][stride]
__device__ __forceinline__ void rd_stage(const RowsDenseArgs& a, const RdGeom& g, int k0, int kc, __half* xs, float* sxs, int stride) {
    const int c8 = kc >> 3, g64 = kc >> 6;
    if (a.x) {                                                // the arithmetic of rows_store(), two units of 256 inputs in flight per warp
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, chunks = kc >> 8, units = g.nrows * chunks;
        for (int u0 = warp; u0 < units; u0 += 2 * nw) {
            uint4 v[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int u = u0 + i * nw, row = u / chunks, ch = u - row * chunks;
                if (u < units) v[i] = __ldcg(reinterpret_cast<const uint4*>(a.x + (size_t)(g.row0 + row) * a.ldx + k0 + ch * 256 + lane * 8));
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int u = u0 + i * nw, row = u / chunks, ch = u - row * chunks;
                if (u >= units) break;
                float s;                                      // (of lanes 0, 8, 16, 24: one group each)
                rows_store(xs + (size_t)row * (kc + 8) + ch * 256 + lane * 8, &s, 0, v[i], lane);
                if ((lane & 7) == 0) sxs[(ch * 4 + (lane >> 3)) * stride + row] = s;
            }
        }
        cp_async_wait<0>();
        __syncthreads();
        return;
    }
    for (int i = threadIdx.x; i < g.nrows * c8; i += blockDim.x) {
        const int row = i / c8, c = i - row * c8;
        cp_async16(xs + (size_t)row * (kc + 8) + c * 8, a.xq + (size_t)(g.row0 + row) * a.K + k0 + c * 8);
    }
    cp_async_commit();
    for (int i = threadIdx.x; i < g.nrows * g64; i += blockDim.x) {
        const int row = i / g64, c = i - row * g64;
        sxs[c * stride + row] = __ldcg(a.sxq + (size_t)(g.row0 + row) * (a.K >> 6) + (k0 >> 6) + c);
    }
    cp_async_wait<0>();
    __syncthreads();
}
template <int EPI>
__device__ __forceinline__ void rd_store(const RowsDenseArgs& a, int row, int n, float v) {
    const size_t idx = (size_t)row * a.ldy + n;
    __half val = f2h(v);
    if (EPI == EPI_RESID) val = hadd_rn(a.y[idx], val);
    a.y[idx] = val;
}
// Tile form: a warp takes every NW-th tile of the run over the whole K.  The block's rows are staged in chunks of kc inputs:
// once when the whole K fits, else again for every round of NW tiles (the totals stay in registers meanwhile).
template <int RG, int NW>
__host__ __device__ constexpr size_t rd_smem(int kc) { return (size_t)NW * XR_DEPTH * XR_UNIT + (size_t)8 * RG * (kc + 8) * 2 + (size_t)(kc >> 6) * (8 * RG + 2) * 4; }
template <int EPI, int RG, int NW>
__global__ void __launch_bounds__(NW * 32, 1) k_gemv_rows(RowsDenseArgs a, int kc) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NR = 8 * RG, SXS = NR + 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, t = lane & 3;
    const int slices = a.K >> 8, cslices = kc >> 8, XS = kc + 8;
    unsigned char* ring = smem + (size_t)warp * XR_DEPTH * XR_UNIT;
    __half* xs = reinterpret_cast<__half*>(smem + (size_t)NW * XR_DEPTH * XR_UNIT);
    float* sxs = reinterpret_cast<float*>(xs + (size_t)NR * XS);
    const RdGeom geo = rd_geom(a, NR);
    const size_t wstep = q4r_w_uint4(a.K), sstep = q4r_s_uint4(a.K);
    int rt = geo.lo + warp, rs = 0, slot = 0;                 // the request cursor: tile, slice; the ring slot read next
    auto request = [&](int to) {
        if (rt < geo.hi) ring_request(ring + to * XR_UNIT, a.q.wr + (size_t)rt * wstep, a.q.sr + (size_t)rt * sstep, rs, lane);
        cp_async_commit();
        if (++rs == slices) { rs = 0; rt += NW; }
    };
    static_assert(XR_DEPTH == 2, "two ring slots");
    request(0); request(1);                                   // weights: ahead of the programmatic-launch wait
    pdl_wait();
    pdl_launch_dependents();
    if (kc == a.K) rd_stage(a, geo, 0, kc, xs, sxs, SXS);
    const __half* xp = xs + (size_t)r * XS + 16 * t;
#pragma unroll 1
    for (int t0 = geo.lo; t0 < geo.hi; t0 += NW) {
        const int tile = t0 + warp;
        float tot[RG][4];
#pragma unroll
        for (int q = 0; q < RG; ++q) { tot[q][0] = 0.f; tot[q][1] = 0.f; tot[q][2] = 0.f; tot[q][3] = 0.f; }
#pragma unroll 1
        for (int c = 0; c < slices; c += cslices) {
            if (kc != a.K) { __syncthreads(); rd_stage(a, geo, c << 8, kc, xs, sxs, SXS); }
            if (tile >= geo.hi) continue;
#pragma unroll 1
            for (int s = 0; s < cslices; ++s) {
                cp_async_wait<XR_DEPTH - 1>();
                __syncwarp();                                 // every lane's part of the slice is there
                float accS[RG][4], accB[RG][4];
#pragma unroll
                for (int q = 0; q < RG; ++q)
#pragma unroll
                    for (int i = 0; i < 4; ++i) { accS[q][i] = 0.f; accB[q][i] = 0.f; }
                compute_rows<RG>(ring + slot * XR_UNIT, xp + s * 256, XS, sxs + s * 4 * SXS + 2 * t, SXS, lane, accS, accB);
                add_slice<RG>(tot, accS, accB);
                __syncwarp();                                 // every lane has read the slot: it may be filled again
                request(slot);
                slot ^= 1;
            }
        }
        if (tile >= geo.hi) continue;
#pragma unroll
        for (int q = 0; q < RG; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int xrow = q * 8 + 2 * t + (i & 1);
                if (xrow < geo.nrows) rd_store<EPI>(a, geo.row0 + xrow, tile * 16 + r + 8 * (i >> 1), tot[q][i]);
            }
    }
}
// Split form, for runs of few tiles: the warps share out the (tile, slice) pairs of the run; the slice values meet in shared
// memory and are added in ascending order (as reduce_tiles() does).  With a tile per warp, four tiles of 16 slices were 10 us
// of waiting for two slices at a time.
constexpr int RD_SPLIT_WARPS = 16, RD_PART = 8 * 20;          // floats of a pair's values: [column][16 rows + 4], conflict-free stores
__host__ __device__ constexpr size_t rd_split_smem(int K, int units) { return rd_smem<1, RD_SPLIT_WARPS>(K) + (size_t)units * RD_PART * 4; }
template <int EPI>
__global__ void __launch_bounds__(RD_SPLIT_WARPS * 32, 1) k_gemv_rows_split(RowsDenseArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NW = RD_SPLIT_WARPS, SXS = 8 + 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, t = lane & 3;
    const int slices = a.K >> 8, XS = a.K + 8;
    unsigned char* ring = smem + (size_t)warp * XR_DEPTH * XR_UNIT;
    __half* xs = reinterpret_cast<__half*>(smem + (size_t)NW * XR_DEPTH * XR_UNIT);
    float* sxs = reinterpret_cast<float*>(xs + (size_t)8 * XS);
    float* part = sxs + (size_t)(a.K >> 6) * SXS;
    const RdGeom geo = rd_geom(a, 8);
    const int units = (geo.hi - geo.lo) * slices;
    auto request = [&](int u, int to) {
        if (u < units) {
            const int tl = u / slices, tile = geo.lo + tl;
            ring_request(ring + to * XR_UNIT, a.q.wr + (size_t)tile * q4r_w_uint4(a.K), a.q.sr + (size_t)tile * q4r_s_uint4(a.K), u - tl * slices, lane);
        }
        cp_async_commit();
    };
    request(warp, 0); request(warp + NW, 1);                  // weights: ahead of the programmatic-launch wait
    pdl_wait();
    pdl_launch_dependents();
    rd_stage(a, geo, 0, a.K, xs, sxs, SXS);
    const __half* xp = xs + (size_t)r * XS + 16 * t;
    int slot = 0;
#pragma unroll 1
    for (int u = warp; u < units; u += NW) {
        const int s = u % slices;
        cp_async_wait<XR_DEPTH - 1>();
        __syncwarp();
        float accS[1][4] = {{0.f, 0.f, 0.f, 0.f}}, accB[1][4] = {{0.f, 0.f, 0.f, 0.f}};
        compute_rows<1>(ring + slot * XR_UNIT, xp + s * 256, XS, sxs + s * 4 * SXS + 2 * t, SXS, lane, accS, accB);
        __syncwarp();
        request(u + 2 * NW, slot);
        slot ^= 1;
        float* p = part + (size_t)u * RD_PART + 2 * t * 20 + r;
#pragma unroll
        for (int i = 0; i < 4; ++i) p[(i & 1) * 20 + 8 * (i >> 1)] = __fadd_rn(accS[0][i], accB[0][i]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (geo.hi - geo.lo) * 128; i += NW * 32) {
        const int tl = i >> 7, col = (i >> 4) & 7, row = i & 15;
        if (col >= geo.nrows) continue;
        const float* p = part + (size_t)tl * slices * RD_PART + col * 20 + row;
        float v = 0.f;
        for (int s = 0; s < slices; ++s) v = __fadd_rn(v, p[(size_t)s * RD_PART]);
        rd_store<EPI>(a, geo.row0 + col, (geo.lo + tl) * 16 + row, v);
    }
}
constexpr size_t RD_ROOM = (size_t)227 * 1024;
// CTAs that share a block of nr rows: all multiprocessors divided by the blocks
static int rd_ctas(int M, int nr, int ntiles) {
    const int c = sm_count() / ((M + nr - 1) / nr);
    return c < 1 ? 1 : (c > ntiles ? ntiles : c);
}
template <int EPI, int RG, int NW>
static void launch_gemv_rows_t(const RowsDenseArgs& a, cudaStream_t st, bool pdl) {
    static bool configured = false;
    if (!configured) { cudaFuncSetAttribute(k_gemv_rows<EPI, RG, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RD_ROOM); configured = true; }
    int kc = a.K;                                              // (K: a multiple of 256 up to 4096, so of 512 where halves are needed -- see rd_fits)
    if (rd_smem<RG, NW>(kc) > RD_ROOM) kc = a.K / 2;
    const dim3 grid((unsigned)rd_ctas(a.M, 8 * RG, a.N >> 4), (unsigned)((a.M + 8 * RG - 1) / (8 * RG)));
    profile_launch(EPI == EPI_RESID ? "k_gemv_rows_outproj" : "k_gemv_rows_inproj", st, [&] {
        return launch_pdl(pdl, k_gemv_rows<EPI, RG, NW>, grid, NW * 32, rd_smem<RG, NW>(kc), st, a, kc);
    });
}
template <int EPI>
static void launch_gemv_rows(const RowsDenseArgs& a, cudaStream_t st, bool pdl) {
    const int ntiles = a.N >> 4, slices = a.K >> 8;
    auto tiles_of = [&](int nr) { const int c = rd_ctas(a.M, nr, ntiles); return (ntiles + c - 1) / c; };      // tiles of a CTA
    // split form: up to 8 tiles a run, a third of the tile form's warps (17 rows: 3 tiles of 16 slices 16.1 -> 12.7 us by events,
    // 16 tiles of 8 slices 15.5 -> 17.1)
    const size_t split = rd_split_smem(a.K, tiles_of(8) * slices);
    if (tiles_of(8) <= 8 && split <= RD_ROOM) {
        static bool configured = false;
        if (!configured) { cudaFuncSetAttribute(k_gemv_rows_split<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RD_ROOM); configured = true; }
        profile_launch(EPI == EPI_RESID ? "k_gemv_rows_outproj" : "k_gemv_rows_inproj", st, [&] {
            return launch_pdl(pdl, k_gemv_rows_split<EPI>, dim3((unsigned)rd_ctas(a.M, 8, ntiles), (unsigned)((a.M + 7) / 8)), RD_SPLIT_WARPS * 32, split, st, a);
        });
        return;
    }
    // 8, 16 or 32 rows per CTA: a tile of 8 slices takes 0.41, 0.60 or 1.0 us, the staging 3, 4 or 6 (more rows per block: fewer
    // expansions of the weights, but fewer CTAs per block and a longer start); waves of CTAs where the blocks are more than the multiprocessors
    const int nrs[3] = {8, 16, 32}, per_tile[3] = {41, 60, 100}, start[3] = {300, 400, 600};
    int best = 0; long best_cost = 0;
    for (int i = 0; i < 3; ++i) {
        if (i == 2 && rd_smem<4, 16>(a.K) > RD_ROOM && a.K % 512) continue;
        const long waves = ((a.M + nrs[i] - 1) / nrs[i] + sm_count() - 1) / sm_count();
        const long cost = waves * ((long)tiles_of(nrs[i]) * slices * per_tile[i] / 8 + start[i]);
        if (i == 0 || cost <= best_cost) { best = i; best_cost = cost; }
    }
    if (best == 2) launch_gemv_rows_t<EPI, 4, 16>(a, st, pdl);
    else if (best == 1) launch_gemv_rows_t<EPI, 2, 16>(a, st, pdl);
    else launch_gemv_rows_t<EPI, 1, 24>(a, st, pdl);
}
// dense projection of M > 1 rows (a.direct: of any number): prologue rows, then the tile kernel.  Returns false when the shape is not covered.
bool launch_dense_rows(int pro, int epi, const DenseArgs& a, cudaStream_t st, bool pdl) {
    // plain rows need no prologue kernel; of more than 32 the preparation in every CTA costs more than the launch
    const bool plain = pro == PRO_PLAIN && !a.prepared && (a.direct || a.M <= 32);
    if (!(a.xq && a.sxq) && !(plain && a.direct)) return false;
    if (!dense_rows_shape(a.direct ? 2 : a.M, a.N, a.K) || (epi != EPI_STORE && epi != EPI_RESID)) return false;
    RowsPrepArgs p{a.x, a.ldx, a.nw, a.nw32, a.z, a.ldz, a.eps, a.K, a.xq, a.sxq};
    if (!a.prepared && !plain) launch_rows_prep_args(pro, p, a.M, st, pdl);
    RowsDenseArgs d{a.q, a.N, a.K, a.M, a.xq, a.sxq, a.y, a.ldy, plain ? a.x : nullptr, a.ldx};
    if (epi == EPI_RESID) launch_gemv_rows<EPI_RESID>(d, st, pdl); else launch_gemv_rows<EPI_STORE>(d, st, pdl);
    return true;
}

// ================================================================================ lm_head + argmax
// The tile form with the argmax of k_head: per tile the largest logit of each row (lower index on a tie) is merged into the
// warp's table in shared memory, the CTAs' maxima meet in the CTA that finishes last.  k_head reads the whole matrix once per
// 8 rows (47 us each at 248320 x 2048, the memory's pace); here once per 16, 24 or 32 rows.
__device__ __forceinline__ bool head_better(float v, int i, float bv, int bi) { return v > bv || (v == bv && i < bi); }
template <int RG>
__global__ void __launch_bounds__(512, 1) k_head_rows(RowsDenseArgs a, __half* logits, float* pval, int* pidx, int* out_tok, unsigned* counter) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NW = 16, NR = 8 * RG, SXS = NR + 2;
    __shared__ float s_val[NW][NR];
    __shared__ int s_idx[NW][NR];
    __shared__ int s_last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, t = lane & 3;
    const int slices = a.K >> 8, XS = a.K + 8;
    unsigned char* ring = smem + (size_t)warp * XR_DEPTH * XR_UNIT;
    __half* xs = reinterpret_cast<__half*>(smem + (size_t)NW * XR_DEPTH * XR_UNIT);
    float* sxs = reinterpret_cast<float*>(xs + (size_t)NR * XS);
    const RdGeom geo = rd_geom(a, NR);
    const size_t wstep = q4r_w_uint4(a.K), sstep = q4r_s_uint4(a.K);
    int rt = geo.lo + warp, rs = 0, slot = 0;
    auto request = [&](int to) {
        if (rt < geo.hi) ring_request(ring + to * XR_UNIT, a.q.wr + (size_t)rt * wstep, a.q.sr + (size_t)rt * sstep, rs, lane);
        cp_async_commit();
        if (++rs == slices) { rs = 0; rt += NW; }
    };
    request(0); request(1);                                   // weights: ahead of the programmatic-launch wait
    if (lane < NR) { s_val[warp][lane] = -INFINITY; s_idx[warp][lane] = 0x7fffffff; }
    pdl_wait();
    pdl_launch_dependents();
    rd_stage(a, geo, 0, a.K, xs, sxs, SXS);
    const __half* xp = xs + (size_t)r * XS + 16 * t;
#pragma unroll 1
    for (int tile = geo.lo + warp; tile < geo.hi; tile += NW) {
        float tot[RG][4];
#pragma unroll
        for (int q = 0; q < RG; ++q) { tot[q][0] = 0.f; tot[q][1] = 0.f; tot[q][2] = 0.f; tot[q][3] = 0.f; }
#pragma unroll 1
        for (int s = 0; s < slices; ++s) {
            cp_async_wait<XR_DEPTH - 1>();
            __syncwarp();
            float accS[RG][4], accB[RG][4];
#pragma unroll
            for (int q = 0; q < RG; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i) { accS[q][i] = 0.f; accB[q][i] = 0.f; }
            compute_rows<RG>(ring + slot * XR_UNIT, xp + s * 256, XS, sxs + s * 4 * SXS + 2 * t, SXS, lane, accS, accB);
            add_slice<RG>(tot, accS, accB);
            __syncwarp();
            request(slot);
            slot ^= 1;
        }
#pragma unroll
        for (int q = 0; q < RG; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int row = q * 8 + 2 * t + j, n = tile * 16 + r;
                const __half lo = f2h(tot[q][j]), hi = f2h(tot[q][2 + j]);
                if (logits && row < geo.nrows) {
                    logits[(size_t)(geo.row0 + row) * a.N + n] = lo;
                    logits[(size_t)(geo.row0 + row) * a.N + n + 8] = hi;
                }
                float v = -INFINITY; int i = 0x7fffffff;      // (a NaN is never better: it must not stand for the lane's other logit)
                if (head_better(h2f(lo), n, v, i)) { v = h2f(lo); i = n; }
                if (head_better(h2f(hi), n + 8, v, i)) { v = h2f(hi); i = n + 8; }
#pragma unroll
                for (int off = 4; off <= 16; off <<= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, v, off);
                    const int oi = __shfl_xor_sync(0xffffffffu, i, off);
                    if (head_better(ov, oi, v, i)) { v = ov; i = oi; }
                }
                if (r == 0 && head_better(v, i, s_val[warp][row], s_idx[warp][row])) { s_val[warp][row] = v; s_idx[warp][row] = i; }
            }
    }
    __syncthreads();
    const int parts = gridDim.x;
    if ((int)threadIdx.x < geo.nrows) {
        const int row = threadIdx.x;
        float bv = -INFINITY; int bi = 0x7fffffff;
        for (int w = 0; w < NW; ++w) if (head_better(s_val[w][row], s_idx[w][row], bv, bi)) { bv = s_val[w][row]; bi = s_idx[w][row]; }
        pval[(size_t)(geo.row0 + row) * parts + blockIdx.x] = bv;
        pidx[(size_t)(geo.row0 + row) * parts + blockIdx.x] = bi;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(counter, 1u) == gridDim.x * gridDim.y - 1) ? 1 : 0;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int m = warp; m < a.M; m += NW) {                    // one warp per row over the CTAs' maxima
        float bv = -INFINITY; int bi = 0x7fffffff;
        for (int p = lane; p < parts; p += 32) {
            const float v = __ldcg(pval + (size_t)m * parts + p); const int i = __ldcg(pidx + (size_t)m * parts + p);
            if (head_better(v, i, bv, bi)) { bv = v; bi = i; }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
            if (head_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) out_tok[m] = bi;
    }
    if (threadIdx.x == 0) *counter = 0u;
}
template <int RG>
static void launch_head_rows_t(const RowsDenseArgs& d, const DenseArgs& a, cudaStream_t st, bool pdl) {
    static bool configured = false;
    if (!configured) { cudaFuncSetAttribute(k_head_rows<RG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(RD_ROOM - 8192)); configured = true; }
    const dim3 grid((unsigned)rd_ctas(d.M, 8 * RG, d.N >> 4), (unsigned)((d.M + 8 * RG - 1) / (8 * RG)));
    profile_launch("k_head", st, [&] { return launch_pdl(pdl, k_head_rows<RG>, grid, 512, rd_smem<RG, 16>(d.K), st, d, a.logits, a.pval, a.pidx, a.out_tok, a.counter); });
}
// lm_head of M > 8 rows with the final norm.  Returns false when the shape is not covered.
bool launch_head_rows(const DenseArgs& a, cudaStream_t st, bool pdl) {
    if (!a.xq || !a.sxq || a.K % 256 || a.K > 4096 || a.N % 16) return false;
    // by the pace of a block (tiles x 60, 80 or 100), blocks one after the other
    const int per_tile[3] = {60, 80, 100};
    int best = -1; long best_cost = 0;
    for (int i = 0; i < 3; ++i) {
        const size_t smem = i == 0 ? rd_smem<2, 16>(a.K) : i == 1 ? rd_smem<3, 16>(a.K) : rd_smem<4, 16>(a.K);
        const long cost = (long)((a.M + 16 + 8 * i - 1) / (16 + 8 * i)) * per_tile[i];
        if (smem <= RD_ROOM - 8192 && (best < 0 || cost < best_cost)) { best = i; best_cost = cost; }
    }
    if (best < 0) return false;
    RowsPrepArgs p{a.x, a.ldx, a.nw, nullptr, nullptr, 0, a.eps, a.K, a.xq, a.sxq};
    launch_rows_prep_args(PRO_RMSNORM, p, a.M, st, pdl);
    const RowsDenseArgs d{a.q, a.N, a.K, a.M, a.xq, a.sxq, nullptr, 0, nullptr, 0};
    if (best == 2) launch_head_rows_t<4>(d, a, st, pdl);
    else if (best == 1) launch_head_rows_t<3>(d, a, st, pdl);
    else launch_head_rows_t<2>(d, a, st, pdl);
    return true;
}

// ================================================================================ experts
// Work: (expert slot, block of 8 or 16 of its rows) x tiles of 16 weight rows, block-major; slot n_active is the shared expert
// (all rows).  A CTA per multiprocessor takes an equal, contiguous run of the tiles (one to three blocks at decode sizes)
// and its 24 (16) consumer warps walk that run, a tile over the whole K each.  A producer warp gathers the rows of the next block
// into a ring of shared-memory stages with bulk copies (mbarrier full / empty): no CTA-wide barrier between experts, which
// is what bounded the pass kernels when every expert has one or two rows.
// Bound: instruction issue first (the 4-bit expansion is about 150 of the 260 instructions that a slice of 16 x 256 weights
// needs), the weight stream second.  So: as many warps as the registers allow (six per sub-partition; four left 40 % of
// the issue slots empty), whole runs instead of items of 16 tiles (seven rounds for the work of 6.2), and a slice's weights
// by 16-byte asynchronous copies two slices ahead (110 KB per SM in flight; bulk copies of 2 KB arrive later; rows
// straight from L1 instead of staged: eight lines per load, 89 us for gate/up).  Batch of 64 (event times, 4.5 us of
// them the events'): gate/up 73.6 -> 64 us, down 53.4 -> 43.
// Blocks of 16 rows share the expansion (512 rows: 152 + 94 -> 129 + 80 us); the second half of a block of at most 8 rows is not computed.
__host__ __device__ constexpr int xr_blocks(int RG) { return 64 / RG; }        // most (slot, block) entries of a CTA's run
__host__ __device__ constexpr int xr_warps(int RG) { return RG == 1 ? 24 : 16; }       // consumer warps
template <int NR>
struct XrBlock { int expert, count; int src[NR], dst[NR]; };   // expert -1: the shared one; count: rows; src, dst -1: no row
struct XrStage {                              // the NR rows of a block in shared memory
    __half* xs;                               // [NR][K + 8]
    float* sxs;                               // [NR][K/64 + 4]
    float* craw;                              // down: [NR][K/8] chunk sums as written by the gate/up kernel
};
template <bool DOWN>
__host__ __device__ constexpr size_t xr_stage_bytes(int K, int NR) { return (size_t)NR * (K + 8) * 2 + (size_t)NR * (K / 64 + 4) * 4 + (DOWN ? (size_t)NR * (K / 8) * 4 : 0); }
template <int NR>
__device__ __forceinline__ XrStage xr_carve(unsigned char* base, int K) {
    XrStage s;
    s.xs = reinterpret_cast<__half*>(base); base += (size_t)NR * (K + 8) * 2;
    s.sxs = reinterpret_cast<float*>(base); base += (size_t)NR * (K / 64 + 4) * 4;
    s.craw = reinterpret_cast<float*>(base);
    return s;
}
// One slice of a tile, in a ring slot, against RG x 8 rows of a stage (xp: this lane's row of the first eight, sx: the slice's group
// sums of column 2t, of column 2t + 1 SXS floats on).  The order of operations per column is that of compute_slice_x().
template <int RG, int XS, int SXS>
__device__ __forceinline__ void xr_slice(const unsigned char* slot, const __half* xp, const float* sx, int lane, float (*tot)[4]) {
    const uint4* w = reinterpret_cast<const uint4*>(slot);
    float4 sa[RG], sb[RG];
    float accS[RG][4], accB[RG][4];
#pragma unroll
    for (int q = 0; q < RG; ++q) {
        sa[q] = *reinterpret_cast<const float4*>(sx + q * 8 * SXS); sb[q] = *reinterpret_cast<const float4*>(sx + (q * 8 + 1) * SXS);
#pragma unroll
        for (int i = 0; i < 4; ++i) accS[q][i] = accB[q][i] = 0.f;
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const uint4 wv = w[g * 32 + lane];
        uint32_t a0[4], b0[4], a1[4], b1[4];
        dequant8(wv.x, a0); dequant8(wv.z, b0); dequant8(wv.y, a1); dequant8(wv.w, b1);
        const uint2 sv = *reinterpret_cast<const uint2*>(slot + 2048 + (g >> 1) * 128 + (lane >> 2) * 16 + (g & 1) * 8);
        const float2 fa = __half22float2(*reinterpret_cast<const __half2*>(&sv.x)), fb = __half22float2(*reinterpret_cast<const __half2*>(&sv.y));
#pragma unroll
        for (int q = 0; q < RG; ++q) {
            const uint4 X0 = *reinterpret_cast<const uint4*>(xp + q * 8 * XS + 64 * g), X1 = *reinterpret_cast<const uint4*>(xp + q * 8 * XS + 64 * g + 8);
            float c[4];
            mma_f16_z(c, a0[0], b0[0], a0[1], b0[1], X0.x, X0.y);
            mma_f16(c, a0[2], b0[2], a0[3], b0[3], X0.z, X0.w);
            mma_f16(c, a1[0], b1[0], a1[1], b1[1], X1.x, X1.y);
            mma_f16(c, a1[2], b1[2], a1[3], b1[3], X1.z, X1.w);
            const float sx0 = g == 0 ? sa[q].x : g == 1 ? sa[q].y : g == 2 ? sa[q].z : sa[q].w, sx1 = g == 0 ? sb[q].x : g == 1 ? sb[q].y : g == 2 ? sb[q].z : sb[q].w;
            scale_group<false>(c, fa, fb, make_float2(sx0, sx1), accS[q], accB[q]);
        }
    }
    add_slice<RG>(tot, accS, accB);
}
// The routing of a call of at most XR_ROUTE rows, done by every CTA from the logits (a warp per row) in place of a kernel that routes and
// leaves lists: the choices, the slots in the order of their experts and the pairs of each slot in the order of their rows (all CTAs
// must agree on which pairs are a block).  All threads; rows, first: 256 words each; the caller synchronises before it reads t and pairs.
// Returns n_active.
constexpr int XR_ROUTE = 24;
__device__ __forceinline__ int slot_route(SlotTable& t, unsigned* rows, int* first, int* pairs, const ExpertArgs& a, int rows_per_block, int nshared) {
    const int tid = threadIdx.x, m = tid >> 5, lane = tid & 31;
    if (tid < 256) rows[tid] = 0u;
    int id = 0;
    if (m < a.M) id = route_select(route_load<false>(a.rlogits + (size_t)m * a.E, a.E, lane), a.E, a.topk, lane);
    const bool mine = m < a.M && lane < a.topk;
    __syncthreads();
    if (mine) atomicOr(&rows[id], 1u << m);
    __syncthreads();
    // pairs (at most 24 x 32), slots and blocks (at most 256) of the experts so far, ten bits each
    unsigned c = 0, own = 0, inc = 0;
    if (tid < 256) {
        c = (unsigned)__popc(rows[tid]);                        // (the choices are slots below E: top_k is at most E)
        own = c | (c > 0 ? 1u << 10 : 0u) | ((c + rows_per_block - 1) / rows_per_block) << 20;
        inc = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const unsigned o = __shfl_up_sync(0xffffffffu, inc, d); if (lane >= d) inc += o; }
        if (lane == 31) t.ws[m] = (int)inc;
    }
    __syncthreads();
    unsigned all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) { const unsigned o = (unsigned)t.ws[w]; all += o; if (w < m) inc += o; }
    const int n_active = (int)(all >> 10 & 1023u), blocks = (int)(all >> 20);
    if (tid < 256 && c > 0) {
        const unsigned before = inc - own;
        const int slot = (int)(before >> 10 & 1023u), off = (int)(before & 1023u);
        t.cnt[slot] = (int)c; t.expert[slot] = tid; t.off[slot] = off; t.base[slot + 1] = (int)(inc >> 20);
        first[tid] = off;
    }
    if (tid == 0) { t.base[0] = 0; t.base[n_active + 1] = blocks + (nshared + rows_per_block - 1) / rows_per_block; }
    __syncthreads();
    if (mine) pairs[first[id] + __popc(rows[id] & ((1u << m) - 1u))] = m * a.topk + lane;
    return n_active;
}
// S: slices of K.  RG: blocks of 8 or 16 rows.  STALL: a test's form, in which no row is ever fetched, so that every consumer's wait runs out, and soon
template <bool DOWN, int S, int RG, bool STALL>
__global__ void __launch_bounds__((xr_warps(RG) + 1) * 32, 1) k_expert_rows(ExpertArgs a, int lg_tiles, int nstages) {
    extern __shared__ __align__(16) unsigned char smem[];        // weight rings, then nstages stages
    __shared__ __align__(8) uint64_t s_full[8], s_empty[8], s_raw[8];
    __shared__ SlotTable s_tab;
    constexpr int XR_WARPS = xr_warps(RG), XR_THREADS = (XR_WARPS + 1) * 32, NR = 8 * RG;
    __shared__ XrBlock<NR> s_blk[xr_blocks(RG)];
    __shared__ int s_sig, s_abort, s_pairs[XR_ROUTE * 32];
    constexpr int K = S << 8, G64 = K >> 6, SXS = G64 + 4, XS = K + 8;
    constexpr size_t stage_bytes = xr_stage_bytes<DOWN>(K, NR);
    unsigned char* stages = smem + (size_t)XR_WARPS * XR_DEPTH * XR_UNIT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, t = lane & 3;
    const int ntiles = 1 << lg_tiles, npair = a.M * a.topk;
    const int nshared = a.M_shared >= 0 ? a.M_shared : a.M;
    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < nstages; ++i) { mbar_init(&s_full[i], DOWN ? 1 : NR); mbar_init(&s_empty[i], XR_WARPS); mbar_init(&s_raw[i], NR); }
        mbar_fence_init();
    }
    if (!DOWN) pdl_wait();                                      // the lists, or the logits (down: they were there before gate/up started)
    pdl_launch_dependents();
    unsigned* scratch = reinterpret_cast<unsigned*>(s_blk);     // (filled below)
    static_assert(sizeof(s_blk) >= 512 * sizeof(int), "counters of slot_route()");
    const int n_active = RG == 1 && a.route_here ? slot_route(s_tab, scratch, reinterpret_cast<int*>(scratch + 256), s_pairs, a, NR, nshared) : slot_table(s_tab, a.lists, NR, nshared);
    const int* pairs = RG == 1 && a.route_here ? s_pairs : a.lists.pairs;
    __syncthreads();
    const long total = (long)s_tab.base[n_active + 1] << lg_tiles;
    const int lo = (int)(total * blockIdx.x / gridDim.x), hi = (int)(total * (blockIdx.x + 1) / gridDim.x);
    const int b0 = lo >> lg_tiles, nb = hi > lo ? ((hi - 1) >> lg_tiles) - b0 + 1 : 0;
    for (int i = tid; i < nb * NR; i += XR_THREADS) {           // the rows of the run's blocks
        const int sb = b0 + i / NR, n = i % NR, j = slot_of(s_tab, n_active, sb), first = (sb - s_tab.base[j]) * NR, ridx = first + n;
        const bool shared = (j == n_active);
        const int cnt = shared ? nshared : s_tab.cnt[j];
        const bool have = ridx < cnt;
        int dst = -1, src = -1;
        if (have && shared) { dst = npair + ridx; src = DOWN ? dst : a.shared_row0 + ridx; }
        else if (have) { dst = pairs[s_tab.off[j] + ridx]; src = DOWN ? dst : dst / a.topk; }
        XrBlock<NR>& b = s_blk[i / NR];
        b.src[n] = src; b.dst[n] = dst;
        if (n == 0) { b.count = cnt - first; b.expert = shared ? -1 : s_tab.expert[j]; }
    }
    __syncthreads();
    unsigned fail_code = 0;          // which wait ran out: 16 producer/empty, 32 producer/chunk sums, 64 consumer/full
    if (warp == XR_WARPS) {
        // ------------------------------------------------------------ producer: the rows of the run's blocks, stage after stage
        if (DOWN) pdl_wait();                                  // the gate/up kernel's rows
        for (int k = 0; k < nb && !STALL; ++k) {
            const int stg = k % nstages, use = k / nstages;
            const XrStage St = xr_carve<NR>(stages + (size_t)stg * stage_bytes, K);
            if (use > 0 && !xr_wait<STALL>(&s_empty[stg], (uint32_t)((use - 1) & 1), &s_abort)) { fail_code |= 16u; break; }
            if (lane < NR) {
                uint64_t* bar = DOWN ? &s_raw[stg] : &s_full[stg];
                const int src = s_blk[k].src[lane];
                if (src >= 0) {
                    const __half* xsrc = (DOWN ? a.hbuf : a.xq) + (size_t)src * K;
                    constexpr uint32_t sums = (DOWN ? K / 8 : G64) * 4;
                    mbar_expect_tx(bar, (uint32_t)(K * 2) + sums);
                    bulk_g2s(St.xs + (size_t)lane * XS, xsrc, (uint32_t)K * 2, bar);
                    if (DOWN) bulk_g2s(St.craw + (size_t)lane * (K / 8), a.csum + (size_t)src * (K / 8), sums, bar);
                    else bulk_g2s(St.sxs + (size_t)lane * SXS, a.sxq + (size_t)src * G64, sums, bar);
                } else mbar_arrive(bar);                              // (a column without a row keeps what was there: nobody reads its result)
            }
            if (DOWN) {
                // group sums from the chunk sums: eight of them combined in the butterfly order of rows_store()
                if (!xr_wait<STALL>(&s_raw[stg], (uint32_t)(use & 1), &s_abort)) { fail_code |= 32u; break; }
                for (int i = lane; i < NR * G64; i += 32) {
                    const int row = i / G64, g = i - row * G64;
                    const float* c = St.craw + (size_t)row * (K / 8) + g * 8;
                    const float4 lo4 = *reinterpret_cast<const float4*>(c), hi4 = *reinterpret_cast<const float4*>(c + 4);
                    const float e = __fadd_rn(__fadd_rn(lo4.x, hi4.x), __fadd_rn(lo4.z, hi4.z));       // (s0 + s4) + (s2 + s6)
                    const float o = __fadd_rn(__fadd_rn(lo4.y, hi4.y), __fadd_rn(lo4.w, hi4.w));       // (s1 + s5) + (s3 + s7)
                    St.sxs[(size_t)row * SXS + g] = __fadd_rn(e, o);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_full[stg]);
            }
        }
        // the choices and gates of row m, for the combine, from CTA m (nobody waits for them here)
        if (RG == 1 && !DOWN && a.route_here) {
            __shared__ float s_gate[256];
            for (int m = blockIdx.x; m < a.M; m += gridDim.x) {
                __syncwarp();
                route_row_warp(a.rlogits + (size_t)m * a.E, a.E, a.topk, a.inds_out + m * a.topk, a.scores_out + m * a.topk, s_gate, lane);
            }
        }
    } else {
    // ---------------------------------------------------------------- consumers
    unsigned char* ring = smem + (size_t)warp * XR_DEPTH * XR_UNIT;
    const size_t wstep = q4r_w_uint4(K), sstep = q4r_s_uint4(K);
    // nibbles and scales of tile task `i` (nullptr past the run's end)
    auto tile_of = [&](int i, const uint4*& w, const uint4*& sc) {
        w = nullptr; sc = nullptr;
        if (i >= hi) return;
        const int e = s_blk[(i >> lg_tiles) - b0].expert;
        const Q4R& q = DOWN ? (e < 0 ? a.sh_down : a.down) : (e < 0 ? a.sh_gu : a.gu);
        const size_t T = ((size_t)max(e, 0) << lg_tiles) + (i & (ntiles - 1));
        w = q.wr + T * wstep; sc = q.sr + T * sstep;
    };
    auto request = [&](int slot, const uint4* w, const uint4* sc, int s) {      // slice s of a tile into a ring slot: one copy group
        if (w) ring_request(ring + slot * XR_UNIT, w, sc, s, lane);
        cp_async_commit();
    };
    constexpr int NB = XR_DEPTH > S ? XR_DEPTH / S : 1;           // tiles the ring holds at least the start of
    const uint4 *w0, *c0, *wn, *cn;                               // this tile, and the one whose slices are requested ahead
    tile_of(lo + warp, w0, c0);
    if (S >= XR_DEPTH) { request(0, w0, c0, 0); request(1, w0, c0, 1); }
    else { request(0, w0, c0, 0); tile_of(lo + warp + XR_WARPS, wn, cn); request(1, wn, cn, 0); }
    int odd = 0, cur = 0;                                         // cur: the block whose stage this warp holds
    bool here = false;                                            // its rows have arrived
#pragma unroll 1
    for (int i = lo + warp; i < hi; i += XR_WARPS) {
        tile_of(i + NB * XR_WARPS, wn, cn);
        const int bi = (i >> lg_tiles) - b0, tile = i & (ntiles - 1);
        const XrBlock<NR>& b = s_blk[bi];
        if (bi != cur) {                                          // done with the stages of the blocks before
            __syncwarp();
            if (lane == 0) for (int u = cur; u < bi; ++u) mbar_arrive(&s_empty[u % nstages]);
            cur = bi; here = false;
        }
        if (!here && !xr_wait<STALL>(&s_full[bi % nstages], (uint32_t)((bi / nstages) & 1), &s_abort)) { fail_code |= 64u; break; }
        here = true;
        const XrStage St = xr_carve<NR>(stages + (size_t)(bi % nstages) * stage_bytes, K);
        const __half* xp = St.xs + (size_t)r * XS + 16 * t;
        const float *sx0 = St.sxs + 2 * t * SXS, *sx1 = sx0 + SXS;
        float tot[RG][4];
#pragma unroll
        for (int i = 0; i < RG * 4; ++i) tot[i >> 2][i & 3] = 0.f;
        const bool full = RG == 1 || b.count > 8;                 // (16 rows: of a block's last eight there may be none)
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int slot = S >= XR_DEPTH ? s % XR_DEPTH : odd;
            if constexpr (RG == 1) {
                XRegs xr;
                const float4 sa = *reinterpret_cast<const float4*>(sx0 + s * 4), sb = *reinterpret_cast<const float4*>(sx1 + s * 4);
                xr.sx[0] = make_float2(sa.x, sb.x); xr.sx[1] = make_float2(sa.y, sb.y); xr.sx[2] = make_float2(sa.z, sb.z); xr.sx[3] = make_float2(sa.w, sb.w);
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    xr.x[2 * g] = *reinterpret_cast<const uint4*>(xp + s * 256 + 64 * g);
                    xr.x[2 * g + 1] = *reinterpret_cast<const uint4*>(xp + s * 256 + 64 * g + 8);
                }
                cp_async_wait<XR_DEPTH - 1>();
                __syncwarp();                                         // every lane's part of the slice is there
                SliceRegs rg;
                load_slice_smem(rg, reinterpret_cast<const uint4*>(ring + slot * XR_UNIT), reinterpret_cast<const uint4*>(ring + slot * XR_UNIT + 2048), lane);
                float accS[1][4] = {{0.f, 0.f, 0.f, 0.f}}, accB[1][4] = {{0.f, 0.f, 0.f, 0.f}};
                compute_slice_x(rg, xr, accS[0], accB[0]);
                add_slice<1>(tot, accS, accB);
            } else {
                cp_async_wait<XR_DEPTH - 1>();
                __syncwarp();
                if (full) xr_slice<RG, XS, SXS>(ring + slot * XR_UNIT, xp + s * 256, sx0 + s * 4, lane, tot);
                else xr_slice<1, XS, SXS>(ring + slot * XR_UNIT, xp + s * 256, sx0 + s * 4, lane, tot);
            }
            __syncwarp();                                         // every lane has read the slot: it may be filled again
            if (S > XR_DEPTH && s + XR_DEPTH < S) request(slot, w0, c0, s + XR_DEPTH);
            else request(slot, wn, cn, S > XR_DEPTH ? s + XR_DEPTH - S : s);
        }
        w0 = wn; c0 = cn; odd ^= 1;
        if (DOWN) {
#pragma unroll
            for (int u = 0; u < 4 * RG; ++u) {
                const int dst = b.dst[(u >> 2) * 8 + 2 * t + (u & 1)];
                if (dst >= 0) {
                    __half* rowp = a.dbuf + (size_t)dst * a.H;
                    if (a.ep_pairs_per_rank > 0 && dst < npair) {       // routed pair in expert-parallel mode: the owner's buffer
                        const int own = dst / a.ep_pairs_per_rank;
                        rowp = a.peer_dbuf[own] + (size_t)(dst - own * a.ep_pairs_per_rank) * a.H;
                    }
                    rowp[tile * 16 + r + 8 * (u >> 1 & 1)] = f2h(tot[u >> 2][u & 3]);
                }
            }
        } else {
            // SwiGLU of (gate row r, up row r) per column; the 8 outputs of a column (lanes with the same t) form one
            // 8-chunk of the down projection's input: stored in the products' order with its chunk sum
#pragma unroll
            for (int j = 0; j < 2 * RG; ++j) {
                const int q = j >> 1, jc = j & 1;
                if (q > 0 && !full) break;
                const __half hv = swiglu_h(f2h(tot[q][jc]), f2h(tot[q][2 + jc]));
                const unsigned hb = __half_as_ushort(hv);
                unsigned v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = __shfl_sync(0xffffffffu, hb, u * 4 + t);
                const int dst = b.dst[q * 8 + 2 * t + jc];
                if (r == 0 && dst >= 0) {
                    const uint4 nat = make_uint4(v[0] | (v[1] << 16), v[2] | (v[3] << 16), v[4] | (v[5] << 16), v[6] | (v[7] << 16));
                    *reinterpret_cast<uint4*>(a.hbuf + (size_t)dst * a.I + tile * 8) = make_uint4(nat.x, nat.z, nat.y, nat.w);
                    a.csum[(size_t)dst * (a.I / 8) + tile] = sum8_f32(nat);
                }
            }
        }
    }
    __syncwarp();
    if (lane == 0) for (int u = cur; u < nb; ++u) mbar_arrive(&s_empty[u % nstages]);      // (also of blocks in which this warp had no tile)
    }
    if (fail_code && a.err && lane == 0) atomicOr(a.err, fail_code | (DOWN ? 8u : 4u));
    if (fail_code) {                           // bulk copies this CTA started may still be landing in its shared memory: outlast them
        const long long t0 = clock64();
        while (clock64() - t0 < 200000ll) { }
    }
    if (DOWN && a.ep_sig.world > 0) {
        // expert-parallel: every CTA makes its peer stores visible system-wide and draws a ticket; the last one raises this
        // rank's combine flag at every peer
        __threadfence_system();
        __syncthreads();
        if (tid == 0) {
            const unsigned ticket = atomicAdd(a.ep_sig.ticket, 1u);
            s_sig = (ticket == gridDim.x - 1) ? 1 : 0;
            if (s_sig) *a.ep_sig.ticket = 0u;
        }
        __syncthreads();
        if (s_sig && tid < a.ep_sig.world)
            st_release_sys(a.ep_sig.flags[tid] + 8 + a.ep_sig.rank, ep_seq(a.ep_sig.ctr, a.ep_sig.layer, 1));
    }
}
// the tiles (their binary logarithm) and the stages of a launch with blocks of 8 RG rows; false: shape not covered
template <bool DOWN>
static bool expert_rows_shape(const ExpertArgs& a, int RG, int& lg, int& nstages) {
    const int ntiles = DOWN ? a.H / 16 : a.I / 8, K = DOWN ? a.I : a.H, NR = 8 * RG;
    if (!a.csum || (!DOWN && (!a.xq || !a.sxq)) || (K != 256 && K != 512 && K != 1024 && K != 2048 && K != 4096)) return false;
    lg = 0; while ((1 << lg) < ntiles) ++lg;
    const long pairs = (long)a.M * a.topk, blocks = pairs / NR + (pairs < 256 ? pairs : 256) + a.M / NR + 1;    // at most one partial block per expert
    nstages = (int)(((size_t)216 * 1024 - (size_t)xr_warps(RG) * XR_DEPTH * XR_UNIT) / xr_stage_bytes<DOWN>(K, NR));
    if (nstages > 8) nstages = 8;
    return (1 << lg) == ntiles && blocks / sm_count() + 2 <= xr_blocks(RG) && nstages >= RG;
}
// A warp per row: more rows would be routed in turns by every CTA, and a kernel of its own is done sooner.
bool expert_rows_route(const ExpertArgs& a) {
    int lg, nstages;
    return a.M <= XR_ROUTE && a.E <= 256 && a.topk <= 32 && a.ep_pairs_per_rank == 0 && expert_rows_shape<false>(a, 1, lg, nstages) && expert_rows_shape<true>(a, 1, lg, nstages);
}
template <bool DOWN, int S, int RG, bool STALL = false>
static bool launch_expert_rows_t(const ExpertArgs& a, cudaStream_t st, bool pdl) {
    const int grid = sm_count();
    int lg, nstages;
    if (!expert_rows_shape<DOWN>(a, RG, lg, nstages)) return false;
    const size_t smem = (size_t)xr_warps(RG) * XR_DEPTH * XR_UNIT + xr_stage_bytes<DOWN>(S << 8, 8 * RG) * nstages;
    static bool configured = false;
    if (!configured) { cudaFuncSetAttribute(k_expert_rows<DOWN, S, RG, STALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); configured = true; }
    profile_launch(DOWN ? "k_expert_rows_down" : "k_expert_rows_gateup", st, [&] { return launch_pdl(pdl, k_expert_rows<DOWN, S, RG, STALL>, dim3((unsigned)grid), (xr_warps(RG) + 1) * 32, smem, st, a, lg, nstages); });
    return true;
}
// Blocks of 16 rows from a mean of more than 8 rows an expert: with fewer most blocks would be half empty, and the 16 warps that
// two stages of 16 rows leave room for are slower than 24 (gate/up + down, 256 experts, 8 a row, evenly: 192 rows 121 us in blocks of 8,
// 136 in blocks of 16, 256 rows 150 and 150, 320 rows 174 and 154, 512 rows 245 and 208).  For K = 4096 there is no room.
// Expert-parallel calls too: their rows are those of all ranks, and the mean over all experts is that of the rank's own.
template <bool DOWN, int S>
static bool launch_expert_rows_s(const ExpertArgs& a, cudaStream_t st, bool pdl) {
    if ((long)a.M * a.topk > 8l * a.E && !a.route_here && launch_expert_rows_t<DOWN, S, 2>(a, st, pdl)) return true;
    return launch_expert_rows_t<DOWN, S, 1>(a, st, pdl);
}
template <bool DOWN>
static bool launch_expert_rows_d(const ExpertArgs& a, cudaStream_t st, bool pdl) {
    switch (DOWN ? a.I : a.H) {
        case 256: return launch_expert_rows_s<DOWN, 1>(a, st, pdl);
        case 512: return !DOWN && a.stall ? launch_expert_rows_t<DOWN, 2, 1, !DOWN>(a, st, pdl) : launch_expert_rows_s<DOWN, 2>(a, st, pdl);
        case 1024: return launch_expert_rows_s<DOWN, 4>(a, st, pdl);
        case 2048: return launch_expert_rows_s<DOWN, 8>(a, st, pdl);
        case 4096: return launch_expert_rows_t<DOWN, 16, 1>(a, st, pdl);
        default: return false;
    }
}
bool launch_expert_rows_gateup(const ExpertArgs& a, cudaStream_t st, bool pdl) { return launch_expert_rows_d<false>(a, st, pdl); }
bool launch_expert_rows_down(const ExpertArgs& a, cudaStream_t st, bool pdl) { return launch_expert_rows_d<true>(a, st, pdl); }

// ================================================================================ router for many rows
// k_router_rows   logits of all rows: a CTA keeps 8 router rows (or the shared gate) in registers and walks the row
//                 groups of 8, whose normed rows arrive in shared memory by cp.async two groups ahead of their use.
//                 The dot product is the one of k_moe_router (lane l owns 8 consecutive inputs of every 256-wide block,
//                 sequential f32 accumulate, butterfly over the lanes), so the logits are the same bits.
// k_route_rows    one warp per row: top-k + gates (route_row_warp), and the row's pairs go to their experts' places; the last CTA
//                 lists the experts that have pairs.  (Expert-parallel: a CTA per row, which sends the indices to every rank.)
// Input rows are already normed (k_final_norm), so no CTA repeats the norm.
template <bool Q8>
__global__ void __launch_bounds__(256, 2) k_router_rows(RouterArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];                   // [2][8][H] halves
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nblk = a.H >> 8;
    const bool tail = (blockIdx.x == gridDim.x - 1);
    const int e = blockIdx.x * 8 + warp;
    const bool wvalid = tail ? (warp == 0) : (e < a.E);
    uint4 wreg[16]; uint2 qreg[16]; __half2 sbreg[16];
    if constexpr (Q8) {
        const uint8_t* qrow = tail ? a.sg_q8 : (a.router_q8 + (size_t)e * a.H);
        const __half* srow = tail ? a.sg_qs : (a.router_qs + (size_t)e * (a.H >> 6));
        const __half* brow = tail ? a.sg_qb : (a.router_qb + (size_t)e * (a.H >> 6));
#pragma unroll
        for (int kb = 0; kb < 16; ++kb) {
            const bool ok = wvalid && kb < nblk;
            qreg[kb] = ok ? *reinterpret_cast<const uint2*>(qrow + kb * 256 + lane * 8) : make_uint2(0, 0);
            sbreg[kb] = ok ? __halves2half2(srow[kb * 4 + (lane >> 3)], brow[kb * 4 + (lane >> 3)]) : __halves2half2(f2h(0.f), f2h(0.f));
        }
    } else {
        const __half* wrow = tail ? a.shared_gate : (a.router + (size_t)e * a.H);
#pragma unroll
        for (int kb = 0; kb < 16; ++kb)
            wreg[kb] = (wvalid && kb < nblk) ? *reinterpret_cast<const uint4*>(wrow + kb * 256 + lane * 8) : make_uint4(0, 0, 0, 0);
    }
    const int ngroups = (a.M + 7) >> 3;
    auto stage = [&](int rg, int b) {
        __half* dst = reinterpret_cast<__half*>(smem) + (size_t)b * 8 * a.H;
        const int mr = min(8, a.M - rg * 8);
        for (int i = tid; i < mr * (a.H >> 3); i += 256) cp_async16(dst + (size_t)i * 8, a.h + (size_t)rg * 8 * a.ldh + (size_t)(i / (a.H >> 3)) * a.ldh + (size_t)(i % (a.H >> 3)) * 8);
        cp_async_commit();
    };
    int it = 0;
    pdl_wait();
    pdl_launch_dependents();
    if ((int)blockIdx.y < ngroups) stage(blockIdx.y, 0);
    for (int rg = blockIdx.y; rg < ngroups; rg += gridDim.y, ++it) {
        const int b = it & 1;
        if (rg + (int)gridDim.y < ngroups) { stage(rg + gridDim.y, b ^ 1); cp_async_wait<1>(); } else cp_async_wait<0>();
        __syncthreads();
        const __half* ps = reinterpret_cast<const __half*>(smem) + (size_t)b * 8 * a.H;
        const int m0 = rg * 8, mr = min(8, a.M - m0);
        if (wvalid) {
            for (int c = 0; c < mr; ++c) {
                const __half* xrow = ps + (size_t)c * a.H;
                float acc = 0.f;
#pragma unroll
                for (int kb = 0; kb < 16; ++kb) {
                    if (kb < nblk) {
                        const uint4 xv = *reinterpret_cast<const uint4*>(xrow + kb * 256 + lane * 8);
                        const __half* xh = reinterpret_cast<const __half*>(&xv);
                        if constexpr (Q8) {
                            float sum = 0.f, accum = 0.f;
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const float xf = h2f(xh[i]);
                                const unsigned q = ((i < 4 ? qreg[kb].x : qreg[kb].y) >> (8 * (i & 3))) & 0xffu;
                                sum = __fadd_rn(sum, xf);
                                accum = fmaf(xf, (float)q, accum);
                            }
                            const float2 sb = __half22float2(sbreg[kb]);
                            acc = __fadd_rn(acc, __fadd_rn(__fmul_rn(sb.x, accum), __fmul_rn(sum, sb.y)));
                        } else {
                            const __half* wh = reinterpret_cast<const __half*>(&wreg[kb]);
#pragma unroll
                            for (int i = 0; i < 8; ++i) acc = fmaf(h2f(xh[i]), h2f(wh[i]), acc);
                        }
                    }
                }
                const float d = warp_sum(acc);
                if (lane == 0) { if (tail) a.sgl[m0 + c] = f2h(d); else a.logits[(size_t)(m0 + c) * a.E + e] = f2h(d); }
            }
        }
        __syncthreads();                       // the buffer is refilled by the next iteration's stage()
    }
}
// The fp16 router for H <= 2048.  Bound by instruction issue: with one expert per warp and halves in registers and shared
// memory every multiply-add came with two conversions (131 us at 512 rows).  Here a warp keeps TWO router rows as f32
// registers, the rows of a group are converted once per CTA, and two rows run side by side: four independent chains of
// the same multiply-adds in the same order.  gr: rows of a group (fewer for short calls, so that more CTAs share the work).
template <int NB>
__global__ void __launch_bounds__(256, 1) k_router_rows2(RouterArgs a, int gr) {
    extern __shared__ __align__(16) unsigned char smem[];                   // [2][gr][H] halves, [gr][NB][2][128] f32
    constexpr int H = NB * 256;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    __half* raw = reinterpret_cast<__half*>(smem);
    float* xf = reinterpret_cast<float*>(smem + (size_t)2 * gr * H * 2);
    const bool tail = (blockIdx.x == gridDim.x - 1);                        // the shared gate: warp w takes row w of a group
    const int e0 = blockIdx.x * 16 + warp * 2;
    float w[2][NB * 8];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const bool ok = tail ? j == 0 : e0 + j < a.E;
        const __half* wrow = tail ? a.shared_gate : a.router + (size_t)(e0 + j) * H;
#pragma unroll
        for (int kb = 0; kb < NB; ++kb) {
            const uint4 v = ok ? *reinterpret_cast<const uint4*>(wrow + kb * 256 + lane * 8) : make_uint4(0, 0, 0, 0);
            const __half* vh = reinterpret_cast<const __half*>(&v);
#pragma unroll
            for (int i = 0; i < 8; ++i) w[j][kb * 8 + i] = h2f(vh[i]);
        }
    }
    const int ngroups = (a.M + gr - 1) / gr;
    auto stage = [&](int rg, int b) {
        const int mr = min(gr, a.M - rg * gr);
        for (int i = tid; i < mr * (H / 8); i += 256)
            cp_async16(raw + (size_t)b * gr * H + (size_t)i * 8, a.h + ((size_t)rg * gr + i / (H / 8)) * a.ldh + (size_t)(i % (H / 8)) * 8);
        cp_async_commit();
    };
    auto dots = [&](const float* x0, const float* x1, float& a00, float& a01, float& a10, float& a11) {
        a00 = 0.f; a01 = 0.f; a10 = 0.f; a11 = 0.f;                         // aRE: row R, expert E
#pragma unroll
        for (int kb = 0; kb < NB; ++kb) {
            float p[8], q[8];
            *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(x0 + kb * 256 + lane * 4);
            *reinterpret_cast<float4*>(p + 4) = *reinterpret_cast<const float4*>(x0 + kb * 256 + 128 + lane * 4);
            *reinterpret_cast<float4*>(q) = *reinterpret_cast<const float4*>(x1 + kb * 256 + lane * 4);
            *reinterpret_cast<float4*>(q + 4) = *reinterpret_cast<const float4*>(x1 + kb * 256 + 128 + lane * 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                a00 = fmaf(p[i], w[0][kb * 8 + i], a00); a01 = fmaf(p[i], w[1][kb * 8 + i], a01);
                a10 = fmaf(q[i], w[0][kb * 8 + i], a10); a11 = fmaf(q[i], w[1][kb * 8 + i], a11);
            }
        }
    };
    int it = 0;
    pdl_wait();
    pdl_launch_dependents();
    if ((int)blockIdx.y < ngroups) stage(blockIdx.y, 0);
    for (int rg = blockIdx.y; rg < ngroups; rg += gridDim.y, ++it) {
        const int b = it & 1;
        if (rg + (int)gridDim.y < ngroups) { stage(rg + gridDim.y, b ^ 1); cp_async_wait<1>(); } else cp_async_wait<0>();
        __syncthreads();
        const int m0 = rg * gr, mr = min(gr, a.M - m0);
        for (int i = tid; i < mr * (H / 8); i += 256) {                     // 8 inputs: 4 into each plane of their 256-wide block
            const uint4 v = *reinterpret_cast<const uint4*>(raw + (size_t)b * gr * H + (size_t)i * 8);
            const __half2* h = reinterpret_cast<const __half2*>(&v);
            const float2 f0 = __half22float2(h[0]), f1 = __half22float2(h[1]), f2 = __half22float2(h[2]), f3 = __half22float2(h[3]);
            float* d = xf + (size_t)(i >> 5) * 256 + (i & 31) * 4;
            *reinterpret_cast<float4*>(d) = make_float4(f0.x, f0.y, f1.x, f1.y);
            *reinterpret_cast<float4*>(d + 128) = make_float4(f2.x, f2.y, f3.x, f3.y);
        }
        __syncthreads();
        if (tail) {
            if (warp < mr) {
                float d, x, y, z;
                dots(xf + (size_t)warp * H, xf + (size_t)warp * H, d, x, y, z);
                d = warp_sum(d);
                if (lane == 0) a.sgl[m0 + warp] = f2h(d);
            }
        } else if (e0 < a.E) {
            for (int c = 0; c < mr; c += 2) {
                const int c1 = min(c + 1, mr - 1);
                float a00, a01, a10, a11;
                dots(xf + (size_t)c * H, xf + (size_t)c1 * H, a00, a01, a10, a11);
                const float s = warp_sum4(a00, a01, a10, a11, lane);
                const int row = m0 + c + (lane >> 4), e = e0 + ((lane >> 3) & 1);
                if ((lane & 7) == 0 && row < m0 + mr && e < a.E) a.logits[(size_t)row * a.E + e] = f2h(s);
            }
        }
    }
}
template <int NB>
static void launch_router_rows2(const RouterArgs& a, cudaStream_t st, bool pdl) {
    const int gx = (a.E + 15) / 16 + 1, want = sm_count() / gx > 0 ? sm_count() / gx : 1;
    int gr = 2; while (gr < 8 && gr * want < a.M) gr *= 2;
    const int ngroups = (a.M + gr - 1) / gr, gy = ngroups < want ? ngroups : want;
    const size_t smem = (size_t)gr * NB * 256 * 8;
    static bool configured = false;
    if (!configured) { cudaFuncSetAttribute(k_router_rows2<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * NB * 256 * 8); configured = true; }
    profile_launch("k_router_rows", st, [&] { return launch_pdl(pdl, k_router_rows2<NB>, dim3((unsigned)gx, (unsigned)gy), 256, smem, st, a, gr); });
}
// grid (ceil(M / 8)), 256 threads: one warp per row.  Expert-parallel: grid (M), one row per CTA.
__global__ void __launch_bounds__(256) k_route_rows(RouterArgs a) {
    __shared__ float s_route[8][512 + 32];
    __shared__ int s_wact[8];
    __shared__ int s_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_wait();
    pdl_launch_dependents();
    if (a.epd.sig.world > 0) {
        // expert-parallel (grid = M, one row per CTA): warp 0 routes the row, then warp w stores the normed row and its
        // routing indices into rank w's gather buffers over peer memory; the CTA that finishes last raises this rank's
        // dispatch flag at every rank.  The pair lists are built from the gathered indices by k_ep_lists.
        const EpSignal& sg = a.epd.sig;
        const int m = blockIdx.x;
        if (warp == 0) route_row_warp(a.logits + (size_t)m * a.E, a.E, a.topk, a.inds + m * a.topk, a.scores + m * a.topk, s_route[0], lane);
        __syncthreads();
        for (int d = warp; d < sg.world; d += 8) {
            if (!a.ep_rows_sent) {
                const uint4* src = reinterpret_cast<const uint4*>(a.p + (size_t)m * a.H);
                uint4* dst = reinterpret_cast<uint4*>(a.epd.pbuf[d] + ((size_t)sg.rank * a.M + m) * a.H);
                for (int i = lane; i < a.H / 8; i += 32) dst[i] = __ldcg(src + i);
            }
            int* di = a.epd.ibuf[d] + ((size_t)sg.rank * a.M + m) * a.topk;
            if (lane < a.topk) di[lane] = a.inds[m * a.topk + lane];
        }
        __threadfence_system();
        __syncthreads();
        if (tid == 0) { const unsigned ticket = atomicAdd(a.counter, 1u); s_last = (ticket == gridDim.x - 1) ? 1 : 0; }
        __syncthreads();
        if (!s_last) return;
        __threadfence_system();
        if (tid == 0) *a.counter = 0u;
        if (tid < sg.world) st_release_sys(sg.flags[tid] + sg.rank, ep_seq(sg.ctr, sg.layer, 0));
        return;
    }
    const int m = blockIdx.x * 8 + warp;
    if (m < a.M) {
        route_row_warp(a.logits + (size_t)m * a.E, a.E, a.topk, a.inds + m * a.topk, a.scores + m * a.topk, s_route[warp], lane);
        // the row's pairs to its experts' places.  (Counted, scanned and placed by the last CTA, the 8192 pairs of 1024 rows were half of
        // 18.6 us by events; now 11.)
        if (lane < a.topk) {
            const int ex = a.inds[m * a.topk + lane];                         // (written by this lane)
            a.lists.pairs[(size_t)ex * a.lists.cap + atomicAdd(a.lists.counts + ex, 1)] = m * a.topk + lane;
        }
    }
    __threadfence();
    __syncthreads();
    if (gridDim.x > 1) {
        if (tid == 0) { const unsigned ticket = atomicAdd(a.counter, 1u); s_last = (ticket == gridDim.x - 1) ? 1 : 0; }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        if (tid == 0) *a.counter = 0u;
    }
    // ---- the experts that have pairs as slots, in ascending order (thread = expert)
    const int cnt = tid < a.E ? __ldcg(a.lists.counts + tid) : 0;
    const unsigned have = __ballot_sync(0xffffffffu, cnt > 0);
    if (lane == 0) s_wact[warp] = __popc(have);
    __syncthreads();
    int slot = __popc(have & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) slot += s_wact[w];
    if (cnt > 0) { a.lists.slot_expert[slot] = tid; a.lists.slot_off[slot] = tid * a.lists.cap; a.lists.slot_cnt[slot] = cnt; a.lists.counts[tid] = 0; }
    if (tid == 255) *a.lists.n_active = slot + (cnt > 0 ? 1 : 0);
}
// Prefill mode: the fp16 router logits as a small tensor-core GEMM (mma.sync m16n8k16, f32 accumulators): a CTA of 4 warps
// computes 32 rows x 32 experts, K in chunks of 128 through three cp.async stages (16-byte pieces swizzled by the row).
// Bound by latency: 64 x 64 tiles left 12 CTAs at 129 rows and 64 at 1024, with one chunk of 64 in flight and the
// shared-gate rows of a tile in one CTA.
// Not the bit pattern of the strict router (the f32 sums run in MMA order), but a row's logits depend on that row only
// and K is walked in a fixed order, so they do not depend on how a prompt is cut into calls.  The shared-gate logit is a
// plain warp dot (the strict order) done by the CTAs of the first expert tile.
__device__ __forceinline__ void rt_ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(smem_u32(p)));
}
constexpr int RT_K = 128, RT_T = 32, RT_ST = 3;               // inputs per chunk, rows / experts per CTA, stages
__device__ __forceinline__ __half* rt_at(__half* base, int row, int chunk) { return base + row * RT_K + ((chunk ^ (row & 7)) << 3); }   // rows of 128 halves
__global__ void __launch_bounds__(128) k_router_mma(RouterArgs a) {
    __shared__ __align__(128) __half sm[RT_ST][2][RT_T * RT_K];               // 48 KB: [stage][rows | experts]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wr = warp >> 1, wc = warp & 1;
    const int m0 = blockIdx.x * RT_T, e0 = blockIdx.y * RT_T;
    const int rows = min(RT_T, a.M - m0), cols = min(RT_T, a.E - e0);
    auto stage = [&](int kc) {
        __half *As = sm[kc % RT_ST][0], *Bs = sm[kc % RT_ST][1];
        for (int i = tid; i < RT_T * (RT_K / 8); i += 128) {
            const int r = i / (RT_K / 8), c = i % (RT_K / 8);
            if (r < rows) cp_async16(rt_at(As, r, c), a.h + (size_t)(m0 + r) * a.ldh + kc * RT_K + c * 8);
            else *reinterpret_cast<uint4*>(rt_at(As, r, c)) = make_uint4(0, 0, 0, 0);
            if (r < cols) cp_async16(rt_at(Bs, r, c), a.router + (size_t)(e0 + r) * a.H + kc * RT_K + c * 8);
            else *reinterpret_cast<uint4*>(rt_at(Bs, r, c)) = make_uint4(0, 0, 0, 0);
        }
    };
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    pdl_wait();
    pdl_launch_dependents();
    const int nk = a.H / RT_K;
    for (int kc = 0; kc < RT_ST - 1; ++kc) { if (kc < nk) stage(kc); cp_async_commit(); }
    for (int kc = 0; kc < nk; ++kc) {
        cp_async_wait<RT_ST - 2>();
        __syncthreads();                       // chunk kc is here, and everyone is done with the chunk whose stage is refilled now
        if (kc + RT_ST - 1 < nk) stage(kc + RT_ST - 1);
        cp_async_commit();
        __half *As = sm[kc % RT_ST][0], *Bs = sm[kc % RT_ST][1];
#pragma unroll
        for (int ks = 0; ks < RT_K / 16; ++ks) {
            uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
            const int mi = lane >> 3;
            rt_ldsm_x4(a0, a1, a2, a3, rt_at(As, wr * 16 + (lane & 7) + (mi & 1) * 8, ks * 2 + (lane >> 4)));
            rt_ldsm_x4(b0, b1, b2, b3, rt_at(Bs, wc * 16 + (mi >> 1) * 8 + (lane & 7), ks * 2 + (mi & 1)));
            mma_f16(acc[0], a0, a1, a2, a3, b0, b1);
            mma_f16(acc[1], a0, a1, a2, a3, b2, b3);
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = wr * 16 + (lane >> 2) + 8 * (i >> 1), c = wc * 16 + n * 8 + 2 * (lane & 3) + (i & 1);
            if (r < rows && c < cols) a.logits[(size_t)(m0 + r) * a.E + e0 + c] = f2h(acc[n][i]);
        }
    // shared-gate logits, the rows dealt to the expert tiles: lane l owns 8 inputs of every 256-wide block
    for (int r = blockIdx.y + warp * gridDim.y; r < rows; r += 4 * gridDim.y) {
        const __half* xrow = a.h + (size_t)(m0 + r) * a.ldh;
        float s = 0.f;
#pragma unroll 8
        for (int kb = 0; kb < (a.H >> 8); ++kb) {
            const uint4 xv = *reinterpret_cast<const uint4*>(xrow + kb * 256 + lane * 8);
            const uint4 wv = *reinterpret_cast<const uint4*>(a.shared_gate + kb * 256 + lane * 8);
            const __half* xh = reinterpret_cast<const __half*>(&xv);
            const __half* wh = reinterpret_cast<const __half*>(&wv);
#pragma unroll
            for (int i = 0; i < 8; ++i) s = fmaf(h2f(xh[i]), h2f(wh[i]), s);
        }
        s = warp_sum(s);
        if (lane == 0) a.sgl[m0 + r] = f2h(s);
    }
}
// prefill mode, fp16 router: logits on the tensor cores, then the routing / pair-list kernel.  false: not covered.
bool launch_router_mma(const RouterArgs& a, cudaStream_t st, bool pdl) {
    if (a.E > 256 || a.H % 256 || a.norm_w || a.router_q8 || a.sg_q8) return false;
    const dim3 grid((unsigned)((a.M + RT_T - 1) / RT_T), (unsigned)((a.E + RT_T - 1) / RT_T));
    profile_launch("k_router_mma", st, [&] { return launch_pdl(pdl, k_router_mma, grid, 128, 0, st, a); });
    profile_launch("k_route_rows", st, [&] { return launch_pdl(pdl, k_route_rows, dim3((unsigned)(a.epd.sig.world > 0 ? a.M : (a.M + 7) / 8)), 256, 0, st, a); });
    return true;
}

// (nothing to launch where the expert kernels route for themselves)
static void launch_route_rows(const RouterArgs& a, cudaStream_t st, bool pdl) {
    if (a.no_route) return;
    const unsigned grid = (unsigned)(a.epd.sig.world > 0 ? a.M : (a.M + 7) / 8);
    profile_launch("k_route_rows", st, [&] { return launch_pdl(pdl, k_route_rows, dim3(grid), 256, 0, st, a); });
}
// rows already normed in a.h (ldh); E <= 256.  Returns false when the shape is not covered.
bool launch_router_rows(const RouterArgs& a, cudaStream_t st, bool pdl) {
    if (a.E > 256 || a.H % 256 || a.H > 4096 || a.norm_w) return false;
    const size_t smem = (size_t)2 * 8 * a.H * 2;
    static bool configured = false;
    if (!configured) {
        cudaFuncSetAttribute(k_router_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
        cudaFuncSetAttribute(k_router_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
        configured = true;
    }
    const int ngroups = (a.M + 7) / 8;
    const int gx = (a.E + 7) / 8 + 1;
    int gy = (2 * sm_count() + gx - 1) / gx; if (gy > ngroups) gy = ngroups; if (gy < 1) gy = 1;
    const dim3 grid((unsigned)gx, (unsigned)gy);
    const bool q8 = a.router_q8 != nullptr;
    if (!q8 && a.H == 512) launch_router_rows2<2>(a, st, pdl);
    else if (!q8 && a.H == 1024) launch_router_rows2<4>(a, st, pdl);
    else if (!q8 && a.H == 2048) launch_router_rows2<8>(a, st, pdl);
    else profile_launch("k_router_rows", st, [&] {
        return launch_pdl(pdl, q8 ? k_router_rows<true> : k_router_rows<false>, grid, 256, smem, st, a);
    });
    launch_route_rows(a, st, pdl);
    return true;
}

// ================================================================================ combine
// grid (M, ceil(H / 2048)), 256 threads, 8 outputs a thread:
// out/resid[m] (+)= sum_k fp16(d[m*topk + k] * score[m,k]) (ascending k) + sigmoid(sgl[m]) * shared[m]
// (swift/Sources/QwispCore/SeedlessFusedVerify.swift:462-484, SeedlessMetalForward.swift:1024-1028)
// Bound by latency: with one output and 2-byte loads per thread and step the eight steps of a thread were 8 dependent
// round trips; all 16-byte loads of a thread are now in flight at once.
// NORM (grid (M), H / 8 threads): the CTA has the whole residual row, and leaves it normed for the next layer's in-projection as
// well, prepared (the arithmetic of k_rows_prep<PRO_RMSNORM>) or, without sxq, as plain rows; a launch less per layer.
template <bool NORM>
__global__ void __launch_bounds__(NORM ? 512 : 256) k_moe_combine(const __half* dbuf, const __half* shared_rows, const __half* scores, const __half* sgl,
                                                                  int H, int topk, __half* resid, __half* out, const __half* nw, float eps, __half* xq, float* sxq) {
    const int m = blockIdx.x, n = (blockIdx.y * 256 + threadIdx.x) * 8;
    uint4 wv = make_uint4(0, 0, 0, 0);
    if (NORM) wv = *reinterpret_cast<const uint4*>(nw + n);
    pdl_wait();
    pdl_launch_dependents();
    if (n >= H) return;
    const uint4 sh = __ldcg(reinterpret_cast<const uint4*>(shared_rows + (size_t)m * H + n));
    uint4 rv = make_uint4(0, 0, 0, 0);
    if (resid) rv = *reinterpret_cast<const uint4*>(resid + (size_t)m * H + n);
    const __half* d0 = dbuf + (size_t)m * topk * H + n;
    __half acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = f2h(0.0f);
#pragma unroll 8
    for (int k = 0; k < topk; ++k) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(d0 + (size_t)k * H));
        const __half sc = scores[m * topk + k];
        const __half* vh = reinterpret_cast<const __half*>(&v);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = hadd_rn(acc[i], hmul_rn(vh[i], sc));
    }
    const __half gate = sigmoid_h(sgl[m]);
    const __half* shh = reinterpret_cast<const __half*>(&sh);
    __half* rh = reinterpret_cast<__half*>(&rv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const __half res = hadd_rn(acc[i], hmul_rn(gate, shh[i]));
        rh[i] = resid ? hadd_rn(rh[i], res) : res;
    }
    *reinterpret_cast<uint4*>((resid ? resid : out) + (size_t)m * H + n) = rv;
    if (NORM) {
        __shared__ float part[16];
        const int ch = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const float ss = warp_sum(sumsq8(rv));
        if (lane == 0) part[ch] = ss;
        __syncthreads();
        float tot = 0.f;
        for (int c = 0; c < (H >> 8); ++c) tot += part[c];
        const float inv = __frsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)H), eps));
        const uint4 o = rms_apply8(rv, wv, inv);
        if (sxq) rows_store(xq + (size_t)m * H, sxq + (size_t)m * (H >> 6), n, o, lane);
        else *reinterpret_cast<uint4*>(xq + (size_t)m * H + n) = o;
    }
}
void launch_moe_combine(const __half* dbuf, const __half* shared_rows, const __half* scores, const __half* sgl, int M, int H, int topk,
                        __half* resid, __half* out, cudaStream_t st, bool pdl, const __half* nw, float eps, __half* xq, float* sxq) {
    profile_launch("k_moe_combine", st, [&] {
        if (xq) return launch_pdl(pdl, k_moe_combine<true>, dim3((unsigned)M), (unsigned)H / 8, 0, st, dbuf, shared_rows, scores, sgl, H, topk, resid, out, nw, eps, xq, sxq);
        return launch_pdl(pdl, k_moe_combine<false>, dim3((unsigned)M, (unsigned)((H + 2047) / 2048)), 256, 0, st, dbuf, shared_rows, scores, sgl, H, topk, resid, out, nw, eps, xq, sxq);
    });
}

}  // namespace sl
