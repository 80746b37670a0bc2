// sampler.cu -- speculative-sampling rows on the device: per verify row a categorical draw by
// Gumbel-max over the (optionally nucleus-truncated) logits, the same draw with the draft token
// excluded, and the accept test coin < p(draft).  Only three int32 per row leave the device.
// Behaviour follows the reference's kernel (swift/Sources/QwispCore/SamplerGPU.swift:39-156):
// counter-based hash noise keyed by (seed, position + row, token), temperature as 1/T (<= 0 means
// greedy with first-index-wins ties, identical to the argmax path), top-p through a 1024-bucket
// histogram of fixed-point softmax weights over the scaled gap (gmax - L)/T.
//
// exp and log are evaluated by the small deterministic routines below (IEEE add / multiply /
// divide only, no fused contraction; ln 2 split in two as by Cody and Waite, then the Taylor series of exp and the
// series of 2 atanh(f / (2 + f)) for log), so the CPU restatement used by the tests reproduces every
// draw and every accept flag bit for bit; their ~1e-7 relative error is irrelevant for sampling.
#include "kernels.h"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace sl {

__device__ __forceinline__ float det_expf(float x) {           // x <= 0
    if (x < -87.0f) return 0.0f;
    const float n = rintf(__fmul_rn(x, 1.44269504f));
    float r = __fsub_rn(x, __fmul_rn(n, 0.693145751953125f));
    r = __fsub_rn(r, __fmul_rn(n, 1.42860682e-6f));
    float p = 1.0f / 720.0f;
    p = __fadd_rn(__fmul_rn(p, r), 1.0f / 120.0f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f / 24.0f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f / 6.0f);
    p = __fadd_rn(__fmul_rn(p, r), 0.5f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f);
    return __fmul_rn(p, __int_as_float(((int)n + 127) << 23));
}
__device__ __forceinline__ float det_logf(float a) {           // a > 0, normal
    int bits = __float_as_int(a);
    int e = ((bits >> 23) & 255) - 127;
    float m = __int_as_float((bits & 0x007fffff) | 0x3f800000);
    if (m > 1.41421354f) { m = __fmul_rn(m, 0.5f); e += 1; }
    const float f = __fsub_rn(m, 1.0f);
    const float s = __fdiv_rn(f, __fadd_rn(2.0f, f));
    const float z = __fmul_rn(s, s);
    float p = 1.0f / 9.0f;
    p = __fadd_rn(__fmul_rn(p, z), 1.0f / 7.0f);
    p = __fadd_rn(__fmul_rn(p, z), 0.2f);
    p = __fadd_rn(__fmul_rn(p, z), 1.0f / 3.0f);
    p = __fadd_rn(__fmul_rn(p, z), 1.0f);
    const float lm = __fmul_rn(__fmul_rn(2.0f, s), p);
    const float fe = (float)e;
    return __fadd_rn(__fmul_rn(fe, 0.693145751953125f), __fadd_rn(lm, __fmul_rn(fe, 1.42860682e-6f)));
}
__device__ __forceinline__ uint32_t qhash(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t h = a * 0x9E3779B1u + 0x165667B1u;
    h ^= b + 0x9E3779B9u + (h << 6) + (h >> 2);
    h ^= c + 0x9E3779B9u + (h << 6) + (h >> 2);
    h ^= h >> 15; h *= 0x2C1B3C6Du; h ^= h >> 12; h *= 0x297A2D39u; h ^= h >> 15;
    return h;
}
__device__ __forceinline__ float u01(uint32_t h) { return fmaxf(__fmul_rn((float)(h >> 8), 1.0f / 16777216.0f), 1e-7f); }

// Eight CTAs, a cluster, share a row: one CTA that walked the vocabulary four times, with a histogram scanned by one thread,
// took 216 us for 4 rows of 151936 (by events), this form 40.  The adjusted logits are read once and stay in shared memory (up to
// 430 thousand), maxima, histograms, sums and candidates meet through distributed shared memory.  The f32 sum of the
// weights keeps its order, that of 1024 threads which each add every 1024th weight, then a butterfly in every warp, then the
// warps in ascending order: a CTA has 128 of those threads' weights, formed by all its threads and added by 128 of them.
constexpr int SAMP_T = 1024;          // threads of a CTA, and strands of the sum
constexpr int SAMP_CL = 8;            // CTAs of a row
constexpr int SAMP_S = SAMP_T / SAMP_CL, SAMP_SUB = SAMP_T / SAMP_S;      // strands of a CTA, threads of a strand
constexpr int SAMP_CAP = 420;         // weights of a strand that fit shared memory
constexpr int SAMP_BINS = 1024;
constexpr float SAMP_SPAN = 40.0f;
static_assert(SAMP_BINS == SAMP_T, "a thread per bin");

__device__ __forceinline__ bool better_si(float s, int i, float bs, int bi) { return s > bs || (s == bs && i < bi); }
struct SampBest { float fs, rs; int fi, ri; };               // best candidate, and best one that is not the draft token
__device__ __forceinline__ void samp_merge(SampBest& a, const SampBest& b) {
    if (better_si(b.fs, b.fi, a.fs, a.fi)) { a.fs = b.fs; a.fi = b.fi; }
    if (better_si(b.rs, b.ri, a.rs, a.ri)) { a.rs = b.rs; a.ri = b.ri; }
}

// grid (SAMP_CL, M) in clusters of SAMP_CL; cap: floats of a strand in shared memory.
// adj: optional [V] f32 penalties / bias added to every row's logits before anything else looks at them
// (the reference's LADJ(v) = float(row[v]) + logitAdj[v], SamplerGPU.swift:41,69); nullptr = none.
__global__ void __launch_bounds__(SAMP_T, 1) k_sample_rows(const __half* logits, const float* adj, const int* draft, int* samp_full, int* samp_resid, int* accept,
                                                           float invT, int V, uint32_t seed_lo, uint32_t seed_hi, uint32_t base_pos, float top_p, int cap) {
    extern __shared__ float buf[];                            // [cap][SAMP_S]: adjusted logits, in the end weights
    __shared__ unsigned hist[SAMP_BINS], s_wsum[32];
    __shared__ float s_mx[SAMP_CL], s_part[32];               // s_part: warp sums of the whole row (in the first CTA)
    __shared__ SampBest s_best[32], s_cta[SAMP_CL];           // s_cta: every CTA's candidates (in the first CTA)
    __shared__ int s_bin;
    const cg::cluster_group cl = cg::this_cluster();
    cl.barrier_arrive();                                      // (waited for before the first look at another CTA's shared memory)
    const int rank = blockIdx.x, m = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int strand = tid & (SAMP_S - 1), sub = tid / SAMP_S, v0 = rank * SAMP_S + strand;
    const int n = (V + SAMP_T - 1) / SAMP_T;                  // weights of a strand: tokens v0 + SAMP_T * i
    const bool cached = n <= cap;
    const __half* row = logits + (size_t)m * V;
    const int d = draft ? draft[m] : -1;
    const bool greedy = invT <= 0.0f, do_top_p = !greedy && top_p < 0.999f;
    const uint32_t salt = seed_hi ^ (base_pos + (uint32_t)m);
    auto ladj = [&](int v) -> float { const float L = h2f(row[v]); return adj ? __fadd_rn(L, adj[v]) : L; };
    auto logit = [&](int i) -> float { return cached ? buf[i * SAMP_S + strand] : ladj(v0 + i * SAMP_T); };
    // maximum (adjusted) logit
    float mx = -INFINITY;
#pragma unroll 4
    for (int i = sub; i < n; i += SAMP_SUB) {
        const int v = v0 + i * SAMP_T;
        const float L = v < V ? ladj(v) : -INFINITY;
        mx = fmaxf(mx, L);
        if (cached) buf[i * SAMP_S + strand] = L;
    }
    mx = warp_max(mx);
    if (lane == 0) s_part[warp] = mx;
    hist[tid] = 0u;
    if (tid == 0) s_bin = SAMP_BINS - 1;
    __syncthreads();
    cl.barrier_wait();
    if (warp == 0) {
        mx = warp_max(s_part[lane]);
        if (lane < SAMP_CL) *cl.map_shared_rank(&s_mx[rank], lane) = mx;
    }
    cl.sync();
    float gmax = -INFINITY;
#pragma unroll
    for (int c = 0; c < SAMP_CL; ++c) gmax = fmaxf(gmax, s_mx[c]);
    auto weight = [&](float L) -> float { return det_expf(-__fmul_rn(__fsub_rn(gmax, L), invT)); };
    float lthr = -INFINITY;
    if (do_top_p) {
        const float bin_w = SAMP_SPAN / (float)SAMP_BINS;
        for (int i = sub; i < n; i += SAMP_SUB) {
            if (v0 + i * SAMP_T >= V) continue;
            const float g = __fmul_rn(__fsub_rn(gmax, logit(i)), invT);
            const unsigned add = (unsigned)__fmul_rn(det_expf(-g), 8192.0f);
            if (add == 0u) continue;                          // (nine tenths of a vocabulary)
            const float q = __fdiv_rn(g, bin_w);
            atomicAdd(&hist[(q >= (float)(SAMP_BINS - 1)) ? (unsigned)(SAMP_BINS - 1) : (unsigned)q], add);
        }
        cl.sync();                                            // the histograms are complete
        unsigned h = 0u;
#pragma unroll
        for (int c = 0; c < SAMP_CL; ++c) h += *cl.map_shared_rank(&hist[tid], c);
        unsigned cum = h;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) { const unsigned o = __shfl_up_sync(0xffffffffu, cum, s); if (lane >= s) cum += o; }
        if (lane == 31) s_wsum[warp] = cum;
        __syncthreads();
        unsigned total = 0u, below = 0u;
#pragma unroll
        for (int w = 0; w < 32; ++w) { const unsigned o = s_wsum[w]; total += o; if (w < warp) below += o; }
        cum += below;
        const unsigned target = (unsigned)__fmul_rn(top_p, (float)total);
        // the first bin that reaches the target.  (Counts wrap from 2^32 on, 524288 tokens as likely as the likeliest: then the sums
        // may pass the target several times)
        if (cum >= target && (tid == 0 || cum - h < target)) atomicMin(&s_bin, tid);
        __syncthreads();
        lthr = __fsub_rn(gmax, __fdiv_rn(__fmul_rn((float)(s_bin + 1), bin_w), invT));
    }
    // Gumbel-max over the nucleus: full, and excluding the draft token
    SampBest best{-INFINITY, -INFINITY, 0x7fffffff, 0x7fffffff};
    for (int i = sub; i < n; i += SAMP_SUB) {
        const int v = v0 + i * SAMP_T;
        if (v >= V) continue;
        const float L = logit(i);
        if (do_top_p && L < lthr) continue;
        float score = L;
        if (!greedy) {
            const float u = u01(qhash(seed_lo, salt, (uint32_t)v));
            score = __fsub_rn(__fmul_rn(L, invT), det_logf(-det_logf(u)));
        }
        samp_merge(best, SampBest{score, v != d ? score : -INFINITY, v, v != d ? v : 0x7fffffff});
    }
    auto reduce = [&](SampBest& b) {
#pragma unroll
        for (int s = 16; s >= 1; s >>= 1) {
            SampBest o;
            o.fs = __shfl_xor_sync(0xffffffffu, b.fs, s); o.fi = __shfl_xor_sync(0xffffffffu, b.fi, s);
            o.rs = __shfl_xor_sync(0xffffffffu, b.rs, s); o.ri = __shfl_xor_sync(0xffffffffu, b.ri, s);
            samp_merge(b, o);
        }
    };
    reduce(best);
    if (lane == 0) s_best[warp] = best;
    __syncthreads();
    if (warp == 0) {
        best = s_best[lane];
        reduce(best);
        if (lane == 0) *cl.map_shared_rank(&s_cta[rank], 0) = best;
    }
    // probability of the draft token: its weight over the sum of the nucleus's
    const float Ld = d >= 0 ? ladj(d) : 0.f;
    const bool want_sum = d >= 0 && !greedy && (!do_top_p || Ld >= lthr);      // (the same in the whole cluster)
    if (want_sum) {
        float z = 0.f;
        for (int c0 = 0; c0 < n; c0 += cap) {
            const int c1 = min(n, c0 + cap);
            if (c0 > 0) __syncthreads();                      // the weights before are added
            for (int i = c0 + sub; i < c1; i += SAMP_SUB) {
                float w = 0.f;                                // (adding +0 changes no sum)
                if (v0 + i * SAMP_T < V) { const float L = logit(i); if (!do_top_p || L >= lthr) w = weight(L); }
                buf[(i - c0) * SAMP_S + strand] = w;
            }
            __syncthreads();
            if (sub == 0) {
#pragma unroll 8
                for (int i = 0; i < c1 - c0; ++i) z = __fadd_rn(z, buf[i * SAMP_S + strand]);
            }
        }
        if (sub == 0) {
#pragma unroll
            for (int s = 16; s >= 1; s >>= 1) z = __fadd_rn(z, __shfl_xor_sync(0xffffffffu, z, s));
            if (lane == 0) *cl.map_shared_rank(&s_part[rank * (SAMP_S / 32) + warp], 0) = z;
        }
    }
    cl.sync();                                                // (the last look at another CTA's shared memory is behind it)
    if (rank == 0 && tid == 0) {
        best = s_cta[0];
        for (int c = 1; c < SAMP_CL; ++c) samp_merge(best, s_cta[c]);
        samp_full[m] = best.fi;
        samp_resid[m] = (d < 0) ? best.fi : best.ri;
        float p_draft = 0.f;
        if (d >= 0 && greedy) p_draft = (d == best.fi) ? 1.0f : 0.0f;
        if (want_sum) {
            float sum = 0.f;
            for (int w = 0; w < SAMP_T / 32; ++w) sum = __fadd_rn(sum, s_part[w]);
            p_draft = __fdiv_rn(det_expf(__fmul_rn(__fsub_rn(Ld, gmax), invT)), sum);
        }
        const float coin = u01(qhash(seed_lo, salt, 0x9999AAAAu));
        accept[m] = (coin < p_draft) ? 1 : 0;
    }
}
void launch_sample_rows(const __half* logits, const float* adj, const int* draft, int* samp_full, int* samp_resid, int* accept, int M, int V,
                        float invT, float top_p, uint32_t seed_lo, uint32_t seed_hi, uint32_t base_pos, cudaStream_t st) {
    const int n = (V + SAMP_T - 1) / SAMP_T, cap = n < SAMP_CAP ? n : SAMP_CAP;
    static bool configured = false;
    if (!configured) { cudaFuncSetAttribute(k_sample_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMP_CAP * SAMP_S * (int)sizeof(float)); configured = true; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(SAMP_CL, (unsigned)M); cfg.blockDim = dim3(SAMP_T); cfg.dynamicSmemBytes = (size_t)cap * SAMP_S * sizeof(float); cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SAMP_CL; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    profile_launch("k_sample_rows", st, [&] {
        return (int)cudaLaunchKernelEx(&cfg, k_sample_rows, logits, adj, draft, samp_full, samp_resid, accept, invT, V, seed_lo, seed_hi, base_pos, top_p, cap);
    });
}

}  // namespace sl
