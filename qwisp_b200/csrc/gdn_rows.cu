// gdn_rows.cu -- the gated delta net of calls with more than one row (prompt chunks, verify rows, batched decode), in two
// kernels:
//   k_gdn_prep   everything that does not depend on the state, for all rows side by side: conv + SiLU of every channel, the
//                q/k norms and scales, decay and beta, the conv history the call leaves.
//   k_gdn_scan   the recurrence alone, the rows of a segment in sequence.
// Every value is formed by the functions of mixer_math.cuh, or by the same operations in the same order, so outputs and
// state are those of k_gdn_core (kernels.cu) bit for bit.
// (conv: swift/Sources/QwispCore/SeedlessFusedVerify.swift:634-663; prep: :839-938; recurrence: GatedDelta.swift:63-124)
#include "kernels.h"
#include "mixer_math.cuh"

namespace sl {

// ---- scratch between the two kernels (records of consecutive rows are contiguous: the scan fetches them with bulk copies)
//   qk  [Hk][M][256] f32   k then q of one key head, each 128 values in the paired order below
//   vg  [Hv * 4][M] records of 144 bytes: 32 f32 of v (one quarter of a value head), decay twice, beta, 4 bytes unused
// Paired order: dk = 4 * leaf + e is stored at (e / 2) * 64 + (leaf % 16) * 4 + (e % 2) * 2 + leaf / 16: the values of leaves
// l and l + 16 form the two halves of one f32x2 operand, and eight lanes that each read 16 bytes read 128 in a row.
constexpr int GS_REC = 144;
__device__ __forceinline__ int gs_paired(int dk) { const int leaf = dk >> 2, e = dk & 3; return (e >> 1) * 64 + (leaf & 15) * 4 + (e & 1) * 2 + (leaf >> 4); }

// The warp's sums of N values at once (N a power of two): the butterfly of warp_sum() on each, the same additions, but a lane
// keeps only half of the values at every level -- N + 5 - log2 N shuffles instead of 5 N.  Lane l gets value l / (32 / N).
template <int N>
__device__ __forceinline__ float warp_sums(float v[N], int lane) {
    int off = 16;
#pragma unroll
    for (int n = N / 2; n >= 1; n /= 2, off /= 2) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) v[i] = __fadd_rn(up ? v[i + n] : v[i], __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + n], off));
    }
    for (; off >= 1; off /= 2) v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], off));
    return v[0];
}
// grid (Hk + Hv, ceil(M / R)), 128 threads: CTAs [0, Hk) own a key head's q and k channels, CTAs [Hk, Hk + Hv) a value
// head's v channels and gates, for R rows.  R = 8 (one segment): the four conv taps of consecutive rows overlap, so a
// thread loads 11 values per channel for its 8 rows, all of them before it uses the first.  R = 2: of fewer rows than fill the
// device that way.  R = 1: rows of several segments.
// Bound by instruction issue (72 % of the slots at 967 rows, memory at a quarter): with a butterfly per value and the two inverse
// norms of a row formed by all 128 threads it took 41 us for 967 rows by events, with neither 27 (129 rows 13.2 -> 10.7).
template <int R>
__global__ void __launch_bounds__(128) k_gdn_prep(GdnArgs a) {
    __shared__ float red_s[2 * R][4], inv_s[2 * R];           // [2 r]: q of row r, [2 r + 1]: k
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * R, nr = min(R, a.M - m0);
    const SegDesc seg = a.segs[a.row_seg[m0]];                // descriptors, history, weights: ahead of the programmatic-launch wait
    const int t0 = m0 - seg.row0;
    const int keyDim = a.Hk * GDN_DK, valDim = a.Hv * GDN_DV, convDim = 2 * keyDim + valDim;
    const int side = a.tab.parity[seg.slot];
    const __half* hist_in = a.tab.conv_hist + (size_t)seg.slot * a.tab.hist_stride_stream + (size_t)side * a.tab.hist_stride_side +
                            (size_t)a.gdn_index * a.tab.hist_stride_layer;
    __half* hist_out = a.tab.conv_hist + (size_t)seg.slot * a.tab.hist_stride_stream + (size_t)(side ^ 1) * a.tab.hist_stride_side +
                       (size_t)a.gdn_index * a.tab.hist_stride_layer;
    // taps of rows m0 .. m0 + R - 1: entries t0 .. t0 + R + 2 of [hist(3) | rows of the segment]
    auto past = [&](int ch, __half x[R + 3]) {
#pragma unroll
        for (int j = 0; j < R + 3; ++j) x[j] = j < CONV_K - 1 && t0 + j < CONV_K - 1 ? hist_in[(size_t)(t0 + j) * convDim + ch] : f2h(0.f);
    };
    const bool inner = t0 >= CONV_K - 1 && nr == R;           // every entry is a row of the call
    auto window = [&](int ch, __half x[R + 3]) {
        const __half* p = a.inproj + ((long)m0 - (CONV_K - 1)) * a.ld + ch;
        if (inner) {
#pragma unroll
            for (int j = 0; j < R + 3; ++j, p += a.ld) x[j] = *p;
        } else {
#pragma unroll
            for (int j = 0; j < R + 3; ++j, p += a.ld) if (t0 + j >= CONV_K - 1 && j < nr + 3) x[j] = *p;
        }
    };
    auto conv = [&](const __half* x, float4 w) { return gdn_conv_silu(h2f(x[0]), h2f(x[1]), h2f(x[2]), h2f(x[3]), w); };
    const int tl = seg.nrows - 1 - t0;                        // the segment's last row, if it is one of this CTA's
    const bool last = tl >= 0 && tl < nr;
    auto leave = [&](int ch, const __half x[R + 3]) {         // the three newest inputs are the next call's history
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r == tl)
                for (int j = 0; j < CONV_K - 1; ++j) hist_out[(size_t)j * convDim + ch] = x[r + 1 + j];
    };
    if ((int)blockIdx.x < a.Hk) {
        const int hk = blockIdx.x, ch_q = hk * GDN_DK + tid, ch_k = keyDim + hk * GDN_DK + tid;
        const float4 wq = *reinterpret_cast<const float4*>(a.conv_w + (size_t)ch_q * 4), wk = *reinterpret_cast<const float4*>(a.conv_w + (size_t)ch_k * 4);
        __half xq[R + 3], xk[R + 3];
        past(ch_q, xq); past(ch_k, xk);
        pdl_wait();
        pdl_launch_dependents();
        window(ch_q, xq); window(ch_k, xk);
        float qc[R], kc[R], sq[2 * R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            qc[r] = conv(xq + r, wq); kc[r] = conv(xk + r, wk);
            sq[2 * r] = qc[r] * qc[r]; sq[2 * r + 1] = kc[r] * kc[r];
        }
        const float sum = warp_sums<2 * R>(sq, lane);
        if (lane % (16 / R) == 0) red_s[lane / (16 / R)][warp] = sum;
        __syncthreads();
        if (tid < 2 * R) inv_s[tid] = gdn_head_inv(red_s[tid][0], red_s[tid][1], red_s[tid][2], red_s[tid][3], a.eps);
        __syncthreads();
        float* rec = a.qk + ((size_t)hk * a.M + m0) * 256 + gs_paired(tid);
#pragma unroll
        for (int r = 0; r < R; ++r, rec += 256) {
            if (r >= nr) break;
            rec[0] = gdn_scale_k(kc[r], inv_s[2 * r + 1]);
            rec[128] = gdn_scale_q(qc[r], inv_s[2 * r]);
        }
        if (last) { leave(ch_q, xq); leave(ch_k, xk); }
    } else {
        const int hv = blockIdx.x - a.Hk, ch_v = 2 * keyDim + hv * GDN_DV + tid;
        const float4 wv = *reinterpret_cast<const float4*>(a.conv_w + (size_t)ch_v * 4);
        const float A_log = a.A_log[hv], dt_bias = a.dt_bias[hv];
        __half xv[R + 3];
        past(ch_v, xv);
        pdl_wait();
        pdl_launch_dependents();
        window(ch_v, xv);
        unsigned char* rec = a.vg + ((size_t)(hv * 4 + warp) * a.M + m0) * GS_REC;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r < nr) *reinterpret_cast<float*>(rec + (size_t)r * GS_REC + lane * 4) = conv(xv + r, wv);
        if (lane < nr) {                                      // every warp makes the gates its quarter's records need
            const __half* gp = a.inproj + (size_t)(m0 + lane) * a.ld + convDim + valDim + hv;
            float g, beta;
            gdn_gate(gp[0], gp[a.Hv], A_log, dt_bias, g, beta);
            *reinterpret_cast<float4*>(rec + (size_t)lane * GS_REC + 128) = make_float4(g, g, beta, 0.f);
        }
        if (last) leave(ch_v, xv);
    }
}

// ---- packed f32 pairs (two independent IEEE operations per instruction)
__device__ __forceinline__ float sum2(f32x2 v) { float lo, hi; asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); return __fadd_rn(lo, hi); }

// (volatile: stays where it is written relative to the shuffles, which share the shared-memory pipe with it)
__device__ __forceinline__ void lds2(const void* p, f32x2& a, f32x2& b) { asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(smem_u32(p)) : "memory"); }

// The recurrence.  A token's update needs kv = S.k over the 128 dk before it can change S, so a row's time is the latency
// of that sum, token after token, as long as the SM keeps up with the operands.  The first form spread a row over a warp
// (4 dk a lane): two butterflies of 5 shuffles each, 0.31 us a token.  Here EIGHT lanes hold a row, and a lane holds 16 dk
// of TWO rows: the butterfly's levels 16 and 8 are adds inside a lane and only levels 4, 2 and 1 are shuffles -- the same
// additions of the same operands, so the same bits -- and the products run as f32x2.  Four lanes a row and one row a lane
// has one level less, but every operand read from shared memory then serves one row instead of two and the shared-memory
// pipe sets the time (0.225 us a token; this form 0.20: a 967-row chunk went from 319 to 197 us, a batch of 64 one-row
// segments from 60 to 48).  The readout's sum is off the chain, see below.
// The loop's code is a limit of its own: eight tokens a turn 196 us for 967 rows, four 187, two 189, three 183 (in chunks of 32 rows;
// 48 rows 179); scalar multiply-adds 188 to 206, the operands' loads moved about no change.
// 32 state rows per CTA (8 per warp), 128 CTAs per stream: one warp per SM sub-partition, which is what the 4096 rows of
// a stream give.  grid (4, Hv, nsegs), 128 threads; k / q / v / gates of CH rows at a time by bulk copies, two buffers.
// STALL: a test's form, in which no operands are ever fetched, so that the wait for them runs out, and soon
template <int CH, bool STALL>
__global__ void __launch_bounds__(128) k_gdn_scan(GdnArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];    // [2][CH][1024] k | q, then [2][CH][144] v | gates
    __shared__ __align__(8) uint64_t bar[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, j = lane & 7;
    const int dvt = blockIdx.x, hv = blockIdx.y;
    const SegDesc seg = a.segs[blockIdx.z];
    const int hk = hv / (a.Hv / a.Hk), valDim = a.Hv * GDN_DV;
    const int side = a.tab.parity[seg.slot];
    const int crow = warp * 8 + (lane >> 3) * 2;              // this lane's first state row inside the CTA's 32
    const size_t base = (size_t)seg.slot * a.tab.state_stride_stream + (size_t)a.gdn_index * a.tab.state_stride_layer + ((size_t)hv * GDN_DV + dvt * 32 + crow) * GDN_DK;
    const float* S_in = a.tab.gdn_state + base + (size_t)side * a.tab.state_stride_side;
    float* S_out = a.tab.gdn_state + base + (size_t)(side ^ 1) * a.tab.state_stride_side;
    const int nchunks = (seg.nrows + CH - 1) / CH;
    auto fetch = [&](int c) {
        if (STALL) return;
        const int b = c & 1, t0 = c * CH, n = min(CH, seg.nrows - t0);
        mbar_expect_tx(&bar[b], (uint32_t)n * (1024 + GS_REC));
        bulk_g2s(smem + (size_t)b * CH * 1024, a.qk + ((size_t)hk * a.M + seg.row0 + t0) * 256, (uint32_t)n * 1024, &bar[b]);
        bulk_g2s(smem + (size_t)2 * CH * 1024 + (size_t)b * CH * GS_REC, a.vg + ((size_t)(hv * 4 + dvt) * a.M + seg.row0 + t0) * GS_REC, (uint32_t)n * GS_REC, &bar[b]);
    };
    if (tid == 0) {
        mbar_init(&bar[0], 1); mbar_init(&bar[1], 1);
        mbar_fence_init();
        fetch(0);
        if (nchunks > 1) fetch(1);
    }
    f32x2 S[2][8];                                            // [row][4 i + e]: dk e of leaves j + 8 i and j + 8 i + 16
#pragma unroll
    for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float4 lo = *reinterpret_cast<const float4*>(S_in + w * GDN_DK + (j + 8 * i) * 4), hi = *reinterpret_cast<const float4*>(S_in + w * GDN_DK + (j + 8 * i + 16) * 4);
            S[w][4 * i] = pk2(lo.x, hi.x); S[w][4 * i + 1] = pk2(lo.y, hi.y); S[w][4 * i + 2] = pk2(lo.z, hi.z); S[w][4 * i + 3] = pk2(lo.w, hi.w);
        }
    auto load = [&](const unsigned char* p, f32x2 x[8]) {     // the lane's operands of a 512-byte vector in paired order
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            lds2(p + (j + 8 * i) * 16, x[4 * i], x[4 * i + 1]);
            lds2(p + 256 + (j + 8 * i) * 16, x[4 * i + 2], x[4 * i + 3]);
        }
    };
    // lane-local part of a row's butterfly: a leaf's four products in the order of gdn_dot4(), then levels 16 and 8
    auto dot = [&](const f32x2 s[8], const f32x2 x[8]) {
        float u[2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
            u[i] = sum2(fma2(s[4 * i + 3], x[4 * i + 3], fma2(s[4 * i + 2], x[4 * i + 2], fma2(s[4 * i], x[4 * i], mul2(s[4 * i + 1], x[4 * i + 1])))));
        return __fadd_rn(u[0], u[1]);
    };
    auto xadd = [](float v, int d) { return __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, d)); };
    const bool up = (lane & 4) != 0;
    const bool writer = (lane & 3) == 0;
    // The two rows' readouts share the shuffles: level 4 leaves row 0 in the lower, row 1 in the upper four lanes.  They run
    // two tokens behind: while the shuffles of token t's kv are in flight, the products of token t-1's readout are issued and
    // the sum of token t-2's readout rides along.
    __half* y = a.y + (size_t)seg.row0 * valDim + (size_t)hv * GDN_DV + dvt * 32 + crow + (up ? 1 : 0);   // token t-2's output
    f32x2 q[8];                                               // operands of token t - 1's readout
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = 0ull;
    float op0 = 0.f, op1 = 0.f;                               // the lane's part of token t - 2's readouts
    bool ok = true;
    int behind = 0;                                           // readouts still inside the pipeline (at most 2)
    // One token.  kq / vg: its records; the next token's k and gates are read from the records behind them (for the last
    // token of a chunk that is whatever follows in shared memory: the chunk's first token is loaded anew).
    auto token = [&](const unsigned char* kq, const unsigned char* vg, f32x2 k[8], f32x2& g2, float& beta, bool store) {
        f32x2 D[2][8];                                        // the decayed state
#pragma unroll
        for (int i = 0; i < 8; ++i) { D[0][i] = mul2(S[0][i], g2); D[1][i] = mul2(S[1][i], g2); }
        float kv0 = dot(D[0], k), kv1 = dot(D[1], k);
        float o = __fadd_rn(up ? op1 : op0, __shfl_xor_sync(0xffffffffu, up ? op0 : op1, 4));
        kv0 = xadd(kv0, 4); kv1 = xadd(kv1, 4);
        op0 = dot(S[0], q); op1 = dot(S[1], q);
        const float2 v = *reinterpret_cast<const float2*>(vg + crow * 4);
        kv0 = xadd(kv0, 2); kv1 = xadd(kv1, 2); o = xadd(o, 2);
        kv0 = xadd(kv0, 1); kv1 = xadd(kv1, 1); o = xadd(o, 1);
        f32x2 kn[8], gn, bn;
        lds2(vg + GS_REC + 128, gn, bn);
        load(kq + 1024, kn);
        load(kq + 512, q);
        const float dl0 = __fmul_rn(__fsub_rn(v.x, kv0), beta), dl1 = __fmul_rn(__fsub_rn(v.y, kv1), beta);
        const f32x2 d0 = pk2(dl0, dl0), d1 = pk2(dl1, dl1);
#pragma unroll
        for (int i = 0; i < 8; ++i) { S[0][i] = fma2(k[i], d0, D[0][i]); S[1][i] = fma2(k[i], d1, D[1][i]); }
        if (store) { if (writer) *y = f2h(o); y += valDim; }
#pragma unroll
        for (int i = 0; i < 8; ++i) k[i] = kn[i];
        g2 = gn; beta = __uint_as_float((unsigned)bn);
    };
    __syncthreads();                                          // the barriers are initialised
    for (int c = 0; c < nchunks; ++c) {
        const int b = c & 1, t0 = c * CH, n = min(CH, seg.nrows - t0);
        ok = ok && mbar_wait_bounded(&bar[b], (uint32_t)((c >> 1) & 1), STALL ? 1 << 10 : 1 << 22);      // (one that ran out is not followed by others)
        const unsigned char* kq = smem + (size_t)b * CH * 1024;
        const unsigned char* vg = smem + (size_t)2 * CH * 1024 + (size_t)b * CH * GS_REC;
        f32x2 k[8];
        load(kq, k);
        const ulonglong2 g0 = *reinterpret_cast<const ulonglong2*>(vg + 128);
        f32x2 g2 = g0.x; float beta = __uint_as_float((unsigned)g0.y);
        int r = 0;
#pragma unroll 1
        while (r < n) {
            if (CH >= 3 && behind == 2 && r + 3 <= n) {       // three tokens at a time: constant offsets, one branch
#pragma unroll
                for (int u = 0; u < 3; ++u) token(kq + u * 1024, vg + u * GS_REC, k, g2, beta, true);
                r += 3; kq += 3 * 1024; vg += 3 * GS_REC;
            } else {
                token(kq, vg, k, g2, beta, behind == 2);
                behind += behind < 2; ++r; kq += 1024; vg += GS_REC;
            }
        }
        __syncthreads();                                      // every warp is done with buffer b
        if (tid == 0 && c + 2 < nchunks) fetch(c + 2);
    }
    {   // the readouts of the last two tokens
        auto finish = [&]() {
            float o = __fadd_rn(up ? op1 : op0, __shfl_xor_sync(0xffffffffu, up ? op0 : op1, 4));
            o = xadd(o, 2); o = xadd(o, 1);
            if (writer) *y = f2h(o);
        };
        if (behind == 2) { finish(); y += valDim; }
        op0 = dot(S[0], q); op1 = dot(S[1], q);
        finish();
    }
#pragma unroll
    for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float4 lo, hi;
            auto out = [&](int e, float& l, float& h) { asm("mov.b64 {%0, %1}, %2;" : "=f"(l), "=f"(h) : "l"(S[w][4 * i + e])); };
            out(0, lo.x, hi.x); out(1, lo.y, hi.y); out(2, lo.z, hi.z); out(3, lo.w, hi.w);
            *reinterpret_cast<float4*>(S_out + w * GDN_DK + (j + 8 * i) * 4) = lo;
            *reinterpret_cast<float4*>(S_out + w * GDN_DK + (j + 8 * i + 16) * 4) = hi;
        }
    if (!ok) {                                 // copies of this CTA may still be landing: outlast them
        if (a.err && lane == 0) atomicOr(a.err, 1u);
        const long long c0 = clock64();
        while (clock64() - c0 < 200000ll) { }
    }
}

size_t gdn_qk_floats(int Hk, int rows) { return (size_t)Hk * rows * 256; }
size_t gdn_vg_bytes(int Hv, int rows) { return (size_t)Hv * 4 * rows * GS_REC; }

constexpr int GS_CH = 48;             // rows a chunk: a multiple of the three tokens of a turn
template <int CH, bool STALL = false>
static void launch_scan_t(const GdnArgs& a, int nsegs, cudaStream_t st) {
    const size_t smem = (size_t)2 * CH * (1024 + GS_REC) + 256;     // (the last token reads one record of gates past its own)
    static bool configured = false;
    if (!configured) { cudaFuncSetAttribute(k_gdn_scan<CH, STALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); configured = true; }
    profile_launch("k_gdn_scan", st, [&] { k_gdn_scan<CH, STALL><<<dim3(4, (unsigned)a.Hv, (unsigned)nsegs), 128, smem, st>>>(a); return 0; });
}
void launch_gdn_rows(const GdnArgs& in, int M, int nsegs, cudaStream_t st, bool pdl) {
    GdnArgs a = in; a.M = M;
    profile_launch("k_gdn_prep", st, [&] {
        // (8 rows per CTA once that fills the device four times over; of fewer rows, 2)
        if (nsegs == 1 && (long)(a.Hk + a.Hv) * ((M + 7) / 8) < 4l * sm_count())
            return launch_pdl(pdl, k_gdn_prep<2>, dim3((unsigned)(a.Hk + a.Hv), (unsigned)((M + 1) / 2)), 128, 0, st, a);
        if (nsegs == 1) return launch_pdl(pdl, k_gdn_prep<8>, dim3((unsigned)(a.Hk + a.Hv), (unsigned)((M + 7) / 8)), 128, 0, st, a);
        return launch_pdl(pdl, k_gdn_prep<1>, dim3((unsigned)(a.Hk + a.Hv), (unsigned)M), 128, 0, st, a);
    });
    // (the scan is an ordinary launch: started early, its CTAs went to the multiprocessors that k_gdn_prep had left free,
    // several to one, and 17 rows took 7 us longer)
    // one row per segment (batched decode): the state's traffic is the time, small buffers leave room for more CTAs per SM
    if (M == nsegs) launch_scan_t<1>(a, nsegs, st);
    else if (a.stall) launch_scan_t<GS_CH, true>(a, nsegs, st);
    else launch_scan_t<GS_CH>(a, nsegs, st);
}

}  // namespace sl
