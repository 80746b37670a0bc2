// gemm_tc.cu -- 4-bit group-64 GEMM for many activation rows ("F2": prompt chunks in prefill mode) on the 5th-generation
// tensor cores: tcgen05.mma (kind::f16) issued by one thread, the expanded weights and the accumulator in tensor memory
// (TMEM), the activations in shared memory.
//
//   y[t, n] (+)= sum_k x[t, k] * fp16(scale[n, k/64] * q[n, k] + bias[n, k/64])
//
// Prefill-mode numerics: every weight is dequantised to fp16 with one rounding (the dequantised-weight GEMM of the
// reference's batched / prefill path, swift/Sources/QwispCore/SeedlessMetalForward.swift:160-185), so the whole K
// range accumulates in ONE f32 accumulator in TMEM and the epilogue runs once.  Like the reference's hybrid prefill
// this is not bit-identical to the GEMV family, but every token column is independent of the others and K is walked in
// a fixed order, so results do not depend on how many rows share a call or on how a prompt is cut into calls.
//
// One kernel, k_tc, serves the dense projections (DenseWork) and the grouped experts (ExpertWork): persistent CTAs, one
// per multiprocessor, each take their items of 128 weight rows x NT activation rows over the whole K, 128 inputs a stage.
// The warps have roles and meet only at mbarriers:
//   mma        1 warp: waits for two full stages, issues their sixteen MMAs (M=128, N=NT, K=16), commits them to the stages'
//             "empty" barriers.  It is warp 0: the other warps keep the issue slots busy;
//   load       4 warps: the NT x 128 activations of the stage, 16-byte asynchronous copies that count themselves in at
//             the stage's "full" barrier;
//   dequant   16 warps: a warp owns 32 weight rows of the item (a lane a row: a lane of tensor memory is a row) and every
//             fourth stage; its words are loaded two of its stages ahead (across items), expanded to fp16 (scale and bias by
//             one fp16x2 multiply-add per pair) and stored to the A operand in TMEM as they are;
//   epilogue   4 warps: read the finished accumulator while the next item accumulates in the other half of its TMEM.
// The first form (256 threads that all loaded, expanded, synchronised and waited in turn, one pair of groups ahead)
// spent 2.5 us on a pair of groups whose MMAs take 0.3: every pair paid the latency of its weights and of its rows.
// With roles but the A operand in shared memory, writing and reading it took most of that memory's bandwidth, and an MMA
// warp that branched on its lane number needed 1200 cycles a stage to compute addresses: uniform code needs 700.
// 1024-token chunk of the 2048 / 512 / 256-expert geometry (alone, back to back, evenly routed): experts 101 + 70 us, dense
// 12352 x 2048 54 us (0.95 PFLOP/s); 129 tokens: 77 + 47 and 18.6 us.  With a fragment of a row a lane, so that a quarter of the
// warp had to exchange its words, the experts took 158 + 109.  The experts are bound by the issue of the expansion (129 tokens,
// gate/up: issue slots 71 %, ALU 48 %, tensor pipe 22 % of the active cycles), the large dense products by rows and weights out of L2.
#include "kernels.h"
#include "gemv.cuh"

namespace sl {

constexpr int TC_ROWS = 128;      // weight rows per item (UMMA M)
constexpr int TC_LD = 4, TC_EPI = 4, TC_DQ = 16;                            // warps of each role (+ 1 for the MMAs)
constexpr int TC_EPI0 = 4, TC_DQ0 = 8;                                      // first warp of the role (load: 1, 2, 3 and the last)
constexpr int TC_THREADS = (1 + TC_LD + TC_EPI + TC_DQ) * 32;

// Activation tiles in shared memory: K-major, 128-byte swizzle.  A row holds 64 halves (128 bytes); 8 rows form a 1024-byte
// atom inside which the 16-byte chunk index is XORed with the row index (conflict-free for the threads that fill it and for
// the tensor core that reads it; an unswizzled layout ran the same MMAs several times slower); atoms of further rows follow
// at 1024-byte steps.  Tiles start on 1024-byte boundaries.
__device__ __forceinline__ uint32_t tc_off(int row, int chunk) { return ((uint32_t)(row >> 3) << 10) + ((row & 7) << 7) + (((chunk ^ row) & 7) << 4); }
__device__ __forceinline__ uint64_t umma_desc_sw128(const void* smem_ptr) {
    // shared-memory matrix descriptor: start address; leading byte offset 1 (unused by swizzled K-major layouts); stride
    // byte offset 1024 (between 8-row atoms); all without their 4 low bits; descriptor version 1; layout type 2 = 128-byte swizzle
    const uint64_t addr = (uint64_t)(smem_u32(smem_ptr) >> 4) & 0x3FFFull;
    return addr | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// D (TMEM) (+)= A (TMEM, 8 columns = 16 halves of K per lane) * B (shared memory)
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        :: "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t r[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 32 lanes (rows) x 16 columns
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t v[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                    "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory"); }

// Bounded wait of a role.  The first that runs out (a poll takes up to 4 us, so some 17 s) raises the CTA's abort word; every
// later wait of the CTA then gives up after 256 polls.  The outcome is a lane's own, but what follows a wait needs whole warps:
// a role goes on to the end of its item whatever its waits said (its results are discarded then) and leaves by tc_agree().
// The lanes' polls, like every branch that is a lane's own (rows or tiles that only half a warp has), are behind a __syncwarp()
// or a vote before the next tcgen05 instruction of the .sync.aligned kind, which a warp has to come to as one.
// Warps need not agree: none waits for another but here and at the end of the kernel.
template <int LIMIT>
__device__ __forceinline__ bool tc_wait(uint64_t* b, uint32_t parity, volatile int* abort_word) {
    if (mbar_try_wait(b, parity)) return true;
    for (int i = 0; i < LIMIT; ++i) {
        if (mbar_try_wait(b, parity)) return true;
        if ((i & 255) == 255 && *abort_word) return false;
    }
    *abort_word = 1;
    return false;
}
__device__ __forceinline__ bool tc_agree(bool ok) { return __all_sync(0xffffffffu, ok); }

// ---- one K group (64 inputs) of a row of a tile: packed words -> A operand.  A lane of tensor memory is a weight row, and the
// weights arrive by rows (gemv.cuh), so a lane expands what it has loaded and stores it as it is: 32 columns of two halves.
// Bound by the issue of these instructions: 13 per word of 8 weights.
__device__ __forceinline__ void tc_expand(uint32_t w, __half2 sc, __half2 bi, uint32_t* c) {
    uint32_t d[4];
    dequant8(w, d);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 h = __hfma2(*reinterpret_cast<const __half2*>(&d[j]), sc, bi);
        c[j == 1 ? 2 : j == 2 ? 1 : j] = *reinterpret_cast<const uint32_t*>(&h);
    }
}
// w: the words of the group; sb: its (scale, bias); taddr: the warp's lanes, the group's first column
__device__ __forceinline__ void tc_group_A(const uint2 w[4], uint32_t sb, uint32_t taddr) {
    const __half2 h = *reinterpret_cast<const __half2*>(&sb), sc = __half2half2(__low2half(h)), bi = __half2half2(__high2half(h));
    uint32_t v[16];
    tc_expand(w[0].x, sc, bi, v); tc_expand(w[0].y, sc, bi, v + 4); tc_expand(w[1].x, sc, bi, v + 8); tc_expand(w[1].y, sc, bi, v + 12);
    tmem_st16(taddr, v);
    tc_expand(w[2].x, sc, bi, v); tc_expand(w[2].y, sc, bi, v + 4); tc_expand(w[3].x, sc, bi, v + 8); tc_expand(w[3].y, sc, bi, v + 12);
    tmem_st16(taddr + 16, v);
}

// ================================================================================ the two kinds of work
// Items are (rows block, 128 weight rows), weight rows fastest.  A work type says which items a CTA has, the weights of a tile of an
// item (moved along by a cursor), the place of a block's activation rows (halves from base(); Place: wide enough for the rows that
// the kind of work can have), and the epilogue.
struct TcRun { int blk, rt, count; };                      // a role's place in its CTA's items, and how many the CTA has
struct TcTile { const uint4 *w, *s; int blk, rt; };   // fragment-major nibbles and scales of a tile (nullptr: none) of weight-row group rt

struct GemmTcArgs {
    Q4R q; int N, K, M;
    const __half* x; int ldx;
    __half* y; int ldy;
    int add_to_y;                    // y += result (residual) instead of y = result
    unsigned* err;
};
// Dense projection: a block is a token tile.
template <int NT>
struct DenseWork {
    using Args = GemmTcArgs;
    static constexpr bool STRIDED = true;                                   // rows of a block lie stride() halves apart
    using Place = size_t;                                                   // (a product of the caller's own size: any M)
    static constexpr Place NO_ROW = ~(Place)0;
    struct Shared {};
    const Args& a;
    int NRT;                                                                // weight-row groups
    __device__ DenseWork(const Args& args, Shared&) : a(args), NRT((args.N + TC_ROWS - 1) / TC_ROWS) {}
    __device__ int items() const { return NRT * ((a.M + NT - 1) / NT); }
    // CTA b of n: a contiguous run, so that most steps stay inside a block
    __device__ TcRun run(int b, int n) const { const int lo = (int)((long)items() * b / n), hi = (int)((long)items() * (b + 1) / n); return {lo / NRT, lo % NRT, hi - lo}; }
    __device__ void next(TcRun& w) const { if (++w.rt == NRT) { w.rt = 0; ++w.blk; } }
    __device__ int inputs() const { return a.K; }
    __device__ unsigned* err() const { return a.err; }
    __device__ bool has_tile(int rt, int tl) const { return rt * 8 + tl < a.N >> 4; }
    __device__ TcTile tile(int blk, int rt, int tl) const {
        const int T = rt * 8 + tl, GP = a.K >> 7;
        if (!has_tile(rt, tl)) return {nullptr, nullptr, blk, rt};          // (a matrix whose rows are not a multiple of 128)
        return {a.q.wr + (size_t)T * GP * 64, a.q.sr + (size_t)T * GP * 8, blk, rt};
    }
    __device__ const __half* base() const { return a.x; }
    __device__ uint32_t stride() const { return (uint32_t)a.ldx; }
    __device__ Place row(int blk, int n) const { return blk * NT + n < a.M ? (Place)(blk * NT + n) * (Place)a.ldx : NO_ROW; }
    struct Epi {};
    __device__ void begin(Epi&, int, int, int) const {}
    // quarter: accumulator lanes 32 * quarter ..; taddr: the item's columns in TMEM; release() once they have been read
    template <class Release>
    __device__ void epilogue(Epi&, int blk, int rt, int quarter, int lane, uint32_t taddr, Release release) const {
        const int row = rt * TC_ROWS + quarter * 32 + lane, t0 = blk * NT, nt = min(NT, a.M - t0);
#pragma unroll 1
        for (int c0 = 0; c0 < nt; c0 += 16) {
            uint32_t d[16];
            __syncwarp();
            tmem_ld16(taddr + (uint32_t)c0, d);
            if (c0 + 16 >= nt) release();
            if (row < a.N) {
                __half* y = a.y + (size_t)(t0 + c0) * a.ldy + row;
                __half old[16];
                if (a.add_to_y) {                                           // sixteen residual values in flight at a time
#pragma unroll
                    for (int n = 0; n < 16; ++n) if (c0 + n < nt) old[n] = y[(size_t)n * a.ldy];
                }
#pragma unroll
                for (int n = 0; n < 16; ++n)
                    if (c0 + n < nt) {
                        const __half v = f2h(__uint_as_float(d[n]));
                        y[(size_t)n * a.ldy] = a.add_to_y ? hadd_rn(old[n], v) : v;
                    }
            }
        }
    }
};
// Routed + shared experts of a prompt chunk: a block is up to NT rows of one expert slot, gathered through the pair lists.
// gate/up: the epilogue applies SwiGLU to (gate row r, up row r) of a paired tile -- they sit 8 accumulator lanes apart --
// and stores the SwiGLU rows in natural order; down: the pair's output row.
template <bool DOWN, int NT>
struct ExpertWork {
    using Args = ExpertArgs;
    static constexpr bool STRIDED = false;
    using Place = uint32_t;                                                 // (an engine has at most 1024 rows: 17k pair rows of 4096)
    static constexpr Place NO_ROW = ~(Place)0;
    static constexpr int MAX_BLK = 1024;
    struct Shared { SlotTable tab; short slot[MAX_BLK]; int dst[TC_EPI][(NT + 31) / 32 * 32]; };      // slot: of a block; dst: a list of each epilogue warp
    const Args& a;
    Shared& sh;
    int n_active, K, ntiles, NRT, npair, nshared, step_b, step_r;
    __device__ ExpertWork(const Args& args, Shared& s) : a(args), sh(s) {
        K = DOWN ? a.I : a.H;
        ntiles = DOWN ? a.H / 16 : a.I / 8;                                 // tiles of 16 weight rows per expert
        NRT = (ntiles + 7) / 8;                                             // groups of 128 weight rows
        npair = a.M * a.topk;
        nshared = a.M_shared >= 0 ? a.M_shared : a.M;
        pdl_wait();                                                         // (the lists)
        n_active = slot_table(sh.tab, a.lists, NT, nshared);
        __syncthreads();
        for (int b = threadIdx.x; b < min(sh.tab.base[n_active + 1], MAX_BLK); b += TC_THREADS) sh.slot[b] = (short)slot_of(sh.tab, n_active, b);
        __syncthreads();
        step_b = (int)gridDim.x / NRT; step_r = (int)gridDim.x % NRT;
    }
    __device__ int items() const { return sh.tab.base[n_active + 1] * NRT; }
    // CTA b of n: every n-th item.  An item's loads and epilogue are as long as its rows, and a routed expert's blocks hold few rows or
    // many, the shared expert's are full: dealt out like this every CTA has some of each.  In contiguous runs with the shared expert's
    // items dealt out among them, a prompt of 2900 tokens took 62.5 ms, now 59.5, one of 129 7.95 and 7.73 ms; 256 experts
    // routed evenly (gate/up, down): 129 rows 79.3, 48.5 -> 76.6, 47.3 us, 1024 rows 103.8, 73.8 -> 101.3, 69.9.
    // A new block with every item asks for its slot and its rows' places each time: the slots in a table, the places an item ahead.
    __device__ TcRun run(int b, int n) const { return {b / NRT, b % NRT, b < items() ? (items() - b + n - 1) / n : 0}; }
    __device__ void next(TcRun& w) const {
        w.blk += step_b; w.rt += step_r;
        if (w.rt >= NRT) { w.rt -= NRT; ++w.blk; }
    }
    __device__ int slot(int blk) const { return blk < MAX_BLK ? sh.slot[blk] : slot_of(sh.tab, n_active, blk); }
    __device__ int inputs() const { return K; }
    __device__ unsigned* err() const { return a.err; }
    __device__ bool has_tile(int rt, int tl) const { return rt * 8 + tl < ntiles; }
    __device__ TcTile tile(int blk, int rt, int tl) const {
        if (!has_tile(rt, tl)) return {nullptr, nullptr, blk, rt};
        const int j = slot(blk);
        const bool shared = (j == n_active);
        const Q4R& q = DOWN ? (shared ? a.sh_down : a.down) : (shared ? a.sh_gu : a.gu);
        const size_t T = (size_t)(shared ? 0 : sh.tab.expert[j]) * ntiles + rt * 8 + tl;
        return {q.wr + T * (K >> 7) * 64, q.sr + T * (K >> 7) * 8, blk, rt};
    }
    // row n of a block: its pair id (shared expert: npair + row), or -1
    __device__ int pair_of(int blk, int n) const {
        const int j = slot(blk), i = (blk - sh.tab.base[j]) * NT + n;
        if (j == n_active) return i < nshared ? npair + i : -1;
        return i < sh.tab.cnt[j] ? a.lists.pairs[sh.tab.off[j] + i] : -1;
    }
    __device__ const __half* base() const { return DOWN ? a.hbuf : a.p; }
    __device__ uint32_t stride() const { return 0; }
    __device__ Place place(int p) const {                                   // of a pair
        if (p < 0) return NO_ROW;
        return (Place)(DOWN ? p : (p >= npair ? a.shared_row0 + p - npair : p / a.topk)) * (Place)K;
    }
    struct Epi { int blk = -1, count = 0; };                                // the block whose rows are listed in sh.dst
    // The rows of a block, listed before its accumulators are waited for.  Each warp makes the list for itself, so that the four
    // have nothing to meet for (behind the wait it cost a prompt 1.2 %).
    __device__ void begin(Epi& e, int blk, int quarter, int lane) const {
        if (blk == e.blk) return;
        e.blk = blk;
        __syncwarp();
#pragma unroll
        for (int n = 0; n < NT; n += 32) sh.dst[quarter][n + lane] = pair_of(blk, n + lane);
        const int j = slot(blk);
        e.count = min(NT, (j == n_active ? nshared : sh.tab.cnt[j]) - (blk - sh.tab.base[j]) * NT);
        __syncwarp();
    }
    template <class Release>
    __device__ void epilogue(Epi& e, int, int rt, int quarter, int lane, uint32_t taddr, Release release) const {
        const int i = quarter * 32 + lane;
        const int* dsts = sh.dst[quarter];
        const int i16 = i & 15, etile = rt * 8 + (i >> 4);
        const bool up = i16 >= 8, have = etile < ntiles;
        __half* out = DOWN ? a.dbuf + (size_t)rt * TC_ROWS + (i & ~1) : a.hbuf + etile * 8 + (i16 & 7);
#pragma unroll 1
        for (int c0 = 0; c0 < e.count; c0 += 16) {
            uint32_t d[16];
            __syncwarp();
            tmem_ld16(taddr + (uint32_t)c0, d);
            if (c0 + 16 >= e.count) release();
            if (DOWN) {
                // two columns at a time: an even lane stores its row and the next of the first, an odd lane of the second
#pragma unroll
                for (int n = 0; n < 16; n += 2) {
                    const __half2 h = __floats2half2_rn(__uint_as_float(d[n]), __uint_as_float(d[n + 1]));
                    const uint32_t mine = *reinterpret_cast<const uint32_t*>(&h), other = __shfl_xor_sync(0xffffffffu, mine, 1);
                    const int dst = dsts[c0 + n + (lane & 1)];
                    if (dst >= 0 && have) *reinterpret_cast<uint32_t*>(out + (size_t)dst * a.H) = __byte_perm(mine, other, (lane & 1) ? 0x3276 : 0x5410);
                }
            } else {
                // two columns at a time: the gate lane finishes the first, the up lane the second; each sends what the other lacks
#pragma unroll
                for (int n = 0; n < 16; n += 2) {
                    const uint32_t other = __shfl_xor_sync(0xffffffffu, up ? d[n] : d[n + 1], 8);
                    const float g = __uint_as_float(up ? other : d[n]), u = __uint_as_float(up ? d[n + 1] : other);
                    const __half v = swiglu_h(f2h(g), f2h(u));
                    const int dst = dsts[c0 + n + (up ? 1 : 0)];
                    if (dst >= 0 && have) out[(size_t)dst * a.I] = v;
                }
            }
        }
    }
};

// ================================================================================ the kernel
// ST: stages (even, at least 4); U: stages whose weights a dequant warp has in flight
// TMEM columns: [2][ACC] accumulators, [ST][64] A operands
// STALL: a test's form, in which no row is ever loaded, so that every wait runs out, and soon
template <class W, int NT, int ST, int U, bool STALL>
__global__ void __launch_bounds__(TC_THREADS, 1) k_tc(typename W::Args a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];             // ST stages x [2 groups][NT rows x 128 B]
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // tiles start on 1024-byte boundaries
    constexpr int TILE = NT * 128, STAGE = 2 * TILE, ACC = NT == 48 ? 64 : NT, LIMIT = STALL ? 1 << 10 : 1 << 22;
    static_assert(2 * ACC + ST * 64 <= 512 && ST >= 4 && ST % 2 == 0, "tensor memory");
    __shared__ __align__(8) uint64_t s_full[ST], s_empty[ST], s_acc_full[2], s_acc_empty[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ typename W::Shared s_work;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // (the shuffle tells the compiler that it is uniform)
    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < ST; ++i) { mbar_init(&s_full[i], TC_DQ / 4 + TC_LD * 32); mbar_init(&s_empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&s_acc_full[i], 1); mbar_init(&s_acc_empty[i], TC_EPI); }
        mbar_fence_init();
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    W work(a, s_work);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    const int KS = work.inputs() >> 7;                                      // stages per item (even)
    const TcRun run = work.run(blockIdx.x, gridDim.x);
    bool ok = true;
    if (warp == 0) {
        // ------------------------------------------------------------ mma
        // The whole warp walks the stages, so that addresses and descriptors stay in uniform registers; one elected lane issues.
        const uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(TC_ROWS >> 4) << 24);   // f32 accumulate, f16 x f16, K-major B
        const uint64_t db0 = umma_desc_sw128(smem);
        const uint32_t ta0 = tmem + 2 * ACC;
        int st = 0; uint32_t ph = 0;
        for (int k = 0; k < run.count && ok; ++k) {
            if (k >= 2) ok = tc_wait<LIMIT>(&s_acc_empty[k & 1], (uint32_t)(((k >> 1) - 1) & 1), &s_abort) && ok;
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)((k & 1) * ACC);
#pragma unroll 1
            for (int s = 0; s < KS; s += 2) {                               // (KS and ST are even)
                ok = tc_wait<LIMIT>(&s_full[st], ph, &s_abort) && ok;
                ok = tc_wait<LIMIT>(&s_full[st + 1], ph, &s_abort) && ok;
                tc_fence_after();
                tc_fence_proxy();                                           // the rows other threads' asynchronous copies wrote are operand data now
                const uint64_t db = db0 + (uint32_t)(st * (STAGE >> 4));    // (the address field counts 16 bytes: a K step of 16 halves is 2)
                const uint32_t ta = ta0 + st * 64;
                if (tc_elect()) {
                    umma_f16_ts(acc, ta, db, idesc, s > 0 ? 1u : 0u);
#pragma unroll
                    for (int j = 1; j < 8; ++j) umma_f16_ts(acc, ta + j * 8, db + (j >> 2) * (TILE >> 4) + (j & 3) * 2, idesc, 1u);
                    umma_commit(&s_empty[st]);
#pragma unroll
                    for (int j = 8; j < 16; ++j) umma_f16_ts(acc, ta + j * 8, db + (j >> 2) * (TILE >> 4) + (j & 3) * 2, idesc, 1u);
                    umma_commit(&s_empty[st + 1]);
                    if (s == KS - 2) umma_commit(&s_acc_full[k & 1]);
                }
                __syncwarp();
                st += 2; if (st == ST) { st = 0; ph ^= 1u; }
            }
            ok = tc_agree(ok);
        }
    } else if (warp >= TC_DQ0 && warp < TC_DQ0 + TC_DQ) {
        // ------------------------------------------------------------ dequant: 32 rows of the item (two tiles), every fourth stage
        // (a warp reaches the TMEM lanes 32 * (warp % 4) ..).  Stages are counted through the run: an item of two stages leaves
        // two of the four warps of a quarter without one.
        const int d = warp - TC_DQ0, quarter = d & 3, tl = quarter * 2 + (lane >> 4), row = lane & 15;
        const uint32_t ta = tmem + 2 * ACC + ((uint32_t)(quarter * 32) << 16);
        uint2 wv[U][8]; uint32_t sv[U][2];                                  // [stage in flight][group, two words], (scale, bias)
        int f_k = 0, f_s = d >> 2;                                          // the fetch cursor: item of the run, stage of it
        TcRun fw = run;
        TcTile ft = run.count > 0 ? work.tile(fw.blk, fw.rt, tl) : TcTile{nullptr, nullptr, 0, 0};
        auto seek = [&] {                                                   // past the end of an item: on to the one that has stage f_s
            while (f_s >= KS) {
                f_s -= KS;
                if (++f_k >= run.count) { ft.w = nullptr; f_s = 0; return; }
                work.next(fw);
                if (ft.w && fw.blk == ft.blk && fw.rt == ft.rt + 1 && work.has_tile(fw.rt, tl)) { ft.w += KS * 512; ft.s += KS * 64; ++ft.rt; }      // eight tiles on
                else ft = work.tile(fw.blk, fw.rt, tl);
            }
        };
        seek();
        auto fetch = [&](uint2 w[8], uint32_t sc[2]) {
            if (ft.w) {
                const uint2* p = reinterpret_cast<const uint2*>(ft.w + f_s * 64 + (row & 7) * 4) + (row >> 3);
#pragma unroll
                for (int i = 0; i < 8; ++i) w[i] = __ldg(p + (i >> 2) * 64 + (i & 3) * 2);
                const uint32_t* q = reinterpret_cast<const uint32_t*>(ft.s + f_s * 8 + (row & 7)) + (row >> 3);
                sc[0] = __ldg(q); sc[1] = __ldg(q + 2);
            }
            if (f_k < run.count) { f_s += 4; seek(); }
        };
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int i = 0; i < 8; ++i) wv[u][i] = make_uint2(0, 0);        // (rows the matrix does not have)
            sv[u][0] = 0; sv[u][1] = 0;
            fetch(wv[u], sv[u]);
        }
        const int total = run.count * KS;                                     // stages of the run
        int n = d >> 2, st = n;
        uint32_t ph = 1;                                                    // parity of the stage's "empty" (a fresh barrier passes at 1)
        while (n < total && ok) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (n < total) {
                    ok = tc_wait<LIMIT>(&s_empty[st], ph, &s_abort) && ok;
                    __syncwarp();
                    tc_fence_after();                                       // (rows the matrix does not have are expanded too: their outputs are not stored)
                    tc_group_A(wv[u], sv[u][0], ta + st * 64);
                    tc_group_A(wv[u] + 4, sv[u][1], ta + st * 64 + 32);
                    fetch(wv[u], sv[u]);
                    __syncwarp();                                           // (N % 32 == 16: only half of the warp has a tile)
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) tc_arrive(&s_full[st]);
                    n += 4;
                    st += 4; if (st >= ST) { st -= ST; ph ^= 1u; }
                }
            }
            ok = tc_agree(ok);
        }
    } else if (warp < TC_EPI0 || warp >= TC_DQ0) {
        // ------------------------------------------------------------ load: the activation rows of every stage
        pdl_wait();
        constexpr int NP = NT / 16;                                         // rows of a stage per thread, 2 pieces of 16 bytes each
        const int lt = (warp < TC_EPI0 ? warp - 1 : 3) * 32 + lane;
        // the 8 lanes of a quarter warp write into the 8 rows of one atom (distinct swizzled chunks) and read 4 x 64 contiguous
        // bytes per row
        const int n0 = ((lt >> 6) << 3) + (lt & 7), chunk = (lt >> 3) & 7;  // rows n0 + 16 h, the same chunk of both groups
        const uint32_t off0 = smem_u32(smem) + tc_off(n0, chunk);
        const __half* base = work.base() + chunk * 8;
        typename W::Place src[W::STRIDED ? 1 : NP];                         // row places (strided: of the first row)
        int st = 0; uint32_t ph = 1;
        TcRun at = run;
        int held = -1, have = 0;                                            // held: the block whose row places are in src; have: its rows (strided)
        int next[W::STRIDED ? 1 : NP];                                      // the next item's pairs, looked up an item ahead
        if constexpr (!W::STRIDED) { for (int h = 0; h < NP; ++h) next[h] = run.count > 0 ? work.pair_of(at.blk, n0 + 16 * h) : -1; }
        for (int k = 0; k < run.count && ok && !STALL; ++k) {
            const int blk = at.blk;
            work.next(at);
            if constexpr (W::STRIDED) {
                if (blk != held) {
                    held = blk;
                    src[0] = work.row(blk, n0); have = 0;
                    for (int h = 0; h < NP; ++h) have += work.row(blk, n0 + 16 * h) != W::NO_ROW;
                }
            } else {
#pragma unroll
                for (int h = 0; h < NP; ++h) {
                    src[h] = work.place(next[h]);
                    if (k + 1 < run.count && at.blk != blk) next[h] = work.pair_of(at.blk, n0 + 16 * h);
                }
            }
#pragma unroll 1
            for (int s = 0; s < KS; ++s) {
                ok = tc_wait<LIMIT>(&s_empty[st], ph, &s_abort) && ok;
                const uint32_t B = off0 + (uint32_t)st * STAGE;
                auto copy = [&](int h, const __half* p) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(B + 2048u * h), "l"(p) : "memory");
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(B + TILE + 2048u * h), "l"(p + 64) : "memory");
                };
                // (a row the item does not have keeps what was there: its column is not stored)
                if (W::STRIDED) {
                    const __half* p = base + src[0] + s * 128;
#pragma unroll 4
                    for (int h = 0; h < NP; ++h, p += (size_t)16 * work.stride()) if (h < have) copy(h, p);
                } else {
#pragma unroll
                    for (int h = 0; h < NP; ++h) {
                        const typename W::Place o = src[W::STRIDED ? 0 : h];
                        if (o != W::NO_ROW) copy(h, base + o + s * 128);
                    }
                }
                // the barrier counts this thread in when its copies have landed: nobody waits for them here
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&s_full[st])) : "memory");
                if (++st == ST) { st = 0; ph ^= 1u; }
            }
            ok = tc_agree(ok);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ------------------------------------------------------------ epilogue
        pdl_wait();                                                         // (residual rows, and rows that the kernel before may still read)
        typename W::Epi epi;
        const int quarter = warp - TC_EPI0;
        TcRun at = run;
        for (int k = 0; k < run.count && ok; ++k) {
            work.begin(epi, at.blk, quarter, lane);
            ok = tc_agree(tc_wait<LIMIT>(&s_acc_full[k & 1], (uint32_t)((k >> 1) & 1), &s_abort));
            tc_fence_after();
            if (ok) work.epilogue(epi, at.blk, at.rt, quarter, lane, tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((k & 1) * ACC), [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) tc_arrive(&s_acc_empty[k & 1]);
            });
            work.next(at);
        }
    }
    if (!ok) {                                 // MMAs of this CTA may still be running: outlast them before TMEM is given back
        if (work.err() && lane == 0) atomicOr(work.err(), 1u);
        const long long c0 = clock64();
        while (clock64() - c0 < 200000ll) { }
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
}
constexpr int TC_U = 2;
template <class W, int NT, int ST, int U, bool STALL = false>
static int launch_tc_t(const typename W::Args& a, int grid, cudaStream_t st, bool pdl) {
    constexpr size_t smem = (size_t)ST * NT * 256 + 1024;
    static bool configured = false;
    if (!configured) {
        cudaError_t err = cudaFuncSetAttribute(k_tc<W, NT, ST, U, STALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return (int)err;
        configured = true;
    }
    return launch_pdl(pdl, k_tc<W, NT, ST, U, STALL>, dim3((unsigned)grid), TC_THREADS, smem, st, a);
}
template <int NT, int ST>
static int launch_gemm_tc_t(const GemmTcArgs& a, cudaStream_t st, bool pdl) {
    const int items = ((a.N + TC_ROWS - 1) / TC_ROWS) * ((a.M + NT - 1) / NT), grid = items < sm_count() ? items : sm_count();
    return launch_tc_t<DenseWork<NT>, NT, ST, TC_U>(a, grid, st, pdl);
}
int launch_gemm_tc(const Q4R& q, int N, int K, int M, const __half* x, int ldx, __half* y, int ldy, bool add_to_y, unsigned* err, cudaStream_t st, bool pdl) {
    if (N % 16 || K % 256) return -1;
    GemmTcArgs a{q, N, K, M, x, ldx, y, ldy, add_to_y ? 1 : 0, err};
    // The token tile is a scheduling choice only (a token's column never interacts with another's).  An item's time is the
    // larger of its MMAs and of the expansion of its weights (whatever the tile), and a multiprocessor does
    // ceil(items / multiprocessors) of them: the cheapest sum, the wider tile on a tie.  Measured, K = 2048, weights from memory:
    // 8.2, 5.7, 6.0 us an item of 128, 64, 32 tokens, the first with a start of about 8 more; the costs are those of the first (16.5, 13, 12.5).
    // 20 row counts from 16 to 1024 of 12352 x 2048, 9216 x 2048 and 2048 x 4096: the chosen tile was the fastest or within 7 % of it,
    // which is also what two runs of one tile differ by (129 rows of 12352: 23.1, 18.6, 24.9; 512: 33.0, 40.7, 59.6; 1024: 59.5, 70.0, 112).
    const long row_tiles = (N + TC_ROWS - 1) / TC_ROWS;
    const int nts[3] = {128, 64, 32}, cost[3] = {320, 260, 260};
    int best = 0; long best_cost = 0;
    for (int i = 0; i < 3; ++i) {
        const long items = row_tiles * ((M + nts[i] - 1) / nts[i]), c = (items + sm_count() - 1) / sm_count() * cost[i];
        if (i == 0 || c < best_cost) { best = i; best_cost = c; }
    }
    if (best == 0) return launch_gemm_tc_t<128, 4>(a, st, pdl);
    if (best == 1) return launch_gemm_tc_t<64, 6>(a, st, pdl);
    return launch_gemm_tc_t<32, 6>(a, st, pdl);
}

// Rows of an expert's block.  Each row beyond the block's is another expansion of the expert's weights, and each column of the
// tile without a row costs its share of the loads and MMAs: the narrowest tile that most experts' rows fit into once.  Prompt
// calls of the 40-layer, 256-expert geometry in ms with 32 / 48 / 64 rows a block: 129 rows (4 an expert) 8.31 / 8.52 / 8.80;
// 512 (16) 14.2 / 14.3 / 14.7; 640 (20) 16.73 / 16.76 / 17.20; 768 (24) 18.6 / 18.4 / 18.9; 1024 (32) 23.0 / 22.2 / 22.5.
template <bool DOWN, int NT>
static int launch_expert_tc_n(const ExpertArgs& a, cudaStream_t st, bool pdl) {
    if constexpr (!DOWN)
        if (a.stall) return launch_tc_t<ExpertWork<DOWN, NT>, NT, 6, TC_U, true>(a, sm_count(), st, pdl);
    return launch_tc_t<ExpertWork<DOWN, NT>, NT, 6, TC_U>(a, sm_count(), st, pdl);
}
template <bool DOWN>
static bool launch_expert_tc_t(const ExpertArgs& a, cudaStream_t st, bool pdl) {
    const int K = DOWN ? a.I : a.H;
    if (K % 256 || a.ep_pairs_per_rank > 0) return false;              // (expert-parallel calls keep the row kernels)
    int rc = 0;
    const int mean = a.M * a.topk / a.E, nt = mean <= 20 ? 32 : mean <= 34 ? 48 : 64;
    profile_launch(DOWN ? "k_expert_umma_down" : "k_expert_umma_gateup", st, [&] {
        return rc = nt == 32 ? launch_expert_tc_n<DOWN, 32>(a, st, pdl) : nt == 48 ? launch_expert_tc_n<DOWN, 48>(a, st, pdl) : launch_expert_tc_n<DOWN, 64>(a, st, pdl);
    });
    return rc == 0;
}
bool launch_expert_tc_gateup(const ExpertArgs& a, cudaStream_t st, bool pdl) { return launch_expert_tc_t<false>(a, st, pdl); }
bool launch_expert_tc_down(const ExpertArgs& a, cudaStream_t st, bool pdl) { return launch_expert_tc_t<true>(a, st, pdl); }

}  // namespace sl
