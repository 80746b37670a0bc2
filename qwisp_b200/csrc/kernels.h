// kernels.h -- argument blocks and host launchers of the Seedless B200 kernels.
#pragma once
#include "gemv.cuh"
#include <functional>

namespace sl {

struct Q4W { const uint32_t* w = nullptr; const __half* s = nullptr; const __half* b = nullptr; int64_t N = 0; int K = 0; };

struct DenseArgs {
    int lg_slices = 0;                   // log2(K/256), filled by the launcher
    unsigned* err = nullptr;             // set to 1 if a bounded wait on a bulk copy gave up
    __half* norm_scratch = nullptr;      // [M][K] scratch for the tensor-core path (normed rows); nullptr keeps the GEMV path
    bool tc = false;                     // prefill mode: dense projections on the tcgen05 GEMM (set per call by the caller)
    __half* xq = nullptr; float* sxq = nullptr;   // [M][K] / [M][K/64] scratch of the many-row kernels (calls with more than one row); nullptr: pass kernels
    bool direct = false;                 // a many-row product of plain rows may run without that scratch
    Q4R q;                                                       // repacked weights (tiles of 16 rows)
    int N, K, M;                                                 // N outputs (= 16 * tiles)
    const __half* x; int ldx;                                    // activations (plain) / residual stream (rmsnorm) / y (normgate)
    const __half* nw;                                            // norm weight
    const float* nw32 = nullptr;                                 // gated norm: f32 norm weight (norm in f32); nw keeps its fp16 cast
    const __half* z; int ldz;                                    // gate input of the gated norm
    float eps;
    __half* y; int ldy;                                          // output rows
    __half* logits;                                              // optional [M][N] (argmax epilogue)
    float* pval; int* pidx; int* out_tok; unsigned* counter;     // argmax partials / result / ticket
    bool prepared = false;                                       // xq / sxq (prefill mode: norm_scratch) already hold the prologue's rows (a many-row call)
    PfList pf;                                                   // weights of later kernels to pull into L2
    MoeRow moe;                                                  // PRO_MOERMS: x is the residual row before the last MoE block's combine
};

// what a kernel needs to raise this rank's flags at its peers (world == 0: not expert-parallel)
struct EpSignal { unsigned* flags[8]; unsigned* ctr; unsigned* ticket; int world = 0, rank = 0, layer = 0; };
// the router's dispatch: peer gather buffers + flags
struct EpDispatch { __half* pbuf[8]; int* ibuf[8]; EpSignal sig; };

struct MoeLists {
    int* n_active;       // [1]
    int* slot_expert;    // [E]
    int* slot_off;       // [E]
    int* slot_cnt;       // [E]
    int* pairs;          // pair ids (row*top_k + k) grouped by expert slot, from slot_off on
    int* counts;         // [E] pairs of each expert so far, zero between launches (k_route_rows)
    int cap;             // its room for an expert's pairs: pair ids of expert e from pairs[e * cap] on
};

struct RouterArgs {
    const __half* h; int ldh;            // input rows
    const __half* norm_w; float eps;     // post-attention norm (nullptr: rows are already normed)
    const __half* router;                // fp16 [E][H]
    const __half* shared_gate;           // fp16 [H]
    // the checkpoint's 8-bit group-64 form of the two (set all six or none; they replace the fp16 pair)
    const uint8_t* router_q8 = nullptr; const __half *router_qs = nullptr, *router_qb = nullptr;   // [E][H] bytes, [E][H/64] scales / biases
    const uint8_t* sg_q8 = nullptr; const __half *sg_qs = nullptr, *sg_qb = nullptr;               // [H] bytes, [H/64]
    int M, H, E;
    __half* p;                           // normed rows out [M][H]
    __half* logits;                      // [M][E]
    __half* sgl;                         // [M] shared-expert gate logit
    int topk; int* inds; __half* scores; // [M][topk] routing result (written by the last CTA)
    MoeLists lists; unsigned* counter;
    unsigned* group_counter;             // [ceil(M/8)] tickets of the row groups, zero between launches
    int no_route = 0;                    // 1: stop after the logits; the consumer (the expert kernel) routes from them itself
    EpDispatch epd;                      // expert-parallel: the last CTA sends the rows and indices to every rank instead of building lists
    int ep_rows_sent = 0;                // expert-parallel, many-row router: the norm kernel has sent the rows already; only the indices remain
    PfList pf;                           // static prefetch (every CTA)
};

// Peer pointers of the expert-parallel exchange (ep_exchange.cu): entry d is rank d's buffer as mapped into this
// process (entry `rank` is the local one).  pbuf: gathered normed rows [world*M][H]; ibuf: gathered routing indices
// [world*M][top_k]; dbuf: the pair outputs of the OWNER's rows [M*top_k][H]; flags: [0,8) dispatch, [8,16) combine.
struct EpPeers {
    __half* pbuf[8]; int* ibuf[8]; __half* dbuf[8]; unsigned* flags[8];
    unsigned* ctr;                       // local step counter (all ranks advance it in lockstep)
    int world, rank;
};

struct ExpertArgs {
    int lg_slices = 0;                   // log2(K/256), filled by the launcher
    unsigned* err = nullptr;             // set to 1 if a bounded wait on a bulk copy gave up
    Q4R gu, down;                        // expert slabs, repacked: gate/up paired tiles (I/8 per expert), down tiles (H/16 per expert)
    Q4R sh_gu, sh_down;
    MoeLists lists;
    const __half* p;                     // [M][H] normed rows
    __half* hbuf;                        // [(M*topk + M)][I]
    __half* dbuf;                        // [(M*topk + M)][H]
    int M, H, I, topk;
    int E = 0;                           // experts of the model (of all ranks): a launch goes by the mean rows of an expert
    const __half* rlogits = nullptr;     // route_here: router logits [M][E]; every CTA routes from them itself (deterministic, so all CTAs
    int route_here = 0;                  //   agree) instead of waiting for a routing kernel or a routing tail in the router kernel
    int* inds_out = nullptr; __half* scores_out = nullptr;   //   the result, published by one CTA (fused kernel) or one CTA per row
    int lg_slices2 = 0;                  // fused kernel: log2(I/256) of the down phase
    unsigned* slot_sync = nullptr;       // fused kernel: [2][top_k + 1] counters, zero between launches
    int nstages = 1;                     // weight stages per CTA (2: a CTA walks several expert slots, filled by the launcher)
    int M_shared = -1;                   // rows the shared expert runs on (-1: all M) and where they start in p:
    int shared_row0 = 0;                 // expert-parallel calls see every rank's rows in p but own only some
    const __half* scores; const __half* sgl;   // combine inputs (down kernel)
    __half* resid;                       // residual stream updated in place, or nullptr ...
    __half* out;                         // ... then the block output goes here
    unsigned* tile_counter;              // [H/16] tickets, zero between launches; nullptr: no fused combine (dbuf only)
    // expert-parallel down projection: a routed pair's output row goes to the pair owner's buffer over peer memory
    // (rank = pair / ep_pairs_per_rank, row inside it = pair % ep_pairs_per_rank); nullptr entries: everything local
    __half* peer_dbuf[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    int ep_pairs_per_rank = 0;
    EpSignal ep_sig;                     // down kernel: its last CTA raises the combine flags
    PfList pf;                           // static prefetch (gate/up kernel: next layer's in-projection)
    // many-row kernels: the normed rows in the products' order (gemv.cuh) + their group sums (gate/up input), and the chunk sums of the
    // SwiGLU rows ([(M*topk + M)][I/8], written by gate/up, read by down; hbuf is then in that order too)
    const __half* xq = nullptr; const float* sxq = nullptr; float* csum = nullptr;
    bool stall = false;                  // test hook: the gate/up kernel in the form whose waits run out
};

struct GdnArgs {
    const __half* inproj; int ld;        // [M][ld]: qkv | z | b | a
    const float* conv_w; const float* A_log; const float* dt_bias;
    int Hk, Hv; float eps;
    StreamTable tab; int gdn_index;      // which GDN layer (index among GDN layers)
    const SegDesc* segs;
    __half* y;                           // [M][Hv*128]
    // two-kernel form (gdn_rows.cu): row -> segment, and the scratch between the kernels
    const int* row_seg = nullptr;
    float* qk = nullptr;                 // gdn_qk_floats(): normed, scaled k | q
    unsigned char* vg = nullptr;         // gdn_vg_bytes(): conv + SiLU of v, (decay, beta)
    int M = 0;                           // rows of the call (filled by the launcher)
    unsigned* err = nullptr;
    bool stall = false;                  // test hook: the scan in the form whose wait runs out
};

struct AttnArgs {
    const __half* inproj; int ld;        // [M][ld]: q(+gate) | k | v
    const __half* q_norm; const __half* k_norm;
    int NH, KV; float eps, theta;
    StreamTable tab; int attn_index;     // index among attention layers
    int n_attn_layers, page_size;
    __half* kv_pool;
    const SegDesc* segs; const int* row_seg; const int* row_off;   // per row: segment, offset inside it
    const int* row_pos_override;         // optional explicit positions (operator tests) or nullptr
    __half* qrot;                        // [M][NH][256]
    float* part_o; float* part_ml;       // split partials
    int nsplit;
    int max_keys = 0;                    // most keys of a row, where the host knows it (0: not): no CTAs for splits that cannot exist
    __half* gated;                       // [M][NH*256]
    int M;
};

#ifdef __CUDACC__
// The slot lists in shared memory with the prefix of their row blocks, for the kernels that walk (slot, block) items.
struct SlotTable { int base[260]; int expert[256], off[256], cnt[256]; int ws[8]; };   // base[n_active] = the shared expert's first block, base[n_active + 1] = total
// All threads of the CTA (256 at least) call it; every list entry is requested at once and the prefix is a block scan, so
// this costs one memory latency (a scan by one warp, 32 slots after 32, cost eight: 4 us ahead of the first weight).
// Returns n_active; the caller synchronises before it reads the table.
__device__ __forceinline__ int slot_table(SlotTable& t, const MoeLists& L, int rows_per_block, int nshared) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int na = *L.n_active;
    int nb = 0, inc = 0;
    if (tid < 256) {
        const int cnt = L.slot_cnt[tid], ex = L.slot_expert[tid], off = L.slot_off[tid];     // (entries past n_active: unused)
        t.cnt[tid] = cnt; t.expert[tid] = ex; t.off[tid] = off;
        nb = tid < na ? (cnt + rows_per_block - 1) / rows_per_block : 0;
        inc = nb;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const int o = __shfl_up_sync(0xffffffffu, inc, d); if (lane >= d) inc += o; }
        if (lane == 31) t.ws[warp] = inc;
    }
    __syncthreads();
    if (tid < 256) {
        for (int w = 0; w < warp; ++w) inc += t.ws[w];
        t.base[tid + 1] = inc;
        if (tid == 0) t.base[0] = 0;
    }
    __syncthreads();
    if (tid == 0) t.base[na + 1] = t.base[na] + (nshared + rows_per_block - 1) / rows_per_block;
    return na;
}
// (slot, block) index -> slot: the last j with base[j] <= sb
__device__ __forceinline__ int slot_of(const SlotTable& t, int n_active, int sb) {
    int lo = 0, hi = n_active;
    while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (t.base[mid] <= sb) lo = mid; else hi = mid - 1; }
    return lo;
}
// position of row m; address of (stream slot, position, K=0 / V=1, kv head) in the paged arena
__device__ __forceinline__ int row_position(const AttnArgs& a, int m) {
    if (a.row_pos_override) return a.row_pos_override[m];
    const SegDesc seg = a.segs[a.row_seg[m]];
    return a.tab.kv_len[seg.slot] + a.row_off[m];
}
__device__ __forceinline__ __half* kv_ptr(const AttnArgs& a, int slot, int pos, int which, int kvh) {
    int page = a.tab.page_table[(size_t)slot * a.tab.max_pages + pos / a.page_size];
    size_t page_elems = (size_t)a.n_attn_layers * 2 * a.KV * a.page_size * ATT_D;
    return a.kv_pool + (size_t)page * page_elems +
           ((((size_t)a.attn_index * 2 + which) * a.KV + kvh) * a.page_size + (pos % a.page_size)) * ATT_D;
}
#endif

struct StepEndArgs {
    StreamTable tab; const SegDesc* segs; int nsegs;
    const int* out_tok; int* tok_in; int* hist; int* hist_pos; int hist_cap; int M;
};

int sm_count();
// ---- the one-kernel decode step (step_persistent.cu) ----
struct PsGeom {
    int G;                                  // CTAs (one per multiprocessor)
    int H, I, E, topk, V;
    int Hk, Hv, NH, KV;
    int keyDim, valDim, convDim, gdn_in, attn_in, attn_out;
    int S_h, S_i;                           // 256-wide slices of K = H, K = I
    int gu_spp;                             // CTAs per expert slot in the gate/up phase
    int rows_per_sm;                        // gdn state rows per CTA (multiple of 4)
    int router_spr;                         // ring slots per router row
};
struct PLayer {                             // one layer's weights as the step kernel reads them (an array of these lives on the device)
    int is_attn, type_index;
    const __half *in_norm, *post_norm;
    Q4R r_in, r_out;
    const float *conv_w, *A_log, *dt_bias; const __half* gdn_norm; const float* gdn_norm32;
    const __half *q_norm, *k_norm;
    const __half *router, *shared_gate;     // fp16 forms only
    Q4R r_gu, r_down, r_sh_gu, r_sh_down;
};
struct PStepArgs {
    PsGeom geom;
    const PLayer* layers; int n_layers;
    const __half* embed; const __half* final_norm; Q4R lm_head;
    float eps, theta;
    StreamTable tab; const SegDesc* segs;
    __half* kv_pool; int n_attn_layers, page_size, nsplit;
    int *tok_in, *out_tok, *hist, *hist_pos; int hist_cap;
    unsigned* step_seq;                     // sequence number of the next step (device word, >= 1)
    // exchange lines (16 B each): per layer a block of x_stride lines, plus one block after the last layer
    int x_reps; size_t x_rep_stride;        // every exchange line exists in x_reps copies, x_rep_stride lines apart
    uint4* xbuf; size_t x_stride; int x_off_h, x_off_in, x_off_mix, x_off_hm, x_off_lg, x_off_hb, x_off_arg;
    uint4* xatt; size_t xatt_stride;        // attention partials, one block per attention layer
    unsigned* err; unsigned* abort_flag;
    uint32_t* timeline;                     // profiling: [CTA][layer + 1][24] nanosecond stamps, or nullptr
};
bool ps_plan(PsGeom& g, int n_sm);           // fills the derived fields; false if the step kernel cannot run this geometry here
int launch_step_persistent(const PStepArgs& a, cudaStream_t st);   // cooperative launch; returns a cudaError_t

void launch_dense(int pro, int epi, const DenseArgs& a, cudaStream_t st, bool pdl);
// many-row forms (more than one row per call); the bool launchers return false when the shape is not covered
inline bool dense_rows_shape(int M, int N, int K) { return M > 1 && K % 256 == 0 && K <= 4096 && N % 16 == 0; }
bool launch_dense_rows(int pro, int epi, const DenseArgs& a, cudaStream_t st, bool pdl);
bool launch_head_rows(const DenseArgs& a, cudaStream_t st, bool pdl);      // lm_head + argmax behind the final norm
void launch_rows_prep_plain(const __half* x, int ldx, int M, int K, __half* xq, float* sxq, cudaStream_t st, bool pdl);
// prefill mode: the experts of a prompt chunk as grouped GEMMs on the tensor cores (pair lists as built by the router); hbuf in natural order
bool launch_expert_tc_gateup(const ExpertArgs& a, cudaStream_t st, bool pdl);
bool launch_expert_tc_down(const ExpertArgs& a, cudaStream_t st, bool pdl);
// router for many rows: a.h holds rows that are already normed; logits kernel + routing / pair lists kernel
bool launch_router_rows(const RouterArgs& a, cudaStream_t st, bool pdl);
bool launch_router_mma(const RouterArgs& a, cudaStream_t st, bool pdl);    // prefill mode, fp16 router: logits on the tensor cores
bool expert_rows_route(const ExpertArgs& a);     // may the expert kernels of this call route for themselves (route_here)?
bool launch_expert_rows_gateup(const ExpertArgs& a, cudaStream_t st, bool pdl);
bool launch_expert_rows_down(const ExpertArgs& a, cudaStream_t st, bool pdl);
// xq / sxq (optional): the rows also normed with nw and prepared for the next layer's in-projection (H a multiple of 256, <= 4096);
// xq alone: normed as plain rows
void launch_moe_combine(const __half* dbuf, const __half* shared_rows, const __half* scores, const __half* sgl, int M, int H, int topk,
                        __half* resid, __half* out, cudaStream_t st, bool pdl, const __half* nw = nullptr, float eps = 0.f, __half* xq = nullptr, float* sxq = nullptr);
// many-row GEMM on tcgen05 tensor cores with the accumulator in tensor memory (N % 16 == 0, K % 256 == 0); 0 or an error code
int launch_gemm_tc(const Q4R& q, int N, int K, int M, const __half* x, int ldx, __half* y, int ldy, bool add_to_y, unsigned* err, cudaStream_t st, bool pdl);
// speculative-sampling rows on fp16 logits [M][V]: categorical draw, draw without the draft token, accept flag
void launch_sample_rows(const __half* logits, const float* adj /*[V] added to every row, or nullptr*/, const int* draft, int* samp_full, int* samp_resid, int* accept, int M, int V,
                        float invT, float top_p, uint32_t seed_lo, uint32_t seed_hi, uint32_t base_pos, cudaStream_t st);
// lm_head + argmax whose scratch is a fixed module-scope device array; returns 0 or a cudaError_t
int launch_head_static(const DenseArgs& a, cudaStream_t st);
int head_static_max_rows();
void launch_embed(const __half* embed, const int* tokens, int M, int H, int vocab, __half* h, cudaStream_t st);
void launch_embed_dequant_q4(const uint32_t* w, const __half* s, const __half* b, __half* out, int64_t vocab, int H, cudaStream_t st);
void launch_router(const RouterArgs& a, cudaStream_t st, bool pdl);
void launch_expert_gateup(const ExpertArgs& a, int nslots, cudaStream_t st, bool pdl);
void launch_expert_down(const ExpertArgs& a, int nslots, cudaStream_t st, bool pdl);
// batch-1 decode: gate/up and down in ONE launch (a per-slot barrier between the phases); false if the shapes do not fit it
bool launch_expert_fused(const ExpertArgs& a, cudaStream_t st, bool pdl);
bool expert_fused_applicable(const ExpertArgs& a);      // the shape test launch_expert_fused applies
// expert-parallel exchange (ep_exchange.cu)
void launch_ep_lists(const EpPeers& P, int npairs, int e0, int e1, const MoeLists& lists, int layer, unsigned* err, cudaStream_t st);
void launch_ep_combine(const EpPeers& P, const __half* shared_rows, const __half* scores, const __half* sgl, int M, int H, int topk,
                       __half* resid, __half* out, int layer, unsigned* err, cudaStream_t st);
void launch_ep_step_end(unsigned* ctr, cudaStream_t st);
void launch_gdn_core(const GdnArgs& a, int nsegs, cudaStream_t st, bool pdl);
// prefill-mode attention of one stream's chunk on the tensor cores (after launch_attn_prep); false: call not covered
bool launch_attn_prefill(const AttnArgs& a, int nsegs, cudaStream_t st, bool pdl);
void launch_gdn_rows(const GdnArgs& a, int M, int nsegs, cudaStream_t st, bool pdl);   // the same result by k_gdn_prep + k_gdn_scan (needs the scratch fields)
size_t gdn_qk_floats(int Hk, int rows); size_t gdn_vg_bytes(int Hv, int rows);
void launch_attn_prep(const AttnArgs& a, cudaStream_t st, bool pdl);
// q/k prep (when every row is its stream's only row) + split-KV decode + merge in one launch; counters: 2*M*KV zeros
void launch_attn_fused(const AttnArgs& a, bool prep, unsigned* counters, cudaStream_t st, bool pdl);
void launch_step_end(const StepEndArgs& a, cudaStream_t st);
// xq / sxq (optional): the normed rows also in the prepared form of the many-row kernels
void launch_final_norm(const __half* h, const __half* w, float eps, int M, int H, __half* out, cudaStream_t st, bool pdl, __half* xq = nullptr, float* sxq = nullptr);
// expert-parallel: the normed rows also go into every rank's gather buffer (RouterArgs::ep_rows_sent then tells the routing kernel)
void launch_final_norm_ep(const __half* h, const __half* w, float eps, int M, int H, __half* out, const EpDispatch& epd, cudaStream_t st);
void launch_wait_probe(unsigned* err, cudaStream_t st);   // test hook: a bounded wait that runs out sets bit 2 of *err
int64_t kernel_launch_count();
void count_launch();
void count_launches(int64_t n);
// run `fn` (one kernel launch) between the profiling events of `tag` when profiling is on, and count it
void profile_launch(const char* tag, cudaStream_t st, const std::function<int()>& fn);
// k<<<grid, threads, smem, st>>>(args...); pdl: as a programmatic dependent launch (k waits for its predecessor itself)
template <class... P, class... A>
inline int launch_pdl(bool pdl, void (*k)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    if (pdl) { cfg.attrs = attr; cfg.numAttrs = 1; }
    return (int)cudaLaunchKernelEx(&cfg, k, P(args)...);
}
void profile_start();
int profile_report(char* buf, size_t cap);

// ---- stream state <-> host blob (state_io.cu) ----
struct StateIoArgs {
    int n_layers, attn_every, n_attn, kv_heads, page_size, len;
    uint32_t hist_words, state_words;       // 4-byte words of one GDN layer's conv history / state
    float* state; __half* hist;             // current side of the stream, GDN layers in order
    __half* kv_pool; const int* pages;      // the stream's page table row (device)
};
struct StateIoRing {                        // page-locked slots and their device counterparts (32 MB each), made at the first use
    uint8_t *pinned = nullptr, *dev = nullptr;
    cudaEvent_t done[16] = {};
    int init();                             // 0 or a cudaError_t; after a failure nothing is held, and it may be tried again
    void destroy();
};
// (the ring initialised) copies the whole blob out of (save) or into the stream's caches; when it returns, a save is complete in `host` and a
// restore has read all of `host` (its device work may still be in flight on st).  0 or a cudaError_t.
int state_io(StateIoRing& ring, const StateIoArgs& a, bool save, uint8_t* host, size_t bytes, cudaStream_t st);
void launch_set_pages(int* dst, const int* pages, int n, cudaStream_t st);     // dst[i] = pages[i]; pages (host) is read before the call returns
void launch_set_len_parity(const StreamTable& tab, int slot, int len, int parity, cudaStream_t st);

// synthetic data + quantiser (synth.cu)
uint64_t tensor_seed(uint64_t base_seed, const char* name);
void launch_synth_f16(uint64_t tseed, int64_t n, float mean, float std, __half* out, cudaStream_t st);
void launch_synth_f32(uint64_t tseed, int64_t n, float mean, float std, float* out, cudaStream_t st);
void launch_synth_q4(uint64_t tseed, int64_t N, int64_t K, float std, uint32_t* packed, __half* s, __half* b, cudaStream_t st);
void launch_quantize_q4(const __half* w, int64_t N, int64_t K, uint32_t* packed, __half* s, __half* b, cudaStream_t st);
void host_synth_tokens(uint64_t tseed, int64_t n, int32_t vocab, int32_t* out);
// MLX affine layout -> fragment-major layout; pair != 0: tile = 8 rows of A + the same 8 rows of B
void launch_repack_q4(const Q4W& a, const Q4W* b_pair, uint4* wr, uint4* sr, cudaStream_t st);

}  // namespace sl
