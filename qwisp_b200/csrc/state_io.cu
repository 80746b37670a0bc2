// state_io.cu -- a stream's caches as the self-describing "QWS1" blob (persistentStateData / restorePersistentState,
// swift/Sources/QwispCore/SeedlessFusedVerify.swift:4077-4154), moved between the device and pageable host memory.
//
// The blob is a sequence of 4-byte words: file header, then per layer its header and its data (conv history and state of a
// GDN layer; K and V of every kv head, positions in order, of an attention layer).  Its pieces lie in some 700 places of
// the device memory of a 1024-token stream, and the host buffer is pageable.  One copy call per piece took 36 ms for an
// 85 MB save + restore: each is staged by the driver on one host thread.  Here the word -> place map is arithmetic, so a
// kernel packs (or unpacks) any range of the blob, and the ranges travel through page-locked slots that several host
// threads fill or drain (the host's page faults and copies are what takes the time; the link needs 1.6 ms for 85 MB).
#include "kernels.h"

#include <cstring>
#include <thread>
#include <vector>

namespace sl {

struct BlobPlace { uint32_t* dev; uint32_t header; };         // dev == nullptr: a header word

__device__ __forceinline__ BlobPlace blob_place(const StateIoArgs& a, uint64_t w) {
    if (w < 3) return {nullptr, w == 0 ? 0x31535751u : (w == 1 ? 1u : (uint32_t)a.n_layers)};
    w -= 3;
    const uint64_t gw = 3 + a.hist_words + a.state_words;     // words of a GDN / attention layer
    const uint64_t hw = (uint64_t)a.len * (ATT_D / 2), aw = 4 + 2 * (uint64_t)a.kv_heads * hw;
    const uint64_t period = (a.attn_every - 1) * gw + aw;     // layers come as (attn_every - 1) GDN layers and an attention layer
    const uint64_t p = w / period;
    uint64_t r = w - p * period;
    if (r < (a.attn_every - 1) * gw) {
        const uint64_t i = r / gw, li = p * (a.attn_every - 1) + i;
        r -= i * gw;
        if (r < 3) return {nullptr, r == 0 ? 2u : (r == 1 ? a.hist_words * 2 : a.state_words)};
        r -= 3;
        if (r < a.hist_words) return {reinterpret_cast<uint32_t*>(a.hist) + li * a.hist_words + r, 0u};
        return {reinterpret_cast<uint32_t*>(a.state) + li * a.state_words + (r - a.hist_words), 0u};
    }
    r -= (a.attn_every - 1) * gw;
    if (r < 4) return {nullptr, r == 0 ? 1u : (r == 1 ? (uint32_t)a.kv_heads : (r == 2 ? (uint32_t)ATT_D : (uint32_t)a.len))};
    r -= 4;
    const uint64_t plane = r / hw;                            // which * kv_heads + head
    r -= plane * hw;
    const int pos = (int)(r / (ATT_D / 2));
    const size_t page_elems = (size_t)a.n_attn * 2 * a.kv_heads * a.page_size * ATT_D;
    __half* e = a.kv_pool + (size_t)a.pages[pos / a.page_size] * page_elems + (((size_t)p * 2 * a.kv_heads + plane) * a.page_size + pos % a.page_size) * ATT_D;
    return {reinterpret_cast<uint32_t*>(e) + r % (ATT_D / 2), 0u};
}
template <bool PACK>
__global__ void __launch_bounds__(256) k_state_io(StateIoArgs a, uint64_t w0, unsigned n, uint32_t* buf) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const BlobPlace b = blob_place(a, w0 + i);
        if (PACK) buf[i] = b.dev ? *b.dev : b.header;
        else if (b.dev) *b.dev = buf[i];
    }
}
static void launch_state_io(bool pack, const StateIoArgs& a, uint64_t w0, unsigned n, uint32_t* buf, cudaStream_t st) {
    const unsigned grid = (n + 1023) / 1024;
    if (pack) k_state_io<true><<<grid, 256, 0, st>>>(a, w0, n, buf);
    else k_state_io<false><<<grid, 256, 0, st>>>(a, w0, n, buf);
    count_launch();
}

constexpr size_t SIO_SLOT = (size_t)2 << 20;                  // bytes of a slot: about 40 us on the link
constexpr int SIO_THREADS = 8;

int StateIoRing::init() {
    if (pinned) return 0;
    const size_t bytes = SIO_SLOT * 2 * SIO_THREADS;
    cudaError_t e = cudaMallocHost(&pinned, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&dev, bytes);
    for (int i = 0; i < 2 * SIO_THREADS && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming);
    if (e != cudaSuccess) { destroy(); cudaGetLastError(); }
    return (int)e;
}
void StateIoRing::destroy() {
    for (cudaEvent_t& ev : done) if (ev) { cudaEventDestroy(ev); ev = nullptr; }
    if (pinned) { cudaFreeHost(pinned); pinned = nullptr; }
    if (dev) { cudaFree(dev); dev = nullptr; }
}
// Ranges t, t + T, t + 2T, ... of the blob by thread t through its two slots.
static cudaError_t sio_worker(StateIoRing& ring, const StateIoArgs& a, bool save, uint8_t* host, size_t bytes, int t, int T, int device, cudaStream_t st) {
    cudaError_t e = cudaSetDevice(device);
    const size_t n = (bytes + SIO_SLOT - 1) / SIO_SLOT;
    auto range = [&](size_t c, size_t& off, size_t& len) { off = c * SIO_SLOT; len = bytes - off < SIO_SLOT ? bytes - off : SIO_SLOT; };
    auto slot = [&](size_t k) { return (size_t)t * 2 + (k & 1); };
    auto drain = [&](size_t c, size_t k) {                    // save: the range has arrived in its slot
        size_t off, len; range(c, off, len);
        cudaError_t r = cudaEventSynchronize(ring.done[slot(k)]);
        if (r == cudaSuccess) memcpy(host + off, ring.pinned + slot(k) * SIO_SLOT, len);
        return r;
    };
    size_t k = 0;
    for (size_t c = t; c < n && e == cudaSuccess; c += T, ++k) {
        size_t off, len; range(c, off, len);
        uint8_t* pin = ring.pinned + slot(k) * SIO_SLOT;
        uint8_t* dev = ring.dev + slot(k) * SIO_SLOT;
        if (save) {
            if (k >= 2 && (e = drain(c - 2 * T, k - 2)) != cudaSuccess) break;
            launch_state_io(true, a, off / 4, (unsigned)(len / 4), (uint32_t*)dev, st);
            e = cudaMemcpyAsync(pin, dev, len, cudaMemcpyDeviceToHost, st);
        } else {
            if (k >= 2 && (e = cudaEventSynchronize(ring.done[slot(k)])) != cudaSuccess) break;    // the slot's last range has left it
            memcpy(pin, host + off, len);
            e = cudaMemcpyAsync(dev, pin, len, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) launch_state_io(false, a, off / 4, (unsigned)(len / 4), (uint32_t*)dev, st);
        }
        if (e == cudaSuccess) e = cudaEventRecord(ring.done[slot(k)], st);
    }
    if (save)
        for (size_t i = k < 2 ? 0 : k - 2; i < k && e == cudaSuccess; ++i) e = drain((size_t)t + i * T, i);
    return e;
}
int state_io(StateIoRing& ring, const StateIoArgs& a, bool save, uint8_t* host, size_t bytes, cudaStream_t st) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return (int)e;
    // a thread per four ranges (8 MB): starting one costs about what copying a megabyte does
    int T = (int)(bytes / (4 * SIO_SLOT));
    const int cores = (int)std::thread::hardware_concurrency();
    if (T > SIO_THREADS) T = SIO_THREADS;
    if (cores > 0 && T > cores) T = cores;
    if (T < 1) T = 1;
    std::vector<cudaError_t> rc((size_t)T, cudaSuccess);
    std::vector<std::thread> pool;
    for (int t = 1; t < T; ++t) pool.emplace_back([&, t] { rc[(size_t)t] = sio_worker(ring, a, save, host, bytes, t, T, device, st); });
    rc[0] = sio_worker(ring, a, save, host, bytes, 0, T, device, st);
    for (std::thread& th : pool) th.join();
    for (cudaError_t r : rc) if (r != cudaSuccess) return (int)r;
    return 0;
}

__global__ void k_set_len_parity(StreamTable tab, int slot, int len, int parity) { tab.kv_len[slot] = len; tab.parity[slot] = parity; }
void launch_set_len_parity(const StreamTable& tab, int slot, int len, int parity, cudaStream_t st) {
    k_set_len_parity<<<1, 1, 0, st>>>(tab, slot, len, parity);
    count_launch();
}

struct PageRun { int page[64]; };
__global__ void k_set_pages(int* dst, PageRun r, int n) { if ((int)threadIdx.x < n) dst[threadIdx.x] = r.page[threadIdx.x]; }
void launch_set_pages(int* dst, const int* pages, int n, cudaStream_t st) {
    for (int i = 0; i < n; i += 64) {
        PageRun r; const int m = n - i < 64 ? n - i : 64;
        memcpy(r.page, pages + i, (size_t)m * sizeof(int));
        k_set_pages<<<1, 64, 0, st>>>(dst + i, r, m);
        count_launch();
    }
}

}  // namespace sl
