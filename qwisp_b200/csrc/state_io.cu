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

#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

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
static cudaError_t launch_state_io(bool pack, const StateIoArgs& a, uint64_t w0, unsigned n, uint32_t* buf, cudaStream_t st) {
    const unsigned grid = (n + 1023) / 1024;
    if (pack) k_state_io<true><<<grid, 256, 0, st>>>(a, w0, n, buf);
    else k_state_io<false><<<grid, 256, 0, st>>>(a, w0, n, buf);
    count_launch();
    return cudaGetLastError();
}

constexpr size_t SIO_SLOT = (size_t)2 << 20;                  // bytes of a slot: about 40 us on the link
constexpr int SIO_THREADS = 8, SIO_SLOTS = 2 * SIO_THREADS;
static_assert(sizeof(StateIoRing::done) == SIO_SLOTS * sizeof(cudaEvent_t), "an event per slot");

int StateIoRing::init() {
    if (pinned) return 0;
    const size_t bytes = SIO_SLOT * SIO_SLOTS;
    cudaError_t e = cudaMallocHost(&pinned, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&dev, bytes);
    for (int i = 0; i < SIO_SLOTS && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming);
    if (e != cudaSuccess) { destroy(); cudaGetLastError(); }
    return (int)e;
}
void StateIoRing::destroy() {
    for (cudaEvent_t& ev : done) if (ev) { cudaEventDestroy(ev); ev = nullptr; }
    if (pinned) { cudaFreeHost(pinned); pinned = nullptr; }
    if (dev) { cudaFree(dev); dev = nullptr; }
}
// The copies between the caller's memory and the slots.  Range c of the blob goes by way of slot c % SIO_SLOTS; ranges are posted in
// order, and threads that are started as ranges are posted copy them (the calling thread if there is none).
// These threads make no CUDA call: all of those are the calling thread's, so its stream (a per-thread one, say), its context and
// its error state are the only ones.  It keeps the link and the threads supplied and copies nothing itself meanwhile: with its
// help 85 MB took 8.5 ms there and back, without 7.7 (7.8 when every thread moved its own ranges all the way).
struct SioCopies {
    const bool save;
    uint8_t* const host;
    uint8_t* const slots;
    const size_t bytes;
    int most;                                                 // threads
    std::mutex m;
    std::condition_variable work, copied;
    size_t posted = 0, taken = 0, done[SIO_SLOTS] = {};       // done: ranges copied by way of a slot
    bool stop = false;
    int started = 0;
    std::thread pool[SIO_THREADS];

    SioCopies(bool save_, uint8_t* host_, uint8_t* slots_, size_t bytes_, int most_) : save(save_), host(host_), slots(slots_), bytes(bytes_), most(most_) {}
    ~SioCopies() {
        { std::lock_guard<std::mutex> l(m); stop = true; taken = posted; }
        work.notify_all();
        for (int i = 0; i < started; ++i) pool[i].join();
    }
    size_t length(size_t c) const { return bytes - c * SIO_SLOT < SIO_SLOT ? bytes - c * SIO_SLOT : SIO_SLOT; }
    void copy(size_t c) {
        uint8_t *h = host + c * SIO_SLOT, *p = slots + c % SIO_SLOTS * SIO_SLOT;
        if (save) memcpy(h, p, length(c)); else memcpy(p, h, length(c));
    }
    void take(std::unique_lock<std::mutex>& l) {              // the next posted range; l is held before and after
        const size_t c = taken++;
        l.unlock();
        copy(c);
        l.lock();
        ++done[c % SIO_SLOTS];
        copied.notify_one();
    }
    void run() {
        std::unique_lock<std::mutex> l(m);
        for (;;) {
            work.wait(l, [&] { return stop || taken < posted; });
            if (taken >= posted) return;
            take(l);
        }
    }
    void post() {                                             // range `posted`
        if (started < most) {                                 // (no thread to be had: the ones there are, or the caller, do the work)
            try { pool[started] = std::thread([this] { run(); }); ++started; } catch (...) { most = started; }
        }
        std::unique_lock<std::mutex> l(m);
        ++posted;
        if (started) work.notify_one(); else take(l);
    }
    void wait(size_t c) {                                     // until range c has been copied
        std::unique_lock<std::mutex> l(m);
        copied.wait(l, [&] { return done[c % SIO_SLOTS] > c / SIO_SLOTS; });
    }
};
// Half of the slots are on their way between device and slot, half between slot and caller's memory.
int state_io(StateIoRing& ring, const StateIoArgs& a, bool save, uint8_t* host, size_t bytes, cudaStream_t st) {
    // a thread per four ranges (8 MB): starting one costs about what copying a megabyte does
    int T = (int)(bytes / (4 * SIO_SLOT));
    const int cores = (int)std::thread::hardware_concurrency();
    if (T > SIO_THREADS) T = SIO_THREADS;
    if (cores > 0 && T > cores) T = cores;
    SioCopies copies(save, host, ring.pinned, bytes, T > 1 ? T : 0);
    const size_t n = (bytes + SIO_SLOT - 1) / SIO_SLOT;
    cudaError_t e = cudaSuccess;
    auto enqueue = [&](size_t c) {
        const size_t s = c % SIO_SLOTS, len = copies.length(c);
        uint8_t *pin = ring.pinned + s * SIO_SLOT, *dev = ring.dev + s * SIO_SLOT;
        if (save) {
            e = launch_state_io(true, a, c * (SIO_SLOT / 4), (unsigned)(len / 4), (uint32_t*)dev, st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(pin, dev, len, cudaMemcpyDeviceToHost, st);
        } else {
            e = cudaMemcpyAsync(dev, pin, len, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = launch_state_io(false, a, c * (SIO_SLOT / 4), (unsigned)(len / 4), (uint32_t*)dev, st);
        }
        if (e == cudaSuccess) e = cudaEventRecord(ring.done[s], st);
    };
    auto landed = [&](size_t c) { e = cudaEventSynchronize(ring.done[c % SIO_SLOTS]); };
    if (save) {
        size_t sent = 0;
        for (size_t c = 0; c < n && e == cudaSuccess; ++c) {
            for (; sent < n && sent < c + SIO_SLOTS / 2 && e == cudaSuccess; ++sent) {
                if (sent >= SIO_SLOTS) copies.wait(sent - SIO_SLOTS);            // the slot's last range has left it
                enqueue(sent);
            }
            if (e == cudaSuccess) landed(c);
            if (e == cudaSuccess) copies.post();
        }
        if (e == cudaSuccess) for (size_t c = n < SIO_SLOTS ? 0 : n - SIO_SLOTS; c < n; ++c) copies.wait(c);
    } else {
        const size_t ahead = copies.most ? SIO_SLOTS / 2 : 1;
        size_t posted = 0;
        for (size_t c = 0; c < n && e == cudaSuccess; ++c) {
            for (; posted < n && posted < c + ahead && e == cudaSuccess; ++posted) {
                if (posted >= SIO_SLOTS) landed(posted - SIO_SLOTS);
                if (e == cudaSuccess) copies.post();
            }
            if (e == cudaSuccess) { copies.wait(c); enqueue(c); }
        }
    }
    return (int)e;
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
