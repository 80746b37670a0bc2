// A stand-in for the CUDA runtime on the host, for tests of the library's host side without a GPU: preloaded in front of
// libcudart, it gives "device" memory from the heap, runs copies at once and kernels not at all, and makes the calls fail that a
// test asks it to fail.  Of the kernels only k_state_io is imitated: packing leaves each word's number, unpacking notes what
// arrived for each word.  Found as libnccl.so.2 as well, it is that library for a rank whose peers do not exist.
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
std::mutex mu;
std::map<std::string, long> counts;
std::map<const void*, std::string> kernels;
std::map<std::pair<std::string, unsigned>, long> launched;   // by kernel and threads of a block
std::map<uint64_t, uint32_t> unpacked;
const pthread_t main_thread = pthread_self();
thread_local cudaError_t last = cudaSuccess;              // as the runtime keeps it: per host thread
struct Config { dim3 grid, block; size_t smem; void* stream; };
thread_local Config config;
size_t fail_bytes = 0;
bool fail_graphs = false;
std::atomic<long> threads_left{-1}, launches_left{-1};
bool capturing = false;

void note(const char* what) {
    std::lock_guard<std::mutex> l(mu);
    ++counts[what];
    if (!pthread_equal(pthread_self(), main_thread)) ++counts["other_thread"];
}
cudaError_t ret(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
cudaError_t alloc(const char* what, void** p, size_t n) {
    note(what);
    if (n == fail_bytes) return ret(cudaErrorMemoryAllocation);
    *p = calloc(1, n);
    return ret(*p ? cudaSuccess : cudaErrorMemoryAllocation);
}
cudaError_t launch(const void* f, unsigned threads, void** args) {
    note("launches");
    if (launches_left.load() >= 0 && launches_left.fetch_sub(1) <= 0) return ret(cudaErrorLaunchOutOfResources);
    std::string name;
    { std::lock_guard<std::mutex> l(mu); name = kernels[f]; ++launched[{name, threads}]; }
    if (!capturing && name.find("k_state_io") != std::string::npos) {        // (StateIoArgs, first word, words, slot)
        const uint64_t w0 = *static_cast<uint64_t*>(args[1]);
        const unsigned n = *static_cast<unsigned*>(args[2]);
        uint32_t* buf = *static_cast<uint32_t**>(args[3]);
        if (name.find("ILb1E") != std::string::npos) for (unsigned i = 0; i < n; ++i) buf[i] = (uint32_t)(w0 + i);
        else { std::lock_guard<std::mutex> l(mu); for (unsigned i = 0; i < n; ++i) unpacked[w0 + i] = buf[i]; }
    }
    return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- what a test sees and sets
long fake_count(const char* what) { std::lock_guard<std::mutex> l(mu); return counts[what]; }
void fake_fail_alloc(size_t bytes) { fail_bytes = bytes; }                    // allocations of exactly this size fail (0: none)
void fake_fail_threads(long after) { threads_left = after; }                  // thread starts fail after that many (-1: none)
void fake_fail_launches(long after) { launches_left = after; }                // kernel launches fail after that many (-1: none)
void fake_fail_graphs(int on) { fail_graphs = on != 0; }                      // no memory for graphs
long fake_launched(const char* part, unsigned threads) {                      // launches of kernels with this in their name and blocks of so many threads
    std::lock_guard<std::mutex> l(mu);
    long n = 0;
    for (auto& kv : launched) if (kv.first.second == threads && kv.first.first.find(part) != std::string::npos) n += kv.second;
    return n;
}
long fake_unpacked(uint32_t* out, long n) {                                   // words that arrived, in order; -1 if one is missing
    std::lock_guard<std::mutex> l(mu);
    if ((long)unpacked.size() != n) return -1;
    for (auto& kv : unpacked) { if ((long)kv.first >= n) return -1; out[kv.first] = kv.second; }
    unpacked.clear();
    return n;
}

int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
    using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    static Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
    if (threads_left.load() >= 0 && threads_left.fetch_sub(1) <= 0) return EAGAIN;
    { std::lock_guard<std::mutex> l(mu); ++counts["threads"]; }
    return real(t, a, f, arg);
}

// ---- registration and launches
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { kernels[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) { config = {g, b, s, st}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) { *g = config.grid; *b = config.block; *s = config.smem; *static_cast<void**>(st) = config.stream; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3 b, void** args, size_t, cudaStream_t) { return launch(f, b.x, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) { return launch(f, c->blockDim.x, args); }

// ---- devices
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { note("set_device"); return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char room[1 << 16]; *p = room; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "error of the stand-in"; }

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) { return alloc("malloc", p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return alloc("malloc_host", p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return alloc("malloc_host", p, n); }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { note("memcpy_async"); if (!capturing) memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { if (!capturing) memset(d, v, n); return cudaSuccess; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t* h, void*) { memset(h, 0, sizeof *h); return cudaSuccess; }
cudaError_t cudaIpcOpenMemHandle(void** p, cudaIpcMemHandle_t, unsigned) { *p = calloc(1, 1 << 22); return ret(*p ? cudaSuccess : cudaErrorMemoryAllocation); }      // (a peer's memory, never written)
cudaError_t cudaIpcCloseMemHandle(void* p) { free(p); return cudaSuccess; }

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(new char); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete reinterpret_cast<char*>(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { note("stream_sync"); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(new char); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<char*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { note("event_record"); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { note("event_sync"); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    note("captures");
    if (s == nullptr || s == cudaStreamLegacy) return ret(cudaErrorStreamCaptureUnsupported);
    capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { capturing = false; *g = reinterpret_cast<cudaGraph_t>(new char); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { if (fail_graphs) return ret(cudaErrorMemoryAllocation); note("graphs_made"); *x = reinterpret_cast<cudaGraphExec_t>(new char); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<char*>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { note("graphs_dropped"); delete reinterpret_cast<char*>(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { note("graph_launches"); return cudaSuccess; }

// ---- NCCL
struct FakeNcclId { char bytes[128]; };
int ncclGetUniqueId(FakeNcclId*) { return 0; }
int ncclCommInitRank(void** c, int, FakeNcclId, int) { *c = new char; return 0; }
int ncclCommDestroy(void* c) { delete static_cast<char*>(c); return 0; }
int ncclAllGather(const void*, void*, size_t, int, void*, cudaStream_t) { return 0; }
int ncclReduceScatter(const void*, void*, size_t, int, int, void*, cudaStream_t) { return 0; }
int ncclGroupStart() { return 0; }
int ncclGroupEnd() { return 0; }
const char* ncclGetErrorString(int) { return "error of the stand-in"; }
}
