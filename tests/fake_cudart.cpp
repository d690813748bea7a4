// A CUDA runtime without a GPU for CPU tests of host code: devices, function attributes, launches and the order that events
// give to streams are only recorded. A stream is a count of the work queued on it; an event holds the counts that have to
// be reached before it, and a host that waits for it knows that they are. Nothing else tells the host: cudaFree and
// cudaDeviceSynchronize do not wait here.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdlib>
#include <map>
#include <utility>

namespace {
int device = 0, launches = 0, refused = 0, unordered_frees = 0, recorded_in_capture = 0, blocks = 0;
size_t config_shared = 0;
unsigned long long reserved = 0;
std::map<std::pair<int, const void*>, int> shared_allowed, times_allowed;
using Order = std::map<void*, long>;  // per stream, how much of its work comes before
std::map<void*, Order> streams, events;
Order host;  // what the host has seen finished
std::map<void*, bool> capturing;
template <typename H> H made() { return static_cast<H>(static_cast<void*>(std::malloc(16))); }
void later(Order& a, const Order& b) {
    for (auto& kv : b) a[kv.first] = std::max(a[kv.first], kv.second);
}
}  // namespace

extern "C" {
// Launches in all, those above the shared memory that their device allows them, and the most opt-ins a kernel got on one.
int fake_launches() { return launches; }
int fake_refused() { return refused; }
int fake_most_opt_ins() {
    int most = 0;
    for (auto& kv : times_allowed) most = std::max(most, kv.second);
    return most;
}
// Queues work on a stream (or has a capture record it); blocks given back to a pool while work was queued on some stream
// that the host had not seen finished; events recorded on a stream that a capture had; blocks handed out and not given
// back.
void fake_work(cudaStream_t s) { streams[s][s] += !capturing[s]; }
void fake_capture(cudaStream_t s, int on) { capturing[s] = on != 0; }
int fake_unordered_frees() { return unordered_frees; }
int fake_recorded_in_capture() { return recorded_in_capture; }
int fake_blocks() { return blocks; }
void fake_reserve(unsigned long long n) { reserved = n; }  // what every pool holds

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = made<cudaStream_t>();
    streams[*s][*s] = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* status) {
    *status = capturing[s] ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t s) { return streams[s][s] > host[s] ? cudaErrorNotReady : cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = made<cudaEvent_t>();
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (capturing[s]) ++recorded_in_capture;
    events[e] = streams[s];
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    later(host, events[e]);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    events.erase(e);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    *p = made<cudaMemPool_t>();
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void* v) {
    *static_cast<unsigned long long*>(v) = reserved;
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t) {
    *p = made<void*>();
    ++blocks;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void*, cudaStream_t) {
    --blocks;
    unordered_frees += std::any_of(streams.begin(), streams.end(), [](auto& s) { return s.second[s.first] > host[s.first]; });
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t) {
    *p = made<void*>();
    return cudaSuccess;
}
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t s) {
    fake_work(s);
    return cudaSuccess;
}

cudaError_t cudaGetDevice(int* d) {
    *d = device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    device = d;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        shared_allowed[{device, f}] = v;
        ++times_allowed[{device, f}];
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t shared, cudaStream_t) {
    ++launches;
    const auto it = shared_allowed.find({device, f});
    if (shared <= 48 * 1024 || (it != shared_allowed.end() && (size_t)it->second >= shared)) return cudaSuccess;
    ++refused;
    return cudaErrorInvalidValue;
}
// what nvcc's host code calls
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t shared, void*) {
    config_shared = shared;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* shared, void* stream) {
    *g = *b = dim3(1);
    *shared = config_shared;
    *static_cast<void**>(stream) = nullptr;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 0; }
}
