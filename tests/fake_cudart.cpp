// A CUDA runtime without a GPU for CPU tests of host code: devices, function attributes and launches are only recorded.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <map>
#include <utility>

namespace {
int device = 0, launches = 0, refused = 0;
size_t config_shared = 0;
std::map<std::pair<int, const void*>, int> shared_allowed, times_allowed;
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
