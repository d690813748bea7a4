// hostio.cu -- see hostio.cuh.
#include "hostio.cuh"

#include <algorithm>

#include "context.cuh"

namespace simk {

// ---- freed device blocks ---------------------------------------------------------------------------------------------
// cudaMalloc and cudaFree of a call's temporaries and of a potential's slices took 50-300 us each, half of a small HRTEM
// image, and now and then a fresh block tens of ms on a busy host. (A list of freed blocks that were never split or joined
// missed on each new potential: 512^2 scan, first pass 154-215 ms, now 154; 768^2 phonons 18-36, now 17; a new job table
// 42, now 34.) Blocks of up to kLargest come from one memory pool a device, which splits and joins what it holds and
// grows by whole chunks; at most kKept bytes beyond the blocks in use stay there. Every block goes back only after the
// device has finished everything queued, as cudaFree waits, and the pool's stream is idle when one is handed out, so any
// stream and thread may take it next. When the last context goes, so does what the pool holds free.
namespace {
constexpr size_t kKept = 512u << 20;
constexpr size_t kLargest = 256u << 20;
struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;  // orders the pool's operations
    void* fence = nullptr;          // a small block that wait_as_free trades for a new one
    size_t live = 0;                // bytes handed out
    int contexts = 0;
};
std::mutex g_pools_mutex;
DevicePool& device_pool(int device) {
    static auto* m = new std::map<int, DevicePool>();  // never destroyed: buffers may be released at exit
    return (*m)[device];
}
void open_pool(DevicePool& d, int device) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    SIMK_CUDA(cudaMemPoolCreate(&d.pool, &props));
    unsigned long long hold = ~0ULL;  // what stays is bounded in device_free
    SIMK_CUDA(cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &hold));
    SIMK_CUDA(cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking));
    SIMK_CUDA(cudaMalloc(&d.fence, 512));
}
cudaError_t pool_alloc(DevicePool& d, void** p, size_t n) {
    const cudaError_t e = cudaMallocFromPoolAsync(p, n, d.pool, d.stream);
    return e == cudaSuccess ? cudaStreamSynchronize(d.stream) : e;
}
// Waits for everything queued on the device, as cudaFree does and by cudaFree itself: cudaDeviceSynchronize in one thread
// breaks off the stream capture of another (cudaErrorStreamCaptureUnsupported there, the capture invalidated), cudaFree
// does not. The new block is taken first, so the driver's chunk of small blocks stays: 2.8 us on an idle device.
void wait_as_free(DevicePool& d) {
    void* old = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_pools_mutex);
        void* next = nullptr;
        if (cudaMalloc(&next, 512) != cudaSuccess) {
            cudaGetLastError();
            next = nullptr;
        }
        old = d.fence;
        d.fence = next;
    }
    if (!old || cudaFree(old) != cudaSuccess) {  // (no block: memory had run out at the last trade)
        cudaGetLastError();
        cudaDeviceSynchronize();
    }
}
}  // namespace

void* device_alloc(size_t n, size_t* got, int* device) {
    n = (n + 511) / 512 * 512;
    SIMK_CUDA(cudaGetDevice(device));
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    DevicePool& d = device_pool(*device);
    if (!d.pool) open_pool(d, *device);
    auto take = [&](void** p) { return n > kLargest ? cudaMalloc(p, n) : pool_alloc(d, p, n); };
    void* p = nullptr;
    cudaError_t e = take(&p);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        cudaMemPoolTrimTo(d.pool, 0);
        e = take(&p);
    }
    check_cuda(e, "cudaMalloc");
    if (n <= kLargest) d.live += n;
    *got = n;
    return p;
}

void device_free(void* p, size_t bytes, int device) {
    if (!p) return;
    if (bytes > kLargest) {
        cudaFree(p);
        return;
    }
    int current = device;
    cudaGetDevice(&current);
    if (current != device) cudaSetDevice(device);
    DevicePool* pool = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_pools_mutex);
        pool = &device_pool(device);  // stays where it is: the map never moves its entries
    }
    wait_as_free(*pool);
    {
        std::lock_guard<std::mutex> lk(g_pools_mutex);
        DevicePool& d = *pool;
        cudaFreeAsync(p, d.stream);
        d.live -= bytes;
        unsigned long long held = 0;
        cudaMemPoolGetAttribute(d.pool, cudaMemPoolAttrReservedMemCurrent, &held);
        const size_t keep = d.live + (d.contexts ? kKept : 0);
        if (held > keep) {
            cudaStreamSynchronize(d.stream);
            cudaMemPoolTrimTo(d.pool, keep);
        }
    }
    if (current != device) cudaSetDevice(current);
}

void device_context_made(int device) {
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    ++device_pool(device).contexts;
}

void device_context_gone(int device) {
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    DevicePool& d = device_pool(device);
    if (--d.contexts == 0 && d.pool) {
        cudaStreamSynchronize(d.stream);
        cudaMemPoolTrimTo(d.pool, 0);
    }
}

// ---- pinned staging --------------------------------------------------------------------------------------------------
void HostStage::ensure(size_t n) {
    n = std::min(std::max<size_t>(n, 64 << 10), kHalf);
    if (bytes >= n) return;
    release();
    for (int i = 0; i < 2; ++i) {
        SIMK_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&half[i]), n, cudaHostAllocDefault));
        SIMK_CUDA(cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming));
    }
    bytes = n;
}

void HostStage::release() {
    for (int i = 0; i < 2; ++i) {
        if (done[i]) {
            cudaEventSynchronize(done[i]);  // a copy may still read or write the half
            cudaEventDestroy(done[i]);
        }
        if (half[i]) cudaFreeHost(half[i]);
        done[i] = nullptr;
        half[i] = nullptr;
    }
    bytes = 0;
}

void upload_complex(Context& ctx, float2* dst, const double* re, const double* im, long long n) {
    HostStage& st = ctx.stage;
    st.ensure((size_t)n * sizeof(float2));
    const long long chunk = (long long)(st.bytes / sizeof(float2));
    int h = 0;
    for (long long first = 0; first < n; first += chunk, h ^= 1) {
        const long long m = std::min(chunk, n - first);
        SIMK_CUDA(cudaEventSynchronize(st.done[h]));  // the half's last copy
        float2* const to = reinterpret_cast<float2*>(st.half[h]);
        for (long long i = 0; i < m; ++i) to[i] = make_float2((float)re[first + i], (float)im[first + i]);
        SIMK_CUDA(cudaMemcpyAsync(dst + first, to, m * sizeof(float2), cudaMemcpyHostToDevice, ctx.stream));
        SIMK_CUDA(cudaEventRecord(st.done[h], ctx.stream));
    }
}

void download_complex(Context& ctx, const float2* src, long long n, double* re, double* im, double* intensity) {
    HostStage& st = ctx.stage;
    st.ensure((size_t)n * sizeof(float2));
    const long long chunk = (long long)(st.bytes / sizeof(float2));
    auto fetch = [&](long long first, int h) {
        if (first >= n) return;
        const long long m = std::min(chunk, n - first);
        SIMK_CUDA(cudaMemcpyAsync(st.half[h], src + first, m * sizeof(float2), cudaMemcpyDeviceToHost, ctx.stream));
        SIMK_CUDA(cudaEventRecord(st.done[h], ctx.stream));
    };
    int h = 0;
    SIMK_CUDA(cudaEventSynchronize(st.done[0]));
    SIMK_CUDA(cudaEventSynchronize(st.done[1]));
    fetch(0, 0);
    for (long long first = 0; first < n; first += chunk, h ^= 1) {
        fetch(first + chunk, h ^ 1);
        SIMK_CUDA(cudaEventSynchronize(st.done[h]));
        const long long m = std::min(chunk, n - first);
        const float2* const from = reinterpret_cast<const float2*>(st.half[h]);
        if (re)
            for (long long i = 0; i < m; ++i) {
                re[first + i] = from[i].x;
                im[first + i] = from[i].y;
            }
        if (intensity)
            for (long long i = 0; i < m; ++i) {
                const double x = from[i].x, y = from[i].y;
                intensity[first + i] = x * x + y * y;
            }
    }
}

}  // namespace simk
