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
// grows by whole chunks; at most kKept bytes beyond the blocks in use stay there. A block goes back once the host has seen
// the fences of every context of the device pass (any of them may have used it), and the pool's stream is idle when one is
// handed out, so any stream and thread may take it next. (Neither cudaFree of some other block nor cudaDeviceSynchronize
// waits in place of the fences: that the first waits is not promised, and the second breaks off the stream capture of
// another thread.) When the last context goes, so does what the pool holds free.
namespace {
constexpr size_t kKept = 512u << 20;
constexpr size_t kLargest = 256u << 20;
struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;  // orders the pool's operations
    size_t live = 0;                // bytes handed out
    std::vector<StreamFence*> fences;
};
std::mutex g_pools_mutex;
DevicePool& device_pool(int device) {
    static auto* m = new std::map<int, DevicePool>();  // never destroyed: buffers may be released at exit
    return (*m)[device];
}
thread_local ActiveContext* t_active = nullptr;

void open_pool(DevicePool& d, int device) {
    if (!d.stream) SIMK_CUDA(cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking));
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    SIMK_CUDA(cudaMemPoolCreate(&pool, &props));
    unsigned long long hold = ~0ULL;  // what stays is bounded in device_free
    const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &hold);
    if (e != cudaSuccess) cudaMemPoolDestroy(pool);
    SIMK_CUDA(e);
    d.pool = pool;
}
// Asking how far a stream is, and waiting for it, is refused while another thread captures in the global mode; not in a
// thread whose own mode is the relaxed one.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
// The fence at the end of what the stream holds now, unless a capture is recording it (what is captured has not run).
void fence(Context& c, bool ask) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c.stream, &s) != cudaSuccess || s != cudaStreamCaptureStatusNone) return;
    if (ask && cudaStreamQuery(c.stream) == cudaSuccess) {
        c.fence->pending = false;
        return;
    }
    if (ask) cudaGetLastError();  // (not ready)
    c.fence->pending = true;
    if (cudaEventRecord(c.fence->event.get(), c.stream) != cudaSuccess) cudaStreamSynchronize(c.stream);
}
Event make_event() {
    cudaEvent_t e = nullptr;
    SIMK_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return Event(e, [](cudaEvent_t made) { cudaEventDestroy(made); });
}
}  // namespace

ActiveContext::ActiveContext(Context& c) : before_(t_active), ctx(c) {
    SIMK_CUDA(cudaSetDevice(ctx.device));
    t_active = this;
}

ActiveContext::~ActiveContext() {
    fence(ctx, false);
    t_active = before_;
}

void ActiveContext::fence_all(int device) {
    for (ActiveContext* a = t_active; a; a = a->before_)
        if (a->ctx.device == device) fence(a->ctx, true);
}

void* device_alloc(size_t n, size_t* got, int* device) {
    n = (n + 511) / 512 * 512;
    SIMK_CUDA(cudaGetDevice(device));
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    DevicePool& d = device_pool(*device);
    if (!d.pool) open_pool(d, *device);
    auto take = [&](void** p) {
        if (n > kLargest) return cudaMalloc(p, n);
        const cudaError_t e = cudaMallocFromPoolAsync(p, n, d.pool, d.stream);
        return e == cudaSuccess ? cudaStreamSynchronize(d.stream) : e;
    };
    void* p = nullptr;
    cudaError_t e = take(&p);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        cudaStreamSynchronize(d.stream);
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
    const RelaxedCapture relaxed;
    ActiveContext::fence_all(device);
    std::vector<Event> before;  // waited for without the lock: other threads take and give back meanwhile
    {
        std::lock_guard<std::mutex> lk(g_pools_mutex);
        for (StreamFence* f : device_pool(device).fences) {
            if (f->pending) before.push_back(f->event);
            before.insert(before.end(), f->left.begin(), f->left.end());
        }
    }
    for (const Event& e : before) cudaEventSynchronize(e.get());
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    DevicePool& d = device_pool(device);
    for (StreamFence* f : d.fences)
        for (const Event& e : before) f->left.erase(std::remove(f->left.begin(), f->left.end(), e), f->left.end());
    cudaFreeAsync(p, d.stream);
    d.live -= bytes;
    unsigned long long held = 0;
    cudaMemPoolGetAttribute(d.pool, cudaMemPoolAttrReservedMemCurrent, &held);
    const size_t keep = d.live + (d.fences.empty() ? 0 : kKept);
    if (held > keep) {
        cudaStreamSynchronize(d.stream);
        cudaMemPoolTrimTo(d.pool, keep);
    }
    if (current != device) cudaSetDevice(current);
}

size_t device_held_free(int device) {
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    DevicePool& d = device_pool(device);
    unsigned long long held = 0;
    if (!d.pool || cudaMemPoolGetAttribute(d.pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess) return 0;
    return held > d.live ? (size_t)held - d.live : 0;
}

void device_context_made(Context& ctx) {
    auto fence = std::make_unique<StreamFence>();
    fence->event = make_event();
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    device_pool(ctx.device).fences.push_back(fence.get());
    ctx.fence = std::move(fence);
}

void device_stream_leaves(Context& ctx) {  // (not a call on the stream: its owner may have destroyed it)
    if (!ctx.fence->pending) return;
    int current = ctx.device;
    cudaGetDevice(&current);
    if (current != ctx.device) cudaSetDevice(ctx.device);
    Event next = make_event();
    if (current != ctx.device) cudaSetDevice(current);
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    ctx.fence->left.push_back(std::move(ctx.fence->event));
    ctx.fence->event = std::move(next);
    ctx.fence->pending = false;
}

void device_context_gone(int device, std::unique_ptr<StreamFence> fence) {
    std::lock_guard<std::mutex> lk(g_pools_mutex);
    DevicePool& d = device_pool(device);
    d.fences.erase(std::remove(d.fences.begin(), d.fences.end(), fence.get()), d.fences.end());
    if (d.fences.empty() && d.pool) {
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
