// hostio.cu -- see hostio.cuh.
#include "hostio.cuh"

#include <algorithm>

#include "context.cuh"

namespace simk {

// ---- freed device blocks ---------------------------------------------------------------------------------------------
// cudaMalloc and cudaFree of a call's temporaries and of a potential's slices took 50-300 us each, half of a small HRTEM
// image. A freed block is kept (per device, at most kKept bytes in all, the oldest going first) and handed out again to
// a request it fits within a quarter. Every block comes back only after the device has finished everything queued, as
// cudaFree waits, so any stream and thread may take it next. When the last context goes, so do the blocks.
namespace {
constexpr size_t kKept = 512u << 20;
struct Block {
    void* ptr;
    size_t bytes;
};
struct DeviceBlocks {
    std::vector<Block> kept;  // oldest first
    size_t bytes = 0;
    int contexts = 0;
};
std::mutex g_blocks_mutex;
std::map<int, DeviceBlocks>& device_blocks() {
    static auto* m = new std::map<int, DeviceBlocks>();  // never destroyed: buffers may be released at exit
    return *m;
}
void drop_all(DeviceBlocks& d) {
    for (Block& b : d.kept) cudaFree(b.ptr);
    d.kept.clear();
    d.bytes = 0;
}
}  // namespace

void* device_alloc(size_t n, size_t* got, int* device) {
    n = (n + 511) / 512 * 512;
    SIMK_CUDA(cudaGetDevice(device));
    std::lock_guard<std::mutex> lk(g_blocks_mutex);
    DeviceBlocks& d = device_blocks()[*device];
    size_t best = d.kept.size();
    for (size_t i = 0; i < d.kept.size(); ++i) {
        const size_t b = d.kept[i].bytes;
        if (b >= n && b <= n + std::max<size_t>(n / 4, 4096) && (best == d.kept.size() || b < d.kept[best].bytes)) best = i;
    }
    if (best < d.kept.size()) {
        const Block b = d.kept[best];
        d.kept.erase(d.kept.begin() + best);
        d.bytes -= b.bytes;
        *got = b.bytes;
        return b.ptr;
    }
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, n);
    if (e == cudaErrorMemoryAllocation && !d.kept.empty()) {
        cudaGetLastError();
        drop_all(d);
        e = cudaMalloc(&p, n);
    }
    check_cuda(e, "cudaMalloc");
    *got = n;
    return p;
}

void device_free(void* p, size_t bytes, int device) {
    if (!p) return;
    int current = device;
    cudaGetDevice(&current);
    if (current != device) cudaSetDevice(device);
    {
        std::lock_guard<std::mutex> lk(g_blocks_mutex);
        DeviceBlocks& d = device_blocks()[device];
        if (d.contexts == 0 || bytes > kKept / 2 || cudaDeviceSynchronize() != cudaSuccess) {
            cudaFree(p);
        } else {
            d.kept.push_back({p, bytes});
            d.bytes += bytes;
            while (d.bytes > kKept) {
                cudaFree(d.kept.front().ptr);
                d.bytes -= d.kept.front().bytes;
                d.kept.erase(d.kept.begin());
            }
        }
    }
    if (current != device) cudaSetDevice(current);
}

void device_context_made(int device) {
    std::lock_guard<std::mutex> lk(g_blocks_mutex);
    ++device_blocks()[device].contexts;
}

void device_context_gone(int device) {
    std::lock_guard<std::mutex> lk(g_blocks_mutex);
    DeviceBlocks& d = device_blocks()[device];
    if (--d.contexts == 0) drop_all(d);
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
