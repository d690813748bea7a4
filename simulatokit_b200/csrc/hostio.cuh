// hostio.cuh -- memory that calls would otherwise allocate each time: freed device blocks kept for reuse, and the pinned
// buffers through which split float64 host arrays become interleaved complex64 on the device and back.
#pragma once

#include <atomic>

#include "common.cuh"

namespace simk {

struct Context;

// Where a context's queued work ends, for the blocks that are given back: an event on its stream, recorded when a call
// returns with work still queued, and those of the streams that the context had before.
using Event = std::shared_ptr<std::remove_pointer_t<cudaEvent_t>>;
struct StreamFence {
    Event event;
    std::atomic<bool> pending{false};
    std::vector<Event> left;
};
void device_context_made(Context& ctx);
// The fence of a context that is gone, its work finished and its buffers given back.
void device_context_gone(int device, std::unique_ptr<StreamFence> fence);
// Before the context takes another stream: its work on the present one counts further.
void device_stream_leaves(Context& ctx);

// A call on the context in this thread: its device is the current one, and its fence is up to date at the end.
class ActiveContext {
    ActiveContext* const before_;

public:
    Context& ctx;
    explicit ActiveContext(Context& c);
    ~ActiveContext();
    ActiveContext(const ActiveContext&) = delete;
    ActiveContext& operator=(const ActiveContext&) = delete;
    static void fence_all(int device);  // brings the fences of this thread's calls on the device up to date
};

// A context's pinned staging: two halves, so that one is converted while the other is copied. Grown on demand up to
// kHalf bytes each, freed with the context.
struct HostStage {
    static constexpr size_t kHalf = 8u << 20;
    char* half[2] = {nullptr, nullptr};
    size_t bytes = 0;
    cudaEvent_t done[2] = {nullptr, nullptr};
    HostStage() = default;
    HostStage(const HostStage&) = delete;
    HostStage& operator=(const HostStage&) = delete;
    ~HostStage() { release(); }
    void ensure(size_t n);
    void release();
};

// dst[i] = (re[i], im[i]) rounded to float32, stream-ordered; the host arrays may be reused when it returns.
void upload_complex(Context& ctx, float2* dst, const double* re, const double* im, long long n);
// re[i], im[i] = src[i] (both null: not wanted), and intensity[i] = re^2 + im^2 where it is not null. Returns when the host
// arrays are written (the stream has then reached this point).
void download_complex(Context& ctx, const float2* src, long long n, double* re, double* im, double* intensity = nullptr);

}  // namespace simk
