// hostio.cuh -- memory that calls would otherwise allocate each time: freed device blocks kept for reuse, and the pinned
// buffers through which split float64 host arrays become interleaved complex64 on the device and back.
#pragma once

#include "common.cuh"

namespace simk {

struct Context;

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
// re[i], im[i] = src[i] (either may be null), and intensity[i] = re^2 + im^2 where it is not null. Returns when the host
// arrays are written (the stream has then reached this point).
void download_complex(Context& ctx, const float2* src, long long n, double* re, double* im, double* intensity = nullptr);

}  // namespace simk
