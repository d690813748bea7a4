// linefft_kernels.cuh -- batched line transforms of the lengths in twopass_plans.inc, float32 or float64, in place, with
// one shared-memory exchange: N = R1 R2, item j < R2 takes the R1-point DFT of x[j + R2 r] into row j of M, item k < R1
// column k of M times W_N^{jk} through the R2-point DFT to the points k + R1 s. With BLUE the N points are the padded
// work length of Bluestein's transform of n points: the chirp on the way in, the kernel's spectrum between the DFTs (item
// k has those frequencies in registers), and the way back through the same exchange to the chirp on the way out, all in
// one kernel. The inverse is the conjugate of the transform of the conjugate.
//
// Bound by memory latency and, in float64, by the FP64 pipe; the shared-memory Stockham passes of fft.cu (still taken by
// the other lengths) go through shared memory once per radix-16 or smaller step with run-time index divisions. 16 waves
// of 331 x 250 (Bluestein over 1024 points, and 10 x 25): 68 us a pass there. Figures at the dispatch in fft.cu.
#pragma once

#include "dftreg.cuh"
#include "linefft.cuh"

namespace simk {

template <int N> struct LineLen { static constexpr int R1 = 0, R2 = 0; };
#define SIMK_TWO_PLAN(n, a, b) \
    template <> struct LineLen<n> { static constexpr int R1 = a, R2 = b; };
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN

template <int N, typename V> struct LinePlanCfg {
    static constexpr int R1 = LineLen<N>::R1, R2 = LineLen<N>::R2, LD = R1 | 1;
    // threads an SM: the registers R2 values need
    static constexpr int RM = R1 > R2 ? R1 : R2;
    static constexpr int MAXT = (sizeof(V) == 8 ? (RM <= 16 ? 768 : 512) : (RM <= 16 ? 384 : 256));
    // rows: lines a block
    static constexpr int L = 128 / R2 > 0 ? 128 / R2 : 1;
    static constexpr int NT_ROWS = (L * R2 + 31) / 32 * 32;
    static constexpr int QB_ROWS = (L * R1 + NT_ROWS - 1) / NT_ROWS;
    // columns: 64-byte row segments
    static constexpr int TC = 64 / (int)sizeof(V);
    static constexpr int NT_COLS = ((R1 > R2 ? R1 : R2) * TC + 31) / 32 * 32;
    static constexpr size_t SMEM_ROWS = (size_t)L * R2 * LD * sizeof(V), SMEM_COLS = (size_t)R2 * LD * TC * sizeof(V);
};

// Value `idx` of a line on its way in or out: conjugated for the inverse, times the chirp (BLUE), zero past n.
template <bool BLUE, typename V>
__device__ __forceinline__ V line_in(const V* p, int idx, long long stride, const LineArgs<V>& a) {
    if (BLUE && idx >= a.n) return mk<V>(0, 0);
    V x = p[idx * stride];
    if (a.conj) x.y = -x.y;
    if constexpr (BLUE) x = cmul(x, __ldg(a.chirp + idx));
    return x;
}
template <bool BLUE, typename V>
__device__ __forceinline__ void line_out(V* p, int idx, long long stride, V x, const LineArgs<V>& a) {
    if (BLUE && idx >= a.n) return;
    if constexpr (BLUE) x = cmul(x, __ldg(a.chirp + idx));
    if (a.conj) x.y = -x.y;
    if (a.scale != 1) x = x * a.scale;
    p[idx * stride] = x;
}
// Steps B and C shared by rows and columns: column k of M (slots m[j step]) through the DFT, and for BLUE back again.
template <int N, bool BLUE, typename V>
__device__ __forceinline__ void line_step_b(V* m, int step, int k, V (&v)[LinePlanCfg<N, V>::R2], const LineArgs<V>& a) {
    constexpr int R1 = LinePlanCfg<N, V>::R1, R2 = LinePlanCfg<N, V>::R2;
#pragma unroll
    for (int j = 0; j < R2; ++j) v[j] = j ? cmul(m[j * step], __ldg(a.table + j * R1 + k)) : m[0];
    dft_reg<R2, -1>(v);
    if constexpr (BLUE) {
#pragma unroll
        for (int s = 0; s < R2; ++s) v[s] = cmul(v[s], __ldg(a.khat + k + R1 * s));
        dft_reg<R2, +1>(v);
#pragma unroll
        for (int j = 0; j < R2; ++j) m[j * step] = j ? cmulc(v[j], __ldg(a.table + j * R1 + k)) : v[0];
    }
}

template <int N, bool BLUE, typename V>
__global__ void __launch_bounds__(LinePlanCfg<N, V>::NT_ROWS, LinePlanCfg<N, V>::MAXT / LinePlanCfg<N, V>::NT_ROWS)
    line_rows(LineArgs<V> a) {
    using P = LinePlanCfg<N, V>;
    constexpr int R1 = P::R1, R2 = P::R2, LD = P::LD, L = P::L;
    extern __shared__ __align__(16) unsigned char smem_line[];
    V* const M = reinterpret_cast<V*>(smem_line);
    const int u = threadIdx.x;
    const long long first = (long long)blockIdx.x * L;
    const int l = u / R2, j = u % R2;
    const bool on = l < L && first + l < a.lines;
    V* const line = a.data + (first + l) * a.n;
    if (on) {
        V v[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = line_in<BLUE>(line, j + R2 * r, 1, a);
        dft_reg<R1, -1>(v);
#pragma unroll
        for (int k = 0; k < R1; ++k) M[(l * R2 + j) * LD + k] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < P::QB_ROWS; ++q) {
        const int i = u + P::NT_ROWS * q, lb = i / R1, k = i % R1;
        if (lb >= L || first + lb >= a.lines) continue;
        V v[R2];
        line_step_b<N, BLUE>(M + lb * (R2 * LD) + k, LD, k, v, a);
        if constexpr (!BLUE) {
            V* const out = a.data + (first + lb) * a.n;
#pragma unroll
            for (int s = 0; s < R2; ++s) line_out<false>(out, k + R1 * s, 1, v[s], a);
        }
    }
    if constexpr (BLUE) {
        __syncthreads();
        if (on) {
            V v[R1];
#pragma unroll
            for (int k = 0; k < R1; ++k) v[k] = M[(l * R2 + j) * LD + k];
            dft_reg<R1, +1>(v);
#pragma unroll
            for (int s = 0; s < R1; ++s) line_out<true>(line, j + R2 * s, 1, v[s], a);
        }
    }
}

template <int N, bool BLUE, typename V>
__global__ void __launch_bounds__(LinePlanCfg<N, V>::NT_COLS, LinePlanCfg<N, V>::MAXT / LinePlanCfg<N, V>::NT_COLS > 0
                                                                  ? LinePlanCfg<N, V>::MAXT / LinePlanCfg<N, V>::NT_COLS
                                                                  : 1) line_cols(LineArgs<V> a) {
    using P = LinePlanCfg<N, V>;
    constexpr int R1 = P::R1, R2 = P::R2, LD = P::LD, TC = P::TC;
    extern __shared__ __align__(16) unsigned char smem_line[];
    const int u = threadIdx.x, c = u % TC, item = u / TC;
    V* const M = reinterpret_cast<V*>(smem_line) + c;
    const unsigned groups = (unsigned)(a.ny + TC - 1) / TC;
    const long long b = blockIdx.x / groups;
    const int iy = (int)(blockIdx.x - b * groups) * TC + c;
    const bool live = iy < a.ny;
    V* const col = a.data + b * a.n * a.ny + iy;
    if (live && item < R2) {
        V v[R1];
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = line_in<BLUE>(col, item + R2 * r, a.ny, a);
        dft_reg<R1, -1>(v);
#pragma unroll
        for (int k = 0; k < R1; ++k) M[(item * LD + k) * TC] = v[k];
    }
    __syncthreads();
    if (live && item < R1) {
        V v[R2];
        line_step_b<N, BLUE>(M + item * TC, LD * TC, item, v, a);
        if constexpr (!BLUE) {
#pragma unroll
            for (int s = 0; s < R2; ++s) line_out<false>(col, item + R1 * s, a.ny, v[s], a);
        }
    }
    if constexpr (BLUE) {
        __syncthreads();
        if (live && item < R2) {
            V v[R1];
#pragma unroll
            for (int k = 0; k < R1; ++k) v[k] = M[(item * LD + k) * TC];
            dft_reg<R1, +1>(v);
#pragma unroll
            for (int s = 0; s < R1; ++s) line_out<true>(col, item + R2 * s, a.ny, v[s], a);
        }
    }
}

template <int N, bool BLUE, typename V> void launch_line(const LineArgs<V>& a, bool columns, cudaStream_t stream) {
    using P = LinePlanCfg<N, V>;
    static PerDevice setup;
    setup.get([] {
        return allow_shared(line_rows<N, BLUE, V>, P::SMEM_ROWS) + allow_shared(line_cols<N, BLUE, V>, P::SMEM_COLS);
    });
    if (columns) {
        const long long blocks = a.lines / a.ny * ((a.ny + P::TC - 1) / P::TC);
        SIMK_REQUIRE(blocks < (1LL << 31), "too many FFT lines");
        line_cols<N, BLUE, V><<<(unsigned)blocks, P::NT_COLS, P::SMEM_COLS, stream>>>(a);
    } else {
        const long long blocks = (a.lines + P::L - 1) / P::L;
        SIMK_REQUIRE(blocks < (1LL << 31), "too many FFT lines");
        line_rows<N, BLUE, V><<<(unsigned)blocks, P::NT_ROWS, P::SMEM_ROWS, stream>>>(a);
    }
    SIMK_CUDA(cudaGetLastError());
}

}  // namespace simk
