// linefft.cuh -- batched line transforms with one exchange (kernels in linefft_kernels.cuh): what fft.cu dispatches to.
#pragma once

#include <vector>

#include "common.cuh"

namespace simk {

// `lines` lines of n points in place: rows (line l at data + l n), or the columns of lines / ny fields of n x ny.
template <typename V> struct LineArgs {
    V* data;
    const V* table;  // W_N^{jk} at j R1 + k
    const V* chirp;  // Bluestein: n values; khat: N values
    const V* khat;
    long long lines;
    int n, ny, conj;
    decltype(V::x) scale;
};

template <int N, bool BLUE, typename V> void launch_line(const LineArgs<V>& a, bool columns, cudaStream_t stream);

// The float32 twiddles W_n^{jk} of a plan n = r1 r2, times `scale`, at j r1 + k.
std::vector<float2> line_table(int n, int r1, double scale = 1.0);
// R1 of the plan of N points, 0 where there is none; whether Bluestein's work length N is taken.
int line_first_radix(int N);
bool line_bluestein_length(int N);
template <typename V> void launch_line_any(int N, bool blue, const LineArgs<V>& a, bool columns, cudaStream_t stream);

}  // namespace simk
