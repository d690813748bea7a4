// twopass.cuh -- the fused passes with one shared-memory exchange per transform (engine 6): what fused.cu calls. The
// kernels are in twopass_kernels.cuh, instantiated by twopass_*.cu; the lengths are listed in twopass_plans.inc.
#pragma once

#include "context.cuh"

namespace simk {

struct TwoPassCols {
    float2* psi = nullptr;
    const float2* P = nullptr;
    int mode = 0;  // 0: FFT, x P, IFFT / (nx ny); 1: FFT, x P; 2: the probes' spectrum, IFFT; 3: as 1, with the detection
    int ny = 0, count = 0;
    const float2* spectrum = nullptr;
    const float2* rx = nullptr;
    const float2* ry = nullptr;
    const int* p_row = nullptr;  // job tables: wave b uses the propagator P + p_row[b] N
    const FusedDetect* det = nullptr;
};

// Columns of up to this length stay on the register engine: at 128 points its 4-column tiles took 41.5 us for 512 waves
// and 7.0 us for one, the two-pass engine 45.2 and 8.5; at 256 68.3 against 61.8 for 256 waves.
constexpr int kTwoColsAbove = 128;

// Whether lines of n points have a plan here.
bool twopass_length(int n);
// The plan's twiddle table of n divided by `points` (the inverse transform's 1 / (nx ny) in the columns' way back),
// created on first use (allocates and copies: not inside a stream capture).
const float2* twopass_table(Context& ctx, int n, long long points = 1);
// The row pass over nrows = count nx rows of ny points: [inverse], x t x scale, [forward]. False: no plan for ny.
bool twopass_rows(Context& ctx, float2* psi, const float2* tmul, int nx, int ny, long long nrows, int inv, int fwd,
                  float scale);
// The column pass over lines of nx > kTwoColsAbove points (false otherwise, or without a plan); with mode 3 *groups
// receives the column groups of the partial sums.
bool twopass_cols(Context& ctx, int nx, const TwoPassCols& a, int* groups);

}  // namespace simk
