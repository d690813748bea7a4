// twopass_kernels.cuh -- the fused row and column passes with one shared-memory exchange per transform (engine 6).
//
// A line of N = R1 R2 points is the matrix x[j + R2 r], j < R2, r < R1. Both passes of a slice are a transform, a
// multiplication and the transform back, so the line goes through three steps around two exchanges in one place:
//   A  item j < R2: R1-point DFT over r of the values it loads from memory        -> M[j][0 .. R1)
//   B  item k < R1: column k of M, x W_N^{+-jk}, R2-point DFT: the line's points k + R1 m; x t or P there; the R2-point
//      DFT back, x W_N^{-+jk}                                                      -> the same column of M
//   C  item j < R2: row j of M, R1-point DFT back: points j + R2 s, stored
// Every DFT is in one thread's registers (dftreg.cuh), so a transform exchanges its data through shared memory once
// (the register-resident radix-8 passes of fused.cu do so two or three times), item k rewrites exactly the slots it
// read, and item j of step C reads what it wrote in A of the next line: two barriers a line. Loads and stores go
// straight between global memory and registers (neither staged nor copied back); warps or blocks run free of one
// another, so the latency of one line's loads is covered by the arithmetic of the others.
#pragma once

#include "dftreg.cuh"
#include "tma.cuh"
#include "twopass.cuh"

namespace simk {

// ---- plans -----------------------------------------------------------------------------------------------------------
template <int N> struct TwoPlan { static constexpr int R1 = 0, R2 = 0; };
#define SIMK_TWO_PLAN(n, a, b) \
    template <> struct TwoPlan<n> { static constexpr int R1 = a, R2 = b; static_assert(a * b == n, ""); };
#include "twopass_plans.inc"
#undef SIMK_TWO_PLAN

template <int GT> __device__ __forceinline__ void group_sync(int id) {
    if constexpr (GT == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(GT) : "memory");
}

// n / d for n < 2^31 as a multiplication and a shift (Granlund and Montgomery's round-up method).
struct FastDiv {
    unsigned d, mul, shift;
};
inline FastDiv fast_div(unsigned d) {
    unsigned l = 0;
    while (l < 32 && (1ULL << l) < d) ++l;
    return FastDiv{d, (unsigned)((((1ULL << l) - d) << 32) / d + 1), l};
}
__device__ __forceinline__ unsigned operator/(unsigned n, const FastDiv& f) {
    return (__umulhi(n, f.mul) + n) >> f.shift;
}

// ---- rows ------------------------------------------------------------------------------------------------------------
// Bound by HBM where the DFTs are cheap (512: 5.1 TB/s of the measured 6.5, 424 us for 512 waves; 1024: 4.9), by issue
// and the FMA pipe elsewhere (500 = 20 x 25: 3.6 TB/s, 161 us for 144 waves, FMA pipe near half busy).
// A group of GT threads takes GR rows at a time: one warp where R1 and R2 divide its lanes evenly (256, 512, 1024 and
// 128 points: no barrier beyond __syncwarp), else a block.
// SPREAD: at 512 a warp takes one row instead of two, half of step B's lanes idle, for launches of few rows.
template <int N, bool SPREAD = false> struct RowPlan {
    static constexpr int R1 = TwoPlan<N>::R1, R2 = TwoPlan<N>::R2;
    static constexpr bool EVEN = (32 % R1 == 0) && (32 % R2 == 0), WARP = EVEN || (R2 == 32 && R1 >= 24);
    static constexpr int GR = EVEN ? 32 / (SPREAD ? (R1 > R2 ? R1 : R2) : R1) : WARP ? 1 : 128 / R2;
    static constexpr int GT = WARP ? 32 : (GR * R2 + 31) / 32 * 32;
    static constexpr int NT = WARP ? 128 : GT;
    static constexpr int LD = R1 | 1;  // odd: column walks of M touch every bank pair
    static constexpr int QA = (GR * R2 + GT - 1) / GT, QB = (GR * R1 + GT - 1) / GT;
    // an SM, asked of the compiler: 85, 102 or 128 registers
    static constexpr int BLOCKS = (R2 <= 16 ? 768 : R2 <= 25 ? 640 : 512) / NT;
    static constexpr size_t SMEM = (size_t)(N + NT / GT * GR * R2 * LD) * sizeof(float2);
};

template <int N, bool SPREAD = false>
__global__ void __launch_bounds__(RowPlan<N, SPREAD>::NT, RowPlan<N, SPREAD>::BLOCKS)
    two_rows(float2* __restrict__ psi, const float2* __restrict__ tmul, const float2* __restrict__ table, unsigned nx,
             FastDiv count, int inv, int fwd, float scale, const float2* const* __restrict__ t_of_wave) {
    using P = RowPlan<N, SPREAD>;
    constexpr int R1 = P::R1, R2 = P::R2, GT = P::GT, GR = P::GR, LD = P::LD, QA = P::QA, QB = P::QB;
    extern __shared__ __align__(16) float2 smem_two_rows[];
    float2* const tw = smem_two_rows;
    const int tid = threadIdx.x, grp = tid / GT, u = tid % GT;
    float2* const M = smem_two_rows + N + grp * (GR * R2 * LD);
    // the table comes while the first rows do: waited for before the first step B
    for (int i = tid; i < N / 2; i += P::NT)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(tw + 2 * i)), "l"(table + 2 * i)
                     : "memory");
    bool table_here = false;
    auto wait_table = [&] {
        if (table_here) return;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        table_here = true;
    };
    const unsigned nrows = nx * count.d;
    const unsigned ntiles = (nrows + GR - 1) / GR;
    const unsigned step = gridDim.x * (P::NT / GT);
    const bool with_t = tmul != nullptr || t_of_wave != nullptr;
    for (unsigned tile = blockIdx.x * (P::NT / GT) + grp; tile < ntiles; tile += step) {
        // rows in the order (ix, wave): a group's rows share their row of t, which stays in L1
        const unsigned row0 = tile * GR;
        float2* line[QA];
#pragma unroll
        for (int q = 0; q < QA; ++q) {
            const int i = u + GT * q;
            const unsigned r = row0 + i / R2;
            line[q] = nullptr;
            if ((GR * R2 % GT == 0 || i < GR * R2) && r < nrows) {
                const unsigned ix = r / count;
                line[q] = psi + ((size_t)(r - ix * count.d) * nx + ix) * N + i % R2;
            }
        }
        if (with_t) {  // the rows of t to L1, for step B
            constexpr int LINES = (N + 15) / 16;  // of 128 bytes
            for (int l = u; l < GR * LINES; l += GT) {
                const unsigned r = row0 + l / LINES;
                if (r < nrows) {
                    const unsigned ix = r / count, b = r - ix * count.d;
                    const float2* const t = (t_of_wave ? t_of_wave[b] : tmul) + (size_t)ix * N + 16 * (l % LINES);
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(t));
                }
            }
        }
        if (inv) {
            float2 v[QA][R1];
#pragma unroll
            for (int q = 0; q < QA; ++q)
#pragma unroll
                for (int r = 0; r < R1; ++r) v[q][r] = line[q] ? __ldcg(line[q] + R2 * r) : make_float2(0.0f, 0.0f);
#pragma unroll
            for (int q = 0; q < QA; ++q) {
                const int i = u + GT * q;
                dft_reg<R1, +1>(v[q]);
                if (GR * R2 % GT == 0 || i < GR * R2) {
                    float2* m = M + (i / R2) * (R2 * LD) + (i % R2) * LD;
#pragma unroll
                    for (int k = 0; k < R1; ++k) m[k] = v[q][k];
                }
            }
            group_sync<GT>(1);
        }
        wait_table();
#pragma unroll
        for (int q = 0; q < QB; ++q) {
            const int i = u + GT * q;
            const unsigned r = row0 + i / R1;
            if ((GR * R1 % GT == 0 || i < GR * R1) && r < nrows) {
                const int k = i % R1;
                const unsigned ix = r / count, b = r - ix * count.d;
                float2* const m = M + (i / R1) * (R2 * LD) + k;
                float2* const row = psi + ((size_t)b * nx + ix) * N + k;
                float2 v[R2];
                if (inv) {
#pragma unroll
                    for (int j = 0; j < R2; ++j) v[j] = j ? cmulc(m[j * LD], tw[j * R1 + k]) : m[0];
                    dft_reg<R2, +1>(v);
                } else {
#pragma unroll
                    for (int s = 0; s < R2; ++s) v[s] = __ldcg(row + R1 * s);
                }
                if (with_t) {
                    const float2* const t = (t_of_wave ? t_of_wave[b] : tmul) + (size_t)ix * N + k;
#pragma unroll
                    for (int s = 0; s < R2; ++s) v[s] = cmul(v[s], __ldg(t + R1 * s));
                }
                if (scale != 1.0f) {
#pragma unroll
                    for (int s = 0; s < R2; ++s) v[s] = v[s] * scale;
                }
                if (fwd) {
                    dft_reg<R2, -1>(v);
#pragma unroll
                    for (int j = 0; j < R2; ++j) m[j * LD] = j ? cmul(v[j], tw[j * R1 + k]) : v[0];
                } else {
#pragma unroll
                    for (int s = 0; s < R2; ++s) __stcg(row + R1 * s, v[s]);
                }
            }
        }
        group_sync<GT>(1);
        if (fwd) {
#pragma unroll
            for (int q = 0; q < QA; ++q) {
                if (line[q]) {
                    const int i = u + GT * q;
                    const float2* m = M + (i / R2) * (R2 * LD) + (i % R2) * LD;
                    float2 v[R1];
#pragma unroll
                    for (int k = 0; k < R1; ++k) v[k] = m[k];
                    dft_reg<R1, -1>(v);
#pragma unroll
                    for (int s = 0; s < R1; ++s) __stcg(line[q] + R2 * s, v[s]);
                }
            }
            if (!inv) group_sync<GT>(1);  // the next rows' step B writes what other threads read here
        }
    }
    wait_table();  // (a warp without rows)
}

// ---- columns ---------------------------------------------------------------------------------------------------------
// A sub-block of NT threads takes a tile of TC = 8 adjacent columns (64-byte row segments) of one wave; a block has up
// to SUBS of them, which synchronise apart and share a ring of NB tile buffers: tile i of the block is in buffer i % NB
// and belongs to sub-block i % SUBS. TMA brings a tile in and takes it out; the load of tile i + NB is issued by the
// sub-block that had tile i, once the store of tile i has read its buffer (asked for in the middle of its next tile).
// Bound at 512 by the latency of a tile's three steps at four warps a scheduler (512 waves: 505 us between two slices,
// 4.25 TB/s; 443 us the mean of a 6-slice scan's launches, as the times below; FMA pipe and issue near half busy).
// Tiles loaded and stored from registers instead, without TMA: 541 us, most of it the loads' latency; tiles of 16
// columns that way 550 us; P's first values asked for in step B 482 us, before the tile's wait 440 us. Programmatic
// dependent launch of the passes cost 4 % at 512^2 (5 % at 256^2) and is not used.
// All three steps work in place: step A's value (j, k) lies in the row j + R2 k that item j owns, with the rows of
// j and j ^ 1 exchanged for odd k where R2 is even, so that two neighbouring items always lie in different halves of the
// 128 bytes that a half-warp reads at once, along j as along k (items j and j ^ 1 are in one warp).
template <int N> struct ColPlan {
    static constexpr int R1 = TwoPlan<N>::R1, R2 = TwoPlan<N>::R2, TC = 8;
    static constexpr int TILE = N * TC;  // float2
    static constexpr int NB = (int)((222 * 1024 - 2 * N * sizeof(float2)) / (TILE * sizeof(float2)));
    // threads an SM, by the registers a step-B item needs: 85, 102, 113 or 128 each
    static constexpr int RM = R1 > R2 ? R1 : R2, MAXT = RM <= 16 ? 768 : RM <= 20 ? 640 : RM <= 25 ? 576 : 512;
    static constexpr int subs_of(int nt) { return MAXT / nt < NB - (NB > 3 ? 2 : 1) ? MAXT / nt : NB - (NB > 3 ? 2 : 1); }
    // Threads of a sub-block: the idle share of its rounds of items, weighed against the threads that leaves an SM; the
    // smallest of equals, since more sub-blocks cover each other's barriers (384: 128 threads 77.9 us, 192 threads
    // 83.5 us for 128 waves; 640: 256 threads 132 us, 128 threads with one spare buffer 154 us for 64 waves).
    static constexpr double cost(int nt) {
        const int rounds = (R2 * TC + nt - 1) / nt + (R1 * TC + nt - 1) / nt, all = nt * subs_of(nt);
        return (double)(nt * rounds) / (all < 512 ? all : 512);
    }
    static constexpr int NT = [] {
        int best = 128;
        for (int nt = 160; nt <= 256; nt += 32)
            if (cost(nt) < 0.98 * cost(best)) best = nt;
        return best;
    }();
    static constexpr int SUBS = subs_of(NT);
    static constexpr int QA = (R2 * TC + NT - 1) / NT, QB = (R1 * TC + NT - 1) / NT;
    static constexpr bool SWAP = R2 % 2 == 0;
    static constexpr int BOXH = [] {
        for (int h = 256; h > 2; --h)  // even: every box starts at a multiple of 128 bytes
            if (h % 2 == 0 && N % h == 0) return h;
        return 2;
    }();
    static_assert(N % 2 == 0 && NT % 32 == 0, "whole warps, 16-byte rows");
    static constexpr size_t smem(int buffers) { return ((size_t)2 * N + (size_t)buffers * TILE) * sizeof(float2); }
};

// The wave's mean goes past the transforms of step B: it is taken off the R2 values of item 0 of line 0 beforehand, and
// what P makes of it is added to them afterwards. A plane wave's energy is in that one value, and its rounding at each
// level of the two transforms, slice after slice, was most of the error of sums over an exit wave (energy after 40 weak
// slices, rms: 256^2 3.7e-7, now 4e-8; 640^2 4.1e-7, now 1.1e-7). One tile of a wave in ny / 8 has it. With R2 <= 16 the
// item does this in registers; else in shared memory by functions of their own, as the registers of all items would be
// planned for it (inlined: 512 446 -> 454 us, 640 105 -> 108; functions at 256 62.6 us, registers 60.5). It costs 2 % of
// the pass at 256 (59.2 -> 60.5 us), 6 % at 576 (123 -> 131), elsewhere 1 % or less.
// sum / R to 18 bits: R times that is exact (and only what is near the mean is needed: the rest stays in the values).
template <int R> __device__ __forceinline__ float2 short_mean(float2 sum) {
    static_assert(R <= 64, "18 bits and the radix's fit in 24");
    return make_float2(__int_as_float(__float_as_int(sum.x * (1.0f / R)) & ~63),
                       __int_as_float(__float_as_int(sum.y * (1.0f / R)) & ~63));
}
template <int R, int STEP> __device__ __noinline__ float2 take_mean(float2* x) {
    float2 s = x[0];
#pragma unroll 4
    for (int j = 1; j < R; ++j) s = padd(s, x[j * STEP]);
    s = short_mean<R>(s);
#pragma unroll 4
    for (int j = 0; j < R; ++j) x[j * STEP] = psub(x[j * STEP], s);
    return s;
}
template <int R1, int R2, int STEP>
__device__ __noinline__ void give_mean(float2* x, float2 z, const float2* tw_back, float scale, float rest) {
    x[0] = make_float2(fmaf(z.x, scale, fmaf(z.x, rest, x[0].x)), fmaf(z.y, scale, fmaf(z.y, rest, x[0].y)));
#pragma unroll 4
    for (int j = 1; j < R2; ++j) {
        const float s = tw_back[j * R1].x;
        x[j * STEP] = make_float2(fmaf(z.x, s, x[j * STEP].x), fmaf(z.y, s, x[j * STEP].y));
    }
}

struct TwoDetect {
    const int* ptr = nullptr;   // [groups C + 1]
    const int2* ent = nullptr;  // (row TC + column, weight bits)
    double* partial = nullptr;  // [wave][groups][C]
    int n_ch = 0, store = 0;
};

// Tiles in the order (waves in groups of `subs`, column group, wave in its group): the sub-blocks of a block take the
// same columns of different waves, so their reads of P meet in L1. `waves` of the waves are in whole groups.
struct TileOrder {
    FastDiv round, subs, rest;  // tiles of a group of waves; waves of a group; waves of the last, short one (or 1)
    unsigned groups, waves, tiles;
};

template <int N, int MODE>
__global__ void __launch_bounds__(ColPlan<N>::NT* ColPlan<N>::SUBS, 1)
    two_cols(const __grid_constant__ CUtensorMap map, float2* __restrict__ psi, const float2* __restrict__ prop,
             const float2* __restrict__ table, const float2* __restrict__ back, float scale, float rest, int ny,
             TileOrder order, int buffers, int* err,
             const int* __restrict__ p_row, const float2* __restrict__ rx, const float2* __restrict__ ry, TwoDetect det) {
    using P = ColPlan<N>;
    constexpr int R1 = P::R1, R2 = P::R2, TC = P::TC, NT = P::NT, QA = P::QA, QB = P::QB, TILE = P::TILE,
                  BOXH = P::BOXH;
    constexpr bool SWAP = P::SWAP;
    extern __shared__ __align__(128) float2 smem_two_cols[];
    __shared__ __align__(8) uint64_t full[P::NB];
    __shared__ int failed[P::SUBS], issued[P::NB];
    [[maybe_unused]] __shared__ float2 mean[P::SUBS];
    // W_N^{jk}, and for the way back the same divided by nx ny (so that scaling costs nothing: every value but j = 0
    // takes a twiddle)
    float2* const tw = smem_two_cols + buffers * TILE;
    float2* const tw_back = tw + N;
    const unsigned subs = order.subs.d;
    const int tid = threadIdx.x, sub = tid / NT, u = tid % NT;
    const unsigned ntiles = order.tiles, round = gridDim.x * subs;
    auto place = [&](unsigned tile, unsigned& b, unsigned& g) {
        const unsigned w = tile / order.round * subs;
        const unsigned r = tile - w * order.groups;
        const bool whole = w < order.waves;
        g = whole ? r / order.subs : r / order.rest;
        b = w + (r - g * (whole ? subs : order.rest.d));
    };
    const unsigned first = blockIdx.x * subs;
    auto tile_of = [&](unsigned i) {  // the block's i-th tile
        const unsigned q = i / order.subs;
        return first + q * round + (i - q * subs);
    };
    auto issue = [&](unsigned i) {
        const unsigned tile = tile_of(i);
        if (tile >= ntiles) return;
        unsigned b, g;
        place(tile, b, g);
        const int s = (int)(i % buffers);
        ++issued[s];
        mbar_arrive_expect_tx(&full[s], (uint32_t)(TILE * sizeof(float2)));
#pragma unroll
        for (int k = 0; k < N / BOXH; ++k)
            tma_load_2d(smem_two_cols + s * TILE + k * BOXH * TC, &map, &full[s], 2 * TC * (int)g, (int)b * N + k * BOXH);
    };
    if (tid < (int)subs) failed[tid] = 0;
    if (tid == 0) {
        for (int s = 0; s < buffers; ++s) {
            issued[s] = 0;
            mbar_init(&full[s], 1);
        }
        fence_barrier_init();
        if constexpr (MODE != 2)
            for (int i = 0; i < buffers; ++i) issue(i);
    }
    for (int i = tid; i < N; i += blockDim.x) {
        tw[i] = __ldg(table + i);
        if constexpr (MODE == 0 || MODE == 2) tw_back[i] = __ldg(back + i);
    }
    __syncthreads();
    const int c = u % TC, item = u / TC;
    for (unsigned i = sub; tile_of(i) < ntiles; i += subs) {
        const int s = (int)(i % buffers);
        float2* const M = smem_two_cols + s * TILE + c;
        unsigned b, g;
        place(tile_of(i), b, g);
        const int iy = (int)g * TC + c;
        const bool live = iy < ny;
        // P comes from L2: the first values of step B are asked for ahead, at the start of step B, or where registers are
        // plenty (R2 <= 16) before the wave's tile is waited for (256: 63 -> 59 us for 256 waves; 512 that way 425 -> 452
        // for 512 waves, 768 166 -> 183 for 64)
        constexpr bool SOON = R2 <= 16;
        constexpr int EARLY = MODE == 2 ? 0 : R2 <= 16 ? 8 : R2 == 25 ? 8 : R2 / 2;
        [[maybe_unused]] const float2* const P0 = prop + (MODE != 2 && p_row ? (size_t)__ldg(p_row + b) * N * ny : 0) + iy;
        [[maybe_unused]] float2 pe[EARLY > 0 ? EARLY : 1];
        [[maybe_unused]] auto ask = [&] {
            const float2* p = P0 + (size_t)item * ny;
            const bool on = live && (R1 * TC % NT == 0 || item < R1);
#pragma unroll
            for (int t = 0; t < EARLY; ++t, p += R1 * ny) pe[t] = on ? __ldg(p) : make_float2(0.0f, 0.0f);
        };
        if constexpr (EARLY > 0 && SOON) ask();
        if (u == 0) {
            if constexpr (MODE == 2) bulk_wait_read();  // this buffer's last tile has left
            else if (!mbar_wait_bounded(&full[s], (i / buffers) & 1)) {
                atomicExch(err, 1);
                failed[sub] = 1;
            }
        }
        group_sync<NT>(1 + sub);
        if (failed[sub]) break;
        if constexpr (MODE != 2) {
#pragma unroll
            for (int q = 0; q < QA; ++q) {
                const int j = item + NT / TC * q;
                const bool on = R2 * TC % NT == 0 || j < R2;
                float2 v[R1];
                if (on) {
                    const float2* in = M + j * TC;
#pragma unroll
                    for (int r = 0; r < R1; ++r) v[r] = in[r * (R2 * TC)];
                    dft_reg<R1, -1>(v);
                }
                __syncwarp();  // item j ^ 1 has read the rows written here
                if (on) {
                    float2* const out[2] = {M + j * TC, M + (SWAP ? j ^ 1 : j) * TC};
#pragma unroll
                    for (int r = 0; r < R1; ++r) out[r & 1][r * (R2 * TC)] = v[r];
                }
            }
            group_sync<NT>(1 + sub);
            if (u == 0 && i >= subs) {  // the buffer of this sub-block's last tile: its next load
                bulk_wait_read();
                issue(i - subs + buffers);
            }
        }
        const bool zero = MODE == 0 && u == 0 && g == 0;  // has the wave's zero frequency
        if (!SOON && zero) mean[sub] = take_mean<R2, TC>(M);
#pragma unroll
        for (int q = 0; q < QB; ++q) {
            const int k = item + NT / TC * q, odd = SWAP ? (k & 1) : 0;
            if (R1 * TC % NT != 0 && k >= R1) continue;
            float2* const col = M + k * (R2 * TC);
            float2* const m[2] = {col + odd * TC, col - odd * TC};  // slot of (j, k): m[j & 1][j TC]
            float2 v[R2];
            if constexpr (MODE == 2) {
                const float2 y = live ? __ldg(ry + (size_t)b * ny + iy) : make_float2(0.0f, 0.0f);
                const float2* p = prop + (size_t)k * ny + iy;
                const float2* const x = rx + (size_t)b * N + k;
#pragma unroll
                for (int t = 0; t < R2; ++t, p += R1 * ny)
                    v[t] = live ? cmul(cmul(__ldg(p), __ldg(x + R1 * t)), y) : make_float2(0.0f, 0.0f);
            } else {
                if (EARLY > 0 && !SOON && q == 0) ask();
#pragma unroll
                for (int j = 0; j < R2; ++j) v[j] = j ? cmul(m[j & 1][j * TC], tw[j * R1 + k]) : m[0][0];
                if (SOON && q == 0 && zero) {
                    float2 s = v[0];
#pragma unroll
                    for (int j = 1; j < R2; ++j) s = padd(s, v[j]);
                    s = short_mean<R2>(s);
                    mean[sub] = cmul(make_float2(R2 * s.x, R2 * s.y), pe[0]);
#pragma unroll
                    for (int j = 0; j < R2; ++j) v[j] = psub(v[j], s);
                }
                dft_reg<R2, -1>(v);
                const float2* p = P0 + (size_t)(k + R1 * (q == 0 ? EARLY : 0)) * ny;
#pragma unroll
                for (int t = 0; t < R2; ++t) {
                    if (t < EARLY && q == 0) {
                        v[t] = cmul(v[t], pe[t < EARLY ? t : 0]);
                    } else {
                        v[t] = cmul(v[t], live ? __ldg(p) : make_float2(0.0f, 0.0f));
                        p += R1 * ny;
                    }
                }
            }
            if constexpr (MODE == 0 || MODE == 2) {
                dft_reg<R2, +1>(v);
                if (SOON && q == 0 && zero) {
                    const float2 z = mean[sub];
#pragma unroll
                    for (int j = 0; j < R2; ++j) v[j] = padd(v[j], z);
                }
#pragma unroll
                for (int j = 0; j < R2; ++j) {
                    // (j = 0 has no twiddle: scale + rest is 1 / (nx ny))
                    m[j & 1][j * TC] = j           ? cmulc(v[j], tw_back[j * R1 + k])
                                       : MODE == 0 ? make_float2(fmaf(v[0].x, scale, v[0].x * rest),
                                                                 fmaf(v[0].y, scale, v[0].y * rest))
                                                   : v[0];
                }
            } else {
                if (live && (MODE == 1 || det.store)) {
                    float2* out = psi + ((size_t)b * N + k) * ny + iy;
#pragma unroll
                    for (int t = 0; t < R2; ++t, out += R1 * ny) __stcg(out, v[t]);
                }
                if constexpr (MODE == 3) {
#pragma unroll
                    for (int t = 0; t < R2; ++t) m[t & 1][t * TC] = v[t];  // row k + R1 t in the slot of (t, k)
                }
            }
        }
        if (!SOON && zero)
            give_mean<R1, R2, TC>(M, cmul(make_float2(R2 * mean[sub].x, R2 * mean[sub].y), __ldg(P0)), tw_back, scale, rest);
        if constexpr (MODE == 1) fence_proxy_async_shared();
        group_sync<NT>(1 + sub);
        if constexpr (MODE == 0 || MODE == 2) {
#pragma unroll
            for (int q = 0; q < QA; ++q) {
                const int j = item + NT / TC * q;
                const bool on = R2 * TC % NT == 0 || j < R2;
                float2 v[R1];
                if (on) {
                    const float2* const in[2] = {M + j * TC, M + (SWAP ? j ^ 1 : j) * TC};
#pragma unroll
                    for (int r = 0; r < R1; ++r) v[r] = in[r & 1][r * (R2 * TC)];
                    dft_reg<R1, +1>(v);
                }
                __syncwarp();
                if (on) {
                    float2* out = M + j * TC;
#pragma unroll
                    for (int r = 0; r < R1; ++r) out[r * (R2 * TC)] = v[r];
                }
            }
            fence_proxy_async_shared();
            group_sync<NT>(1 + sub);
            if (u == 0) {
#pragma unroll
                for (int n = 0; n < N / BOXH; ++n)
                    tma_store_2d(&map, smem_two_cols + s * TILE + n * BOXH * TC, 2 * TC * (int)g, (int)b * N + n * BOXH);
                bulk_commit();
            }
        }
        if constexpr (MODE == 3) {
            // every channel's share of this tile, summed in float64 in a fixed order: a thread's entries, its warp by
            // shuffles, the warps in order
            constexpr int NW = NT / 32;
            __shared__ double sums[P::SUBS][NW];
            const float2* const T = smem_two_cols + s * TILE;
            const int* ptr = det.ptr + (size_t)g * det.n_ch;
            for (int ch = 0; ch < det.n_ch; ++ch) {
                const int e1 = __ldg(ptr + ch + 1);
                double sum = 0.0;
                for (int e = __ldg(ptr + ch) + u; e < e1; e += NT) {
                    const int2 q = __ldg(det.ent + e);
                    const int row = q.x / TC, kk = row % R1, t = row / R1;
                    const float2 v = T[((SWAP ? t ^ (kk & 1) : t) + R2 * kk) * TC + q.x % TC];
                    sum += (double)((v.x * v.x + v.y * v.y) * __int_as_float(q.y));
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (u % 32 == 0) sums[sub][u / 32] = sum;
                if (ch + 1 == det.n_ch) fence_proxy_async_shared();
                group_sync<NT>(1 + sub);
                if (u == 0) {
                    double t = 0.0;
                    for (int w = 0; w < NW; ++w) t += sums[sub][w];
                    det.partial[((size_t)b * order.groups + g) * det.n_ch + ch] = t;
                }
                group_sync<NT>(1 + sub);
            }
        }
    }
    if (u == 0) bulk_wait_all();  // the stores read this block's shared memory: finish them before it is freed
    __syncthreads();
    // after an abandoned wait: no copy into this block's shared memory may be in flight when it ends
    if (MODE != 2 && tid == 0) {
        int any = 0;
        for (unsigned q = 0; q < subs; ++q) any |= failed[q];
        if (any)
            for (int s = 0; s < buffers; ++s)
                if (issued[s]) mbar_wait_bounded(&full[s], (issued[s] - 1) & 1);
    }
}

// ---- launches --------------------------------------------------------------------------------------------------------
template <int N, bool SPREAD>
void launch_two_rows_s(Context& ctx, const float2* table, float2* psi, const float2* tmul, int nx, long long nrows, int inv,
                       int fwd, float scale) {
    using P = RowPlan<N, SPREAD>;
    static PerDevice setup;
    const int resident = setup.get([] {
        allow_shared(two_rows<N, SPREAD>, P::SMEM);
        int n = 0;
        SIMK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, two_rows<N, SPREAD>, P::NT, P::SMEM));
        return std::max(1, n);
    });
    const long long tiles = (nrows + P::GR - 1) / P::GR, per = P::NT / P::GT;
    const int grid = (int)std::min<long long>((tiles + per - 1) / per, (long long)resident * ctx.sm_count);
    two_rows<N, SPREAD><<<grid, P::NT, P::SMEM, ctx.stream>>>(psi, tmul, table, (unsigned)nx,
                                                              fast_div((unsigned)(nrows / nx)), inv, fwd, scale,
                                                              ctx.wave_t);
    SIMK_CUDA(cudaGetLastError());
    ++ctx.launches;
}

template <int N>
bool launch_two_rows(Context& ctx, const float2* table, float2* psi, const float2* tmul, int nx, long long nrows, int inv,
                     int fwd, float scale) {
    if (nrows >= (1LL << 31) - (1 << 20)) return false;
    // Up to four rows a multiprocessor (one 512^2 wave) a launch is one tile's chain of steps long: one row a warp is the
    // shorter chain (512^2, one wave: 7.23 -> 6.90 us a pass, rows and columns; from two waves on no difference). Each row's
    // arithmetic is the same.
    if constexpr (RowPlan<N, true>::GR == 1 && RowPlan<N>::GR == 2) {
        if (nrows <= 4LL * ctx.sm_count) {
            launch_two_rows_s<N, true>(ctx, table, psi, tmul, nx, nrows, inv, fwd, scale);
            return true;
        }
    }
    launch_two_rows_s<N, false>(ctx, table, psi, tmul, nx, nrows, inv, fwd, scale);
    return true;
}

template <int N, int MODE> bool launch_two_cols_m(Context& ctx, const float2* table, const TwoPassCols& a, int* groups) {
    using P = ColPlan<N>;
    const long long g = (a.ny + P::TC - 1) / P::TC, tiles = g * a.count;
    if (tiles >= (1LL << 31) - (1 << 20) || a.ny % 2) return false;  // rows of a multiple of 16 bytes
    static PerDevice setup;
    setup.get([] { return allow_shared(two_cols<N, MODE>, P::smem(P::NB)); });
    TwoDetect d{};
    if constexpr (MODE == 3) {
        const DetectorPlan::TileChannels& t = a.det->plan->tiles(P::TC);
        d.ptr = t.ptr.as<int>();
        d.ent = t.ent.as<int2>();
        d.partial = a.det->partial;
        d.n_ch = a.det->plan->n_channels;
        d.store = a.det->store;
        *groups = (int)g;
    }
    // a small launch spreads over the SMs: no more sub-blocks a block than its tiles give work, no more buffers than
    // its share of them
    const long long share = (tiles + ctx.sm_count - 1) / ctx.sm_count;
    const int subs = (int)std::min<long long>(P::SUBS, share);
    const int buffers = MODE == 2 ? subs : (int)std::min<long long>(P::NB, std::max<long long>(subs + 1, share));
    const int grid = (int)std::min<long long>((tiles + subs - 1) / subs, ctx.sm_count);
    TileOrder order;
    order.round = fast_div((unsigned)(subs * g));
    order.subs = fast_div((unsigned)subs);
    order.rest = fast_div((unsigned)std::max(1, a.count % subs));
    order.groups = (unsigned)g;
    order.waves = (unsigned)(a.count / subs * subs);
    order.tiles = (unsigned)tiles;
    const double inverse = MODE == 0 ? 1.0 / ((double)N * a.ny) : 1.0;
    const float scale = (float)inverse;
    const float2* const back = MODE == 0 ? twopass_table(ctx, N, (long long)N * a.ny) : table;
    const CUtensorMap map = encode_tensor_map_2d(a.psi, 2ULL * a.ny, (unsigned long long)a.count * N, 2 * P::TC, P::BOXH);
    two_cols<N, MODE><<<grid, P::NT * subs, P::smem(buffers), ctx.stream>>>(
        map, a.psi, MODE == 2 ? a.spectrum : a.P, table, back, scale, (float)(inverse - (double)scale), a.ny, order,
        buffers, ctx.err_flag.as<int>(), a.p_row, a.rx, a.ry, d);
    SIMK_CUDA(cudaGetLastError());
    ++ctx.launches;
    return true;
}

template <int N> bool launch_two_cols(Context& ctx, const float2* table, const TwoPassCols& a, int* groups) {
    switch (a.mode) {
        case 0: return launch_two_cols_m<N, 0>(ctx, table, a, groups);
        case 1: return launch_two_cols_m<N, 1>(ctx, table, a, groups);
        case 2: return launch_two_cols_m<N, 2>(ctx, table, a, groups);
        default: return launch_two_cols_m<N, 3>(ctx, table, a, groups);
    }
}

}  // namespace simk
