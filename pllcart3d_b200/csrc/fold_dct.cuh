// DCT passes of the Poisson solve (phisolver_dct, pllcart3d.c:2035, 2104
// through fftw_3d.h:45-106) along an axis whose length has no FFT form here:
// the dense product with FFTW's REDFT10 / REDFT01 cosine matrix, folded.
//
// cos(pi k (2j+1) / 2n) at n-1-j is (-1)^k times its value at j, so the DCT-II
// of a line is two products of half the size, the even k from x_j + x_{n-1-j}
// and the odd k from x_j - x_{n-1-j}; the DCT-III forms the sums over even and
// odd k for the first half of the line and combines them by sum and difference
// into both halves: half the multiplications of the full matrix.
//
// A block holds 32 whole lines in shared memory, folded (or sorted by parity)
// on the way in as FP64, and multiplies them on the FP64 tensor pipe (mma.sync
// m8n8k4: 8 outputs x 8 lines x 4 terms; tcgen05 has no FP64 kind).  A warp
// takes 8 outputs of both parities for all 32 lines, so that each matrix
// fragment, read from a table in fragment order, serves 4 products.  The
// storage type is T, the arithmetic FP64 in every form.
// Both operand fragments put element (lane / 4, lane % 4) of an 8 x 4 piece on
// a lane, so data and matrix trade places by swapping the operands: lines
// along the contiguous axis (CONTIG) are the rows of the product and leave 4
// neighbouring outputs on a lane; otherwise the outputs are, and neighbouring
// lines do.
#pragma once

#include <cuda_runtime.h>

#include "dct_kernels.cuh"
#include "fft_dct.cuh"

namespace pll {
namespace {

constexpr int FOLD_LINES = 32;
constexpr int FOLD_MAX = 512;   // longest line (its 32 lines fill 152 KB)

// n values: half of them, in 4-term and 8-output groups
__host__ __device__ constexpr int fold_kb(int n) { return ((n + 1) / 2 + 3) / 4; }
__host__ __device__ constexpr int fold_mb(int n) { return ((n + 1) / 2 + 7) / 8; }
// warps of a block: no more than 8, the output groups spread evenly over them
inline int fold_warps(int n)
{
    const int mb = fold_mb(n), rounds = (mb + 7) / 8;
    return (mb + rounds - 1) / rounds;
}
// doubles of one table: [parity][output group][term group][lane]
inline long fold_table(int n) { return 2L * fold_mb(n) * fold_kb(n) * 32; }

template <bool CONTIG>
struct FoldPitch {   // row of FOLD_LINES doubles: fragment reads (and the
    // transposing stores of contiguous lines) spread over the banks
    static constexpr int value = CONTIG ? FOLD_LINES + 5 : FOLD_LINES + 4;
};
template <bool CONTIG>
size_t fold_smem(int n)
{
    return sizeof(double) * 2 * (size_t)fold_kb(n) * 4 * FoldPitch<CONTIG>::value;
}

// KIND 0: DCT-II, 1: DCT-III of n points, lines as FftLines
template <int KIND, bool CONTIG, typename T>
__device__ __forceinline__ void k_dct_fold_run(const uint3 blockIdx, const dim3 gridDim, FftLines d, int n,
                                               const T* __restrict__ in, T* __restrict__ out,
                                               const double* __restrict__ table)
{
    constexpr int P = FoldPitch<CONTIG>::value;
    extern __shared__ __align__(16) unsigned char fold_raw[];
    double* X = (double*)fold_raw;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const int half = (n + 1) / 2, KB = fold_kb(n), MB = fold_mb(n);
    double* X1 = X + KB * 4 * P;
    const int L0 = blockIdx.x * FOLD_LINES, nl = min(FOLD_LINES, d.lines - L0);
    auto line_in = [&](int l) { return in + (long)((L0 + l) / d.inner) * d.sa_in + (long)((L0 + l) % d.inner) * d.sb_in; };
    auto line_out = [&](int l) {
        return out + (long)((L0 + l) / d.inner) * d.sa_out + (long)((L0 + l) % d.inner) * d.sb_out;
    };

    auto fetch = [&](const T* x, int j, int l) {
        const long se = CONTIG ? 1 : d.se_in;
        double e = 0.0, o = 0.0;
        if (l < nl) {
            if (KIND == 0) {
                if (j < half) {
                    const double a = (double)x[j * se], b = (double)x[(n - 1 - j) * se];
                    const bool mid = 2 * j + 1 == n;
                    e = mid ? a : a + b;
                    o = a - b;
                }
            } else {
                if (2 * j < n) e = (double)x[2 * j * se];
                if (2 * j + 1 < n) o = (double)x[(2 * j + 1) * se];
            }
        }
        X[j * P + l] = e;
        X1[j * P + l] = o;
    };
    if (CONTIG) {
        for (int l = warp; l < FOLD_LINES; l += W) {
            const T* x = line_in(l < nl ? l : 0);
#pragma unroll 4
            for (int j = lane; j < KB * 4; j += 32) fetch(x, j, l);
        }
    } else {
        const T* x = line_in(lane < nl ? lane : 0);
#pragma unroll 4
        for (int j = warp; j < KB * 4; j += W) fetch(x, j, lane);
    }
    __syncthreads();

    const int g = lane >> 2, tg = lane & 3;
    for (int mb = warp; mb < MB; mb += W) {
        double acc[2][4][2];
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int f = 0; f < 4; ++f) acc[p][f][0] = acc[p][f][1] = 0.0;
        const double* t0 = table + (long)mb * KB * 32 + lane;
        const double* t1 = t0 + (long)MB * KB * 32;
        const double* x0 = X + tg * P + g;
        const double* x1 = X1 + tg * P + g;
#pragma unroll 4
        for (int kb = 0; kb < KB; ++kb) {
            const double m0 = __ldg(t0 + kb * 32), m1 = __ldg(t1 + kb * 32);
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const double e = x0[kb * 4 * P + f * 8], o = x1[kb * 4 * P + f * 8];
                if (CONTIG) {
                    dmma_8x8x4(acc[0][f][0], acc[0][f][1], e, m0);
                    dmma_8x8x4(acc[1][f][0], acc[1][f][1], o, m1);
                } else {
                    dmma_8x8x4(acc[0][f][0], acc[0][f][1], m0, e);
                    dmma_8x8x4(acc[1][f][0], acc[1][f][1], m1, o);
                }
            }
        }
#pragma unroll
        for (int f = 0; f < 4; ++f)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int l = f * 8 + (CONTIG ? g : 2 * tg + h), j = mb * 8 + (CONTIG ? 2 * tg + h : g);
                if (l >= nl || j >= half) continue;
                T* y = line_out(l);
                const long se = CONTIG ? 1 : d.se_out;
                const double e = acc[0][f][h], o = acc[1][f][h];
                if (KIND == 0) {
                    y[2 * j * se] = (T)(e * d.scale);
                    if (2 * j + 1 < n) y[(2 * j + 1) * se] = (T)(o * d.scale);
                } else {
                    y[j * se] = (T)((e + o) * d.scale);
                    if (2 * j + 1 < n) y[(n - 1 - j) * se] = (T)((e - o) * d.scale);
                }
            }
    }
}
template <int KIND, bool CONTIG, typename T>
__global__ void __launch_bounds__(256) k_dct_fold(FftLines d, int n, const T* __restrict__ in, T* __restrict__ out,
                                                  const double* __restrict__ table)
{
    if (!after_previous()) return;
    k_dct_fold_run<KIND, CONTIG, T>(blockIdx, gridDim, d, n, in, out, table);
}
template <int KIND, bool CONTIG, typename T>
struct k_dct_fold_b {
    static constexpr auto run = &k_dct_fold_run<KIND, CONTIG, T>;
    static constexpr int maxt = 256, minb = 0;
    static constexpr bool chained = true;
};

}  // namespace
}  // namespace pll
