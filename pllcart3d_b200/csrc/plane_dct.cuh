// The Poisson solve's transforms plane by plane: both DCT axes of an x plane
// in shared memory, the right-hand side formed on the way in (divergence,
// pllcart3d.c:1976-2033) and phi's ghost points written on the way out
// (update_phi_ghosts), so that between the velocities and phi the field is
// written and read twice (around the x-tridiagonals) instead of six times and
// three launches stand where seven did.  For planes of 32, 64 or 128 points a
// side and at most 4096 (34 KB): there a pass over the lines is launch and
// load latency.  64x32x32 FP64 265 -> 235 us a step, 128x64x64 0.536 -> 0.505
// ms, 24 members in FP32 13.3 -> 12.9 ms for 4 steps.  A 128 x 128 plane (133
// KB) leaves one block per SM with nothing beside it while it loads, and its
// two transforms took 77 + 46 us where the line passes take 73 + 57; larger
// planes stay with those (fft_dct.cuh, fold_dct.cuh).
//
// A plane's lines are transformed in place, by the method and the factors of
// fft_dct.cuh: along y the neighbouring columns 2q, 2q+1 share a complex DFT
// (one 16-byte word), along z the rows q, q + NY/2.  Frequency k1 + R1 k2 of a
// line stays at position k2 + R2 k1, where the four steps leave it: the modes
// are stored, solved and read back in that order (their eigenvalues are laid
// out to match), so both copies are contiguous and no step permutes.
#pragma once

#include <cuda_runtime.h>

#include "fft_dct.cuh"
#include "step_kernels.cuh"

namespace pll {
namespace {

template <int NY, int NZ>
struct PlaneShape {
    static constexpr int CELLS = NY * NZ, PITCH = NZ + 2;
    static constexpr int TH = CELLS >= 4096 ? 512 : 256;
    static constexpr size_t SMEM = sizeof(double) * NY * PITCH;
};

// lines along y (columns 2q, 2q+1) and along z (rows q, q + NY/2)
template <int NY, int NZ>
struct PlaneY {
    static constexpr int N = NY, Q = NZ / 2;
    double* P;
    __device__ __forceinline__ cplx<double> get(int q, int p) const
    {
        const double2 v = *(const double2*)(P + p * PlaneShape<NY, NZ>::PITCH + 2 * q);
        return {v.x, v.y};
    }
    __device__ __forceinline__ void set(int q, int p, cplx<double> v) const
    {
        *(double2*)(P + p * PlaneShape<NY, NZ>::PITCH + 2 * q) = make_double2(v.re, v.im);
    }
};
template <int NY, int NZ>
struct PlaneZ {
    static constexpr int N = NZ, Q = NY / 2, HALF = (NY / 2) * PlaneShape<NY, NZ>::PITCH;
    double* P;
    __device__ __forceinline__ cplx<double> get(int q, int p) const
    {
        const double* a = P + q * PlaneShape<NY, NZ>::PITCH + p;
        return {a[0], a[HALF]};
    }
    __device__ __forceinline__ void set(int q, int p, cplx<double> v) const
    {
        double* a = P + q * PlaneShape<NY, NZ>::PITCH + p;
        a[0] = v.re;
        a[HALF] = v.im;
    }
};

// position of frequency k
template <int N>
__device__ __forceinline__ int plane_pos(int k)
{
    return k / FftShape<N>::R1 + FftShape<N>::R2 * (k % FftShape<N>::R1);
}

// DCT-II of every line, from Makhoul's order to plane_pos
template <int TH, typename L>
__device__ __forceinline__ void plane_forward(const L& A, const double2* __restrict__ tw,
                                              const double2* __restrict__ wq)
{
    constexpr int N = L::N, Q = L::Q, R1 = FftShape<N>::R1, R2 = FftShape<N>::R2;
    for (int t = threadIdx.x; t < Q * R2; t += TH) {
        const int q = t % Q, n2 = t / Q;
        cplx<double> v[R1];
#pragma unroll
        for (int n1 = 0; n1 < R1; ++n1) v[n1] = A.get(q, n2 + R2 * n1);
        Dft<double, R1, -1>::run(v);
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) {
            const double2 w = tw[n2 * k1];
            A.set(q, n2 + R2 * k1, k1 == 0 ? v[k1] : cmul(v[k1], w.x, -w.y));
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < Q * R1; t += TH) {
        const int q = t % Q, k1 = t / Q;
        cplx<double> v[R2];
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) v[n2] = A.get(q, n2 + R2 * k1);
        Dft<double, R2, -1>::run(v);
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) A.set(q, k2 + R2 * k1, v[k2]);
    }
    __syncthreads();
    // split the two lines, k and N-k together (fft_dct.cuh)
    for (int t = threadIdx.x; t < Q * (N / 2 + 1); t += TH) {
        const int q = t % Q, k = t / Q, km = (N - k) & (N - 1);
        const int pk = plane_pos<N>(k), pm = plane_pos<N>(km);
        const cplx<double> zk = A.get(q, pk), zm = A.get(q, pm);
        const double2 w = wq[k], w2 = wq[km];
        const cplx<double> p1 = cmul(zk, w.x, -w.y), p2 = cmul(cplx<double>{zm.re, -zm.im}, w.x, -w.y);
        const cplx<double> r1 = cmul(zm, w2.x, -w2.y), r2 = cmul(cplx<double>{zk.re, -zk.im}, w2.x, -w2.y);
        A.set(q, pk, {p1.re + p2.re, p1.im - p2.im});
        if (pm != pk) A.set(q, pm, {r1.re + r2.re, r1.im - r2.im});
    }
    __syncthreads();
}

// DCT-III of every line, from plane_pos to Makhoul's order: the same steps
// backwards
template <int TH, typename L>
__device__ __forceinline__ void plane_inverse(const L& A, const double2* __restrict__ tw,
                                              const double2* __restrict__ wq)
{
    constexpr int N = L::N, Q = L::Q, R1 = FftShape<N>::R1, R2 = FftShape<N>::R2;
    for (int t = threadIdx.x; t < Q * (N / 2 + 1); t += TH) {
        const int q = t % Q, k = t / Q, km = (N - k) & (N - 1);
        const int pk = plane_pos<N>(k), pm = plane_pos<N>(km);
        const cplx<double> xk = A.get(q, pk);
        const cplx<double> xm = k == 0 ? cplx<double>{0.0, 0.0} : A.get(q, pm);   // x_N = 0
        const double2 w = wq[k], w2 = wq[km];
        A.set(q, pk, cmul(cplx<double>{xk.re + xm.im, xk.im - xm.re}, w.x, w.y));
        if (pm != pk) A.set(q, pm, cmul(cplx<double>{xm.re + xk.im, xm.im - xk.re}, w2.x, w2.y));
    }
    __syncthreads();
    for (int t = threadIdx.x; t < Q * R1; t += TH) {
        const int q = t % Q, k1 = t / Q;
        cplx<double> v[R2];
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) v[k2] = A.get(q, k2 + R2 * k1);
        Dft<double, R2, 1>::run(v);
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) {
            const double2 w = tw[n2 * k1];
            A.set(q, n2 + R2 * k1, n2 == 0 ? v[n2] : cmul(v[n2], w.x, w.y));
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < Q * R2; t += TH) {
        const int q = t % Q, n2 = t / Q;
        cplx<double> v[R1];
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) v[k1] = A.get(q, n2 + R2 * k1);
        Dft<double, R1, 1>::run(v);
#pragma unroll
        for (int n1 = 0; n1 < R1; ++n1) A.set(q, n2 + R2 * n1, v[n1]);
    }
    __syncthreads();
}

// one x plane per block: hat[x][..][..] = both DCT-IIs of Re / (dt alpha) div u
template <typename T, int NY, int NZ>
__device__ __forceinline__ void k_dct_plane_fwd_run(const uint3 blockIdx, const dim3 gridDim, Geo G, Rng R, Consts K,
                                                    const T* __restrict__ u, const T* __restrict__ v,
                                                    const T* __restrict__ w, T* __restrict__ hat,
                                                    const double* __restrict__ scal, double alpha,
                                                    const double2* __restrict__ twy, const double2* __restrict__ wqy,
                                                    const double2* __restrict__ twz, const double2* __restrict__ wqz)
{
    using S = PlaneShape<NY, NZ>;
    extern __shared__ __align__(16) unsigned char pd_raw[];
    double* P = (double*)pd_raw;
    const long sx = G.sx, sy = G.sy;
    const long base = (long)(R.is + blockIdx.x) * sx + (long)R.js * sy + R.ks;
    const T ihx = (T)K.ihx, ihy = (T)K.ihy, ihz = (T)K.ihz, fac = (T)(K.Re / (scal[S_DT] * alpha));
#pragma unroll
    for (int t = 0; t < S::CELLS / S::TH; ++t) {
        const int e = threadIdx.x + t * S::TH, z = e % NZ, y = e / NZ;
        const long id = base + (long)y * sy + z;
        const T dx = u[id + sx] - u[id], dy = v[id + sy] - v[id], dz = w[id + 1] - w[id];
        P[mperm<NY>(y) * S::PITCH + mperm<NZ>(z)] =
            (double)mul_rn_(fac, fma(dz, ihz, fma(dy, ihy, mul_rn_(dx, ihx))));
    }
    __syncthreads();
    plane_forward<S::TH>(PlaneY<NY, NZ>{P}, twy, wqy);
    plane_forward<S::TH>(PlaneZ<NY, NZ>{P}, twz, wqz);
    T* out = hat + (long)blockIdx.x * S::CELLS;
#pragma unroll
    for (int e = threadIdx.x; e < S::CELLS; e += S::TH) out[e] = (T)P[(e / NZ) * S::PITCH + e % NZ];
}
template <typename T, int NY, int NZ>
__global__ void __launch_bounds__(PlaneShape<NY, NZ>::TH)
    k_dct_plane_fwd(Geo G, Rng R, Consts K, const T* __restrict__ u, const T* __restrict__ v, const T* __restrict__ w,
                    T* __restrict__ hat, const double* __restrict__ scal, double alpha,
                    const double2* __restrict__ twy, const double2* __restrict__ wqy, const double2* __restrict__ twz,
                    const double2* __restrict__ wqz)
{
    if (!after_previous()) return;
    k_dct_plane_fwd_run<T, NY, NZ>(blockIdx, gridDim, G, R, K, u, v, w, hat, scal, alpha, twy, wqy, twz, wqz);
}
template <typename T, int NY, int NZ>
struct k_dct_plane_fwd_b {
    static constexpr auto run = &k_dct_plane_fwd_run<T, NY, NZ>;
    static constexpr int maxt = PlaneShape<NY, NZ>::TH, minb = 0;
    static constexpr bool chained = true;
};

// and back: phi = both DCT-IIIs of hat times scale, with its ghost points
template <typename T, int NY, int NZ>
__device__ __forceinline__ void k_dct_plane_inv_run(const uint3 blockIdx, const dim3 gridDim, Geo G, Rng R,
                                                    const T* __restrict__ hat, T* __restrict__ phi, double scale,
                                                    const double2* __restrict__ twy, const double2* __restrict__ wqy,
                                                    const double2* __restrict__ twz, const double2* __restrict__ wqz)
{
    using S = PlaneShape<NY, NZ>;
    extern __shared__ __align__(16) unsigned char pd_raw[];
    double* P = (double*)pd_raw;
    const T* in = hat + (long)blockIdx.x * S::CELLS;
#pragma unroll
    for (int e = threadIdx.x; e < S::CELLS; e += S::TH) P[(e / NZ) * S::PITCH + e % NZ] = (double)in[e];
    __syncthreads();
    plane_inverse<S::TH>(PlaneZ<NY, NZ>{P}, twz, wqz);
    plane_inverse<S::TH>(PlaneY<NY, NZ>{P}, twy, wqy);
    const int i = R.is + blockIdx.x;
    const long sx = G.sx, sy = G.sy, base = (long)i * sx + (long)R.js * sy + R.ks;
#pragma unroll 2
    for (int e = threadIdx.x; e < S::CELLS; e += S::TH) {
        const int z = e % NZ, y = e / NZ;
        const long id = base + (long)y * sy + z;
        const T x = (T)mul_rn_(P[mperm<NY>(y) * S::PITCH + mperm<NZ>(z)], scale);
        phi[id] = x;
        if (z == 0) phi[id - 1] = x;
        if (z == NZ - 1) phi[id + 1] = x;
        if (y == 0) phi[id - sy] = x;
        if (y == NY - 1) phi[id + sy] = x;
        if (i == R.is) phi[id - sx] = x;
        if (i == R.ie) phi[id + sx] = x;
    }
}
template <typename T, int NY, int NZ>
__global__ void __launch_bounds__(PlaneShape<NY, NZ>::TH)
    k_dct_plane_inv(Geo G, Rng R, const T* __restrict__ hat, T* __restrict__ phi, double scale,
                    const double2* __restrict__ twy, const double2* __restrict__ wqy, const double2* __restrict__ twz,
                    const double2* __restrict__ wqz)
{
    if (!after_previous()) return;
    k_dct_plane_inv_run<T, NY, NZ>(blockIdx, gridDim, G, R, hat, phi, scale, twy, wqy, twz, wqz);
}
template <typename T, int NY, int NZ>
struct k_dct_plane_inv_b {
    static constexpr auto run = &k_dct_plane_inv_run<T, NY, NZ>;
    static constexpr int maxt = PlaneShape<NY, NZ>::TH, minb = 0;
    static constexpr bool chained = true;
};

}  // namespace
}  // namespace pll
