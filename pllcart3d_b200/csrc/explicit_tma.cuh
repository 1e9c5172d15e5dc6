// Explicit operator + ADI right-hand side (Hc_op/Hu_op/Hv_op/Hw_op,
// pllcart3d.c:1539-1980, with the source assembly of concentration / xmom /
// ymom / zmom, L573-590, L970-989, L1127-1146, L1280-1298) as a
// plane-marching kernel with TMA-staged shared-memory tiles.
//
// A block owns a tile of XT_TJ rows (j) x XT_TK cells (k) and walks ni planes
// along x (chosen per launch, launch_explicit_tma).  Every plane's tiles arrive by cp.async.bulk.tensor (one
// thread issues them; an mbarrier per ring slot counts the bytes): q with a
// +-3 halo in j and k (the WENO5 stencils along y and z), and, with a +-1
// halo, each field the variable reads at a j or k offset (velocities,
// viscosity edges, c).  A ring of XT_NS plane slots keeps planes i-1, i, i+1
// resident while plane i+2 is in flight.  Values read only along x at the
// thread's own (j, k) -- the x WENO5 window q(i-3 .. i+3), the x-face
// viscosity and velocity, c, pg, H_old -- stay in registers, one plain
// coalesced load per plane.  Closures and the stale-D2 hazard are
// k_explicit's, and so are the formulas in other words: differences undivided,
// the stencils read in the upwind direction, WENO5 as the central difference
// plus one weighted correction (weno_corr), stresses as fluxes.
// TMA boxes start on 16-byte boundaries: the k tiles start at k0 = 1 + 32 b,
// so the +-1 box starts at k0-1 (a multiple of 32 elements) and the q box at
// k0-3 (FP64: a multiple of 2) or k0-5 (FP32: a multiple of 4).  No
// multicast.  Every mbarrier wait is bounded; a wait that runs out sets
// ST_TIMEOUT, and the issuing thread drains its copies before the block ends.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "step_kernels.cuh"

namespace pll {
namespace {

constexpr int XT_TK = 32;   // k cells per tile (one warp across)
constexpr int XT_TJ = 8;    // j rows per tile (one warp each)
constexpr int XT_NS = 4;    // plane slots of the ring
constexpr int XT_THREADS = XT_TK * XT_TJ;
constexpr long long XT_WAIT_CYCLES = 2000000000LL;   // ~1 s of SM clock

// blocks per SM asked of the compiler.  With FP32 weights v and w fit three
// (80 registers, 12-20 bytes spilled): 0.92 -> 0.87 and 0.87 -> 0.81 ms per
// launch at 512x256x256.  u (0.76 -> 0.87) and the FP64 weights (0.13 -> 0.18
// at 256x128x128) spill more and lose; c has three by itself (0: no demand).
template <int VAR, typename real>
struct XtBlocks {
    static constexpr int value = PLL_WENO_F32 && sizeof(real) == 8 && VAR >= VV ? 3 : 0;
};

// fields staged with a +-1 halo, per variable (the ones read at a j or k
// offset besides q); order fixes the slot layout
//   VC: v, w            VU: v, w, mu_xy, mu_xz
//   VV: u, w, mu_yz, mu_cell, c_new            VW: u, v, mu_yz, mu_cell
template <int VAR>
struct XtSet {
    static constexpr int NA = VAR == VC ? 2 : VAR == VV ? 5 : 4;
};

template <typename real>
struct XtGeom {
    static constexpr int KB1 = sizeof(real) == 8 ? XT_TK + 2 : XT_TK + 4;   // +-1 box width (16-byte multiple)
    static constexpr int JB1 = XT_TJ + 2;
    static constexpr int H3 = sizeof(real) == 8 ? 3 : 5;                   // q box starts at k0 - H3
    static constexpr int KB3 = sizeof(real) == 8 ? XT_TK + 6 : XT_TK + 8;
    static constexpr int JB3 = XT_TJ + 6;
    static constexpr int T1 = ((JB1 * KB1 * (int)sizeof(real)) + 127) / 128 * 128;
    static constexpr int T3 = ((JB3 * KB3 * (int)sizeof(real)) + 127) / 128 * 128;
};

template <typename real, int VAR>
struct XtSmem {
    static constexpr int NA = XtSet<VAR>::NA;
    static constexpr int SLOT = NA * XtGeom<real>::T1 + XtGeom<real>::T3;
    static constexpr int BAR_OFF = XT_NS * SLOT;
    static constexpr int TOTAL = BAR_OFF + 64;
    static constexpr int DYN = TOTAL + 128;   // slack for 128-byte alignment
};

// the tensor maps of one launch: q (+-3 halo box) and the +-1 fields
struct XtMaps {
    CUtensorMap q;
    CUtensorMap a[5];
};

__device__ __forceinline__ uint32_t xt_saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void xt_tma_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
        "[%2];\n" ::"r"(xt_saddr(dst)),
        "l"((uint64_t)map), "r"(xt_saddr(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

__device__ __forceinline__ bool xt_try_wait(uint64_t* b, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(xt_saddr(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait for the completion of phase `parity`
__device__ __noinline__ bool xt_wait(uint64_t* b, uint32_t parity)
{
    if (xt_try_wait(b, parity)) return true;
    const long long t0 = clock64();
    while (!xt_try_wait(b, parity))
        if (clock64() - t0 > XT_WAIT_CYCLES) return false;
    return true;
}

// the type that evaluates the WENO5 weights of a state in `real`
template <typename real>
struct XtWeno {
    using type = real;
};
#if PLL_WENO_F32
template <>
struct XtWeno<double> {
    using type = float;
};
#endif

// the ENO-2 closure's correction (the first and last two points of a range):
// half the smaller of the two second differences, b behind and c ahead of the
// point in the upwind sense; ties go to the lower line index, b for up
template <typename real>
__device__ __forceinline__ real eno_corr(real b, real c, bool up)
{
    const bool first = up ? fabs(b) <= fabs(c) : !(fabs(c) <= fabs(b));
    return (real)0.5 * (first ? b : c);
}

// b of the closure where it lies outside the range: what an earlier pass of
// the routine left in its scratch line, in undivided differences of this axis
template <int AXIS, typename real>
__device__ __forceinline__ real eno_behind(const real* __restrict__ qg, const Geo& G, const Rng& R, const Consts& K,
                                           int m, bool up, real b)
{
    const int s = AXIS == 0 ? R.is : AXIS == 1 ? R.js : R.ks;
    const int e = AXIS == 0 ? R.ie : AXIS == 1 ? R.je : R.ke;
    const double h = AXIS == 0 ? K.hx : AXIS == 1 ? K.hy : K.hz;
    if (up ? m == s : m == e) return stale_d2<real>(qg, G, R, K, AXIS, up ? s - 1 : e + 1) * (real)(2.0 * h * h);
    return b;
}

template <int AXIS>
__device__ __forceinline__ bool eno_band(const Rng& R, int m)
{
    const int s = AXIS == 0 ? R.is : AXIS == 1 ? R.js : R.ks;
    const int e = AXIS == 0 ? R.ie : AXIS == 1 ? R.je : R.ke;
    return (m <= s + 1) | (m >= e - 1);
}

// WENO5 correction in the form's weight type
template <typename real>
__device__ __forceinline__ real xt_weno(real v0, real v1, real v2, real v3, real v4, real a, real b, real c, real d,
                                        real floor4)
{
    if constexpr (std::is_same<typename XtWeno<real>::type, float>::value) {
        return (real)weno_corr((float)v2, (float)a, (float)b, (float)c, (float)d);
    } else {
        const real vmax = fmax(fmax(fmax(fabs(v0), fabs(v1)), fmax(fabs(v2), fabs(v3))), fabs(v4));
        return weno_corr(a, b, c, d, vmax, floor4);
    }
}

// h x |upwind derivative| sense along y or z: p is the point in its shared
// tile, st the tile's step along the axis.  The window is read in the upwind
// direction (up: increasing), so that neither the differences nor anything
// made of them is selected by the sign; the derivative times the velocity is
// |velocity| / h times the result.  c2: the second difference at the point.
template <int AXIS, typename real>
__device__ __forceinline__ real xt_upwind(const real* p, int st, const real* __restrict__ qg, const Geo& G,
                                          const Rng& R, const Consts& K, int m, bool up, real floor4, real& c2)
{
    const int s = up ? st : -st;
    const real* w = p - 3 * s;
    real d[5];
    real q0 = w[0];
#pragma unroll
    for (int t = 0; t < 5; ++t) {
        const real q1 = w[(t + 1) * s];
        d[t] = q1 - q0;
        q0 = q1;
    }
    const real b = d[2] - d[1], c = d[3] - d[2];
    c2 = c;
    if (eno_band<AXIS>(R, m)) return d[2] + eno_corr<real>(eno_behind<AXIS, real>(qg, G, R, K, m, up, b), c, up);
    return d[2] + xt_weno<real>(d[0], d[1], d[2], d[3], d[4], d[1] - d[0], b, c, d[4] - d[3], floor4);
}

// the same along x from the register window D[t] = q(i-2+t) - q(i-3+t)
template <typename real>
__device__ __forceinline__ real xt_upwind_x(const real* D, const real* __restrict__ qg, const Geo& G, const Rng& R,
                                            const Consts& K, int i, bool up, real floor4, real& c2)
{
    const real v2 = up ? D[2] : -D[3], c = D[3] - D[2];
    const real b = (up ? D[2] : D[4]) - (up ? D[1] : D[3]);
    c2 = c;
    if (eno_band<0>(R, i)) return v2 + eno_corr<real>(eno_behind<0, real>(qg, G, R, K, i, up, b), c, up);
    const real a = (up ? D[1] : D[5]) - (up ? D[0] : D[4]), d = (up ? D[4] : D[2]) - (up ? D[3] : D[1]);
    return v2 + xt_weno<real>(up ? D[0] : D[5], D[1], D[2], D[3], D[4], a, b, c, d, floor4);
}

template <int VAR, typename real>
__global__ void __launch_bounds__(XT_THREADS, XtBlocks<VAR, real>::value) k_explicit_tma(const __grid_constant__ XtMaps maps, Geo G, Rng R,
                                                             Consts K, ExplicitArgs<real> A, int ni, int* status)
{
    using GM = XtGeom<real>;
    using SM = XtSmem<real, VAR>;
    constexpr int NA = XtSet<VAR>::NA;
    constexpr int KB1 = GM::KB1, KB3 = GM::KB3;
    extern __shared__ unsigned char xt_raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)xt_raw + 127) & ~(uintptr_t)127);
    uint64_t* bar = (uint64_t*)(sm + SM::BAR_OFF);
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int k0 = 1 + blockIdx.x * XT_TK;
    const int j0 = R.js + blockIdx.y * XT_TJ;
    const int i0 = R.is + blockIdx.z * ni;
    const int i1 = min(i0 + ni - 1, R.ie);
    const int k = k0 + tx, j = j0 + ty;
    const bool live = k >= R.ks && k <= R.ke && j <= R.je;
    const long sx = G.sx, sy = G.sy;
    constexpr uint32_t STAGE_BYTES = (uint32_t)(NA * GM::JB1 * GM::KB1 + GM::JB3 * GM::KB3) * sizeof(real);

    auto slot_of = [&](int p) { return (p - (i0 - 1)) % XT_NS; };
    auto parity_of = [&](int p) { return (uint32_t)(((p - (i0 - 1)) / XT_NS) & 1); };
    auto tile1 = [&](int p, int a) { return (real*)(sm + slot_of(p) * SM::SLOT + a * GM::T1); };
    auto tile3 = [&](int p) { return (real*)(sm + slot_of(p) * SM::SLOT + NA * GM::T1); };
    auto issue = [&](int p) {   // plane p of every staged field into its slot
        uint64_t* b = &bar[slot_of(p)];
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(xt_saddr(b)),
                     "r"(STAGE_BYTES)
                     : "memory");
#pragma unroll
        for (int a = 0; a < NA; ++a) xt_tma_3d(tile1(p, a), &maps.a[a], b, k0 - 1, j0 - 1, p);
        xt_tma_3d(tile3(p), &maps.q, b, k0 - GM::H3, j0 - 3, p);
    };

    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < XT_NS; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(xt_saddr(&bar[s])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        issue(i0 - 1);
        issue(i0);
        issue(i0 + 1);
    }
    __syncthreads();

    // register windows along x at (j, k)
    const long col = (long)j * sy + k;
    const real* __restrict__ q = A.q;
    real D[6], ql;   // differences of q(i-3 .. i+3), and q(i+3)
    {
        real q0 = live ? q[(long)(i0 - 3) * sx + col] : (real)0;
#pragma unroll
        for (int t = 0; t < 6; ++t) {
            ql = live ? q[(long)(i0 - 2 + t) * sx + col] : (real)0;
            D[t] = ql - q0;
            q0 = ql;
        }
    }
    real xa0 = 0, xa1 = 0, xb0 = 0, xb1 = 0;   // VC: u(i), u(i+1); VU: mu_cell(i-1), (i), c(i-1), c(i);
                                               // VV: mu_xy(i), (i+1); VW: mu_xz(i), (i+1)
    const real* __restrict__ xa = VAR == VC ? A.un : VAR == VU ? A.mu.cell : VAR == VV ? A.mu.xy : A.mu.xz;
    if (live) {
        if (VAR == VU) {
            xa0 = xa[(long)(i0 - 1) * sx + col];
            xa1 = xa[(long)i0 * sx + col];
            xb0 = A.cn[(long)(i0 - 1) * sx + col];
            xb1 = A.cn[(long)i0 * sx + col];
        } else {
            xa0 = xa[(long)i0 * sx + col];
            xa1 = xa[(long)(i0 + 1) * sx + col];
        }
    }
    bool ok = true;
    const int o1 = (ty + 1) * KB1 + tx + 1;        // own cell in a +-1 tile
    const int o3 = (ty + 3) * KB3 + tx + GM::H3;   // own cell in the q tile
    const real dt = (real)A.scal[S_DT];
    const real alpha = (real)A.alpha;

    int issued = i0 + 1;   // last plane issued
    for (int i = i0; i <= i1; ++i) {
        // planes i-1, i (waited before) and i+1 resident; one block-wide
        // verdict, so that every thread leaves the ring together
        bool w = true;
        if (i == i0) w = xt_wait(&bar[slot_of(i - 1)], parity_of(i - 1)) && xt_wait(&bar[slot_of(i)], parity_of(i));
        w = w && xt_wait(&bar[slot_of(i + 1)], parity_of(i + 1));
        if (!__syncthreads_and(w)) {
            ok = false;
            break;
        }
        // every thread is past plane i-2 (read last in the previous step):
        // its slot takes plane i+2, the last plane this block needs being i1+1
        if (i + 2 <= i1 + 1) {
            if (tid == 0) issue(i + 2);
            issued = i + 2;
        }
        // the next plane's x-window values
        real qn = 0, xan = 0, xbn = 0, pgv = 0, hmv = 0;
        if (live) {
            const long id = (long)i * sx + col;
            if (i + 4 < G.NX) qn = q[id + 4 * sx];
            if (VAR == VU) {
                xan = xa[id + sx];
                xbn = A.cn[id + sx];
            } else if (i + 2 < G.NX) {
                xan = xa[id + 2 * sx];
            }
            if (VAR != VC) pgv = A.pg[id];
            hmv = A.Hm[id];
        }
        if (live) {
            const long id = (long)i * sx + col;
            const real* Q = tile3(i);
            auto T = [&](int a, int dp, int dj, int dk) -> real {
                return tile1(i + dp, a)[o1 + dj * KB1 + dk];
            };
            auto QT = [&](int dj, int dk) -> real { return Q[o3 + dj * KB3 + dk]; };
            // advecting velocities (adv_vel), up to their factor of 1/2 or 1/4
            const real q0 = QT(0, 0);
            real ux, uy, uz;
            if (VAR == VC) {
                ux = xa1 + xa0;
                uy = T(0, 0, 1, 0) + T(0, 0, 0, 0);
                uz = T(1, 0, 0, 1) + T(1, 0, 0, 0);
            } else if (VAR == VU) {
                ux = q0;
                uy = T(0, -1, 0, 0) + T(0, 0, 0, 0) + T(0, 0, 1, 0) + T(0, -1, 1, 0);
                uz = T(1, -1, 0, 0) + T(1, 0, 0, 0) + T(1, 0, 0, 1) + T(1, -1, 0, 1);
            } else if (VAR == VV) {
                ux = T(0, 0, -1, 0) + T(0, 1, -1, 0) + T(0, 0, 0, 0) + T(0, 1, 0, 0);
                uy = q0;
                uz = T(1, 0, -1, 0) + T(1, 0, -1, 1) + T(1, 0, 0, 0) + T(1, 0, 0, 1);
            } else {
                ux = T(0, 0, 0, -1) + T(0, 1, 0, -1) + T(0, 0, 0, 0) + T(0, 1, 0, 0);
                uy = T(1, 0, 0, -1) + T(1, 0, 0, 0) + T(1, 0, 1, -1) + T(1, 0, 1, 0);
                uz = q0;
            }
            const real fx = (real)(VAR == VC ? K.hix : VAR == VU ? K.ihx : K.qix);
            const real fy = (real)(VAR == VC ? K.hiy : VAR == VV ? K.ihy : K.qiy);
            const real fz = (real)(VAR == VC ? K.hiz : VAR == VW ? K.ihz : K.qiz);
            // velocity x upwind derivative = |velocity| / h x the upwind-sense
            // difference; one axis at a time keeps register use low
            real c2x, c2y, c2z;
            real ct = fabs(ux) * fx * xt_upwind_x<real>(D, q, G, R, K, i, ux >= (real)0, (real)K.wfx, c2x);
            ct = fma(fabs(uy) * fy, xt_upwind<1, real>(Q + o3, KB3, q, G, R, K, j, uy >= (real)0, (real)K.wfy, c2y), ct);
            ct = fma(fabs(uz) * fz, xt_upwind<2, real>(Q + o3, 1, q, G, R, K, k, uz >= (real)0, (real)K.wfz, c2z), ct);
            // cross stress, and the implicit operator on q_old (acoef) as
            // fluxes: c (q+ - q) - a (q - q-)
            real H = -ct, diff;
            if (VAR == VC) {
                diff = fma((real)K.cdx, c2x, fma((real)K.cdy, c2y, (real)K.cdz * c2z));
            } else {
                const real yp = QT(1, 0) - q0, ym = q0 - QT(-1, 0), zp = QT(0, 1) - q0, zm = q0 - QT(0, -1);
                if (VAR == VU) {   // tiles: 0 v, 1 w, 2 mu_xy, 3 mu_xz
                    const real my = T(2, 0, 0, 0), my1 = T(2, 0, 1, 0), mz = T(3, 0, 0, 0), mz1 = T(3, 0, 0, 1);
                    H = fma((real)K.xuv, fma(my1, T(0, 0, 1, 0) - T(0, -1, 1, 0), -my * (T(0, 0, 0, 0) - T(0, -1, 0, 0))),
                            H);
                    H = fma((real)K.xuw, fma(mz1, T(1, 0, 0, 1) - T(1, -1, 0, 1), -mz * (T(1, 0, 0, 0) - T(1, -1, 0, 0))),
                            H);
                    diff = (real)K.e2x * fma(xa1, D[3], -xa0 * D[2]);
                    diff = fma((real)K.e1y, fma(my1, yp, -my * ym), diff);
                    diff = fma((real)K.e1z, fma(mz1, zp, -mz * zm), diff);
                } else if (VAR == VV) {   // tiles: 0 u, 1 w, 2 mu_yz, 3 mu_cell, 4 c
                    const real mz = T(2, 0, 0, 0), mz1 = T(2, 0, 0, 1);
                    H = fma((real)K.xvu, fma(xa1, T(0, 1, 0, 0) - T(0, 1, -1, 0), -xa0 * (T(0, 0, 0, 0) - T(0, 0, -1, 0))),
                            H);
                    H = fma((real)K.xvw, fma(mz1, T(1, 0, 0, 1) - T(1, 0, -1, 1), -mz * (T(1, 0, 0, 0) - T(1, 0, -1, 0))),
                            H);
                    diff = (real)K.e1x * fma(xa1, D[3], -xa0 * D[2]);
                    diff = fma((real)K.e2y, fma(T(3, 0, 0, 0), yp, -T(3, 0, -1, 0) * ym), diff);
                    diff = fma((real)K.e1z, fma(mz1, zp, -mz * zm), diff);
                } else {   // tiles: 0 u, 1 v, 2 mu_yz, 3 mu_cell
                    const real my = T(2, 0, 0, 0), my1 = T(2, 0, 1, 0);
                    H = fma((real)K.xwu, fma(xa1, T(0, 1, 0, 0) - T(0, 1, 0, -1), -xa0 * (T(0, 0, 0, 0) - T(0, 0, 0, -1))),
                            H);
                    H = fma((real)K.xwv, fma(my1, T(1, 0, 1, 0) - T(1, 0, 1, -1), -my * (T(1, 0, 0, 0) - T(1, 0, 0, -1))),
                            H);
                    diff = (real)K.e1x * fma(xa1, D[3], -xa0 * D[2]);
                    diff = fma((real)K.e1y, fma(my1, yp, -my * ym), diff);
                    diff = fma((real)K.e2z, fma(T(3, 0, 0, 0), zp, -T(3, 0, 0, -1) * zm), diff);
                }
            }
            A.H[id] = H;

            // dt*(gamma H + rho H_old + alpha (A q_old + body))
            if (VAR != VC) {
                diff = fma(-pgv, (real)K.iRe, diff);
                if (VAR == VU) diff = fma((real)K.FxRe, (real)0.5 * (xb1 + xb0), diff);
                if (VAR == VV) diff = fma((real)K.FyRe, (real)0.5 * (T(4, 0, 0, 0) + T(4, 0, -1, 0)), diff);
            }
            A.S[id] = dt * fma(alpha, diff, rk_comb<real>((real)A.g, H, (real)A.r, hmv));
        }
        // slide the windows one plane along x
#pragma unroll
        for (int t = 0; t < 5; ++t) D[t] = D[t + 1];
        D[5] = qn - ql;
        ql = qn;
        xa0 = xa1;
        xa1 = xan;
        if (VAR == VU) {
            xb0 = xb1;
            xb1 = xbn;
        }
    }
    if (!ok && tid == 0) {
        // a wait ran out: report it, and drain (bounded) every copy this
        // block issued before its shared memory goes away
        atomicOr(status, ST_TIMEOUT);
        for (int p = i0 - 1; p <= issued; ++p) (void)xt_wait(&bar[slot_of(p)], parity_of(p));
    }
}

}  // namespace
}  // namespace pll
