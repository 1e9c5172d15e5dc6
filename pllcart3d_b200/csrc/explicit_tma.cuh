// Explicit operator + ADI right-hand side (Hc_op/Hu_op/Hv_op/Hw_op,
// pllcart3d.c:1539-1980, with the source assembly of concentration / xmom /
// ymom / zmom, L573-590, L970-989, L1127-1146, L1280-1298) as a
// plane-marching kernel with TMA-staged shared-memory tiles.
//
// A block owns a tile of TJ rows (j) x XT_TK cells (k) and walks ni planes
// along x (chosen per launch, launch_explicit_tma).  An FP64 thread computes one
// cell of a plane (TJ = 8); an FP32 thread two, rows j and j + 8 (TJ = 16), in
// sm_100's paired instructions (one for two FP32 operations).  Every plane's
// tiles arrive by cp.async.bulk.tensor (one thread issues them; an mbarrier per
// ring slot counts the bytes): q with a
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
constexpr int XT_WJ = 8;    // warps per block: rows of one cell per thread
constexpr int XT_NS = 4;    // plane slots of the ring
constexpr int XT_THREADS = XT_TK * XT_WJ;

// what a thread computes at once: an FP64 cell, or a pair of FP32 cells
template <typename real>
struct XtLane {
    using V = double;
    static constexpr int NC = 1;
};
template <>
struct XtLane<float> {
    using V = f2;
    static constexpr int NC = 2;
};
struct XtUp {   // upwind sense of each cell
    bool a, b;
};
__device__ __forceinline__ double xld(const double* p, long) { return *p; }
__device__ __forceinline__ f2 xld(const float* p, long second) { return F2(p[0], p[second]); }
__device__ __forceinline__ void xset(double& v, double a) { v = a; }
__device__ __forceinline__ void xset(f2& v, float a) { v = S2(a); }
__device__ __forceinline__ double xfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ f2 xfma(f2 a, f2 b, f2 c) { return fma2(a, b, c); }
__device__ __forceinline__ double xabs(double a) { return fabs(a); }
__device__ __forceinline__ f2 xabs(f2 a) { return F2(fabsf(a.v.x), fabsf(a.v.y)); }
__device__ __forceinline__ XtUp xup(double a) { return {a >= 0.0, true}; }
__device__ __forceinline__ XtUp xup(f2 a) { return {a.v.x >= 0.f, a.v.y >= 0.f}; }
__device__ __forceinline__ double xpick(XtUp u, double up, double dn) { return u.a ? up : dn; }
__device__ __forceinline__ f2 xpick(XtUp u, f2 up, f2 dn) { return F2(u.a ? up.v.x : dn.v.x, u.b ? up.v.y : dn.v.y); }
__device__ __forceinline__ double xneg(double a) { return -a; }
__device__ __forceinline__ f2 xneg(f2 a) { return F2(-a.v.x, -a.v.y); }
// g a + r b (rk_comb)
__device__ __forceinline__ double xcomb(double g, double a, double r, double b) { return rk_comb<double>(g, a, r, b); }
__device__ __forceinline__ f2 xcomb(f2 g, f2 a, f2 r, f2 b) { return fma2(g, a, r * b); }

// One variable's constants in its own arithmetic type: -1/h of the advecting
// velocities' sums (with their 1/2 or 1/4), the WENO5 floors, the implicit
// operator's scales, the cross stresses', half the body force, 1/Re, the RK
// coefficients
template <typename real>
struct XtConst {
    real fx, fy, fz, wx, wy, wz, kx, ky, kz, c1, c2, body, iRe, g, r, alpha;
};
template <typename real>
inline XtConst<real> xt_const(int var, const Consts& K, double g, double r)
{
    const double one[3] = {K.ihx, K.ihy, K.ihz}, half[3] = {K.hix, K.hiy, K.hiz}, quarter[3] = {K.qix, K.qiy, K.qiz};
    double f[3];
    for (int a = 0; a < 3; ++a) f[a] = -(var == VC ? half[a] : var == a + 1 ? one[a] : quarter[a]);
    XtConst<real> c;
    c.fx = (real)f[0], c.fy = (real)f[1], c.fz = (real)f[2];
    c.wx = (real)K.wfx, c.wy = (real)K.wfy, c.wz = (real)K.wfz;
    c.kx = (real)(var == VC ? K.cdx : var == VU ? K.e2x : K.e1x);
    c.ky = (real)(var == VC ? K.cdy : var == VV ? K.e2y : K.e1y);
    c.kz = (real)(var == VC ? K.cdz : var == VW ? K.e2z : K.e1z);
    c.c1 = (real)(var == VU ? K.xuv : var == VV ? K.xvu : K.xwu);
    c.c2 = (real)(var == VU ? K.xuw : var == VV ? K.xvw : K.xwv);
    c.body = (real)(0.5 * (var == VU ? K.FxRe : K.FyRe));
    c.iRe = (real)K.iRe;
    c.g = (real)g, c.r = (real)r, c.alpha = (real)(g + r);
    return c;
}
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
    static constexpr int TJ = XT_WJ * XtLane<real>::NC;                     // rows of a tile
    static constexpr int KB1 = sizeof(real) == 8 ? XT_TK + 2 : XT_TK + 4;   // +-1 box width (16-byte multiple)
    static constexpr int JB1 = TJ + 2;
    static constexpr int H3 = sizeof(real) == 8 ? 3 : 5;                   // q box starts at k0 - H3
    static constexpr int KB3 = sizeof(real) == 8 ? XT_TK + 6 : XT_TK + 8;
    static constexpr int JB3 = TJ + 6;
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

// the ENO-2 closure's upwind-sense difference (the first and last two points of
// a range): v2 and half the smaller of the two second differences, b behind and c ahead of the
// point in the upwind sense; ties go to the lower line index, b for up
template <typename real>
__device__ __forceinline__ real eno_diff(real v2, real b, real c, bool up)
{
    const bool first = up ? fabs(b) <= fabs(c) : !(fabs(c) <= fabs(b));
    return fma((real)0.5, first ? b : c, v2);
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

// The upwind-sense difference of one cell from the window's differences
// v0 .. v4 (v2 behind the point; with FP32 weights a FP64 cell re-forms the others) and
// their own a, b, c, d: ENO-2 in the band at the ends of a range, else WENO5
// in the form's weight type.
template <int AXIS, typename real>
__device__ __forceinline__ real xt_diff(real v0, real v1, real v2, real v3, real v4, real a, real b, real c, real d,
                                        const real* __restrict__ qg, const Geo& G, const Rng& R, const Consts& K, int m,
                                        bool up, real floor4)
{
    if (eno_band<AXIS>(R, m)) return eno_diff<real>(v2, eno_behind<AXIS, real>(qg, G, R, K, m, up, b), c, up);
    if constexpr (std::is_same<typename XtWeno<real>::type, float>::value) {
        return v2 + (real)weno_corr((float)v2, (float)a, (float)b, (float)c, (float)d);
    } else {
        const real vmax = fmax(fmax(fmax(fabs(v0), fabs(v1)), fmax(fabs(v2), fabs(v3))), fabs(v4));
        return weno_diff(v2, a, b, c, d, vmax, floor4);
    }
}

// of a thread's FP64 cell, or of its two FP32 cells: their positions along
// the axis differ along y only
template <int AXIS>
__device__ __forceinline__ double xt_diffs(const double* v, double v0, double a, double b, double c, double d,
                                           const double* __restrict__ qg, const Geo& G, const Rng& R, const Consts& K,
                                           int m, XtUp up, double floor4)
{
    return xt_diff<AXIS, double>(v0, v[0], v[1], v[2], v[3], a, b, c, d, qg, G, R, K, m, up.a, floor4);
}
template <int AXIS>
__device__ __forceinline__ f2 xt_diffs(const f2* v, f2 v0, f2 a, f2 b, f2 c, f2 d, const float* __restrict__ qg,
                                       const Geo& G, const Rng& R, const Consts& K, int m, XtUp up, float)
{
    const int m2 = AXIS == 1 ? m + XT_WJ : m;
    if (eno_band<AXIS>(R, m) | eno_band<AXIS>(R, m2))
        return F2(xt_diff<AXIS, float>(0.f, 0.f, v[1].v.x, 0.f, 0.f, a.v.x, b.v.x, c.v.x, d.v.x, qg, G, R, K, m, up.a, 0.f),
                  xt_diff<AXIS, float>(0.f, 0.f, v[1].v.y, 0.f, 0.f, a.v.y, b.v.y, c.v.y, d.v.y, qg, G, R, K, m2, up.b,
                                       0.f));
    const float mx = weno_vmax(v0.v.x, v[0].v.x, v[1].v.x, v[2].v.x, v[3].v.x);
    const float my = weno_vmax(v0.v.y, v[0].v.y, v[1].v.y, v[2].v.y, v[3].v.y);
    return v[1] + weno_corr2(mx, my, a, b, c, d);
}

__device__ __forceinline__ double xt_window(const double* p, int st, XtUp up, int t, long)
{
    return p[(up.a ? st : -st) * (t - 3)];
}
__device__ __forceinline__ f2 xt_window(const float* p, int st, XtUp up, int t, long second)
{
    return F2(p[(up.a ? st : -st) * (t - 3)], p[second + (up.b ? st : -st) * (t - 3)]);
}

// h x the upwind derivative in the upwind sense along y or z: p is the point
// in its shared tile, st the tile's step along the axis.  The window is read
// in the upwind direction (up: increasing), so that neither the differences
// nor anything made of them is selected by the sign; the derivative times the
// velocity is |velocity| / h times the result.  c2: the second difference at
// the point.
template <int AXIS, typename real, typename V = typename XtLane<real>::V>
__device__ __forceinline__ V xt_upwind(const real* p, int st, long second, const real* __restrict__ qg, const Geo& G,
                                       const Rng& R, const Consts& K, int m, XtUp up, real floor4, V& c2)
{
    V d[5], q0 = xt_window(p, st, up, 0, second);
#pragma unroll
    for (int t = 0; t < 5; ++t) {
        const V q1 = xt_window(p, st, up, t + 1, second);
        d[t] = q1 - q0;
        q0 = q1;
    }
    c2 = d[3] - d[2];
    return xt_diffs<AXIS>(d + 1, d[0], d[1] - d[0], d[2] - d[1], c2, d[4] - d[3], qg, G, R, K, m, up, floor4);
}

// the same along x from the register window D[t] = q(i-2+t) - q(i-3+t)
template <typename real, typename V = typename XtLane<real>::V>
__device__ __forceinline__ V xt_upwind_x(const V* D, const real* __restrict__ qg, const Geo& G, const Rng& R,
                                         const Consts& K, int i, XtUp up, real floor4, V& c2)
{
    c2 = D[3] - D[2];
    const V b = xpick(up, D[2], D[4]) - xpick(up, D[1], D[3]);
    const V a = xpick(up, D[1], D[5]) - xpick(up, D[0], D[4]), d = xpick(up, D[4], D[2]) - xpick(up, D[3], D[1]);
    const V v2 = xpick(up, D[2], xneg(D[3]));
    // the window's other differences enter by their magnitude: D1 .. D4 whichever the sense
    const V v[4] = {D[1], v2, xpick(up, D[3], D[2]), D[4]};
    return xt_diffs<0>(v, xpick(up, D[0], D[5]), a, b, c2, d, qg, G, R, K, i, up, floor4);
}

template <int VAR, typename real>
__device__ __forceinline__ void k_explicit_tma_run(const uint3 blockIdx, const dim3 gridDim, const XtMaps& maps, Geo G,
                                                   Rng R, Consts K, XtConst<real> C, ExplicitArgs<real> A, int ni,
                                                   int* status)
{
    using GM = XtGeom<real>;
    using SM = XtSmem<real, VAR>;
    constexpr int NA = XtSet<VAR>::NA;
    using V = typename XtLane<real>::V;
    constexpr int KB1 = GM::KB1, KB3 = GM::KB3;
    extern __shared__ unsigned char xt_raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)xt_raw + 127) & ~(uintptr_t)127);
    uint64_t* bar = (uint64_t*)(sm + SM::BAR_OFF);
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    const int k0 = 1 + blockIdx.x * XT_TK;
    const int j0 = R.js + blockIdx.y * GM::TJ;
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

    // register windows along x at (j, k).  A pair's second cell, XT_WJ rows on,
    // may lie past the last row: it then reads the first one's column (and in
    // the shared tiles its own row, zero-filled past the box) and stores nothing
    const long col = (long)j * sy + k, r2 = XT_WJ * sy;
    const bool live2 = XtLane<real>::NC == 2 && j + XT_WJ <= R.je;
    const real* __restrict__ q = A.q;
    const real* __restrict__ xa = VAR == VC ? A.un : VAR == VU ? A.mu.cell : VAR == VV ? A.mu.xy : A.mu.xz;
    auto at = [&](const real* p, int i) -> V {   // plane i of a field at this thread's cells
        V v;
        xset(v, (real)0);
        if (live) v = xld(p + (long)i * sx + col, live2 ? r2 : 0);
        return v;
    };
    V D[6], ql;   // differences of q(i-3 .. i+3), and q(i+3)
    {
        V q0 = at(q, i0 - 3);
#pragma unroll
        for (int t = 0; t < 6; ++t) {
            ql = at(q, i0 - 2 + t);
            D[t] = ql - q0;
            q0 = ql;
        }
    }
    V xa0, xa1, xb0, xb1;   // VC: u(i), u(i+1); VU: mu_cell(i-1), (i), c(i-1), c(i); VV: mu_xy(i), (i+1);
                            // VW: mu_xz(i), (i+1)
    xa0 = at(xa, VAR == VU ? i0 - 1 : i0);
    xa1 = at(xa, VAR == VU ? i0 : i0 + 1);
    if (VAR == VU) {
        xb0 = at(A.cn, i0 - 1);
        xb1 = at(A.cn, i0);
    }
    auto K2 = [](real a) -> V {   // a constant for every cell of the thread
        V v;
        xset(v, a);
        return v;
    };
    bool ok = true;
    const int o1 = (ty + 1) * KB1 + tx + 1;        // own cell in a +-1 tile
    const int o3 = (ty + 3) * KB3 + tx + GM::H3;   // own cell in the q tile
    const V dt = K2((real)A.scal[S_DT]);

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
        V qn, xan, xbn, pgv, hmv;
        qn = at(q, i + 4 < G.NX ? i + 4 : i);
        xan = at(xa, VAR == VU ? i + 1 : i + 2 < G.NX ? i + 2 : i);
        if (VAR == VU) xbn = at(A.cn, i + 1);
        if (VAR != VC) pgv = at(A.pg, i);
        hmv = at(A.Hm, i);
        if (live) {
            const real* Q = tile3(i) + o3;
            auto T = [&](int a, int dp, int dj, int dk) -> V {
                return xld(tile1(i + dp, a) + o1 + dj * KB1 + dk, XT_WJ * KB1);
            };
            auto QT = [&](int dj, int dk) -> V { return xld(Q + dj * KB3 + dk, XT_WJ * KB3); };
            // advecting velocities (adv_vel), up to their factor of 1/2 or 1/4
            const V q0 = QT(0, 0);
            V ux, uy, uz;
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
            // - velocity x upwind derivative = - |velocity| / h x the upwind-
            // sense difference; one axis at a time keeps register use low
            V c2x, c2y, c2z;
            V H = xabs(ux) * K2(C.fx) * xt_upwind_x<real>(D, q, G, R, K, i, xup(ux), C.wx, c2x);
            H = xfma(xabs(uy) * K2(C.fy), xt_upwind<1, real>(Q, KB3, XT_WJ * KB3, q, G, R, K, j, xup(uy), C.wy, c2y), H);
            H = xfma(xabs(uz) * K2(C.fz), xt_upwind<2, real>(Q, 1, XT_WJ * KB3, q, G, R, K, k, xup(uz), C.wz, c2z), H);
            // cross stress, and the implicit operator on q_old (acoef) as
            // fluxes: c (q+ - q) + a (q- - q)
            V diff;
            if (VAR == VC) {
                diff = xfma(K2(C.kx), c2x, xfma(K2(C.ky), c2y, K2(C.kz) * c2z));
            } else {
                const V yp = QT(1, 0) - q0, ym = QT(-1, 0) - q0, zp = QT(0, 1) - q0, zm = QT(0, -1) - q0;
                V s1, s2, dy, dz;
                if (VAR == VU) {   // tiles: 0 v, 1 w, 2 mu_xy, 3 mu_xz
                    const V my = T(2, 0, 0, 0), my1 = T(2, 0, 1, 0), mz = T(3, 0, 0, 0), mz1 = T(3, 0, 0, 1);
                    s1 = xfma(my1, T(0, 0, 1, 0) - T(0, -1, 1, 0), my * (T(0, -1, 0, 0) - T(0, 0, 0, 0)));
                    s2 = xfma(mz1, T(1, 0, 0, 1) - T(1, -1, 0, 1), mz * (T(1, -1, 0, 0) - T(1, 0, 0, 0)));
                    dy = xfma(my1, yp, my * ym);
                    dz = xfma(mz1, zp, mz * zm);
                } else if (VAR == VV) {   // tiles: 0 u, 1 w, 2 mu_yz, 3 mu_cell, 4 c
                    const V mz = T(2, 0, 0, 0), mz1 = T(2, 0, 0, 1);
                    s1 = xfma(xa1, T(0, 1, 0, 0) - T(0, 1, -1, 0), xa0 * (T(0, 0, -1, 0) - T(0, 0, 0, 0)));
                    s2 = xfma(mz1, T(1, 0, 0, 1) - T(1, 0, -1, 1), mz * (T(1, 0, -1, 0) - T(1, 0, 0, 0)));
                    dy = xfma(T(3, 0, 0, 0), yp, T(3, 0, -1, 0) * ym);
                    dz = xfma(mz1, zp, mz * zm);
                } else {   // tiles: 0 u, 1 v, 2 mu_yz, 3 mu_cell
                    const V my = T(2, 0, 0, 0), my1 = T(2, 0, 1, 0);
                    s1 = xfma(xa1, T(0, 1, 0, 0) - T(0, 1, 0, -1), xa0 * (T(0, 0, 0, -1) - T(0, 0, 0, 0)));
                    s2 = xfma(my1, T(1, 0, 1, 0) - T(1, 0, 1, -1), my * (T(1, 0, 0, -1) - T(1, 0, 0, 0)));
                    dy = xfma(my1, yp, my * ym);
                    dz = xfma(T(3, 0, 0, 0), zp, T(3, 0, 0, -1) * zm);
                }
                H = xfma(K2(C.c1), s1, H);
                H = xfma(K2(C.c2), s2, H);
                diff = K2(C.kx) * xfma(xa1, D[3], xneg(xa0 * D[2]));
                diff = xfma(K2(C.ky), dy, diff);
                diff = xfma(K2(C.kz), dz, diff);
                // with the body force and the accumulated pressure gradient
                diff = xfma(pgv, K2(-C.iRe), diff);
                if (VAR == VU) diff = xfma(K2(C.body), xb1 + xb0, diff);
                if (VAR == VV) diff = xfma(K2(C.body), T(4, 0, 0, 0) + T(4, 0, -1, 0), diff);
            }
            // dt*(gamma H + rho H_old + alpha (A q_old + body))
            const V S = dt * xfma(K2(C.alpha), diff, xcomb(K2(C.g), H, K2(C.r), hmv));
            const long id = (long)i * sx + col;
            if constexpr (XtLane<real>::NC == 2) {
                A.H[id] = H.v.x;
                A.S[id] = S.v.x;
                if (live2) {
                    A.H[id + r2] = H.v.y;
                    A.S[id + r2] = S.v.y;
                }
            } else {
                A.H[id] = H;
                A.S[id] = S;
            }
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

template <int VAR, typename real>
__global__ void __launch_bounds__(XT_THREADS, XtBlocks<VAR, real>::value)
    k_explicit_tma(const __grid_constant__ XtMaps maps, Geo G, Rng R, Consts K, XtConst<real> C, ExplicitArgs<real> A,
                   int ni, int* status)
{
    if (!after_previous()) return;
    k_explicit_tma_run<VAR, real>(blockIdx, gridDim, maps, G, R, K, C, A, ni, status);
}
template <int VAR, typename real>
struct k_explicit_tma_b {
    static constexpr auto run = &k_explicit_tma_run<VAR, real>;
    static constexpr bool maps = true;   // the first argument: tensor maps
    static constexpr int maxt = XT_THREADS, minb = 0, bminb = sizeof(real) == 4 ? 2 : 0;
    static constexpr bool chained = true;
};

}  // namespace
}  // namespace pll
