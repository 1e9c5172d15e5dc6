// Partitioned tridiagonal solves: the ADI lines along x, y and z and the
// Poisson modes along x (tridiag_1rhs pllcart3d.c:3511-3536, pll_tridiag's
// one-rank form pll_tridiag.c:21-47 and 96-110, phisolver_dct L2040-2091) of
// every form but the exact one.
//
// A line of up to E * L rows is cut into L segments of E rows, one thread
// each.  A segment's first row is a separator; the thread eliminates its other
// rows in terms of its own separator and the next segment's, the L separator
// equations are solved by parallel cyclic reduction over warp shuffles, and
// the interior rows follow.  Every input is read once and every output written
// once; the sequential sweep also writes and re-reads c' and the eliminated
// right-hand side, and its one thread per line leaves most of the chip idle on
// all but the largest grids.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "step_kernels.cuh"

namespace pll {
namespace {

// 16 bytes global -> shared
__device__ __forceinline__ void lp_cp16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}

// couplings below this are dropped: far below the rounding of anything they
// could still multiply
template <typename real>
__device__ __forceinline__ real pcr_tiny() { return (real)1e-36; }
template <>
__device__ __forceinline__ float pcr_tiny<float>() { return 1e-24f; }

// The rows are row(e, a, b, c, r): a x_{m-1} + b x_m + c x_{m+1} = r,
// m = E seg + e, with a of a line's first row and c of its last 0 (rows past
// the line may hold anything finite that does not couple back).  Products with
// several uses are rounded on their own, so that a compiler's choice of what
// to fuse cannot differ between two kernels around these bodies.
//
// Eliminate rows 1 .. E-1: x_e = rh - ah S_l - ch S_{l+1}.
template <typename real, int E, typename Row>
__device__ __forceinline__ void part_eliminate(const Row& row, real* rh, real* ah, real* ch)
{
    real a, b, c, r;
    {
        row(1, a, b, c, r);
        const real ib = rcp_<real>(b);
        ch[1] = mul_rn_(c, ib);
        rh[1] = mul_rn_(r, ib);
        ah[1] = mul_rn_(a, ib);
    }
#pragma unroll
    for (int e = 2; e < E; ++e) {
        row(e, a, b, c, r);
        const real ib = rcp_<real>(fma(-a, ch[e - 1], b));
        const real t = mul_rn_(a, ib);
        ch[e] = mul_rn_(c, ib);
        rh[e] = fma(-t, rh[e - 1], mul_rn_(r, ib));
        ah[e] = -mul_rn_(t, ah[e - 1]);
    }
#pragma unroll
    for (int e = E - 2; e >= 1; --e) {
        rh[e] = fma(-ch[e], rh[e + 1], rh[e]);
        ah[e] = fma(-ch[e], ah[e + 1], ah[e]);
        ch[e] = -mul_rn_(ch[e], ch[e + 1]);
    }
}

// The separator's own row with the segment's rows eliminated, before the
// previous segment's last row (gp, vp, wp) is: a x_{-1} + b S + c S_{l+1} = r
template <typename real>
struct SepRow {
    real a, b, c, r;
};
template <typename real, typename Row>
__device__ __forceinline__ SepRow<real> part_separator(const Row& row, real rh1, real ah1, real ch1)
{
    real a, b, c, r;
    row(0, a, b, c, r);
    return {a, fma(-c, ah1, b), -mul_rn_(c, ch1), fma(-c, rh1, r)};
}

// Solve the separator equations, lane seg of an L-lane group holding S_l's.
// The cyclic reduction stops as soon as no lane of the warp has a coupling
// left: each round squares them, and the ADI systems' (diagonally dominant)
// are gone after two or three of the log2(L) rounds.
template <typename real, int L>
__device__ __forceinline__ real part_pcr(const SepRow<real>& s, real gp, real vp, real wp)
{
    constexpr unsigned FULLM = 0xffffffffu;
    real ib = rcp_<real>(fma(-s.a, wp, s.b));
    real al = -mul_rn_(mul_rn_(s.a, vp), ib);
    real ga = mul_rn_(s.c, ib);
    real rho = mul_rn_(fma(-s.a, gp, s.r), ib);
    // al S_{l-d} + S_l + ga S_{l+d} = rho.  A lane without a partner at
    // distance d has a zero coupling there (its shuffle returns its own,
    // finite values).
#pragma unroll
    for (int d = 1; d < L; d <<= 1) {
        if (__all_sync(FULLM, fabs(al) + fabs(ga) < pcr_tiny<real>())) break;
        const real al_m = __shfl_up_sync(FULLM, al, d, L), ga_m = __shfl_up_sync(FULLM, ga, d, L);
        const real rho_m = __shfl_up_sync(FULLM, rho, d, L);
        const real al_p = __shfl_down_sync(FULLM, al, d, L), ga_p = __shfl_down_sync(FULLM, ga, d, L);
        const real rho_p = __shfl_down_sync(FULLM, rho, d, L);
        ib = rcp_<real>(fma(-ga, al_p, fma(-al, ga_m, (real)1)));
        rho = mul_rn_(fma(-ga, rho_p, fma(-al, rho_m, rho)), ib);
        al = -mul_rn_(mul_rn_(al, al_m), ib);
        ga = -mul_rn_(mul_rn_(ga, ga_p), ib);
    }
    return rho;
}

// Rows of a segment by an L-lane group of one warp: x[0 .. E-1]
template <typename real, int E, int L, typename Row>
__device__ __forceinline__ void part_solve(const Row& row, real* x)
{
    constexpr unsigned FULLM = 0xffffffffu;
    real ch[E], rh[E], ah[E];
    part_eliminate<real, E>(row, rh, ah, ch);
    const real gp = __shfl_up_sync(FULLM, rh[E - 1], 1, L);
    const real vp = __shfl_up_sync(FULLM, ah[E - 1], 1, L);
    const real wp = __shfl_up_sync(FULLM, ch[E - 1], 1, L);
    const real sl = part_pcr<real, L>(part_separator<real>(row, rh[1], ah[1], ch[1]), gp, vp, wp);
    const real sn = __shfl_down_sync(FULLM, sl, 1, L);
    x[0] = sl;
#pragma unroll
    for (int e = 1; e < E; ++e) x[e] = fma(-ch[e], sn, fma(-ah[e], sl, rh[e]));
}

// The same with a segment per thread of a block, thread (seg, ln) = (tid / TL,
// tid % TL): the separator equations pass through shared memory (ex, PART_EX
// values a thread, free once every thread has read its rows) to the warps that
// hold one line's segments side by side, put(e, x) takes the rows.
constexpr int PART_EX = 8;
template <typename real, int E, int L, int TL, typename Row, typename Put>
__device__ __forceinline__ void part_solve_block(const Row& row, const Put& put, real* ex)
{
    constexpr int P = TL + 1, N = L * P;   // pitch and size of one exchanged value
    const int tid = threadIdx.x;
    real ch[E], rh[E], ah[E];
    part_eliminate<real, E>(row, rh, ah, ch);
    SepRow<real> s = part_separator<real>(row, rh[1], ah[1], ch[1]);
    const int own = (tid / TL) * P + tid % TL;
    __syncthreads();   // every row has been read
    ex[own] = s.a;
    ex[N + own] = s.b;
    ex[2 * N + own] = s.c;
    ex[3 * N + own] = s.r;
    ex[4 * N + own] = rh[E - 1];
    ex[5 * N + own] = ah[E - 1];
    ex[6 * N + own] = ch[E - 1];
    __syncthreads();
    {
        const int seg = tid % L, at = seg * P + tid / L, pv = at - (seg ? P : 0);
        s = {ex[at], ex[N + at], ex[2 * N + at], ex[3 * N + at]};
        ex[7 * N + at] = part_pcr<real, L>(s, ex[4 * N + pv], ex[5 * N + pv], ex[6 * N + pv]);
    }
    __syncthreads();
    const real sl = ex[7 * N + own], sn = tid / TL < L - 1 ? ex[7 * N + own + P] : (real)0;
    put(0, sl);
#pragma unroll
    for (int e = 1; e < E; ++e) put(e, fma(-ch[e], sn, fma(-ah[e], sl, rh[e])));
}

// Rows of an ADI line's segment in shared memory, ST elements apart: s[] the
// right-hand side and m[] the viscosity family (the next segment's first value
// NX elements further); the line's closures applied.
template <int VAR, int AXIS, typename real, int E, int ST, int NX>
struct AdiRow {
    const real* s;
    const real* m;
    real kap;         // -fac x (operator scale); la = kap mu_m, lc = kap mu_{m+1}
    real boun;        // outflow increment (x)
    bool first, last; // this segment holds the line's first / last row
    int el;           // position of the last row in its segment
    __device__ __forceinline__ void operator()(int e, real& la, real& lb, real& lc, real& lr) const
    {
        constexpr int LO = Closure<VAR, AXIS>::lo, HI = Closure<VAR, AXIS>::hi;
        if (VAR == VC) {
            la = lc = kap;
        } else {
            la = mul_rn_(kap, m[e * ST]);
            lc = mul_rn_(kap, m[e + 1 < E ? (e + 1) * ST : NX]);
        }
        lb = ((real)1 - la) - lc;
        lr = s[e * ST];
        if (e == 0 && first) {
            if (LO == 1) lb += la;
            else if (LO == 2) lb -= la;
            la = (real)0;
        }
        if (e == el && last) {
            if (AXIS == 0) lr = fma(-lc, boun, lr);
            else if (HI == 1) lb += lc;
            else if (HI == 2) lb -= lc;
            lc = (real)0;
        }
    }
};

// -fac x the scale of the implicit operator of VAR along AXIS
template <int VAR, int AXIS, typename real>
__device__ __forceinline__ real adi_kappa(const Consts& K, double dt, double alpha)
{
    const double fac = 0.5 * dt * alpha;
    if (VAR == VC) return (real)(-fac * (AXIS == 0 ? K.cdx : AXIS == 1 ? K.cdy : K.cdz));
    const double ih = AXIS == 0 ? K.ihx : AXIS == 1 ? K.ihy : K.ihz;
    const double d = LineCoef<VAR, AXIS>::twice ? (AXIS == 0 ? K.d2x : AXIS == 1 ? K.d2y : K.d2z)
                                                : (AXIS == 0 ? K.d1x : AXIS == 1 ? K.d1y : K.d1z);
    return (real)(-fac * (d * ih));
}

// ---- x and y lines ---------------------------------------------------------------
// A block owns TL neighbouring lines (adjacent k, the tile aligned so that
// every 16-byte piece of a row is).  All of its inputs (the right-hand side,
// the viscosity family and, along x, q_old) are fetched by 16-byte cp.async at
// once; a thread then holds one segment of one line, neighbouring lanes
// neighbouring lines, and writes its rows straight to global memory, where TL
// lanes make one row piece.  Along x the block also does what surrounds the
// solve: the convective outflow, q_new = q_old + delta and, for c, its Neumann
// ghosts (pllcart3d.c:677-683, 700-712).
template <int VAR, int AXIS, typename real, int E, int L, int TL>
struct LinePart {
    static constexpr int T = TL * L;
    // a tile of rows: TL elements of skew after each segment keep the
    // segments of a warp in different banks; one more row for the family
    static constexpr int TILE = (L * E + 1) * TL + L * TL;
    static constexpr int EX = PART_EX * L * (TL + 1);   // overlays the rhs and the family
    static constexpr int HEAD = (VAR == VC ? 1 : 2) * TILE < EX ? EX : (VAR == VC ? 1 : 2) * TILE;
    static constexpr size_t SMEM = sizeof(real) * (HEAD + (AXIS == 0 ? TILE : 0));
};

template <int VAR, int AXIS, typename real, int E, int L, int TL>
__device__ __forceinline__ void k_line_seg_run(const uint3 blockIdx, const dim3 gridDim, Geo G, Rng R, Consts K,
                                               XsweepArgs<real> A)
{
    using LP = LinePart<VAR, AXIS, real, E, L, TL>;
    constexpr int T = LP::T, OFF = LineCoef<VAR, AXIS>::off;
    constexpr int EPC = 16 / (int)sizeof(real), CPR = TL / EPC;   // elements per piece, pieces per row
    constexpr int SEGP = (E + 1) * TL;                            // from one segment to the next
    extern __shared__ __align__(16) unsigned char lp_raw[];
    real* tS = (real*)lp_raw;
    real* tM = tS + LP::TILE;
    real* tQ = tS + LP::HEAD;
    const int tid = threadIdx.x;
    const int k0 = blockIdx.x * TL;
    const int o = blockIdx.y;   // j (x lines) or i (y lines) offset
    if (o > (AXIS == 0 ? R.je - R.js : R.ie - R.is)) return;   // past a component's shorter extent
    const int n = AXIS == 0 ? R.ie - R.is + 1 : R.je - R.js + 1;
    const long st = AXIS == 0 ? G.sx : G.sy;
    const long base0 = AXIS == 0 ? (long)R.is * G.sx + (long)(R.js + o) * G.sy + k0
                                 : (long)(R.is + o) * G.sx + (long)R.js * G.sy + k0;
    {
        const real* __restrict__ fam = VAR == VC ? nullptr : line_family<VAR, AXIS, real>(A.mu);
        const int c = (tid % CPR) * EPC, r0 = tid / CPR;
        const bool any = k0 + c <= R.ke && k0 + c + EPC > R.ks;   // the piece holds a line of the range
        const real* sp = A.S + base0 + c;
        const real* mp = VAR == VC ? nullptr : fam + base0 + c + OFF * st;
        const real* qp = AXIS == 0 ? A.q + base0 + c : nullptr;
#pragma unroll 2
        for (int m = r0; m <= E * L; m += T / CPR) {
            const int at = m * TL + (m / E) * TL + c;
            const long d = (long)m * st;
            if (any && m < n) {
                lp_cp16(tS + at, sp + d);
                if (VAR != VC) lp_cp16(tM + at, mp + d);
                if (AXIS == 0) lp_cp16(tQ + at, qp + d);
            } else {
#pragma unroll
                for (int t = 0; t < EPC; ++t) {
                    if (m < E * L) tS[at + t] = (real)0;
                    if (VAR != VC && !(any && m == n)) tM[at + t] = (real)0;
                }
                if (VAR != VC && any && m == n) lp_cp16(tM + at, mp + d);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const int ln = tid % TL, seg = tid / TL, k = k0 + ln;
    const bool live = k >= R.ks && k <= R.ke;
    const long base = base0 + ln;
    const double dt = A.scal[S_DT];
    const bool last = seg == (n - 1) / E;
    real boun = (real)0;
    if (AXIS == 0 && last && live) {
        const long rb = base + (long)n * st;
        const real qb = A.q[rb];
        real Hb = -(real)A.scal[S_VBULK] * (qb - A.q[rb - st]);
        Hb = over_h<real>(Hb, K.hx, K.ihx, K.pow2);
        A.H[rb] = Hb;
        boun = rk_step<real>((real)dt, (real)A.g, Hb, (real)A.r, A.Hm[rb]);
        A.qn[rb] = qb + boun;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    const int at = seg * SEGP + ln;
    const AdiRow<VAR, AXIS, real, E, TL, SEGP> row{tS + at, tM + at, adi_kappa<VAR, AXIS, real>(K, dt, A.alpha), boun,
                                                   seg == 0, last, (n - 1) % E};
    const int rows = live ? n - seg * E : 0;   // of this segment on the line
    if (AXIS == 1) {
        real* sp = A.S + base + (long)(seg * E) * st;
        part_solve_block<real, E, L, TL>(row, [&](int e, real x) {
            if (e < rows) sp[e * st] = x;
        }, tS);
        return;
    }
    // q_new, and for c its Neumann ghosts in y (pllcart3d.c:700-705) then z
    // (L707-712; its corners copy the y ghosts, which equal this line's value)
    const int jl = R.js + o;
    const bool jlo = VAR == VC && jl == R.js, jhi = VAR == VC && jl == R.je;
    const bool klo = VAR == VC && k == R.ks, khi = VAR == VC && k == R.ke;
    const bool edge = jlo | jhi | klo | khi;
    real* qn = A.qn + base + (long)(seg * E) * st;
    const real* q = tQ + at;
    const long sy = G.sy;
    part_solve_block<real, E, L, TL>(row, [&](int e, real x) {
        if (e >= rows) return;
        const real v = q[e * TL] + x;
        real* p = qn + e * st;
        *p = v;
        if (edge) {
            if (jlo) p[-sy] = v;
            if (jhi) p[sy] = v;
            if (klo) {
                p[-1] = v;
                if (jlo) p[-sy - 1] = v;
                if (jhi) p[sy - 1] = v;
            }
            if (khi) {
                p[1] = v;
                if (jlo) p[-sy + 1] = v;
                if (jhi) p[sy + 1] = v;
            }
        }
    }, tS);
}
template <int VAR, int AXIS, typename real, int E, int L, int TL>
__global__ void __launch_bounds__(LinePart<VAR, AXIS, real, E, L, TL>::T)
    k_line_seg(Geo G, Rng R, Consts K, XsweepArgs<real> A)
{
    if (!after_previous()) return;
    k_line_seg_run<VAR, AXIS, real, E, L, TL>(blockIdx, gridDim, G, R, K, A);
}
template <int VAR, int AXIS, typename real, int E, int L, int TL>
struct k_line_seg_b {
    static constexpr auto run = &k_line_seg_run<VAR, AXIS, real, E, L, TL>;
    static constexpr int maxt = LinePart<VAR, AXIS, real, E, L, TL>::T, minb = 0;
    static constexpr bool chained = true;
};

// the three momentum components' lines in one launch, component VU + blockIdx.z
template <typename real>
struct Sweeps3 {
    Rng R[3];
    XsweepArgs<real> A[3];
};
template <int AXIS, typename real, int E, int L, int TL>
__device__ __forceinline__ void k_line_seg3_run(const uint3 blockIdx, const dim3 gridDim, Geo G, Consts K,
                                                Sweeps3<real> S)
{
    if (blockIdx.z == 0) k_line_seg_run<VU, AXIS, real, E, L, TL>(blockIdx, gridDim, G, S.R[0], K, S.A[0]);
    else if (blockIdx.z == 1) k_line_seg_run<VV, AXIS, real, E, L, TL>(blockIdx, gridDim, G, S.R[1], K, S.A[1]);
    else k_line_seg_run<VW, AXIS, real, E, L, TL>(blockIdx, gridDim, G, S.R[2], K, S.A[2]);
}
template <int AXIS, typename real, int E, int L, int TL>
__global__ void __launch_bounds__(LinePart<VU, AXIS, real, E, L, TL>::T) k_line_seg3(Geo G, Consts K, Sweeps3<real> S)
{
    if (!after_previous()) return;
    k_line_seg3_run<AXIS, real, E, L, TL>(blockIdx, gridDim, G, K, S);
}
template <int AXIS, typename real, int E, int L, int TL>
struct k_line_seg3_b {
    static constexpr auto run = &k_line_seg3_run<AXIS, real, E, L, TL>;
    static constexpr int maxt = LinePart<VU, AXIS, real, E, L, TL>::T, minb = 0;
    static constexpr bool chained = true;
};

// ---- z lines ---------------------------------------------------------------------
// The contiguous axis: a warp moves its own 32 / L lines (consecutive j)
// through a skewed shared buffer, whole rows at a time, in place.
template <int VAR, typename real, int E, int L>
__device__ __forceinline__ void k_adi_z_part_run(const uint3 blockIdx, const dim3 gridDim, Geo G, Rng R, Consts K,
                                                 MuPtrs<real> mu, real* __restrict__ S,
                                                 const double* __restrict__ scal, double alpha)
{
    constexpr int LPW = 32 / L, PITCH = L * (E + 1) + 1;
    extern __shared__ __align__(16) unsigned char lp_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j0 = R.js + (blockIdx.x * 4 + warp) * LPW;
    const int i = R.is + blockIdx.y;
    if (j0 > R.je || i > R.ie) return;   // warp-uniform
    const int nl = min(LPW, R.je - j0 + 1);
    const int n = R.ke - R.ks + 1;
    const real* __restrict__ mz = VAR == VU ? mu.xz : VAR == VV ? mu.yz : mu.cell;
    const int moff = VAR == VW ? -1 : 0;
    const long base = (long)i * G.sx + (long)j0 * G.sy + R.ks;
    real* sS = (real*)lp_raw + warp * LPW * PITCH;
    real* sM = sS + 4 * LPW * PITCH;
    auto skew = [](int m) { return m + m / E; };
#pragma unroll
    for (int q = 0; q < LPW; ++q) {
        const long b = base + (long)(q < nl ? q : 0) * G.sy;   // lines past the plane repeat the first
#pragma unroll
        for (int t = 0; t < E * L / 32; ++t) {
            const int m = t * 32 + lane;
            sS[q * PITCH + skew(m)] = m < n ? S[b + m] : (real)0;
            if (VAR != VC) sM[q * PITCH + skew(m)] = m <= n ? mz[b + moff + m] : (real)0;
        }
    }
    // the family's value past a full line: of line q by lane q, outside the
    // loop, whose loads a branch would put one after the other (64x32x32
    // FP64 9.1 -> 4.8 us)
    if (VAR != VC && lane < LPW)
        sM[lane * PITCH + skew(E * L)] = n == E * L && lane < nl ? mz[base + (long)lane * G.sy + moff + n] : (real)0;
    __syncwarp();
    const int seg = lane % L;
    real* s = sS + (lane / L) * PITCH + seg * (E + 1);
    const AdiRow<VAR, 2, real, E, 1, E + 1> row{s, sM + (lane / L) * PITCH + seg * (E + 1),
                                      adi_kappa<VAR, 2, real>(K, scal[S_DT], alpha), (real)0, seg == 0,
                                      seg == (n - 1) / E, (n - 1) % E};
    real x[E];
    part_solve<real, E, L>(row, x);
#pragma unroll
    for (int e = 0; e < E; ++e) s[e] = x[e];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < LPW; ++q) {
        if (q >= nl) break;
        const long b = base + (long)q * G.sy;
#pragma unroll
        for (int t = 0; t < E * L / 32; ++t) {
            const int m = t * 32 + lane;
            if (m < n) S[b + m] = sS[q * PITCH + skew(m)];
        }
    }
}
template <int VAR, typename real, int E, int L>
constexpr size_t z_part_smem()
{
    return sizeof(real) * 4 * (32 / L) * (L * (E + 1) + 1) * (VAR == VC ? 1 : 2);
}
template <int VAR, typename real, int E, int L>
__global__ void __launch_bounds__(128) k_adi_z_part(Geo G, Rng R, Consts K, MuPtrs<real> mu, real* __restrict__ S,
                                                    const double* __restrict__ scal, double alpha)
{
    if (!after_previous()) return;
    k_adi_z_part_run<VAR, real, E, L>(blockIdx, gridDim, G, R, K, mu, S, scal, alpha);
}
template <int VAR, typename real, int E, int L>
struct k_adi_z_part_b {
    static constexpr auto run = &k_adi_z_part_run<VAR, real, E, L>;
    static constexpr int maxt = 128, minb = 0;
    static constexpr bool chained = true;
};

template <typename real, int E, int L>
__device__ __forceinline__ void k_adi_z_part3_run(const uint3 blockIdx, const dim3 gridDim, Geo G, Consts K,
                                                  Sweeps3<real> S)
{
    // constant indexes: a batched copy's arguments would go to local memory
    const XsweepArgs<real>&U = S.A[0], &V = S.A[1], &W = S.A[2];
    if (blockIdx.z == 0)
        k_adi_z_part_run<VU, real, E, L>(blockIdx, gridDim, G, S.R[0], K, U.mu, U.S, U.scal, U.alpha);
    else if (blockIdx.z == 1)
        k_adi_z_part_run<VV, real, E, L>(blockIdx, gridDim, G, S.R[1], K, V.mu, V.S, V.scal, V.alpha);
    else
        k_adi_z_part_run<VW, real, E, L>(blockIdx, gridDim, G, S.R[2], K, W.mu, W.S, W.scal, W.alpha);
}
template <typename real, int E, int L>
__global__ void __launch_bounds__(128) k_adi_z_part3(Geo G, Consts K, Sweeps3<real> S)
{
    if (!after_previous()) return;
    k_adi_z_part3_run<real, E, L>(blockIdx, gridDim, G, K, S);
}
template <typename real, int E, int L>
struct k_adi_z_part3_b {
    static constexpr auto run = &k_adi_z_part3_run<real, E, L>;
    static constexpr int maxt = 128, minb = 0;
    static constexpr bool chained = true;
};

// ---- Poisson modes ---------------------------------------------------------------
// The x-tridiagonal of each (ky, kz) mode, in place: 1/dx^2 off the diagonal,
// -2/dx^2 + lam_y + lam_z on it, Neumann at the inlet and, except for mode
// (0, 0) whose right ghost holds phi = 0 (the pressure gauge), at the outlet.
// Modes are stored as T; the solve is FP64.
// Laid out as the x lines above; a piece of a row that is not 16-byte aligned
// (ny nz not a multiple of it) is fetched element by element.
template <typename T, int E, int L, int TL>
struct PoissonPart {
    static constexpr int TH = TL * L;
    static constexpr int TILE = L * E * TL + L * TL;
    static constexpr size_t ROWS = sizeof(T) * TILE, EX = sizeof(double) * PART_EX * L * (TL + 1);
    static constexpr size_t SMEM = ROWS < EX ? EX : ROWS;
};

// The rows over 1/dx^2, negated: (A + C + s) x_m = A x_{m-1} + C x_{m+1} + r,
// A and C 1 or 0 and s >= 0 the row's excess.  Solved for x = al S_l + ga
// S_{l+1} + rho with the deficit de = 1 - al - ga carried along: every
// coefficient is then a sum of products of non-negative numbers, and the
// lowest modes, whose s is down to 1e-6 of the diagonal, lose nothing to
// cancellation: phi's relative error at 512x128x120 is 7e-14, where the
// sequential sweep has 5e-13 and the general elimination above 1e-12.
template <typename T, int E, int ST>
struct PoissonRow {
    const T* t;
    double scale, excess;
    bool first, last, gauge;
    int rows;   // this segment's rows that lie on the line; those past it are x = 0
    __device__ __forceinline__ void operator()(int e, double& A, double& C, double& s, double& r) const
    {
        const bool in = e < rows;
        A = C = in ? 1.0 : 0.0;
        s = in ? excess : 1.0;
        r = mul_rn_((double)t[e * ST], scale);
        if (e == 0 && first) A = 0.0;
        if (last && e == rows - 1) {
            if (gauge) s += 1.0;
            C = 0.0;
        }
    }
};

// as part_solve_block
template <int E, int L, int TL, typename Row, typename Put>
__device__ __forceinline__ void poisson_solve_block(const Row& row, const Put& put, double* ex)
{
    constexpr unsigned FULLM = 0xffffffffu;
    constexpr int P = TL + 1, N = L * P;
    const int tid = threadIdx.x;
    double ga[E], rh[E], al[E], A, C, s, r;
    double de, de1, chain;   // deficits of the current row and of row 1, product of ga from row 1 on
    {
        row(1, A, C, s, r);
        const double i = rcp_<double>((A + C) + s);
        al[1] = mul_rn_(A, i);
        ga[1] = chain = mul_rn_(C, i);
        de = de1 = mul_rn_(s, i);
        rh[1] = mul_rn_(r, i);
    }
#pragma unroll
    for (int e = 2; e < E; ++e) {
        row(e, A, C, s, r);
        const double i = rcp_<double>(fma(A, al[e - 1] + de, C + s)), t = mul_rn_(A, i);
        al[e] = mul_rn_(t, al[e - 1]);
        ga[e] = mul_rn_(C, i);
        de = fma(t, de, mul_rn_(s, i));
        rh[e] = fma(t, rh[e - 1], mul_rn_(r, i));
        de1 = fma(chain, de, de1);
        chain = mul_rn_(chain, ga[e]);
    }
#pragma unroll
    for (int e = E - 2; e >= 1; --e) {
        rh[e] = fma(ga[e], rh[e + 1], rh[e]);
        al[e] = fma(ga[e], al[e + 1], al[e]);
        ga[e] = mul_rn_(ga[e], ga[e + 1]);
    }
    row(0, A, C, s, r);
    const int own = (tid / TL) * P + tid % TL;
    __syncthreads();   // every row has been read
    ex[own] = mul_rn_(C, ga[1]);
    ex[N + own] = fma(C, de1, s);
    ex[2 * N + own] = fma(C, rh[1], r);
    ex[3 * N + own] = al[E - 1];
    ex[4 * N + own] = de;
    ex[5 * N + own] = rh[E - 1];
    __syncthreads();
    {
        const int seg = tid % L, at = seg * P + tid / L, pv = at - (seg ? P : 0);
        // a separator past the line may couple back: nothing couples to it
        const double back = seg ? 1.0 : 0.0;
        double a = mul_rn_(back, ex[3 * N + pv]), g = ex[at], d = fma(back, ex[4 * N + pv], ex[N + at]);
        double i = rcp_<double>((a + g) + d);
        a = mul_rn_(a, i);
        g = mul_rn_(g, i);
        d = mul_rn_(d, i);
        double rho = mul_rn_(fma(back, ex[5 * N + pv], ex[2 * N + at]), i);
        // S_l = a S_{l-h} + g S_{l+h} + rho, a + g + d = 1
#pragma unroll
        for (int h = 1; h < L; h <<= 1) {
            if (__all_sync(FULLM, a + g < pcr_tiny<double>())) break;
            const double a_m = __shfl_up_sync(FULLM, a, h, L), d_m = __shfl_up_sync(FULLM, d, h, L);
            const double g_p = __shfl_down_sync(FULLM, g, h, L), d_p = __shfl_down_sync(FULLM, d, h, L);
            const double r_m = __shfl_up_sync(FULLM, rho, h, L), r_p = __shfl_down_sync(FULLM, rho, h, L);
            i = rcp_<double>(fma(a, a_m + d_m, fma(g, g_p + d_p, d)));
            rho = mul_rn_(fma(g, r_p, fma(a, r_m, rho)), i);
            d = mul_rn_(fma(g, d_p, fma(a, d_m, d)), i);
            a = mul_rn_(mul_rn_(a, a_m), i);
            g = mul_rn_(mul_rn_(g, g_p), i);
        }
        ex[6 * N + at] = rho;
    }
    __syncthreads();
    const double sl = ex[6 * N + own], sn = tid / TL < L - 1 ? ex[6 * N + own + P] : 0.0;
    put(0, sl);
#pragma unroll
    for (int e = 1; e < E; ++e) put(e, fma(ga[e], sn, fma(al[e], sl, rh[e])));
}

template <typename T, int E, int L, int TL>
__device__ __forceinline__ void k_poisson_part_run(const uint3 blockIdx, const dim3 gridDim, int nx, int ny, int nz,
                                                   Consts K, const double* __restrict__ lam_y,
                                                   const double* __restrict__ lam_z, T* __restrict__ hat, int kz_major)
{
    constexpr int TH = PoissonPart<T, E, L, TL>::TH, EPC = 16 / (int)sizeof(T), CPR = TL / EPC;
    extern __shared__ __align__(16) unsigned char lp_raw[];
    T* tS = (T*)lp_raw;
    const int tid = threadIdx.x;
    const int N = ny * nz, t0 = blockIdx.x * TL;
    {
        const int c = (tid % CPR) * EPC, r0 = tid / CPR, left = N - (t0 + c);   // modes from this piece on
        const bool whole = left >= EPC && N % EPC == 0;
        const T* hp = hat + t0 + c;
#pragma unroll 2
        for (int m = r0; m < E * L; m += TH / CPR) {
            T* at = tS + m * TL + (m / E) * TL + c;
            const T* from = hp + (long)m * N;
            if (whole && m < nx) {
                lp_cp16(at, from);
            } else {
#pragma unroll
                for (int t = 0; t < EPC; ++t) at[t] = (m < nx && t < left) ? from[t] : (T)0;
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const int ln = tid % TL, seg = tid / TL;
    // modes stored [x][ky][kz] (kz_major 0) or [x][kz][ky] (kz_major 1)
    const int t = min(t0 + ln, N - 1);
    const int jy = kz_major ? t % ny : t / nz, kz = kz_major ? t / ny : t % nz;
    const double dx2 = rcp_<double>(K.dx2i);
    const double excess = -mul_rn_(lam_y[jy] + lam_z[kz], dx2);
    const int rows = nx - E * seg;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    const PoissonRow<T, E, TL> row{tS + seg * (E + 1) * TL + ln, -dx2, excess, seg == 0, seg == (nx - 1) / E, t == 0,
                                   rows};
    T* out = hat + t0 + ln + (long)(seg * E) * N;
    const int put = t0 + ln < N ? rows : 0;
    poisson_solve_block<E, L, TL>(row, [&](int e, double x) {
        if (e < put) out[(long)e * N] = (T)x;
    }, (double*)lp_raw);
}
template <typename T, int E, int L, int TL>
__global__ void __launch_bounds__(PoissonPart<T, E, L, TL>::TH)
    k_poisson_part(int nx, int ny, int nz, Consts K, const double* __restrict__ lam_y,
                   const double* __restrict__ lam_z, T* __restrict__ hat, int kz_major)
{
    if (!after_previous()) return;
    k_poisson_part_run<T, E, L, TL>(blockIdx, gridDim, nx, ny, nz, K, lam_y, lam_z, hat, kz_major);
}
template <typename T, int E, int L, int TL>
struct k_poisson_part_b {
    static constexpr auto run = &k_poisson_part_run<T, E, L, TL>;
    static constexpr int maxt = PoissonPart<T, E, L, TL>::TH, minb = 0;
    static constexpr bool chained = true;
};

}  // namespace
}  // namespace pll
