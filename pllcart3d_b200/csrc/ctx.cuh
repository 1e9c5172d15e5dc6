// Device context of the pllcart3d B200 step: the state buffers of both
// precision forms and the bookkeeping shared by the orchestration units.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/pllcart3d_gpu.h"
#include "aux_kernels.cuh"
#include "batch.cuh"
#include "common.cuh"
#include "dct_kernels.cuh"
#include "host_util.h"
#include "step_kernels.cuh"


namespace pll {

template <typename real>
struct Bufs {
    real* q[4][2] = {};     // c, u, v, w : [buffer]
    real* H[4][2] = {};
    real* mu[2][4] = {};    // [buffer][cell, xy, xz, yz]
    real* pg[4] = {};       // u, v, w at 1..3
    real* phi = nullptr;
    real* div = nullptr;
    real* S[4] = {};        // ADI right-hand side / eliminated rhs of each variable
                            // (the exact form: one array for all; else v's and
                            // w's are dct1 and dct2)
    real* cc = nullptr;     // Thomas scratch, where a sequential sweep runs
    real* dct1 = nullptr;   // compact nx*ny*nz Poisson buffers (a field's size
    real* dct2 = nullptr;   // where they also hold right-hand sides)
    real *Ty = nullptr, *Tz = nullptr, *Tiy = nullptr, *Tiz = nullptr;
};

// tcgen05 DCT passes of the precision form: tensor maps of the four passes
// (A = the data, Bh / Bl = the cosine matrix's TF32 head and tail)
struct UmmaPlan {
    bool on = false;
    int sms = 148;   // persistent grid: one CTA per SM
    CUtensorMap a[4], bh[4], bl[4];
    float* Thi[4] = {};
    float* Tlo[4] = {};
};

// One axis's DCT passes outside the exact form and the tcgen05 path: by FFT
// (cos / sin of 2 pi m / N and of pi k / (2N)) or by the folded dense product
// (its tables of both kinds in fragment order)
struct DctAxis {
    enum Mode { NONE, FFT, FOLD } mode = NONE;
    double2 *tw = nullptr, *wq = nullptr;
    int r1 = 0, r2 = 0;   // FFT: the length's two factors
    double* table[2] = {nullptr, nullptr};
};

}  // namespace pll

using namespace pll;

struct pllgpu_ctx {
    pllgpu_params P;
    Geo G;
    Rng Rg, Rv[4];
    Consts K;
    int dev = 0;
    bool mixed = false;
    cudaStream_t st = nullptr;
    // side branches of a step (kernels that do not depend on one another),
    // forked from and joined back into st; `at` is where go() launches
    static constexpr int NSIDE = 3;
    cudaStream_t side[NSIDE] = {}, at = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join[NSIDE] = {};
    bool follows[1 + NSIDE] = {};   // the last thing enqueued on st, side[i] is a kernel of the step
    bool chaining = false;          // a whole step is being enqueued
    long nelem = 0;             // elements of one padded field
    Bufs<double> b64;           // state of the FP64 form
    Bufs<float> b32;            // state of the mixed form
    // scratch of the sequential Poisson mode solve, where it runs
    double *mode_cc = nullptr, *mode_rr = nullptr;
    double* stage64 = nullptr;  // one padded FP64 field (mixed-form transfers)
    double *lam_y = nullptr, *lam_z = nullptr;
    DctAxis dct[2];             // the DCT passes along y and z
    bool planes = false;        // ... both at once, plane by plane (plane_dct.cuh)
    double *lam_py = nullptr, *lam_pz = nullptr;   // lam_y, lam_z in the planes' mode order
    bool xt_on = false;         // TMA-staged marching explicit operator
    int xt_cap[4] = {};         // its blocks resident at once, per variable
    UmmaPlan um;                // precision form's tensor-core DCT (when shapes allow)
    double* scal = nullptr;     // device scalars (S_*)
    int* status = nullptr;      // device sticky status bits
    double* work = nullptr;     // slope-parameter scratch
    double* red = nullptr;      // multi-block reduction partials (RED_DOUBLES)
    unsigned* ticket = nullptr; // last-block tickets of those reductions (3, self-resetting)
    double* diag = nullptr;     // per-plane diagnostics + results
    int cur = 0;                // buffer index holding the "old" role
    bool resync_c = false;      // after a restart: copy c's buffers once (resume)
    int tune_exp = 0;           // launch-shape variants (autotuner): explicit-
    int tune_line = 1;          // operator block, x/y line-solve block
    bool tunes_exp = false;     // ... and whether this context launches a kernel
    bool tunes_line = false;    // that takes its shape from them
    bool rotated = false;       // fast steps ran: "new" roles are stale and
                                // logically equal to "old" (see materialize)
    cudaGraphExec_t gexec[2] = {nullptr, nullptr};
    int stream_steps = 0;       // steps taken launch by launch
    double timestep = 0;
    int err = PLLGPU_OK;
    int launches_per_step = 0;
    int counting = 0;
    bool profiling = false;
    std::vector<pll::LaunchRec*>* rec = nullptr;   // recording: launches are stored, not issued
    std::vector<cudaEvent_t> ev_pool;
    std::vector<const char*> ev_label;
    std::vector<void*> allocs;
};

namespace pll {

template <typename real> Bufs<real>& bufs(pllgpu_ctx* c);
template <> inline Bufs<double>& bufs<double>(pllgpu_ctx* c) { return c->b64; }
template <> inline Bufs<float>& bufs<float>(pllgpu_ctx* c) { return c->b32; }

template <typename real> real* q_old(pllgpu_ctx* c, int v) { return bufs<real>(c).q[v][c->cur]; }
template <typename real> real* q_new(pllgpu_ctx* c, int v) { return bufs<real>(c).q[v][1 - c->cur]; }
template <typename real> real* h_n(pllgpu_ctx* c, int v) { return bufs<real>(c).H[v][1 - c->cur]; }
template <typename real> real* h_nm1(pllgpu_ctx* c, int v) { return bufs<real>(c).H[v][c->cur]; }
template <typename real> MuPtrs<real> mu_old(pllgpu_ctx* c)
{
    Bufs<real>& B = bufs<real>(c);
    return {B.mu[c->cur][0], B.mu[c->cur][1], B.mu[c->cur][2], B.mu[c->cur][3]};
}
template <typename real> MuPtrs<real> mu_new(pllgpu_ctx* c)
{
    Bufs<real>& B = bufs<real>(c);
    return {B.mu[1 - c->cur][0], B.mu[1 - c->cur][1], B.mu[1 - c->cur][2], B.mu[1 - c->cur][3]};
}

}  // namespace pll
