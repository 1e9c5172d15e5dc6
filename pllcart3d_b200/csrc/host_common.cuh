// Host-side helpers shared by the runtime and the two precision-form
// orchestration units (each translation unit keeps its own copy).
#pragma once

#include <cstdio>

#include "ctx.cuh"

namespace pll {
namespace {

int fail(pllgpu_ctx* c, int code)
{
    if (c && c->err == PLLGPU_OK) c->err = code;
    return code;
}

#define CK(call)                                                                     \
    do {                                                                             \
        cudaError_t e_ = (call);                                                     \
        if (e_ != cudaSuccess) {                                                     \
            std::fprintf(stderr, "pllgpu: %s failed: %s (%s:%d)\n", #call,           \
                         cudaGetErrorString(e_), __FILE__, __LINE__);                \
            return fail(ctx, PLLGPU_ECUDA);                                          \
        }                                                                            \
    } while (0)

// Side branches of the step.  fork(n) lets side streams 0 .. n-1 start after
// everything enqueued so far, on_side(i) sends the following launches there
// (on_side(-1): back to the main stream), join(n) makes the main stream wait
// for them.  A step recorded for an ensemble, or profiled launch by launch, has
// no branches: its launches stay in order.
bool branches(const pllgpu_ctx* c) { return !c->rec && !c->profiling; }

// whether a spec's own kernel (not its batched copy) begins with after_previous()
template <typename B, typename = void>
struct Chained : std::false_type {};
template <typename B>
struct Chained<B, std::void_t<decltype(B::chained)>> : std::bool_constant<B::chained> {};

// every kernel launch of the step: launched, or recorded while the context
// records (B: the kernel's batching spec, NoBatch where it has none)
template <typename B, typename... P, typename... A>
void go(pllgpu_ctx* ctx, void (*k)(P...), dim3 grid, dim3 blk, size_t smem, A&&... a)
{
    if (ctx->rec) {
        auto* r = new LaunchRecT<B, P...>();
        r->fn = (const void*)k;
        r->k = k;
        r->grid = grid;
        r->blk = blk;
        r->smem = smem;
        tup_fill(r->a, std::forward<A>(a)...);
        ctx->rec->push_back(r);
        return;
    }
    // On the same stream as the launch before it, a kernel that begins with
    // after_previous() is let in while that one still drains.
    const int at = ctx->at == ctx->st ? 0 : ctx->at == ctx->side[0] ? 1 : ctx->at == ctx->side[1] ? 2 : 3;
    const bool early = Chained<B>::value && ctx->chaining && ctx->follows[at] && branches(ctx);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = blk;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->at;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, k, static_cast<P>(std::forward<A>(a))...) != cudaSuccess) fail(ctx, PLLGPU_ECUDA);
    ctx->follows[at] = true;
}

void fork(pllgpu_ctx* ctx, int n)
{
    if (!branches(ctx)) return;
    bool ok = cudaEventRecord(ctx->ev_fork, ctx->st) == cudaSuccess;
    for (int i = 0; i < n && ok; ++i) {
        ok = cudaStreamWaitEvent(ctx->side[i], ctx->ev_fork, 0) == cudaSuccess;
        ctx->follows[1 + i] = false;
    }
    if (!ok) fail(ctx, PLLGPU_ECUDA);
}

void on_side(pllgpu_ctx* ctx, int i)
{
    if (branches(ctx)) ctx->at = i < 0 ? ctx->st : ctx->side[i];
}

void join(pllgpu_ctx* ctx, int n)
{
    if (!branches(ctx)) return;
    ctx->at = ctx->st;
    ctx->follows[0] = false;
    bool ok = true;
    for (int i = 0; i < n && ok; ++i)
        ok = cudaEventRecord(ctx->ev_join[i], ctx->side[i]) == cudaSuccess &&
             cudaStreamWaitEvent(ctx->st, ctx->ev_join[i], 0) == cudaSuccess;
    if (!ok) fail(ctx, PLLGPU_ECUDA);
}

// every kernel launch of the step goes through mark(): it counts launches
// and, in profiling mode, records an event after the launch so that the
// device time of each kernel is the gap to the previous event
void mark(pllgpu_ctx* ctx, const char* label)
{
    ctx->counting++;
    if (!ctx->profiling) return;
    const size_t i = ctx->ev_label.size();
    if (i >= ctx->ev_pool.size()) {
        cudaEvent_t e;
        cudaEventCreate(&e);
        ctx->ev_pool.push_back(e);
    }
    cudaEventRecord(ctx->ev_pool[i], ctx->st);
    ctx->ev_label.push_back(label);
}

template <typename T>
T* dalloc(pllgpu_ctx* ctx, long n)
{
    void* p = nullptr;
    // 1 KB of zeroed slack past the end: kernels that compute cell pairs
    // (k_explicit2) read, and never write, up to 66 elements beyond a field
    const size_t bytes = sizeof(T) * (size_t)(n > 0 ? n : 1) + 1024;
    if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
    cudaMemset(p, 0, bytes);
    ctx->allocs.push_back(p);
    return (T*)p;
}

dim3 box_grid(int nk, int nj, int ni, dim3 blk)
{
    return dim3((nk + blk.x - 1) / blk.x, (nj + blk.y - 1) / blk.y, ni);
}

int ni(const Rng& r) { return r.ie - r.is + 1; }
int nj(const Rng& r) { return r.je - r.js + 1; }
int nk(const Rng& r) { return r.ke - r.ks + 1; }

int set_scalar(pllgpu_ctx* ctx, int slot, double v)
{
    CK(cudaMemcpyAsync(ctx->scal + slot, &v, sizeof(double), cudaMemcpyHostToDevice, ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
    return PLLGPU_OK;
}

double get_scalar(pllgpu_ctx* ctx, int slot)
{
    double v = NAN;
    if (cudaMemcpyAsync(&v, ctx->scal + slot, sizeof(double), cudaMemcpyDeviceToHost, ctx->st) != cudaSuccess ||
        cudaStreamSynchronize(ctx->st) != cudaSuccess)
        fail(ctx, PLLGPU_ECUDA);
    return v;
}

int check_launch(pllgpu_ctx* ctx)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        std::fprintf(stderr, "pllgpu: kernel launch failed: %s\n", cudaGetErrorString(e));
        return fail(ctx, PLLGPU_ECUDA);
    }
    return PLLGPU_OK;
}

int read_status(pllgpu_ctx* ctx)
{
    int s = 0;
    CK(cudaMemcpyAsync(&s, ctx->status, sizeof(int), cudaMemcpyDeviceToHost, ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
    if (s & ST_NAN) return fail(ctx, PLLGPU_ENAN);
    if (s & ST_NOCONV) return fail(ctx, PLLGPU_ENOCONV);
    if (s & ST_BOUNDS) return fail(ctx, PLLGPU_EBOUNDS);
    if (s & ST_TIMEOUT) return fail(ctx, PLLGPU_ETIMEOUT);
    return PLLGPU_OK;
}

__global__ void k_convert_to_f32(long n, const double* __restrict__ a, float* __restrict__ b)
{
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) b[t] = (float)a[t];
}

__global__ void k_convert_to_f64(long n, const float* __restrict__ a, double* __restrict__ b)
{
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) b[t] = (double)a[t];
}

}  // namespace
}  // namespace pll
