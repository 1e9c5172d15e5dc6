// Kernels of the learned surrogate (a 3-d convolutional U-Net that advances
// the cell-centred state of a fingering run by 8 steps): forward, backward
// and Adam, hand-written for the BF16 tensor cores (mma.sync m16n8k16, BF16
// operands, FP32 accumulation).
//
// The forward convolution (and so the input gradient) and the weight gradient
// run on the 5th-generation tensor cores where the shapes allow (nn_umma.cuh:
// tcgen05.mma with a TMEM accumulator, TMA-staged operands whose out-of-bounds
// fill is the zero padding; w rows of up to 128 voxels, channels in sixteens),
// else on the mma.sync kernels below.
//
// Layout: activations are channels-last [n][d][h][w][c] (voxel-major, c
// contiguous), BF16 as operands of the convolutions, FP32 for
// pre-activations and gradients that are accumulated.  Weights are
// [cout][tap][cin] with tap = (dz*3 + dy)*3 + dx.
//
//  * 3x3x3 (and 1x1x1) convolution, zero padding, stride 1, as an implicit
//    GEMM: rows = voxels (128 per CTA), columns = output channels, K = taps x
//    input channels in chunks of 16; the shifted input rows are gathered
//    straight from global memory (16-byte loads, zero outside the volume),
//    double-buffered through shared memory, bias and leaky-ReLU fused in the
//    epilogue.
//  * the input gradient is the same convolution of the output gradient with
//    the weights flipped in space and transposed in channels;
//  * the weight gradient is a GEMM over voxels (cout x cin per tap), split
//    over voxel chunks, FP32 atomics into the gradient;
//  * 2x average pooling, 2x nearest upsampling, channel concatenation,
//    activation backward with the bias-gradient reduction, MSE loss, Adam.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <initializer_list>
#include <type_traits>

#include "nn_umma.cuh"

typedef __nv_bfloat16 bf16;

namespace {

struct Vol {
    int N, D, H, W;
};

__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, const uint32_t* b)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float leaky(float x, float slope) { return x > 0.f ? x : slope * x; }

constexpr int CBM = 128;   // voxels per CTA
constexpr int CBK = 16;    // K chunk (input channels of one tap)
constexpr int CPAD = 24;   // shared row pitch in bf16 (48 bytes: conflict-free fragments)

// Y = act(conv(X, W) + bias): Y32 (pre-activation, FP32) and/or Y16 (post,
// BF16); Cin % 16 == 0, pointers 16-byte aligned
template <int BN>
__global__ void __launch_bounds__(256) k_conv_fwd(const bf16* __restrict__ X, Vol g, int Cin,
                                                  const bf16* __restrict__ Wt, const float* __restrict__ bias,
                                                  int Cout, int ksize, float* __restrict__ Y32,
                                                  bf16* __restrict__ Y16, int act, float slope)
{
    __shared__ __align__(16) bf16 As[2][CBM][CPAD];
    __shared__ __align__(16) bf16 Bs[2][BN][CPAD];
    const long V = (long)g.N * g.D * g.H * g.W;
    const long m0 = (long)blockIdx.x * CBM;
    const int n0 = blockIdx.y * BN;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp & 3, wn = warp >> 2;
    const int gq = lane >> 2, tq = lane & 3;
    constexpr int WN = BN / 2;      // warp tile columns
    constexpr int NQ = WN / 8;      // n8 fragments per warp

    // A loader: row ar (voxel), 8 channels (half ah of the 16-chunk)
    const int ar = tid >> 1, ah = tid & 1;
    const long av = m0 + ar;
    const bool avalid = av < V;
    int an = 0, ad = 0, ahh = 0, aw = 0;
    if (avalid) {
        long t = av;
        aw = (int)(t % g.W);
        t /= g.W;
        ahh = (int)(t % g.H);
        t /= g.H;
        ad = (int)(t % g.D);
        an = (int)(t / g.D);
    }
    const int br = tid >> 1, bh = tid & 1;
    const int ntaps = ksize * ksize * ksize;
    const int kchunks = Cin / CBK;
    const int nk = ntaps * kchunks;

    float acc[2][NQ][4];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[p][q][e] = 0.f;

    uint4 ra, rb;
    auto load = [&](int kk) {
        const int tap = kk / kchunks, c0 = (kk - tap * kchunks) * CBK;
        int dz = 0, dy = 0, dx = 0;
        if (ksize == 3) {
            dz = tap / 9 - 1;
            dy = (tap / 3) % 3 - 1;
            dx = tap % 3 - 1;
        }
        ra = make_uint4(0, 0, 0, 0);
        const int d2 = ad + dz, h2 = ahh + dy, w2 = aw + dx;
        if (avalid && d2 >= 0 && d2 < g.D && h2 >= 0 && h2 < g.H && w2 >= 0 && w2 < g.W) {
            const long nv = (((long)an * g.D + d2) * g.H + h2) * g.W + w2;
            ra = *(const uint4*)(X + nv * Cin + c0 + 8 * ah);
        }
        rb = make_uint4(0, 0, 0, 0);
        if (tid < BN * 2) {
            const int co = n0 + br;
            if (co < Cout) rb = *(const uint4*)(Wt + ((long)co * ntaps + tap) * Cin + c0 + 8 * bh);
        }
    };
    load(0);
    for (int kk = 0; kk < nk; ++kk) {
        const int s = kk & 1;
        *(uint4*)&As[s][ar][8 * ah] = ra;
        if (tid < BN * 2) *(uint4*)&Bs[s][br][8 * bh] = rb;
        __syncthreads();
        if (kk + 1 < nk) load(kk + 1);
        uint32_t a[2][4], b[NQ][2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int r = wm * 32 + p * 16 + gq;
            a[p][0] = *(const uint32_t*)&As[s][r][2 * tq];
            a[p][1] = *(const uint32_t*)&As[s][r + 8][2 * tq];
            a[p][2] = *(const uint32_t*)&As[s][r][2 * tq + 8];
            a[p][3] = *(const uint32_t*)&As[s][r + 8][2 * tq + 8];
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int cn = wn * WN + q * 8 + gq;
            b[q][0] = *(const uint32_t*)&Bs[s][cn][2 * tq];
            b[q][1] = *(const uint32_t*)&Bs[s][cn][2 * tq + 8];
        }
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int q = 0; q < NQ; ++q) mma16816(acc[p][q], a[p], b[q]);
    }
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int q = 0; q < NQ; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const long row = m0 + wm * 32 + p * 16 + gq + 8 * h;
                const int col = n0 + wn * WN + q * 8 + 2 * tq;
                if (row >= V) continue;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (col + e >= Cout) continue;
                    float v = acc[p][q][2 * h + e] + (bias ? bias[col + e] : 0.f);
                    if (Y32) Y32[row * Cout + col + e] = v;
                    if (act) v = leaky(v, slope);
                    if (Y16) Y16[row * Cout + col + e] = __float2bfloat16(v);
                }
            }
}

// dW[co][tap][ci] += sum over voxels of G[v][co] * X[v + o(tap)][ci]
__global__ void __launch_bounds__(256) k_conv_wgrad(const bf16* __restrict__ G, const bf16* __restrict__ X,
                                                    Vol g, int Cin, int Cout, int ksize, long vchunk,
                                                    float* __restrict__ dW)
{
    __shared__ __align__(16) bf16 As[64][CPAD];   // [co][voxel]
    __shared__ __align__(16) bf16 Bs[64][CPAD];   // [ci][voxel]
    const long V = (long)g.N * g.D * g.H * g.W;
    const long v0 = (long)blockIdx.x * vchunk;
    const long v1 = v0 + vchunk < V ? v0 + vchunk : V;
    const int tap = blockIdx.y;
    const int ntc = (Cin + 63) / 64;
    const int co0 = (blockIdx.z / ntc) * 64, ci0 = (blockIdx.z % ntc) * 64;
    const int ntaps = ksize * ksize * ksize;
    int dz = 0, dy = 0, dx = 0;
    if (ksize == 3) {
        dz = tap / 9 - 1;
        dy = (tap / 3) % 3 - 1;
        dx = tap % 3 - 1;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp & 3, wn = warp >> 2;   // warp tile 16 (co) x 32 (ci)
    const int gq = lane >> 2, tq = lane & 3;
    float acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[q][e] = 0.f;
    // loaders: threads 0-127 read 16 voxels x 64 output channels of G,
    // threads 128-255 the same voxels' shifted inputs, 8 channels each
    const int lr = (tid & 127) >> 3, lc = (tid & 7) * 8;
    for (long vb = v0; vb < v1; vb += 16) {
        const long v = vb + lr;
        bf16 vals[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) vals[e] = __float2bfloat16(0.f);
        if (v < v1) {
            if (tid < 128) {
                if (co0 + lc < Cout) {
                    const uint4 u = *(const uint4*)(G + v * Cout + co0 + lc);
                    const bf16* pv = (const bf16*)&u;
#pragma unroll
                    for (int e = 0; e < 8; ++e) vals[e] = pv[e];
                }
            } else {
                long t = v;
                const int w = (int)(t % g.W);
                t /= g.W;
                const int h = (int)(t % g.H);
                t /= g.H;
                const int d = (int)(t % g.D);
                const int n = (int)(t / g.D);
                const int d2 = d + dz, h2 = h + dy, w2 = w + dx;
                if (ci0 + lc < Cin && d2 >= 0 && d2 < g.D && h2 >= 0 && h2 < g.H && w2 >= 0 && w2 < g.W) {
                    const long nv = (((long)n * g.D + d2) * g.H + h2) * g.W + w2;
                    const uint4 u = *(const uint4*)(X + nv * Cin + ci0 + lc);
                    const bf16* pv = (const bf16*)&u;
#pragma unroll
                    for (int e = 0; e < 8; ++e) vals[e] = pv[e];
                }
            }
        }
        __syncthreads();   // previous chunk's fragments are consumed
        if (tid < 128) {
#pragma unroll
            for (int e = 0; e < 8; ++e) As[lc + e][lr] = vals[e];
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) Bs[lc + e][lr] = vals[e];
        }
        __syncthreads();
        uint32_t a[4], b[4][2];
        const int r = wm * 16 + gq;
        a[0] = *(const uint32_t*)&As[r][2 * tq];
        a[1] = *(const uint32_t*)&As[r + 8][2 * tq];
        a[2] = *(const uint32_t*)&As[r][2 * tq + 8];
        a[3] = *(const uint32_t*)&As[r + 8][2 * tq + 8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int cn = wn * 32 + q * 8 + gq;
            b[q][0] = *(const uint32_t*)&Bs[cn][2 * tq];
            b[q][1] = *(const uint32_t*)&Bs[cn][2 * tq + 8];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) mma16816(acc[q], a, b[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int co = co0 + wm * 16 + gq + (e >= 2 ? 8 : 0);
            const int ci = ci0 + wn * 32 + q * 8 + 2 * tq + (e & 1);
            if (co < Cout && ci < Cin) atomicAdd(&dW[((long)co * ntaps + tap) * Cin + ci], acc[q][e]);
        }
}

// Wf[ci][t][co] = W[co][ntaps-1-t][ci]
__global__ void k_flip(const bf16* __restrict__ W, int Cout, int ntaps, int Cin, bf16* __restrict__ Wf)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long n = (long)Cout * ntaps * Cin;
    if (i >= n) return;
    const int ci = (int)(i % Cin);
    const int t = (int)((i / Cin) % ntaps);
    const int co = (int)(i / ((long)Cin * ntaps));
    Wf[((long)ci * ntaps + (ntaps - 1 - t)) * Cout + co] = W[i];
}

// dZ = dY * act'(Z) as BF16, and db[c] += sum_v dZ[v][c]
__global__ void k_act_bwd(const float* __restrict__ dY, const float* __restrict__ Z, long V, int C, int act,
                          float slope, bf16* __restrict__ dZ, float* __restrict__ db)
{
    // block: 256 threads over (voxel chunk, channels); one channel per
    // thread column, voxels strided
    const int c = blockIdx.y * 32 + (threadIdx.x & 31);
    const int vr = threadIdx.x >> 5;   // 0..7
    float s = 0.f;
    if (c < C) {
        for (long v = (long)blockIdx.x * 8 + vr; v < V; v += (long)gridDim.x * 8) {
            float gv = dY[v * C + c];
            if (act && Z[v * C + c] <= 0.f) gv *= slope;
            dZ[v * C + c] = __float2bfloat16(gv);
            s += gv;
        }
    }
    __shared__ float red[8][33];
    red[vr][threadIdx.x & 31] = s;
    __syncthreads();
    if (vr == 0 && c < C) {
        float t = 0.f;
        for (int r = 0; r < 8; ++r) t += red[r][threadIdx.x & 31];
        if (db) atomicAdd(&db[c], t);
    }
}

// The pooling, upsampling and concatenation kernels move VE channels of one
// voxel per thread (16 bytes where the channel counts and the pointers allow,
// else one) and index with IX (32 bits where the array's pieces fit): with one
// element and 64-bit divisions per thread they ran at a tenth of the copy rate
// (2x upsampling of 64 channels to 8 x 128x64x64: 1.6 ms for 0.6 GB).
template <typename T, int VE>
struct __align__(sizeof(T) * VE) Piece {
    T v[VE];
};

template <typename IX>
__device__ __forceinline__ void voxel_of(IX t, const Vol& g, int& b, int& d, int& h, int& w)
{
    w = (int)(t % (unsigned)g.W);
    t /= (unsigned)g.W;
    h = (int)(t % (unsigned)g.H);
    t /= (unsigned)g.H;
    d = (int)(t % (unsigned)g.D);
    b = (int)(t / (unsigned)g.D);
}

__device__ __forceinline__ long voxel_at(const Vol& g, int b, int d, int h, int w)
{
    return (((long)b * g.D + d) * g.H + h) * g.W + w;
}

__device__ __forceinline__ Vol doubled(const Vol& g) { return Vol{g.N, 2 * g.D, 2 * g.H, 2 * g.W}; }
__device__ __forceinline__ Vol halved(const Vol& g) { return Vol{g.N, g.D / 2, g.H / 2, g.W / 2}; }

// child a (0..7) of voxel (b, d, h, w) in the volume f twice as fine
__device__ __forceinline__ long child_at(const Vol& f, int b, int d, int h, int w, int a)
{
    return voxel_at(f, b, 2 * d + (a >> 2), 2 * h + ((a >> 1) & 1), 2 * w + (a & 1));
}

// 2x average pooling of X[N][D][H][W][C] (BF16 in and out)
template <int VE, typename IX>
__global__ void k_pool_fwd(const bf16* __restrict__ X, Vol g, int C, bf16* __restrict__ Y)
{
    using P = Piece<bf16, VE>;
    const Vol q = halved(g);
    const unsigned pc = C / VE;
    const IX i = (IX)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (IX)q.N * q.D * q.H * q.W * pc) return;
    const int c = (int)(i % pc) * VE;
    int b, d, h, w;
    voxel_of<IX>(i / pc, q, b, d, h, w);
    float s[VE];
#pragma unroll
    for (int e = 0; e < VE; ++e) s[e] = 0.f;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const P x = *(const P*)(X + child_at(g, b, d, h, w, a) * C + c);
#pragma unroll
        for (int e = 0; e < VE; ++e) s[e] += __bfloat162float(x.v[e]);
    }
    P y;
#pragma unroll
    for (int e = 0; e < VE; ++e) y.v[e] = __float2bfloat16(0.125f * s[e]);
    *(P*)(Y + (long)i * VE) = y;
}

// gradient of the pooling into dX (FP32, X's volume g), accumulating when acc
template <int VE, typename IX>
__global__ void k_pool_bwd(const float* __restrict__ dY, Vol g, int C, float* __restrict__ dX, int acc)
{
    using P = Piece<float, VE>;
    const unsigned pc = C / VE;
    const IX i = (IX)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (IX)g.N * g.D * g.H * g.W * pc) return;
    const int c = (int)(i % pc) * VE;
    int b, d, h, w;
    voxel_of<IX>(i / pc, g, b, d, h, w);
    P v = *(const P*)(dY + voxel_at(halved(g), b, d / 2, h / 2, w / 2) * C + c);
    P* x = (P*)(dX + (long)i * VE);
    const P o = acc ? *x : P{};
#pragma unroll
    for (int e = 0; e < VE; ++e) v.v[e] = acc ? o.v[e] + 0.125f * v.v[e] : 0.125f * v.v[e];
    *x = v;
}

// [2x nearest upsampling of A (CA channels, volume g) | B (CB channels)] into
// Y (volume 2g); CB = 0: the upsampling alone
template <int VE, typename IX>
__global__ void k_upcat_fwd(const bf16* __restrict__ A, Vol g, int CA, const bf16* __restrict__ B, int CB,
                            bf16* __restrict__ Y)
{
    using P = Piece<bf16, VE>;
    const Vol f = doubled(g);
    const unsigned pc = (CA + CB) / VE;
    const IX i = (IX)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (IX)f.N * f.D * f.H * f.W * pc) return;
    const int c = (int)(i % pc) * VE;
    const IX t = i / pc;
    if (c >= CA) {
        *(P*)(Y + (long)i * VE) = *(const P*)(B + (long)t * CB + (c - CA));
        return;
    }
    int b, d, h, w;
    voxel_of<IX>(t, f, b, d, h, w);
    *(P*)(Y + (long)i * VE) = *(const P*)(A + voxel_at(g, b, d / 2, h / 2, w / 2) * CA + c);
}

// its gradient: dA (volume g) (+)= the sum of the 8 children of dY's first CA
// channels, dB = the other CB (one thread piece each, the copies after the
// sums); dY has CA + CB channels in volume 2g
template <int VE, typename IX>
__global__ void k_upcat_bwd(const float* __restrict__ dY, Vol g, int CA, int CB, float* __restrict__ dA, int accA,
                            float* __restrict__ dB)
{
    using P = Piece<float, VE>;
    const Vol f = doubled(g);
    const int C = CA + CB;
    const unsigned pa = CA / VE, pb = CB / VE;
    const IX sums = (IX)g.N * g.D * g.H * g.W * pa;
    IX i = (IX)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= sums) {
        i -= sums;
        if (i >= (IX)f.N * f.D * f.H * f.W * pb) return;
        *(P*)(dB + (long)i * VE) = *(const P*)(dY + (long)(i / pb) * C + CA + (int)(i % pb) * VE);
        return;
    }
    const int c = (int)(i % pa) * VE;
    int b, d, h, w;
    voxel_of<IX>(i / pa, g, b, d, h, w);
    P s{};
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const P y = *(const P*)(dY + child_at(f, b, d, h, w, a) * C + c);
#pragma unroll
        for (int e = 0; e < VE; ++e) s.v[e] += y.v[e];
    }
    P* x = (P*)(dA + (long)i * VE);
    if (accA) {
        const P o = *x;
#pragma unroll
        for (int e = 0; e < VE; ++e) s.v[e] = o.v[e] + s.v[e];
    }
    *x = s;
}

// Y[v] = [A[v] (CA channels) | B[v] (CB channels)]
template <int VE, typename IX>
__global__ void k_cat_fwd(const bf16* __restrict__ A, int CA, const bf16* __restrict__ B, int CB, long V,
                          bf16* __restrict__ Y)
{
    using P = Piece<bf16, VE>;
    const unsigned pc = (CA + CB) / VE;
    const IX i = (IX)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (IX)V * pc) return;
    const long v = i / pc;
    const int c = (int)(i % pc) * VE;
    *(P*)(Y + (long)i * VE) = c < CA ? *(const P*)(A + v * CA + c) : *(const P*)(B + v * CB + (c - CA));
}

template <int VE, typename IX>
__global__ void k_cat_bwd(const float* __restrict__ dY, int CA, int CB, long V, float* __restrict__ dA, int accA,
                          float* __restrict__ dB, int accB)
{
    using P = Piece<float, VE>;
    const unsigned pc = (CA + CB) / VE;
    const IX i = (IX)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (IX)V * pc) return;
    const long v = i / pc;
    const int c = (int)(i % pc) * VE;
    const bool first = c < CA;
    float* to = first ? dA : dB;
    if (!to) return;
    P* x = (P*)(to + (first ? v * CA + c : v * CB + (c - CA)));
    P y = *(const P*)(dY + (long)i * VE);
    if (first ? accA : accB) {
        const P o = *x;
#pragma unroll
        for (int e = 0; e < VE; ++e) y.v[e] = o.v[e] + y.v[e];
    }
    *x = y;
}

// loss += scale * sum (p - t)^2 ; grad = 2 scale (p - t)
// (a block's terms are summed before its one atomic: an atomic per warp on the
// one address took 3.5 ms over 67 M terms)
__global__ void __launch_bounds__(256) k_mse(const float* __restrict__ P, const float* __restrict__ T, long n,
                                             float scale, float* __restrict__ grad, float* __restrict__ loss)
{
    float s = 0.f;
    for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long)gridDim.x * 256) {
        const float d = P[i] - T[i];
        if (grad) grad[i] = 2.f * scale * d;
        s += scale * d * d;
    }
    if (!loss) return;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ float part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < 8; ++w) t += part[w];
        atomicAdd(loss, t);
    }
}

// sum of squares of x into *out (global gradient norm for clipping)
__global__ void k_sumsq(const float* __restrict__ x, long n, float* __restrict__ out)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    float s = i < n ? x[i] * x[i] : 0.f;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// Adam (Kingma & Ba 2015) on FP32 master weights, BF16 copy out; with
// sumsq given, the gradient is scaled by min(1, clip / ||g||) (global norm
// clipping) and a non-finite norm skips the update
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, long n, float lr, float b1, float b2, float eps, float bc1, float bc2,
                       bf16* __restrict__ w16, const float* __restrict__ sumsq, float clip)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float scale = 1.f;
    if (sumsq) {
        const float nrm = sqrtf(*sumsq);
        if (!isfinite(nrm)) return;
        if (nrm > clip) scale = clip / nrm;
    }
    const float gi = g[i] * scale;
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    w[i] = wi;
    if (w16) w16[i] = __float2bfloat16(wi);
}

__global__ void k_cast(const float* __restrict__ x, long n, bf16* __restrict__ y)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16(x[i]);
}

// network input: cell-centred (u, v, w, c) FP32 [V][4] of one sample plus
// the constant channels -> BF16 [V][16]: (c, u, v, w, r, p, 0 ... 0) after
// the per-channel affine normalisation (x - mean) / std
__global__ void k_pack_input(const float* __restrict__ cells, long V, float r, float p,
                             const float* __restrict__ norm /* mean[4], std[4] */, bf16* __restrict__ out)
{
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const float4 q = ((const float4*)cells)[v];   // u, v, w, c
    const float ch[4] = {q.w, q.x, q.y, q.z};       // c, u, v, w
    bf16* o = out + v * 16;
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = __float2bfloat16((ch[k] - norm[k]) / norm[4 + k]);
    o[4] = __float2bfloat16(r);
    o[5] = __float2bfloat16(p);
#pragma unroll
    for (int k = 6; k < 16; ++k) o[k] = __float2bfloat16(0.f);
}

// training target: the 8-step change of (c, u, v, w) over its scale,
// [V][16] with channels 4-15 zero
__global__ void k_pack_target(const float* __restrict__ a, const float* __restrict__ b, long V,
                              const float* __restrict__ scale /* c, u, v, w */, float* __restrict__ out)
{
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const float4 p = ((const float4*)a)[v], q = ((const float4*)b)[v];   // u, v, w, c
    float* o = out + v * 16;
    o[0] = (q.w - p.w) / scale[0];
    o[1] = (q.x - p.x) / scale[1];
    o[2] = (q.y - p.y) / scale[2];
    o[3] = (q.z - p.z) / scale[3];
#pragma unroll
    for (int k = 4; k < 16; ++k) o[k] = 0.f;
}

// prediction: cells + scale * out[:, 0:4] (out channels c, u, v, w)
__global__ void k_apply_delta(const float* __restrict__ a, const float* __restrict__ out, long V,
                              const float* __restrict__ scale, float* __restrict__ b)
{
    const long v = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    const float4 p = ((const float4*)a)[v];
    const float* o = out + v * 16;
    float4 q;
    q.w = p.w + scale[0] * o[0];
    q.x = p.x + scale[1] * o[1];
    q.y = p.y + scale[2] * o[2];
    q.z = p.z + scale[3] * o[3];
    ((float4*)b)[v] = q;
}

inline unsigned nblk(long n, int b) { return (unsigned)((n + b - 1) / b); }

// ---- the tcgen05 convolution: tensor maps, shape checks, dispatch ----------
int g_conv_path = 0;   // 0: tcgen05 where the shapes allow, 1: mma.sync, 2: tcgen05 or fail

// pieces of VE channels where every count is a multiple of VE and every
// pointer 16-byte aligned, else of one; 32-bit indexes where the pieces fit.
// f(VE, IX) launches over `elems / VE` pieces.
template <int VE, typename F>
int by_piece(long elems, std::initializer_list<int> counts, std::initializer_list<const void*> ptrs, const F& f)
{
    bool wide = true;
    for (int c : counts) wide = wide && c % VE == 0;
    for (const void* p : ptrs) wide = wide && ((uintptr_t)p & 15) == 0;
    const long n = wide ? elems / VE : elems;
    const unsigned blocks = nblk(n, 256);
    const bool small = n + 256 < (1L << 32);
    if (wide && small) f(std::integral_constant<int, VE>(), (unsigned)0, blocks);
    else if (wide) f(std::integral_constant<int, VE>(), (unsigned long)0, blocks);
    else if (small) f(std::integral_constant<int, 1>(), (unsigned)0, blocks);
    else f(std::integral_constant<int, 1>(), (unsigned long)0, blocks);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn nn_encode()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// voxel tiles of the tcgen05 kernels: the whole-row box of at most 128 voxels
// that needs the fewest tiles, of equal ones the one tallest in h; false
// where a w row is longer than a tile
bool cu_boxes(int N, int D, int H, int W, CuGeom& g)
{
    if (W > CU_BM || N < 1 || D < 1 || H < 1 || W < 1) return false;
    g.N = N, g.D = D, g.H = H, g.W = W;
    long best = -1;
    for (int hb = CU_BM / W < H ? CU_BM / W : H; hb >= 1; --hb) {
        const int fit = CU_BM / (W * hb), db = fit < D ? fit : D;
        const long tiles = (long)((H + hb - 1) / hb) * ((D + db - 1) / db);
        if (best < 0 || tiles < best) {
            best = tiles;
            g.hb = hb;
            g.db = db;
        }
    }
    g.th = (H + g.hb - 1) / g.hb;
    g.td = (D + g.db - 1) / g.db;
    return cu_tiles(g) < (1L << 31);
}

// the geometry of the tcgen05 forward path, false when the shapes do not fit
// it: Cout a multiple of the column tile, Cin a multiple of 16
bool cu_geom(int N, int D, int H, int W, int Cin, int Cout, int ksize, CuGeom& g, int& BN, int& CK)
{
    if (Cin % 16 || Cout % 16 || !cu_boxes(N, D, H, W, g)) return false;
    BN = Cout % 128 == 0 ? 128 : Cout % 96 == 0 ? 96 : Cout % 64 == 0 ? 64 : Cout % 32 == 0 ? 32 : 16;
    CK = Cin % 64 == 0 ? 64 : Cin % 32 == 0 ? 32 : 16;
    g.Cin = Cin, g.Cout = Cout, g.ksize = ksize;
    return true;
}

// channels-last [n][d][h][w][C] BF16 array, boxes of CB channels x the tile's
// voxels, swizzled by the box row's width
bool cu_act_map(const CuGeom& g, int C, int CB, const void* X, CUtensorMap* m)
{
    EncodeTiledFn fn = nn_encode();
    if (!fn) return false;
    const CUtensorMapSwizzle sw = CB == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                                : CB == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    const cuuint64_t c2 = (cuuint64_t)C * 2;
    const cuuint64_t xd[5] = {(cuuint64_t)C, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.D, (cuuint64_t)g.N};
    const cuuint64_t xs[4] = {c2, c2 * g.W, c2 * g.W * g.H, c2 * g.W * g.H * g.D};
    const cuuint32_t xb[5] = {(cuuint32_t)CB, (cuuint32_t)g.W, (cuuint32_t)g.hb, (cuuint32_t)g.db, 1};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, (void*)X, xd, xs, xb, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool cu_maps(const CuGeom& g, int BN, int CK, const void* X, const void* Wt, CUtensorMap* mx, CUtensorMap* mw)
{
    EncodeTiledFn fn = nn_encode();
    if (!fn || !cu_act_map(g, g.Cin, CK, X, mx)) return false;
    const CUtensorMapSwizzle sw = CK == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                                : CK == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    const cuuint64_t c2 = (cuuint64_t)g.Cin * 2;
    const cuuint32_t es[3] = {1, 1, 1};
    const int taps = g.ksize * g.ksize * g.ksize;
    const cuuint64_t wd[3] = {(cuuint64_t)g.Cin, (cuuint64_t)taps, (cuuint64_t)g.Cout};
    const cuuint64_t ws[2] = {c2, c2 * taps};
    const cuuint32_t wb[3] = {(cuuint32_t)CK, 1, (cuuint32_t)BN};
    return fn(mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)Wt, wd, ws, wb, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int CK>
bool cu_launch(const CUtensorMap& mx, const CUtensorMap& mw, const CuGeom& g, const float* bias, float* Y32,
               void* Y16, int act, float slope, cudaStream_t st)
{
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_conv_umma<BN, CK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)CuSmem<BN, CK>::DYN) != cudaSuccess)
            return false;
        attr = true;
    }
    const dim3 grid((unsigned)cu_tiles(g), (unsigned)(g.Cout / BN));
    k_conv_umma<BN, CK><<<grid, CU_THREADS, CuSmem<BN, CK>::DYN, st>>>(mx, mw, g, bias, Y32, (__nv_bfloat16*)Y16,
                                                                         act, slope);
    return true;
}

template <int BN>
bool cu_launch_ck(int CK, const CUtensorMap& mx, const CUtensorMap& mw, const CuGeom& g, const float* bias,
                  float* Y32, void* Y16, int act, float slope, cudaStream_t st)
{
    if (CK == 64) return cu_launch<BN, 64>(mx, mw, g, bias, Y32, Y16, act, slope, st);
    if (CK == 32) return cu_launch<BN, 32>(mx, mw, g, bias, Y32, Y16, act, slope, st);
    return cu_launch<BN, 16>(mx, mw, g, bias, Y32, Y16, act, slope, st);
}

// the forward convolution on tcgen05; false when the shapes or the tensor
// maps do not fit (the caller then runs the mma.sync kernel)
bool conv_umma(const void* X, int N, int D, int H, int W, int Cin, const void* Wt, const float* bias, int Cout,
               int ksize, float* Y32, void* Y16, int act, float slope, cudaStream_t st)
{
    CuGeom g;
    int BN = 0, CK = 0;
    if (!cu_geom(N, D, H, W, Cin, Cout, ksize, g, BN, CK)) return false;
    if (((uintptr_t)Y32 & 15) || ((uintptr_t)Y16 & 15) || ((uintptr_t)bias & 3)) return false;
    CUtensorMap mx, mw;
    std::memset(&mx, 0, sizeof(mx));
    std::memset(&mw, 0, sizeof(mw));
    if (!cu_maps(g, BN, CK, X, Wt, &mx, &mw)) return false;
    if (BN == 128) return cu_launch_ck<128>(CK, mx, mw, g, bias, Y32, Y16, act, slope, st);
    if (BN == 96) return cu_launch_ck<96>(CK, mx, mw, g, bias, Y32, Y16, act, slope, st);
    if (BN == 64) return cu_launch_ck<64>(CK, mx, mw, g, bias, Y32, Y16, act, slope, st);
    if (BN == 32) return cu_launch_ck<32>(CK, mx, mw, g, bias, Y32, Y16, act, slope, st);
    return cu_launch_ck<16>(CK, mx, mw, g, bias, Y32, Y16, act, slope, st);
}

// partial sums over the voxels that the weight gradient of one weight is
// split into
long wgrad_chunks(int taps, int Cin, int Cout)
{
    const long n = 4096 / ((long)taps * ((Cout + 63) / 64) * ((Cin + 63) / 64));
    return n < 1 ? 1 : n;
}

// volumes too small for the tcgen05 kernel, whose time hardly depends on the
// volume until the CTAs are full (it sets up and empties one accumulator per
// CTA: 13 us for 16 channels, 17 to 24 from 32 on, 11 for a 1x1x1 kernel), where
// the warp-level kernel takes 7 us and 1 more per 15 voxels: it takes 8 voxels
// in 7 us (13 to 24), 64 in 11 (13 to 24), 128 in 15 to 17
bool wgrad_few(long V, int Cin, int ksize)
{
    return V < (ksize != 3 ? 64 : Cin < 32 ? 96 : 160);
}

template <int GA, int GN>
bool wg_launch(const CuGeom& g, const WgPlan& p, dim3 grid, const CUtensorMap& mx, const CUtensorMap& mg, float* dW,
               cudaStream_t st)
{
    const int smem = (int)WgSmem<GA, GN>::bytes(p.nb);
    // a per-device attribute, set on every launch: the largest block's need
    if (cudaFuncSetAttribute(k_wgrad_umma<GA, GN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)WgSmem<GA, GN>::bytes(128)) != cudaSuccess)
        return false;
    k_wgrad_umma<GA, GN><<<grid, CU_THREADS, smem, st>>>(mx, mg, g, p, dW);
    return true;
}

// the weight gradient on tcgen05; false when the shapes do not fit (the
// caller then runs the mma.sync kernel)
bool wgrad_umma(const void* G, const void* X, int N, int D, int H, int W, int Cin, int Cout, int ksize, float* dW,
                cudaStream_t st)
{
    CuGeom g;
    if (Cin % 16 || Cout % 16 || ((uintptr_t)G & 15) || ((uintptr_t)X & 15) || !cu_boxes(N, D, H, W, g)) return false;
    g.Cin = Cin, g.Cout = Cout, g.ksize = ksize;
    const int GA = Cin % 64 == 0 ? 64 : Cin % 32 == 0 ? 32 : 16;
    WgPlan p;
    p.nb = Cout % 128 == 0 ? 128 : Cout % 64 == 0 ? 64 : Cout % 32 == 0 ? 32 : 16;
    const int GN = p.nb >= 64 ? 64 : p.nb;
    p.taps = ksize * ksize * ksize;
    p.groups = p.taps * (Cin / GA);
    const int tiles = (p.groups * GA + 127) / 128, most = 512 / p.nb;   // row tiles in all; a CTA's accumulators
    p.splits = (tiles + most - 1) / most;
    p.mt = (tiles + p.splits - 1) / p.splits;
    p.splits = (tiles + p.mt - 1) / p.mt;
    p.cols = 32;
    while (p.cols < p.mt * p.nb) p.cols *= 2;
    CUtensorMap mx, mg;
    std::memset(&mx, 0, sizeof(mx));
    std::memset(&mg, 0, sizeof(mg));
    if (!cu_act_map(g, Cin, GA, X, &mx) || !cu_act_map(g, Cout, GN, G, &mg)) return false;
    const long T = cu_tiles(g);
    const int ny = p.splits * (Cout / p.nb);
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // one CTA per SM, the voxel tiles split between the CTAs of a row-tile set
    const long nx = sms / ny < 1 ? 1 : sms / ny;
    const dim3 grid((unsigned)(nx < T ? nx : T), (unsigned)ny);
    // runs a weight's voxels are summed in (wgrad_chunks), in whole runs per CTA
    const long per = (wgrad_chunks(p.taps, Cin, Cout) + grid.x / 2) / grid.x, most_runs = T / grid.x;
    p.runs = (int)(per < 1 ? 1 : per > most_runs ? most_runs : per);
    if (GA == 64) {
        if (GN == 64) return wg_launch<64, 64>(g, p, grid, mx, mg, dW, st);
        if (GN == 32) return wg_launch<64, 32>(g, p, grid, mx, mg, dW, st);
        return wg_launch<64, 16>(g, p, grid, mx, mg, dW, st);
    }
    if (GA == 32) {
        if (GN == 64) return wg_launch<32, 64>(g, p, grid, mx, mg, dW, st);
        if (GN == 32) return wg_launch<32, 32>(g, p, grid, mx, mg, dW, st);
        return wg_launch<32, 16>(g, p, grid, mx, mg, dW, st);
    }
    if (GN == 64) return wg_launch<16, 64>(g, p, grid, mx, mg, dW, st);
    if (GN == 32) return wg_launch<16, 32>(g, p, grid, mx, mg, dW, st);
    return wg_launch<16, 16>(g, p, grid, mx, mg, dW, st);
}

}  // namespace

extern "C" {

// status: 0 ok, 6 invalid argument (shapes), 2 launch failure
int pllnn_conv_fwd(const void* X, int N, int D, int H, int W, int Cin, const void* Wt, const float* bias, int Cout,
                   int ksize, float* Y32, void* Y16, int act, float slope, void* stream)
{
    if (Cin % 16 || (ksize != 1 && ksize != 3) || ((uintptr_t)X & 15) || ((uintptr_t)Wt & 15)) return 6;
    const Vol g{N, D, H, W};
    const long V = (long)N * D * H * W;
    cudaStream_t st = (cudaStream_t)stream;
    if (g_conv_path != 1 && conv_umma(X, N, D, H, W, Cin, Wt, bias, Cout, ksize, Y32, Y16, act, slope, st))
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    if (g_conv_path == 2) return 6;
    if (Cout <= 32) {
        dim3 grid(nblk(V, CBM), nblk(Cout, 32));
        k_conv_fwd<32><<<grid, 256, 0, st>>>((const bf16*)X, g, Cin, (const bf16*)Wt, bias, Cout, ksize, Y32,
                                             (bf16*)Y16, act, slope);
    } else {
        dim3 grid(nblk(V, CBM), nblk(Cout, 64));
        k_conv_fwd<64><<<grid, 256, 0, st>>>((const bf16*)X, g, Cin, (const bf16*)Wt, bias, Cout, ksize, Y32,
                                             (bf16*)Y16, act, slope);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// which kernels the convolutions use: 0 the tcgen05 ones where the shapes
// allow (default), 1 the mma.sync ones, 2 the tcgen05 kernel or status 6
// (forward); returns the previous setting
int pllnn_set_conv_path(int path)
{
    const int old = g_conv_path;
    if (path >= 0 && path <= 2) g_conv_path = path;
    return old;
}

// the library's status bits (0x100: a bounded wait of the tcgen05
// convolution ran out), cleared by the read
int pllnn_status(void)
{
    int v = 0, z = 0;
    if (cudaMemcpyFromSymbol(&v, g_nn_status, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_nn_status, &z, sizeof(int));
    return v;
}

int pllnn_conv_wgrad(const void* G, const void* X, int N, int D, int H, int W, int Cin, int Cout, int ksize,
                     float* dW, void* stream)
{
    if (Cin % 8 || Cout % 8 || (ksize != 1 && ksize != 3)) return 6;
    const Vol g{N, D, H, W};
    const long V = (long)N * D * H * W;
    if ((g_conv_path == 2 || (g_conv_path == 0 && !wgrad_few(V, Cin, ksize))) &&
        wgrad_umma(G, X, N, D, H, W, Cin, Cout, ksize, dW, (cudaStream_t)stream))
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    const int ntaps = ksize * ksize * ksize;
    const int tiles = ((Cout + 63) / 64) * ((Cin + 63) / 64);
    const long chunks = wgrad_chunks(ntaps, Cin, Cout);
    long vchunk = (V + chunks - 1) / chunks;
    vchunk = ((vchunk + 15) / 16) * 16;
    if (vchunk < 256) vchunk = 256;
    dim3 grid((unsigned)((V + vchunk - 1) / vchunk), ntaps, tiles);
    k_conv_wgrad<<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)G, (const bf16*)X, g, Cin, Cout, ksize, vchunk,
                                                         dW);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_flip(const void* Wt, int Cout, int ntaps, int Cin, void* Wf, void* stream)
{
    const long n = (long)Cout * ntaps * Cin;
    k_flip<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>((const bf16*)Wt, Cout, ntaps, Cin, (bf16*)Wf);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_act_bwd(const float* dY, const float* Z, long V, int C, int act, float slope, void* dZ, float* db,
                  void* stream)
{
    long bx = (V + 8 * 64 - 1) / (8 * 64);
    if (bx > 4096) bx = 4096;
    dim3 grid((unsigned)bx, (C + 31) / 32);
    k_act_bwd<<<grid, 256, 0, (cudaStream_t)stream>>>(dY, Z, V, C, act, slope, (bf16*)dZ, db);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_pool_fwd(const void* X, int N, int D, int H, int W, int C, void* Y, void* stream)
{
    if (D % 2 || H % 2 || W % 2) return 6;
    const long n = (long)N * (D / 2) * (H / 2) * (W / 2) * C;
    return by_piece<8>(n, {C}, {X, Y}, [&](auto ve, auto ix, unsigned blocks) {
        k_pool_fwd<ve(), decltype(ix)><<<blocks, 256, 0, (cudaStream_t)stream>>>((const bf16*)X, Vol{N, D, H, W}, C,
                                                                                 (bf16*)Y);
    });
}

int pllnn_pool_bwd(const float* dY, int N, int D, int H, int W, int C, float* dX, int acc, void* stream)
{
    return by_piece<4>((long)N * D * H * W * C, {C}, {dY, dX}, [&](auto ve, auto ix, unsigned blocks) {
        k_pool_bwd<ve(), decltype(ix)><<<blocks, 256, 0, (cudaStream_t)stream>>>(dY, Vol{N, D, H, W}, C, dX, acc);
    });
}

// [2x nearest upsampling of A (CA channels of the volume given) | B] in one pass
int pllnn_upcat_fwd(const void* A, int N, int D, int H, int W, int CA, const void* B, int CB, void* Y, void* stream)
{
    return by_piece<8>((long)N * 8 * D * H * W * (CA + CB), {CA, CB}, {A, B, Y}, [&](auto ve, auto ix, unsigned blocks) {
        k_upcat_fwd<ve(), decltype(ix)><<<blocks, 256, 0, (cudaStream_t)stream>>>(
            (const bf16*)A, Vol{N, D, H, W}, CA, (const bf16*)B, CB, (bf16*)Y);
    });
}

// its gradient: dA (accumulating when accA) and dB
int pllnn_upcat_bwd(const float* dY, int N, int D, int H, int W, int CA, int CB, float* dA, int accA, float* dB,
                    void* stream)
{
    const long V = (long)N * D * H * W;
    return by_piece<4>(V * CA + V * 8 * CB, {CA, CB}, {dY, dA, dB}, [&](auto ve, auto ix, unsigned blocks) {
        k_upcat_bwd<ve(), decltype(ix)><<<blocks, 256, 0, (cudaStream_t)stream>>>(dY, Vol{N, D, H, W}, CA, CB, dA, accA,
                                                                                  dB);
    });
}

int pllnn_up_fwd(const void* X, int N, int D, int H, int W, int C, void* Y, void* stream)
{
    return pllnn_upcat_fwd(X, N, D, H, W, C, nullptr, 0, Y, stream);
}

int pllnn_up_bwd(const float* dY, int N, int D, int H, int W, int C, float* dX, int acc, void* stream)
{
    return pllnn_upcat_bwd(dY, N, D, H, W, C, 0, dX, acc, nullptr, stream);
}

int pllnn_cat_fwd(const void* A, int CA, const void* B, int CB, long V, void* Y, void* stream)
{
    return by_piece<8>(V * (CA + CB), {CA, CB}, {A, B, Y}, [&](auto ve, auto ix, unsigned blocks) {
        k_cat_fwd<ve(), decltype(ix)><<<blocks, 256, 0, (cudaStream_t)stream>>>((const bf16*)A, CA, (const bf16*)B, CB,
                                                                                V, (bf16*)Y);
    });
}

int pllnn_cat_bwd(const float* dY, int CA, int CB, long V, float* dA, int accA, float* dB, int accB, void* stream)
{
    return by_piece<4>(V * (CA + CB), {CA, CB}, {dY, dA, dB}, [&](auto ve, auto ix, unsigned blocks) {
        k_cat_bwd<ve(), decltype(ix)><<<blocks, 256, 0, (cudaStream_t)stream>>>(dY, CA, CB, V, dA, accA, dB, accB);
    });
}

int pllnn_mse(const float* P, const float* T, long n, float scale, float* grad, float* loss, void* stream)
{
    if (n <= 0) return 2;   // no launch of no blocks
    const unsigned blocks = nblk(n, 1024);   // about four terms a thread
    k_mse<<<blocks, 256, 0, (cudaStream_t)stream>>>(P, T, n, scale, grad, loss);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_adam(float* w, const float* g, float* m, float* v, long n, float lr, float b1, float b2, float eps, int t,
               void* w16, const float* sumsq, float clip, void* stream)
{
    const float bc1 = 1.f - powf(b1, (float)t), bc2 = 1.f - powf(b2, (float)t);
    k_adam<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, n, lr, b1, b2, eps, bc1, bc2, (bf16*)w16,
                                                           sumsq, clip);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_sumsq(const float* x, long n, float* out, void* stream)
{
    k_sumsq<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(x, n, out);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_cast(const float* x, long n, void* y, void* stream)
{
    k_cast<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(x, n, (bf16*)y);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_pack_input(const float* cells, long V, float r, float p, const float* norm, void* out, void* stream)
{
    k_pack_input<<<nblk(V, 256), 256, 0, (cudaStream_t)stream>>>(cells, V, r, p, norm, (bf16*)out);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_pack_target(const float* a, const float* b, long V, const float* scale, float* out, void* stream)
{
    k_pack_target<<<nblk(V, 256), 256, 0, (cudaStream_t)stream>>>(a, b, V, scale, out);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int pllnn_apply_delta(const float* a, const float* out, long V, const float* scale, float* b, void* stream)
{
    k_apply_delta<<<nblk(V, 256), 256, 0, (cudaStream_t)stream>>>(a, out, V, scale, b);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // extern "C"
