// Host-side helpers shared by the runtime and the stand-alone primitives.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <mutex>

namespace pll {

inline bool is_pow2(double h)
{
    int e;
    const double m = std::frexp(h, &e);
    return m == 0.5;
}

// FFTW REDFT10 (kind 0) / REDFT01 (kind 1) as dense matrices T[k*n+j]
// (FFTW 3 manual, "1d Real-even DFTs (DCTs)"); the argument is reduced
// mod 4n exactly
inline double dct_entry(int kind, int n, int k, int j)
{
    const double pi = 3.14159265358979323846;
    if (kind == 1 && j == 0) return 1.0;
    const long m = (kind == 0 ? (long)(2 * j + 1) * (long)k : (long)j * (long)(2 * k + 1)) % (4L * n);
    return 2.0 * std::cos(pi * (double)m / (2.0 * n));
}

template <typename T>
inline void dct_matrix(int kind, int n, T* out)
{
    for (int k = 0; k < n; ++k)
        for (int j = 0; j < n; ++j) out[(long)k * n + j] = (T)dct_entry(kind, n, k, j);
}

// Dynamic shared memory of a kernel, opted in for up to `bytes`.  The limit
// belongs to the kernel on the current device, for every context and thread:
// a kernel launched in several sizes (the folded DCT by its length, the batched
// copies by their class) must keep the largest, so it is only ever raised.
inline cudaError_t allow_smem(const void* kernel, size_t bytes)
{
    static std::mutex one;
    std::lock_guard<std::mutex> hold(one);
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
    if (e != cudaSuccess || (long)bytes <= (long)a.maxDynamicSharedSizeBytes) return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// owning device buffer released on scope exit
struct DevBuf {
    void* p = nullptr;
    ~DevBuf()
    {
        if (p) cudaFree(p);
    }
    bool alloc(size_t bytes) { return cudaMalloc(&p, bytes ? bytes : 8) == cudaSuccess; }
    double* d() { return (double*)p; }
};

}  // namespace pll
