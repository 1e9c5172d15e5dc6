// Launch recording and member-batched launches (ensembles).
//
// Every step kernel is written as a body, NAME_run(blockIdx, gridDim, ...),
// whose first two parameters shadow the built-ins, the __global__ NAME that
// calls it with the real ones, and a spec NAME_b (body + launch bounds).
// Stage launchers hand kernel, shape and arguments to go(): normally it
// launches NAME; while a context records (an ensemble building its graphs)
// it stores the launch instead.  Members whose recorded steps match launch
// for launch (same kernels, shapes and shared memory) form a class, and the
// ensemble issues each of the class's launches once: k_members runs the
// same body over a grid whose z extent is the class size times the
// member's, member m = blockIdx.z / gz reading its own arguments from a
// device table.  Each member so computes exactly what it computes alone.
// A body whose first argument is its tensor maps finds them in the launch's
// parameters instead (MapPack): a map that lies in global memory has to be
// acquired by every block before it is used, since a later table may lie at an
// earlier one's address, and with those fences 4 steps of 24 members in FP32
// took 13.8 ms instead of 12.7.  Kernels without a body, the tcgen05 DCT's,
// replay one launch per member.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include "host_util.h"

namespace pll {

// argument pack with one layout on host and device
template <typename... P>
struct Tup {};
template <typename H, typename... T>
struct Tup<H, T...> {
    H h;
    Tup<T...> t;
};

template <size_t I>
struct TupAt {
    template <typename H, typename... T>
    __host__ __device__ static const auto& get(const Tup<H, T...>& x)
    {
        return TupAt<I - 1>::get(x.t);
    }
};
template <>
struct TupAt<0> {
    template <typename H, typename... T>
    __host__ __device__ static const H& get(const Tup<H, T...>& x)
    {
        return x.h;
    }
};

inline void tup_fill(Tup<>&) {}
template <typename H, typename... T, typename A, typename... B>
void tup_fill(Tup<H, T...>& x, A&& a, B&&... b)
{
    x.h = H(std::forward<A>(a));
    tup_fill(x.t, std::forward<B>(b)...);
}

// one recorded launch of one member (the interface the ensemble sees)
struct LaunchRec {
    const void* fn = nullptr;   // the member's own kernel: identity of the launch
    dim3 grid, blk;
    size_t smem = 0;
    virtual ~LaunchRec() {}
    virtual bool batchable() const = 0;
    virtual size_t arg_bytes() const = 0;
    virtual const void* arg_data() const = 0;
    virtual void one(cudaStream_t st) const = 0;
    // before a capture: the batched kernel's shared-memory opt-in
    virtual cudaError_t prepare() const = 0;
    // the most members one launch takes
    virtual unsigned most() const = 0;
    // n members of a class at once: their recorded launches, and member m's
    // argument pack at tab + m * stride
    virtual cudaError_t many(const LaunchRec* const* members, const unsigned char* tab, size_t stride, unsigned n,
                             cudaStream_t st) const = 0;
    bool same_launch(const LaunchRec& o) const
    {
        return fn == o.fn && grid.x == o.grid.x && grid.y == o.grid.y && grid.z == o.grid.z && blk.x == o.blk.x &&
               blk.y == o.blk.y && blk.z == o.blk.z && smem == o.smem && arg_bytes() == o.arg_bytes();
    }
};

namespace {

template <auto RUN, typename... P, size_t... I>
__device__ __forceinline__ void member_run(const Tup<P...>& t, uint3 b, dim3 g, std::index_sequence<I...>)
{
    RUN(b, g, TupAt<I>::get(t)...);
}

// the body over members: grid.z = gz x members
template <auto RUN, typename... P>
__global__ void k_members(const unsigned char* __restrict__ tab, unsigned stride, unsigned gz)
{
    const unsigned m = blockIdx.z / gz;
    const Tup<P...>& t = *reinterpret_cast<const Tup<P...>*>(tab + (size_t)m * stride);
    member_run<RUN, P...>(t, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z - m * gz),
                          dim3(gridDim.x, gridDim.y, gz), std::index_sequence_for<P...>{});
}
template <auto RUN, int MAXT, typename... P>
__global__ void __launch_bounds__(MAXT) k_members_b1(const unsigned char* __restrict__ tab, unsigned stride,
                                                     unsigned gz)
{
    const unsigned m = blockIdx.z / gz;
    const Tup<P...>& t = *reinterpret_cast<const Tup<P...>*>(tab + (size_t)m * stride);
    member_run<RUN, P...>(t, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z - m * gz),
                          dim3(gridDim.x, gridDim.y, gz), std::index_sequence_for<P...>{});
}
template <auto RUN, int MAXT, int MINB, typename... P>
__global__ void __launch_bounds__(MAXT, MINB) k_members_b2(const unsigned char* __restrict__ tab, unsigned stride,
                                                           unsigned gz)
{
    const unsigned m = blockIdx.z / gz;
    const Tup<P...>& t = *reinterpret_cast<const Tup<P...>*>(tab + (size_t)m * stride);
    member_run<RUN, P...>(t, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z - m * gz),
                          dim3(gridDim.x, gridDim.y, gz), std::index_sequence_for<P...>{});
}

// the same for a body whose first argument M is its tensor maps, member m's
// in the launch's own parameters
template <typename M, int N>
struct MapPack {
    M m[N];
};
template <auto RUN, int MAXT, int MINB, int N, typename M, typename... P, size_t... I>
__device__ __forceinline__ void member_run_maps(const M& maps, const Tup<M, P...>& t, uint3 b, dim3 g,
                                                std::index_sequence<I...>)
{
    RUN(b, g, maps, TupAt<I + 1>::get(t)...);
}
template <auto RUN, int MAXT, int MINB, int N, typename M, typename... P>
__global__ void __launch_bounds__(MAXT, MINB) k_members_maps(const __grid_constant__ MapPack<M, N> maps,
                                                             const unsigned char* __restrict__ tab, unsigned stride,
                                                             unsigned gz)
{
    const unsigned m = blockIdx.z / gz;
    const Tup<M, P...>& t = *reinterpret_cast<const Tup<M, P...>*>(tab + (size_t)m * stride);
    member_run_maps<RUN, MAXT, MINB, N, M, P...>(maps.m[m], t, make_uint3(blockIdx.x, blockIdx.y, blockIdx.z - m * gz),
                                                 dim3(gridDim.x, gridDim.y, gz), std::index_sequence_for<P...>{});
}
// A large class's launches carry as many maps as a kernel's 32764 bytes of
// parameters hold, a small one's few: the same time a step, but a graph's nodes
// keep their parameters, and building it for 24 members on 4 grids and running 4
// steps took 21 to 24 ms with 40 maps a launch and 19 with 8.
constexpr int MAPS_FEW = 8, MAPS_MANY = 40;

template <typename B, typename = void>
struct BatchMaps : std::false_type {};
template <typename B>
struct BatchMaps<B, std::void_t<decltype(B::maps)>> : std::bool_constant<B::maps> {};

// minimum blocks per SM of a batched copy: the spec's bminb where it has
// one (a body that reads its arguments from memory holds more registers
// than the kernel that finds them in its parameter bank), else its minb
template <typename B, typename = void>
struct BatchMinb {
    static constexpr int value = B::minb;
};
template <typename B>
struct BatchMinb<B, std::void_t<decltype(B::bminb)>> {
    static constexpr int value = B::bminb;
};

// no body: replayed one launch per member
struct NoBatch {
    static constexpr auto run = nullptr;
    static constexpr int maxt = 0, minb = 0;
};

template <typename B, typename... P>
struct LaunchRecT : LaunchRec {
    void (*k)(P...) = nullptr;
    Tup<P...> a;
    bool batchable() const override { return !std::is_same<B, NoBatch>::value; }
    size_t arg_bytes() const override { return sizeof(Tup<P...>); }
    const void* arg_data() const override { return &a; }
    template <size_t... I>
    void one_(cudaStream_t st, std::index_sequence<I...>) const
    {
        k<<<grid, blk, smem, st>>>(TupAt<I>::get(a)...);
    }
    void one(cudaStream_t st) const override { one_(st, std::index_sequence_for<P...>{}); }
    template <int N, typename M, typename... Q>
    static const void* maps_kernel(const Tup<M, Q...>*)
    {
        static_assert(sizeof(MapPack<M, N>) + 16 <= 32764, "a launch's parameters");
        return (const void*)k_members_maps<B::run, B::maxt, BatchMinb<B>::value, N, M, Q...>;
    }
    const void* batched_kernel(unsigned n) const
    {
        if constexpr (std::is_same<B, NoBatch>::value) return nullptr;
        else if constexpr (BatchMaps<B>::value) return n <= MAPS_FEW ? maps_kernel<MAPS_FEW>(&a) : maps_kernel<MAPS_MANY>(&a);
        else if constexpr (B::maxt == 0) return (const void*)k_members<B::run, P...>;
        else if constexpr (BatchMinb<B>::value == 0) return (const void*)k_members_b1<B::run, B::maxt, P...>;
        else return (const void*)k_members_b2<B::run, B::maxt, BatchMinb<B>::value, P...>;
    }
    unsigned most() const override { return BatchMaps<B>::value ? (unsigned)MAPS_MANY : 65535u; }
    cudaError_t prepare() const override
    {
        // static and dynamic shared memory together above 48 KB need the
        // opt-in: asked for on every build (a host call, once per recorded
        // launch, never per step)
        cudaError_t e = cudaSuccess;
        for (unsigned n : {1u, most()}) {
            const void* kb = batched_kernel(n);
            if (kb && smem > 0 && e == cudaSuccess) e = allow_smem(kb, smem);
        }
        return e;
    }
    template <int N, typename M, typename... Q>
    cudaError_t many_maps(const Tup<M, Q...>*, const LaunchRec* const* members, void** rest, dim3 g, unsigned n,
                          cudaStream_t st) const
    {
        MapPack<M, N> maps;
        std::memset(&maps, 0, sizeof(maps));
        for (unsigned m = 0; m < n; ++m) maps.m[m] = static_cast<const LaunchRecT*>(members[m])->a.h;
        void* args[4] = {&maps, rest[0], rest[1], rest[2]};
        return cudaLaunchKernel(batched_kernel(n), g, blk, args, smem, st);
    }
    cudaError_t many(const LaunchRec* const* members, const unsigned char* tab, size_t stride, unsigned n,
                     cudaStream_t st) const override
    {
        const void* kb = batched_kernel(n);
        if (!kb || n > most()) return cudaErrorInvalidValue;
        unsigned st_ = (unsigned)stride, gz = grid.z;
        const dim3 g(grid.x, grid.y, grid.z * n);
        void* args[3] = {(void*)&tab, (void*)&st_, (void*)&gz};
        if constexpr (BatchMaps<B>::value) {
            if (n <= MAPS_FEW) return many_maps<MAPS_FEW>(&a, members, args, g, n, st);
            return many_maps<MAPS_MANY>(&a, members, args, g, n, st);
        } else {
            return cudaLaunchKernel(kb, g, blk, args, smem, st);
        }
    }
};

}  // namespace
}  // namespace pll
