#pragma once

/*
 * A whole march of a small 1D grid in one launch of one cluster of blocks.
 *
 * The blocks of a cluster run at the same time on up to 16 SMs, and reach each
 * other's shared memory.  A march keeps one point pair per thread in registers:
 * a half step hands what a neighbour needs of each point along by shuffles
 * within a warp, and from warp to warp through a slot of shared memory (of the
 * neighbouring block's, where it lies there), ordered by the cluster's hardware
 * barrier.
 */

#include "common.hpp"

#include <algorithm>
#include <cstdint>

namespace scg
{
namespace cluster
{

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// A slot of shared memory of another block of the cluster, and a store to it.
__device__ __forceinline__ unsigned slot_of(void const * p, unsigned rank)
{
    unsigned out;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(out)
        : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p))), "r"(rank));
    return out;
}
__device__ __forceinline__ void slot_put(unsigned at, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}
__device__ __forceinline__ void slot_put(unsigned at, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}

// Hands N values of each thread's v to the thread before it (Q = 1, into w) or
// after it (Q = 0), over the whole cluster; slots: this half step's, one row of N
// per warp of the block.  Every thread of the cluster calls it.  The threads
// at the cluster's ends receive their own values or an unwritten slot's, which
// they do not use.
template <int N, int Q, typename R>
__device__ __forceinline__ void hand_over(R const * v, R * w, R (*slots)[N])
{
    int const ln = static_cast<int>(threadIdx.x) & 31;
    int const warp = static_cast<int>(threadIdx.x) >> 5;
    int const last = static_cast<int>(blockDim.x >> 5) - 1;
    int const from = Q == 1 ? 0 : 31; // the lane whose values leave the warp
    if (ln == from)
    {
        int const to = Q == 1 ? warp - 1 : warp + 1;
        unsigned const me = blockIdx.x;
        if (to >= 0 && to <= last)
        {
            for (int i = 0; i < N; ++i)
            {
                slots[to][i] = v[i];
            }
        }
        else if (Q == 1 ? me > 0 : me + 1 < gridDim.x)
        {
            unsigned const at = slot_of(slots[Q == 1 ? last : 0], Q == 1 ? me - 1 : me + 1);
            for (int i = 0; i < N; ++i)
            {
                slot_put(at + static_cast<unsigned>(i * sizeof(R)), v[i]);
            }
        }
    }
    cluster_sync();
    for (int i = 0; i < N; ++i)
    {
        R const x = Q == 1 ? __shfl_down_sync(0xffffffffu, v[i], 1) : __shfl_up_sync(0xffffffffu, v[i], 1);
        w[i] = ln == 31 - from ? slots[warp][i] : x;
    }
}

// The largest cluster the current device schedules for a kernel at THREADS
// threads a block: 16 where it can (a non-portable size), else a smaller power of
// two, 0 where it schedules none (part of a GPU may have fewer SMs than a
// portable cluster wants).  Asked once per kernel and device, where the
// permission for 16 holds.
template <auto KERNEL, int THREADS>
inline int cluster_limit()
{
    static PerDevice<int> limit;
    return limit.get([] {
        bool const wide =
            cudaFuncSetAttribute(KERNEL, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        (void)cudaGetLastError();
        for (unsigned size = wide ? 16 : 8; size > 0; size /= 2)
        {
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim = {size, 1, 1};
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(size);
            cfg.blockDim = dim3(THREADS);
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, KERNEL, &cfg) == cudaSuccess && n > 0)
            {
                return static_cast<int>(size);
            }
            (void)cudaGetLastError(); // a refusal is no error of the launch to come
        }
        return 0;
    });
}

// Launch a kernel as one cluster of `blocks` blocks.
template <typename K, typename... A>
void launch_cluster(K * kernel, int blocks, int threads, cudaStream_t stream, A... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim = {static_cast<unsigned>(blocks), 1, 1};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(blocks));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cuda_check(cudaLaunchKernelEx(&cfg, kernel, args...), "cluster launch");
}

// Steps per launch of the cluster kernels (a launch of a few milliseconds).
constexpr int64_t CLUSTER_STEPS = 1024;

// Blocks and warps per block of a cluster of that many threads: as many blocks
// as the limit allows before a second warp per block, so that the warps have
// an SM each as long as there are SMs.  False where they do not fit.
template <auto KERNEL, int MAX_WARPS>
bool cluster_shape(int64_t threads, int & blocks, int & warps)
{
    int const limit = cluster_limit<KERNEL, 32 * MAX_WARPS>();
    if (limit == 0)
    {
        return false;
    }
    int64_t const w = (threads + 31) / 32;
    blocks = 1;
    while (blocks < limit && blocks < w)
    {
        blocks *= 2;
    }
    warps = static_cast<int>(std::min<int64_t>((w + blocks - 1) / blocks, MAX_WARPS + 1));
    return warps <= MAX_WARPS;
}

} // namespace cluster
} // namespace scg
