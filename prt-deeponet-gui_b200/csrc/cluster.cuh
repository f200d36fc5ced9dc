// cluster.cuh -- what the solves that run inside one thread-block cluster share:
// addresses in the cluster's shared memory and the cluster barrier.
//
// A small grid's step is launch, dependent loads and drain, about 2 us
// whatever its size.  When the whole state fits in the shared memory of one
// cluster, the time loop runs in a single kernel: a block per SM holds a part
// of the voxels, one thread each, neighbours in other blocks are reached
// through distributed shared memory, and a step ends with the hardware's
// cluster barrier.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace prt {

// A cluster of 16 blocks needs the non-portable size; what the device can
// place is asked before the first launch.
constexpr int kClusterMax = 16;

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Every thread of every block of the cluster; writes before it are visible
// after it.  The .aligned forms ask that a warp's threads arrive together, and
// the loops come here from branches that part a warp (the last live slot,
// thread 0), so the warp is brought together first; that costs nothing, the
// forms without .aligned 1-5 % of a step.
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::
            : "memory");
}

__device__ __forceinline__ uint32_t shared_address(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
// The same place in the shared memory of block `rank` of the cluster.
__device__ __forceinline__ uint32_t in_block(uint32_t local, unsigned rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}

__device__ __forceinline__ void ld_cluster(uint32_t a, double& v) {
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_cluster(uint32_t a, float& v) {
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_cluster(uint32_t a, int& v) {
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_cluster(uint32_t a, __half& v) {
    unsigned short u;
    asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(u) : "r"(a) : "memory");
    v = __ushort_as_half(u);
}
__device__ __forceinline__ void st_cluster(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, __half v) {
    asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(a), "h"(__half_as_ushort(v)) : "memory");
}

// Blocks for n voxels in parts of whole 128s, at most kClusterMax: a power of
// two (1, 2, 4, 8 or 16).
inline int cluster_blocks(long long n) {
    int c = 1;
    while (c < kClusterMax && (long long)c * 128 < n) c *= 2;
    return c;
}
inline int cluster_span(long long n, int blocks) {
    const long long per = (n + blocks - 1) / blocks;
    return (int)((per + 127) / 128 * 128);
}

// Launches `kern` as one cluster, or returns cudaErrorNotSupported where the
// device cannot place it.  smem_most: the most shared memory that any launch
// of the kernel takes; the limit belongs to the kernel, not to the launch, so
// every launch sets the same one and threads do not lower one another's.
template <class K, class... A>
inline cudaError_t launch_cluster(K kern, int blocks, int threads, size_t smem, size_t smem_most,
                                  cudaStream_t s, A... args) {
    cudaError_t e = cudaSuccess;
    if (smem_most)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_most);
    if (e == cudaSuccess && blocks > 8)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int room = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&room, kern, &cfg);
    if (e != cudaSuccess || room < 1) {
        cudaGetLastError();
        return cudaErrorNotSupported;
    }
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace prt
