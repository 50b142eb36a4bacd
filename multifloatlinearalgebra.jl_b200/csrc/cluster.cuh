// Helpers of the kernels that run a factorization's pivot steps on one
// thread-block cluster: the cluster barrier, stores into other CTAs' shared
// memory, the first-largest reduction, and the launch's cluster size.
#pragma once
#include "mf_device.cuh"
#include "mflab_internal.h"

namespace mfl {

constexpr int MAX_CLUSTER = 16;

// The pivot kernels run each of their long expressions once per column on few
// warps: kept as calls, their code stays in the instruction cache.
template <int N>
__device__ __noinline__ mf<N> div_call(mf<N> x, mf<N> y) {
    return div(x, y);
}

__device__ __forceinline__ void ld_cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t ld_remote(const void *p, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void ld_remote_f64(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void ld_remote_s32(uint32_t a, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void ld_remote_max(uint32_t a, int v) {
    asm volatile("red.relaxed.cluster.shared::cluster.max.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

template <int N>
__device__ __forceinline__ mf<N> ld_get(const double *p) {
    mf<N> v;
#pragma unroll
    for (int l = 0; l < N; ++l) v.v[l] = p[l];
    return v;
}
template <int N>
__device__ __forceinline__ void ld_put(double *p, const mf<N> &v) {
#pragma unroll
    for (int l = 0; l < N; ++l) p[l] = v.v[l];
}

// larger of two candidates: the first strictly larger value in ascending index
// order; index -1 holds no candidate.  The indices of a reduction's candidates
// are distinct: only then do both sides of an exchange pick the same one where
// neither value is the larger.
template <int N>
__device__ __forceinline__ void ld_better(mf<N> &v, int &i, const mf<N> &o, int oi) {
    bool take = oi >= 0;
    if (take && i >= 0) take = gt(o, v) ? true : gt(v, o) ? false : oi < i;
    if (take) {
        v = o;
        i = oi;
    }
}

// best candidate of the lanes' groups of `width` lanes, in every lane
template <int N>
__device__ __forceinline__ void ld_lanes(mf<N> &v, int &i, int width) {
    for (int off = width / 2; off > 0; off >>= 1) {
        mf<N> o;
#pragma unroll
        for (int l = 0; l < N; ++l) o.v[l] = __shfl_xor_sync(0xffffffffu, v.v[l], off);
        const int oi = __shfl_xor_sync(0xffffffffu, i, off);
        ld_better(v, i, o, oi);
    }
}

// The largest cluster of `kern` (threads per CTA, dynamic shared memory) the
// current device can place: sixteen where the larger, non-portable size fits,
// else eight.  `asked` and `sixteen` are the kernel's bit masks over devices.
inline int largest_cluster(const void *kern, int threads, size_t smem,
                           std::atomic<unsigned long long> &asked,
                           std::atomic<unsigned long long> &sixteen, int *most) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return record_cuda_error(e, "cluster device");
    const unsigned long long bit = 1ULL << (dev & 63);
    if (!(asked.load(std::memory_order_acquire) & bit)) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = MAX_CLUSTER;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(MAX_CLUSTER);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0)
            sixteen.fetch_or(bit, std::memory_order_release);
        else
            cudaGetLastError();
        asked.fetch_or(bit, std::memory_order_release);
    }
    *most = sixteen.load(std::memory_order_acquire) & bit ? MAX_CLUSTER : 8;
    return MFLAB_OK;
}

}  // namespace mfl
