// cluster.cuh -- barriers and reductions of the kernels that run a whole solve in one
// thread-block cluster (or in one block: CL false).
#pragma once

#include <cooperative_groups.h>

#include "common.h"

namespace pb {

constexpr int CLUSTER_MAX = 16;  // blocks per cluster (beyond 8 a non-portable size)

// Shared memory of one block's ClusterReduce<THREADS, CL, NV>
template <int THREADS, int NV>
struct ClusterShared {
    double red[2][NV][THREADS / 32];
    double xch[2][CLUSTER_MAX][NV];
};

template <int THREADS, bool CL, int NV>
struct ClusterReduce {
    static constexpr int NW = THREADS / 32;
    ClusterShared<THREADS, NV>& sh;
    cooperative_groups::cluster_group cl;
    int ctas, rank, parity = 0;

    __device__ explicit ClusterReduce(ClusterShared<THREADS, NV>& s) : sh(s), cl(cooperative_groups::this_cluster()) {
        ctas = CL ? (int)cl.num_blocks() : 1;
        rank = CL ? (int)cl.block_rank() : 0;
    }
    __device__ __forceinline__ void barrier() {
        if constexpr (CL) cl.sync();
        else __syncthreads();
    }
    // Sums (MAX: maxima of magnitudes) of v[0, N) over all threads, in every thread; also a
    // barrier. Each block sends its partial results to every other block before it arrives, and
    // all add them in block order: the same bits on every run. The buffers alternate: the next
    // reduction never writes what a slow thread still reads.
    template <int N, bool MAX = false>
    __device__ __forceinline__ void all(double (&v)[NV]) {
        auto join = [](double a, double c) { return MAX ? fmax(a, c) : a + c; };
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] = join(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < N; ++k) sh.red[parity][k][warp] = v[k];
        __syncthreads();
        if constexpr (!CL) {
            // every warp adds the warps' results itself: a barrier less than one warp doing it
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] = sh.red[parity][k][lane % NW];
#pragma unroll
            for (int o = NW / 2; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < N; ++k) v[k] = join(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
        } else {
            if (warp == 0) {
                double u[N];
#pragma unroll
                for (int k = 0; k < N; ++k) u[k] = sh.red[parity][k][lane % NW];
#pragma unroll
                for (int o = NW / 2; o > 0; o >>= 1)
#pragma unroll
                    for (int k = 0; k < N; ++k) u[k] = join(u[k], __shfl_xor_sync(0xffffffffu, u[k], o));
                if (lane < ctas) {
                    double* to = cl.map_shared_rank(&sh.xch[parity][rank][0], lane);
#pragma unroll
                    for (int k = 0; k < N; ++k) to[k] = u[k];
                }
            }
            barrier();
#pragma unroll
            for (int k = 0; k < N; ++k) {
                double u = sh.xch[parity][0][k];
                for (int c = 1; c < ctas; ++c) u = join(u, sh.xch[parity][c][k]);
                v[k] = u;
            }
        }
        parity ^= 1;
    }
};

// Whether the current device places a cluster of CLUSTER_MAX blocks of `kernel` (and allows it to,
// on this device only)
template <typename K>
bool clusterPlaced(K kernel, int threads) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CLUSTER_MAX);
    cfg.blockDim = dim3((unsigned)threads);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CLUSTER_MAX;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    const bool ok = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n >= 1;
    cudaGetLastError();  // a refused query leaves no sticky error
    return ok;
}

// Launches `kernel` as one cluster of ctas blocks; pdl: it releases and awaits its
// neighbours in the stream itself (pdlEnter)
template <typename... KArgs, typename... Args>
void launchCluster(void (*kernel)(KArgs...), int ctas, int threads, cudaStream_t s, bool pdl, const Args&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = pdl && pdlEnabled() ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    PB_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    countLaunch();
}

}  // namespace pb
