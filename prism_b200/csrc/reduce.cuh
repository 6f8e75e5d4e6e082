// reduce.cuh -- deterministic grid-wide reductions shared by the solver kernels.
//
// A reducing kernel accumulates per-thread partial sums (or maxima) of NV
// values, then calls reduceLast(): every block reduces its threads in a fixed
// order and publishes one partial per value, and the last block to arrive
// (an atomic ticket) reduces the block partials in block order. The result is
// bitwise the same on every run for a given grid, with no floating-point
// atomics. The caller's scalar epilogue runs in thread 0 of the last block.
#pragma once

#include "common.h"

namespace pb {

__device__ __forceinline__ double warpSum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warpMax(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Block-reduce NV sums (or maxima; from value MAX_FROM on with that given), publish the block partial, and let the last
// block to arrive reduce all partials in block order. Returns true in the last
// block, where out[] holds the grid totals in every thread. partials holds
// gridDim.x * NV doubles; counter starts at 0 and is left at 0.
template <int NV, bool MAX, int BLOCK = 256, int MAX_FROM = MAX ? 0 : NV>
__device__ bool reduceLast(double (&v)[NV], double* partials, unsigned int* counter, double (&out)[NV]) {
    constexpr int NW = BLOCK / 32;
    __shared__ double sh[NV][NW];
    __shared__ int is_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < NV; ++k) {
        double x = k >= MAX_FROM ? warpMax(v[k]) : warpSum(v[k]);
        if (lane == 0) sh[k][warp] = x;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 0; k < NV; ++k) {
            double s = sh[k][0];
            for (int w = 1; w < NW; ++w) s = k >= MAX_FROM ? fmax(s, sh[k][w]) : s + sh[k][w];
            partials[blockIdx.x * NV + k] = s;
        }
        __threadfence();
        unsigned int t = atomicAdd(counter, 1u);
        is_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    double acc[NV];
    for (int k = 0; k < NV; ++k) {
        acc[k] = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += BLOCK) {
            double x = __ldcg(&partials[b * NV + k]);
            acc[k] = k >= MAX_FROM ? fmax(acc[k], x) : acc[k] + x;
        }
    }
    __syncthreads();
    for (int k = 0; k < NV; ++k) {
        double x = k >= MAX_FROM ? warpMax(acc[k]) : warpSum(acc[k]);
        if (lane == 0) sh[k][warp] = x;
    }
    __syncthreads();
    for (int k = 0; k < NV; ++k) {
        double s = sh[k][0];
        for (int w = 1; w < NW; ++w) s = k >= MAX_FROM ? fmax(s, sh[k][w]) : s + sh[k][w];
        out[k] = s;
    }
    if (threadIdx.x == 0) *counter = 0u;
    return true;
}

// Scale of the FP32 copies of vectors that an FP32 preconditioner of an FP64 iteration reads, from
// the squared norm of the residual at its (re)start. The cycle is linear and the recurrences do
// not depend on a factor in it, so the scale only has to keep the residual's entries, down to 1e-18
// of its first norm, within FP32's 1e-38 to 3e38: 1 from 1e-18 to 1e24, else the power of two that
// brings the norm near 1 (every bit of the results is then that of a system scaled so).
// Kept as what it adds to a double's upper word.
__device__ __forceinline__ int cycleShift(double rr) {
    if (!(rr > 0.0) || !isfinite(rr) || (rr >= 1e-36 && rr <= 1e48)) return 0;
    return -(ilogb(rr) / 2) * (1 << 20);
}
__device__ __forceinline__ float cycleCopy(double v, int shift) {
    const int hi = __double2hiint(v);
    return (float)__hiloint2double((hi & 0x7fffffff) ? hi + shift : hi, __double2loint(v));
}

}  // namespace pb
