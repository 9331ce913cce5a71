// reduce.cuh -- deterministic grid reductions, 16-byte vector views and early launches shared by the
// PCG kernels.
#pragma once

#include "nb2_internal.cuh"

namespace nb2 {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide sum of NV doubles into partials[blockIdx*NV + j]; returns true in the last block
// (after which s_red holds nothing useful and the caller reduces partials itself).
template <int NV>
__device__ bool block_partials(double (&v)[NV], double* partials, unsigned int* counter) {
    __shared__ double red[NV][kRedThreads / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double t = warp_sum(v[j]);
        if (lane == 0) red[j][wid] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            double t = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[j][w];
            partials[blockIdx.x * NV + j] = t;
        }
        __threadfence();
        unsigned int ticket = atomicAdd(counter, 1u);
        last = (ticket == gridDim.x - 1);
    }
    __syncthreads();
    return last;
}

// Fixed-order sum of partials[b*NV + j] over b (called by the whole last block, kRedThreads threads):
// threads, then warps, one barrier.
template <int NV>
__device__ __forceinline__ void final_sum(const double* partials, double (&out)[NV]) {
    __shared__ double red[NV][kRedThreads / 32];
    __threadfence();
    double t[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) t[j] = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kRedThreads)
#pragma unroll
        for (int j = 0; j < NV; ++j) t[j] += __ldcg(partials + b * NV + j);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        t[j] = warp_sum(t[j]);
        if ((threadIdx.x & 31) == 0) red[j][threadIdx.x >> 5] = t[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        out[j] = 0.0;
#pragma unroll
        for (int w = 0; w < kRedThreads / 32; ++w) out[j] += red[j][w];
    }
}

// 16-byte vector view of the CG vectors (float4 / double2): the update kernels move W values
// per load and store when every vector is 16-byte aligned (device allocations are; a caller's
// buffers may not be, then the scalar loop does all of it)
template <typename X>
struct Vec16;
template <>
struct Vec16<float> {
    using T = float4;
    static constexpr int W = 4;
};
template <>
struct Vec16<double> {
    using T = double2;
    static constexpr int W = 2;
};

__device__ __forceinline__ bool aligned16(const void* a, const void* b, const void* c,
                                          const void* d, const void* e) {
    return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
             reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(d) |
             reinterpret_cast<uintptr_t>(e)) & 15) == 0;
}

// wait for the kernels before this one (programmatic dependent launch; nothing to wait for after an
// ordinary one), and let the next one start its own prologue; neither orders anything else: the wait
// returns when they have completed
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// launch a kernel that may start while the one before it runs (pdl); it has to call pdl_wait before
// it touches anything that one writes
template <typename... Args>
cudaError_t launch_early(bool pdl, cudaStream_t stream, unsigned grid, unsigned block,
                         size_t smem, void (*kernel)(Args...), Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace nb2
