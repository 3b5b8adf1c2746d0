// device_util.cuh — device helpers shared by the sampler and the rebuild kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "smem_limit.h"

namespace culda {

// Neumaier-compensated accumulation: s + c carries the running sum.  Both
// error terms are formed and one selected, so lanes that take different sides
// do not diverge.
__device__ __forceinline__ void neumaier(float &s, float &c, float x) {
    const float t = s + x;
    const float a = (s - t) + x, b = (x - t) + s;
    c += fabsf(s) >= fabsf(x) ? a : b;
    s = t;
}

// The GPU-wide nanosecond timer: kernels of one iteration record their first
// start and last end with it (an event node in the iteration's graph costs
// 3 to 5 us of idle GPU instead).
__device__ __forceinline__ unsigned long long global_timer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void clock_start(unsigned long long *clock) {
    if (clock) atomicMin(&clock[0], global_timer());
}
__device__ __forceinline__ void clock_end(unsigned long long *clock) {
    if (clock) atomicMax(&clock[1], global_timer());
}

// Lanes [g*G, g*G+G) of a warp cooperate on one token ("a group").
template <int G>
__device__ __forceinline__ unsigned group_mask(int lane) {
    if constexpr (G == 32)
        return 0xffffffffu;
    else
        return ((1u << G) - 1u) << (lane & ~(G - 1));
}

// Butterfly sum over the group's lanes; every lane ends with the same bits.
template <int G>
__device__ __forceinline__ float group_sum(float v, unsigned m) {
    if constexpr (G > 1) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(m, v, o));
    }
    return v;
}

template <int G, class T>
__device__ __forceinline__ T group_bcast(T v, int src, unsigned m) {
    if constexpr (G == 1)
        return v;
    else
        return __shfl_sync(m, v, src, G);
}

// Ballot restricted to the group, bit j = lane j of the group.
template <int G>
__device__ __forceinline__ unsigned group_ballot(bool pred, unsigned m, int lane) {
    const unsigned b = __ballot_sync(m, pred);
    if constexpr (G == 32)
        return b;
    else
        return (b >> (lane & ~(G - 1))) & ((1u << G) - 1u);
}

// Exclusive prefix of v over the group's lanes (Kogge-Stone).
template <int G>
__device__ __forceinline__ float group_excl(float v, int gl, unsigned m) {
    if constexpr (G == 1) {
        return 0.f;
    } else {
        float incl = v;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const float t = __shfl_up_sync(m, incl, o, G);
            if (gl >= o) incl += t;
        }
        const float ex = __shfl_up_sync(m, incl, 1, G);
        return gl == 0 ? 0.f : ex;
    }
}

// Opts a kernel into at least `smem` bytes of dynamic shared memory on the
// current device (up to the threshold the default, less room for static shared
// memory, will do).  May be called while a stream is captured.
inline cudaError_t allow_smem(const void *fn, size_t smem) {
    if (smem <= 40 * 1024) return cudaSuccess;
    static SmemLimits limits;  // one per process
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    return (cudaError_t)limits.raise(fn, device, smem, (int)cudaErrorMemoryAllocation, [fn](size_t bytes) {
        return (int)cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    });
}

inline int grid_for(int64_t n) {
    int64_t b = (n + 255) / 256;
    return (int)(b < 1 ? 1 : (b > 148 * 32 ? 148 * 32 : b));
}

}  // namespace culda
