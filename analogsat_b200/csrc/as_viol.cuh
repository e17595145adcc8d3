// Exact unsat counts of many states (ISat::GetClauseViolationCount,
// AnalogSAT/cpu_sat/CpuSat.cpp:136-173; CudaSatBase.cu:124-191), up to 32 states at a
// time: a variable's truth values in the states of a group are the bits of one mask, so a
// clause is checked for all of them with one word load, one gather and two logic
// operations per literal, and counted in bit-sliced counters (plane p holds bit p of
// every state's count).  A variable is TRUE when s > 0; the sentinel's mask is 0 (FALSE).
//
//  viol_group_kernel  instances whose masks fit one SM (compact literal words): one CTA
//                     per group, masks in shared memory, internal variable order.
//  viol_mask_kernel + viol_count_kernel
//                     wider instances: masks in global memory, the clauses of a group
//                     spread over many CTAs, counts added up with integer atomics
//                     (order-independent, so still exact and deterministic).
//
// 16,384 states of N = 1000, M = 4250 took 102 us with one state per CTA pass (every literal
// word and every spin gathered again for each state), 25 us here (33 us with eight loads in
// flight per thread instead of sixteen).  The spins' reads, 4 N bytes per FP32 state, are
// 10 us of it at 6.5 TB/s: a CTA's reads and clause checks follow one another, and the
// CTAs of the one wave are in step, so the two add up.
#pragma once

#include "as_device.cuh"

namespace asb {

constexpr int kViolPlanes = 7;                         // counts up to 127 per thread between flushes
constexpr int kViolFlush = (1 << kViolPlanes) - 1;

// 32 x 32 bit transpose across a warp: lane r's bit c becomes lane c's bit r.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x) {
    const int lane = threadIdx.x & 31;
    uint32_t mask = 0x0000FFFFu;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & j) ? ((x & ~mask) | ((y & ~mask) >> j)) : ((x & mask) | ((y & mask) << j));
        mask ^= mask << (j >> 1);
    }
    return x;
}

// A read-only load that stays in program order: the loads of a batch are all issued before
// the first of them is used, whatever the compiler would make of it otherwise.
__device__ __forceinline__ float ld_once(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_once(const double* p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Truth masks of one variable over `cnt` states (row pointer p, rows `stride` apart).
template <typename T>
__device__ __forceinline__ uint32_t truth_mask(const T* __restrict__ p, int cnt, long long stride) {
    constexpr int U = sizeof(T) == 4 ? 16 : 8;  // loads in flight
    uint32_t m = 0;
    int s = 0;
    for (; s + U <= cnt; s += U, p += U * stride) {
        T v[U];
#pragma unroll
        for (int i = 0; i < U; i++) v[i] = ld_once(p + i * stride);
#pragma unroll
        for (int i = 0; i < U; i++) m |= (v[i] > T(0) ? 1u : 0u) << (s + i);
    }
    for (; s < cnt; s++, p += stride) m |= (__ldg(p) > T(0) ? 1u : 0u) << s;
    return m;
}

// States in which clause m is violated.
template <int KMAX, bool EXACT, int ENC>
__device__ __forceinline__ uint32_t clause_open(const DevInstance& I, int m, const uint32_t* masks) {
    Lit<ENC> w[KMAX];
#pragma unroll
    for (int q = 0; q < KMAX; q++)
        if (EXACT || q < I.k) {
            const int idx = q * I.mp + m;
            if constexpr (ENC == 0) w[q].w = __ldg(I.lit + idx);
            else w[q].w = __ldg(I.litw + idx);
        }
    uint32_t sat = 0;
#pragma unroll
    for (int q = 0; q < KMAX; q++)
        if (EXACT || q < I.k) sat |= masks[w[q].var()] ^ (uint32_t)((int)w[q].w >> 31);
    return ~sat;
}

// Violated clauses m0 + tid, m0 + tid + nt, ... < m1 of every state; returns, in lane s of
// every warp, the warp's count for state s.
template <int KMAX, bool EXACT, int ENC>
__device__ __forceinline__ int count_open(const DevInstance& I, int m0, int m1, int tid, int nt,
                                          const uint32_t* masks) {
    int cnt = 0;
    for (int base = m0; base < m1; base += kViolFlush * nt) {
        const int end = min(m1, base + kViolFlush * nt);
        uint32_t c[kViolPlanes];
#pragma unroll
        for (int p = 0; p < kViolPlanes; p++) c[p] = 0;
        for (int m = base + tid; m < end; m += nt) {
            uint32_t u = clause_open<KMAX, EXACT, ENC>(I, m, masks);
#pragma unroll
            for (int p = 0; p < kViolPlanes; p++) {
                const uint32_t t = c[p] & u;
                c[p] ^= u;
                u = t;
            }
        }
#pragma unroll
        for (int p = 0; p < kViolPlanes; p++) cnt += __popc(warp_transpose32(c[p])) << p;
    }
    return cnt;
}

template <typename T, int KMAX, bool EXACT, int BT>
__global__ void __launch_bounds__(BT) viol_group_kernel(DevInstance I, const T* __restrict__ x,
                                                         int* __restrict__ counts, int ntraj, long long stride,
                                                         int per) {
    extern __shared__ __align__(16) uint32_t viol_masks[];
    __shared__ int total[32];
    const int tid = threadIdx.x, n = I.n;
    const long long s0 = (long long)blockIdx.x * per;
    const int cnt = (int)min((long long)per, ntraj - s0);
    for (int i = tid; i < n; i += BT) viol_masks[__ldg(I.iperm + i)] = truth_mask<T>(x + s0 * stride + i, cnt, stride);
    if (tid == 0) viol_masks[n] = 0u;
    if (tid < 32) total[tid] = 0;
    __syncthreads();
    const int c = count_open<KMAX, EXACT, 0>(I, 0, I.m, tid, BT, viol_masks);
    atomicAdd(total + (tid & 31), c);
    __syncthreads();
    if (tid < cnt) counts[s0 + tid] = total[tid];
}

// Masks of group blockIdx.y (n + 1 words each in gmask), its counts set to zero.
template <typename T>
__global__ void __launch_bounds__(256) viol_mask_kernel(DevInstance I, const T* __restrict__ x,
                                                         int* __restrict__ counts, uint32_t* __restrict__ gmask,
                                                         int ntraj, long long stride) {
    const int n = I.n, groups = (ntraj + 31) / 32;
    for (int g = blockIdx.y; g < groups; g += gridDim.y) {
        const long long s0 = 32ll * g;
        const int cnt = (int)min(32ll, ntraj - s0);
        uint32_t* mk = gmask + (long long)g * (n + 1);
        const int i = blockIdx.x * 256 + threadIdx.x;
        if (i < n) mk[__ldg(I.iperm + i)] = truth_mask<T>(x + s0 * stride + i, cnt, stride);
        if (i == n) mk[n] = 0u;
        if (i < cnt) counts[s0 + i] = 0;
    }
}

// A slice of the clauses of group blockIdx.y, added to the group's counts.
template <int KMAX, bool EXACT>
__global__ void __launch_bounds__(256) viol_count_kernel(DevInstance I, int* __restrict__ counts,
                                                          const uint32_t* __restrict__ gmask, int ntraj) {
    __shared__ int total[32];
    const int tid = threadIdx.x, groups = (ntraj + 31) / 32;
    const int m0 = (int)((long long)I.m * blockIdx.x / gridDim.x);
    const int m1 = (int)((long long)I.m * (blockIdx.x + 1) / gridDim.x);
    for (int g = blockIdx.y; g < groups; g += gridDim.y) {
        if (tid < 32) total[tid] = 0;
        __syncthreads();
        const int c = count_open<KMAX, EXACT, 1>(I, m0, m1, tid, 256, gmask + (long long)g * (I.n + 1));
        atomicAdd(total + (tid & 31), c);
        __syncthreads();
        const long long s = 32ll * g + tid;
        if (tid < 32 && s < ntraj) atomicAdd(counts + s, total[tid]);
        __syncthreads();
    }
}

}  // namespace asb
