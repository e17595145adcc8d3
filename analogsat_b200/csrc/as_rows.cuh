// Standalone RHS (ISat::GetDerivatives) of instances that no SM holds: the whole GPU works
// on one group of states at a time, in three kernels per group of L states:
//
//  row_spread_kernel   public spins -> rows [internal variable][L], sentinel row -1;
//  row_clause_kernel   one thread per SUB lanes of a clause: K row gathers, da_m straight to
//                      the public output, the literals' contributions to the rows of their
//                      SELL slots [slot][L];
//  row_var_kernel      one thread per SUB lanes of a variable: its slots' rows in public
//                      clause order (the reference's summation order), ds_i to the output.
//
// An FP32 row of L = 8 lanes (FP64: 4) is one 32-byte sector, so the random accesses -- the
// spin gathers and the contribution stores -- move whole sectors, and the literal words are
// read once per group.  Groups are processed in chunks whose rows stay in L2 where an
// instance allows it.  Bound by those random sectors of L2, one gather and one store per
// literal.  One CTA per state with its vectors in global memory, the form before it (still
// used for the tanh and bias variants, whose clause-weight sum is per CTA), is bound by one
// SM's L2 latency: four states of N = 1e5, M = 1e6, K = 4 took 6,380 us, 100 us here; 2,176
// of N = 3800, K = 3 (compact words, clauses out of public order) 1,296 us, 434 us here (618
// with the clauses taken in the packing's order).
// Arithmetic as clause_phase / var_phase, lane by lane.
#pragma once

#include "as_device.cuh"

namespace asb {

template <typename T, int SUB> struct LaneVec { T v[SUB]; };
template <typename T, int SUB>
__device__ __forceinline__ LaneVec<T, SUB> ld_lanes(const T* p) {
    LaneVec<T, SUB> r;
    if constexpr (SUB * sizeof(T) == 16) {
        *reinterpret_cast<uint4*>(&r) = *reinterpret_cast<const uint4*>(p);
    } else {
        static_assert(SUB == 1, "16-byte or scalar lanes");
        r.v[0] = *p;
    }
    return r;
}
template <typename T, int SUB>
__device__ __forceinline__ void st_lanes(T* p, const LaneVec<T, SUB>& r) {
    if constexpr (SUB * sizeof(T) == 16) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&r);
    else *p = r.v[0];
}

// One chunk of state groups: states s0 .. s0 + ns - 1 in groups of L lanes; group g's spin
// rows at sy + g sy_stride, its contribution rows at cs + g cs_stride.
template <typename T>
struct RowArgs {
    DevInstance I;
    const T* x;
    T* dxdt;
    long long stride;  // values per state
    T *sy, *cs;
    long long sy_stride, cs_stride;
    long long s0;
    int ns;
};

template <typename T, int L>
__global__ void __launch_bounds__(256) row_spread_kernel(RowArgs<T> A) {
    const int n = A.I.n, g = blockIdx.y;
    const int i = blockIdx.x * 256 + threadIdx.x;
    T* sy = A.sy + g * A.sy_stride;
    if (i < n) {
        const int cnt = min(L, A.ns - g * L);
        const T* x = A.x + (A.s0 + (long long)g * L) * A.stride + i;
        T v[L];
#pragma unroll
        for (int l = 0; l < L; l++) v[l] = l < cnt ? __ldg(x + l * A.stride) : T(0);
        T* row = sy + (long long)__ldg(A.I.iperm + i) * L;
#pragma unroll
        for (int l = 0; l < L; l++) row[l] = v[l];
    } else if (i == n) {
#pragma unroll
        for (int l = 0; l < L; l++) sy[(long long)n * L + l] = T(-1);
    }
}

template <typename T, bool LOGA, int KMAX, bool EXACT, int SUB, int R>
__global__ void __launch_bounds__(256) row_clause_kernel(RowArgs<T> A) {
    using Ar = Arith<T>;
    constexpr int L = SUB * R;
    // the power-of-two folding of clause_phase (same roundings)
    constexpr bool kFold = LOGA && sizeof(T) == 4;
    const DevInstance& I = A.I;
    const int g = blockIdx.y;
    const long long it = (long long)blockIdx.x * 256 + threadIdx.x;
    // public clause order: the accesses to x and dxdt are the coalesced ones, the words those
    // that follow the packing's clause order (2 L against 2 K accesses a clause)
    const int j = (int)(it / R), lb = (int)(it % R) * SUB;
    if (j >= I.m) return;
    const int m = __ldg(I.icperm + j);
    const T* sy = A.sy + g * A.sy_stride + lb;
    T* cs = A.cs + g * A.cs_stride + lb;
    const T knorm = (T)ldexp(1.0, -I.k);
    const int cnt = A.ns - g * L - lb;  // this thread's lanes below cnt are states
    const long long at = (A.s0 + (long long)g * L + lb) * A.stride + I.n + j;
    uint32_t w[KMAX], slot[KMAX];
#pragma unroll
    for (int q = 0; q < KMAX; q++)
        if (EXACT || q < I.k) w[q] = __ldg(I.litw + (size_t)q * I.mp + m);
    T am[SUB];
#pragma unroll
    for (int l = 0; l < SUB; l++) am[l] = l < cnt ? __ldg(A.x + at + l * A.stride) : T(0);
    T f[KMAX][SUB];
#pragma unroll
    for (int q = 0; q < KMAX; q++)
        if (EXACT || q < I.k) {
            const LaneVec<T, SUB> s = ld_lanes<T, SUB>(sy + (long long)(w[q] & 0x7fffffffu) * L);
            const bool neg = (w[q] >> 31) != 0;
#pragma unroll
            for (int l = 0; l < SUB; l++) f[q][l] = neg ? Ar::add(T(1), s.v[l]) : Ar::sub(T(1), s.v[l]);
        }
#pragma unroll
    for (int q = 0; q < KMAX; q++)
        if (EXACT || q < I.k) slot[q] = __ldg(I.slotw + (size_t)q * I.mp + m);
    T r[SUB], km[SUB];
#pragma unroll
    for (int l = 0; l < SUB; l++) {
        if constexpr (LOGA) am[l] = exp2_fast(am[l]);
        km[l] = knorm;
#pragma unroll
        for (int q = 0; q < KMAX; q++)
            if (EXACT || q < I.k) km[l] = (kFold && q == 0) ? f[q][l] : Ar::mul(km[l], f[q][l]);
        T da;
        if constexpr (kFold) da = (km[l] * km[l]) * (knorm * knorm * T(kInvLn2));
        else da = Ar::mul(Ar::mul(am[l], km[l]), km[l]);
        if (l < cnt) A.dxdt[at + l * A.stride] = da;
        r[l] = kFold ? km[l] * (am[l] * (T(2) * knorm * knorm)) : Ar::mul(Ar::mul(km[l], knorm), am[l]);
    }
    const bool wide_k = KMAX > 10 && I.k > 10;  // the generic CalculateAll form (CpuSat.cpp:291-349)
#pragma unroll
    for (int q = 0; q < KMAX; q++) {
        if (EXACT || q < I.k) {
            LaneVec<T, SUB> c;
            const bool neg = (w[q] >> 31) != 0;
#pragma unroll
            for (int l = 0; l < SUB; l++) {
                T rr;
                if (!wide_k) {
                    T prod = T(1);
                    bool first = true;
#pragma unroll
                    for (int o = 0; o < KMAX; o++)
                        if (o != q && (EXACT || o < I.k)) {
                            prod = first ? f[o][l] : Ar::mul(prod, f[o][l]);
                            first = false;
                        }
                    rr = Ar::mul(r[l], prod);
                    if constexpr (!kFold) rr = rr + rr;
                } else {
                    T temp = kFold ? knorm * km[l] : km[l];
#pragma unroll
                    for (int o = 0; o < KMAX; o++)
                        if (EXACT || o < I.k) temp = Ar::mul(temp, o == q ? T(1) : f[o][l]);
                    rr = Ar::mul(Ar::mul(Ar::mul(T(2), temp), knorm), am[l]);
                }
                c.v[l] = neg ? -rr : rr;
            }
            st_lanes<T, SUB>(cs + (long long)slot[q] * L, c);
        }
    }
}

template <typename T, int SUB, int R>
__global__ void __launch_bounds__(256) row_var_kernel(RowArgs<T> A) {
    using Ar = Arith<T>;
    constexpr int L = SUB * R;
    const DevInstance& I = A.I;
    const int g = blockIdx.y;
    const long long it = (long long)blockIdx.x * 256 + threadIdx.x;
    const int v = (int)(it / R), lb = (int)(it % R) * SUB;
    if (v >= I.n) return;
    const T* p = A.cs + g * A.cs_stride + ((long long)__ldg(I.srow + (v >> 5)) * 32 + (v & 31)) * L + lb;
    const int deg = __ldg(I.deg + v);  // the slots behind it in the row are never written
    T sum[SUB];
#pragma unroll
    for (int l = 0; l < SUB; l++) sum[l] = T(0);
#pragma unroll 8
    for (int i = 0; i < deg; i++, p += 32 * L) {
        const LaneVec<T, SUB> c = ld_lanes<T, SUB>(p);
#pragma unroll
        for (int l = 0; l < SUB; l++) sum[l] = Ar::add(sum[l], c.v[l]);
    }
    const int cnt = A.ns - g * L - lb;
    T* d = A.dxdt + (A.s0 + (long long)g * L + lb) * A.stride + __ldg(I.perm + v);
#pragma unroll
    for (int l = 0; l < SUB; l++)
        if (l < cnt) d[l * A.stride] = sum[l];
}

}  // namespace asb
