// Discrete adjoint of the RK45 (Cash-Karp) integration: gradients of the final
// potential with respect to the initial state and per-clause weights.
//
// Weighted CTDS (w = 1 is the reference ODE, AnalogSAT/cpu_sat/CpuSat.cpp:199-241):
//   ds_i = sum_m 2 w_m a_m c_mi K_mi K_m,   da_m = a_m K_m^2,
//   L    = V(x(T)) = sum_m w_m a_m(T) K_m(s(T))^2.
// adj_forward_kernel runs the adaptive controller to T (last step clamped to land on
// T), records the accepted step sizes and checkpoints the state before every accepted
// step and at T in global memory; adj_backward_kernel runs the adjoint recursion of that
// frozen step sequence backwards, recomputing each step's stage derivatives from its
// checkpoint:
//   rho_j   = h (c_j lam + sum_{i>j} b_ij sigma_i)        (dL/dk_j)
//   sigma_j = J(y_j)^T rho_j                              (dL/dy_j)
//   lam    <- lam + sum_j sigma_j ,   g_w += (df/dw)(y_j)^T rho_j.
// J^T u is the RHS's vector-Jacobian product -- the Hessian-vector product of V in the
// spin block -- computed with the same clause-phase / var-phase structure as the RHS:
// per clause in registers, per-literal contributions stored into the SELL slots,
// per-variable row sums.  With f_q = 1 - c_q s_q and g_q = c_q u_q, the sums over
// leave-two-out products that it needs are the epsilon parts of leave-one-out products of
// (f_q + epsilon g_q), formed from prefix and suffix products in O(K).
// Linear a in both FP32 and FP64 (over a short horizon a grows at most by e^T).
//
// Bound by instruction issue and the latency of the short phases between barriers, one CTA
// per trajectory.  So each stage is its own code (stage number and tableau row known at
// compile time), a variable phase also forms the spins (and cotangents) of the next stage
// -- two barriers per evaluation --, the checkpoints come from the forward pass instead of a
// second integration, and the shared memory of a trajectory is cut so that two or three
// CTAs share an SM (adjoint_threads).  1,024 trajectories of N = 200, M = 850, T = 5 (38 steps
// each), FP32: forward 1.28 ms, backward 6.45 ms with runtime stage loops and a second
// integration, 0.98 and 2.24 ms here; 153 of N = 151 in FP64 0.59 and 2.61 against 0.35 and
// 0.63 ms.
#pragma once

#include <type_traits>

#include "as_kernels.cuh"

namespace asb {

struct AdjointParams {
    const DevInstance* inst;
    const int* unit_inst;
    const long long* unit_state;   // element offset of each unit's public x0 / grad_x0
    const long long* unit_wofs;    // offset of each unit's clause weights / grad_w (public order)
    const void* x0;                // public layout, solver precision
    const double* weights;         // per clause, public order (null = all 1)
    double* hs;                    // [unit][max_steps] accepted step sizes
    int* nsteps;                   // [unit] steps to reach t_end (-1: more than max_steps, -2 underflow);
                                   // [num_units], [num_units + 1]: work counters of the two kernels
    void* ckpt;                    // checkpoint pool, solver precision, internal element order
    long long ckpt_cap;            // its values
    unsigned long long* ckpt_used; // values asked of it (more than ckpt_cap: the pass has to be repeated)
    long long* ckpt_off;           // [unit][max_steps + 1] pool offset of each checkpoint, the last at T
    double* loss;                  // [unit]
    double* grad_x0;               // public layout, FP64 as the caller's
    double* grad_w;                // per clause, public order
    int num_units, max_steps;
    double eps, t_end;
};

// A literal's sign applied to a value: -a for a negated literal.
__device__ __forceinline__ float flip_sign(float a, uint32_t w) {
    return __int_as_float(__float_as_int(a) ^ (int)(w & 0x80000000u));
}
__device__ __forceinline__ double flip_sign(double a, uint32_t w) {
    return __hiloint2double(__double2hiint(a) ^ (int)(w & 0x80000000u), __double2loint(a));
}

// Weighted RHS clause phase: contributions use w a, the returned da = a K^2.  The
// power-of-two scalings (knorm = 2^-k) are folded: P = f_0 .. f_{k-1}, K = knorm P.
template <typename T, int KMAX, bool EXACT>
__device__ __forceinline__ T wclause_fwd(const DevInstance& I, int m, const T* sy, T* cs, T a, T w, T knorm) {
    Lit<0> L[KMAX];
    T f[KMAX];
    T P = T(1);
#pragma unroll
    for (int q = 0; q < KMAX; q++) {
        if (EXACT || q < I.k) L[q].load(I, q * I.mp + m);
    }
#pragma unroll
    for (int q = 0; q < KMAX; q++) {
        if (EXACT || q < I.k) {
            f[q] = T(1) - flip_sign(sy[L[q].var()], L[q].w);
            P = q == 0 ? f[0] : P * f[q];
        }
    }
    const T r2 = ((T(2) * knorm * knorm) * P * w) * a;
#pragma unroll
    for (int q = 0; q < KMAX; q++) {
        if (EXACT || q < I.k) {
            T prod = T(1);
            bool first = true;
#pragma unroll
            for (int l = 0; l < KMAX; l++)
                if (l != q && (EXACT || l < I.k)) {
                    prod = first ? f[l] : prod * f[l];
                    first = false;
                }
            cs[L[q].slot()] = flip_sign(r2 * prod, L[q].w);
        }
    }
    const T K = knorm * P;
    return a * K * K;
}

// VJP clause phase for clause m at state (spins sy, weight a) with cotangent
// (spins su, weight ua): stores the spin-block contributions into cs, returns the
// a-block entry and the w-gradient in gw.
template <typename T, int KMAX, bool EXACT>
__device__ __forceinline__ T wclause_vjp(const DevInstance& I, int m, const T* sy, const T* su, T* cs, T a,
                                         T ua, T w, T knorm, T& gw) {
    Lit<0> L[KMAX];
    // f[q], g[q]; sP[q] + epsilon sD[q] = prod_{l >= q} (f_l + epsilon g_l)
    T f[KMAX], g[KMAX], sP[KMAX], sD[KMAX];
#pragma unroll
    for (int q = 0; q < KMAX; q++)
        if (EXACT || q < I.k) L[q].load(I, q * I.mp + m);
#pragma unroll
    for (int q = 0; q < KMAX; q++) {
        if (EXACT || q < I.k) {
            f[q] = T(1) - flip_sign(sy[L[q].var()], L[q].w);
            g[q] = flip_sign(su[L[q].var()], L[q].w);  // the sentinel's cotangent slot holds 0
        }
    }
    const int k = EXACT ? KMAX : I.k;
#pragma unroll
    for (int q = KMAX - 1; q >= 0; q--) {
        if (EXACT || q < k) {
            const bool last = EXACT ? q == KMAX - 1 : q == k - 1;
            const int q1 = q + 1 < KMAX ? q + 1 : q;
            sP[q] = last ? f[q] : f[q] * sP[q1];
            sD[q] = last ? g[q] : f[q] * sD[q1] + g[q] * sP[q1];
        }
    }
    const T kn2 = knorm * knorm;
    const T P = sP[0], S = sD[0];  // K = knorm P, sum_q u_q c_q K_q = knorm S
    const T pu = ua * P;
    const T a2 = T(-2) * kn2 * a;
    gw = -a2 * S * P;
    T p = T(1), d = T(0);  // prefix product and its epsilon part
#pragma unroll
    for (int r = 0; r < KMAX; r++) {
        if (EXACT || r < k) {
            const bool last = EXACT ? r == KMAX - 1 : r == k - 1;
            const int r1 = r + 1 < KMAX ? r + 1 : r;
            // K_r = knorm Pr; knorm Dr = sum_{q != r} u_q c_q prod_{l != q, r} f_l knorm
            T Pr, Dr;
            if (r == 0) {
                Pr = last ? T(1) : sP[r1];
                Dr = last ? T(0) : sD[r1];
            } else {
                Pr = last ? p : p * sP[r1];
                Dr = last ? d : d * sP[r1] + p * sD[r1];
            }
            cs[L[r].slot()] = flip_sign(a2 * (w * (Pr * S + P * Dr) + pu * Pr), L[r].w);
            d = r == 0 ? g[0] : d * f[r] + p * g[r];
            p = r == 0 ? f[0] : p * f[r];
        }
    }
    return kn2 * P * (T(2) * w * S + pu);
}

// Cash-Karp tableau rows used by the adjoint (b_ij for stage i, c_j).
__host__ __device__ constexpr double ck_b(int i, int j) {
    switch (i * 8 + j) {
        case 2 * 8 + 1: return ck::b21;
        case 3 * 8 + 1: return ck::b31;
        case 3 * 8 + 2: return ck::b32;
        case 4 * 8 + 1: return ck::b41;
        case 4 * 8 + 2: return ck::b42;
        case 4 * 8 + 3: return ck::b43;
        case 5 * 8 + 1: return ck::b51;
        case 5 * 8 + 2: return ck::b52;
        case 5 * 8 + 3: return ck::b53;
        case 5 * 8 + 4: return ck::b54;
        case 6 * 8 + 1: return ck::b61;
        case 6 * 8 + 2: return ck::b62;
        case 6 * 8 + 3: return ck::b63;
        case 6 * 8 + 4: return ck::b64;
        case 6 * 8 + 5: return ck::b65;
        default: return 0.0;
    }
}
__host__ __device__ constexpr double ck_c(int j) {
    switch (j) {
        case 1: return ck::c1;
        case 3: return ck::c3;
        case 4: return ck::c4;
        case 6: return ck::c6;
        default: return 0.0;
    }
}

// Shared-memory layout (E = n + m, Ep = E rounded to 4):
//   V[0..5]   X, K1..K5 (forward: xnew takes K2's place after stage 6; backward: the stage
//             inputs y_2..y_5 take K2..K5's places at the VJP of stage 6)
//   backward  V[6] lam, V[7..11] sigma_2..sigma_6, gw (m) grad w
//   w         clause weights (m; weighted calls only)
//   sy, su    spins / spin cotangents of the current stage (n+1 each, sentinel at n)
//   cs        contribution slots (nslots + 1)
__host__ __device__ inline size_t adjoint_smem_values(int n, int m, int nslots, bool backward, bool weighted) {
    const size_t Ep = (size_t)((n + m + 3) & ~3), mp = (size_t)((m + 3) & ~3), np = (size_t)((n + 1 + 3) & ~3);
    return (backward ? 12 * Ep + mp + 2 * np : 6 * Ep + np) + (weighted ? mp : 0) + (size_t)nslots + 1;
}
// The largest instance an adjoint call takes.  The kernels need less (adjoint_smem_values); the
// limit of fifteen vectors of E values is that of an earlier layout, kept so that the same
// calls are refused.
__host__ __device__ inline size_t adjoint_limit_values(int n, int m, int nslots) {
    const size_t Ep = (size_t)((n + m + 3) & ~3);
    return 15 * Ep + 2 * (size_t)((n + 1 + 3) & ~3) + (size_t)nslots + 1;
}

template <typename T>
struct AdjSmem {
    T *X, *w, *gw, *sy, *su, *cs;
    int Ep;
    __device__ __forceinline__ T* V(int i) const { return X + (size_t)i * Ep; }
    __device__ void init(unsigned char* raw, int n, int m, bool backward, bool weighted) {
        const int mp = (m + 3) & ~3, np = (n + 1 + 3) & ~3;
        Ep = (n + m + 3) & ~3;
        X = reinterpret_cast<T*>(raw);
        T* b = X + (size_t)(backward ? 12 : 6) * Ep;
        gw = b;
        if (backward) b += mp;
        w = weighted ? b : nullptr;
        if (weighted) b += mp;
        sy = b;
        b += np;
        su = b;
        if (backward) b += np;
        cs = b;
    }
    template <int S> __device__ __forceinline__ T input(int e, T h) const {  // y_S of element e
        return stage_in<S, T>(X[e], S > 1 ? V(1)[e] : T(0), S > 2 ? V(2)[e] : T(0), S > 3 ? V(3)[e] : T(0),
                              S > 4 ? V(4)[e] : T(0), S > 5 ? V(5)[e] : T(0), h);
    }
    // rho_J of element e from lam and the stored sigmas
    template <int J> __device__ __forceinline__ T rho(int e, T h) const {
        T acc = ck_c(J) != 0.0 ? T(ck_c(J)) * V(6)[e] : T(0);
#pragma unroll
        for (int i = J + 1; i <= 6; i++) acc += T(ck_b(i, J)) * V(5 + i)[e];  // sigma_i at V(5 + i)
        return h * acc;
    }
    __device__ __forceinline__ T weight(int m) const { return w ? w[m] : T(1); }
};

// One weighted RHS evaluation at stage S: clause phase over spins sy (formed before), barrier,
// sums.  on_clause(e, d) and on_var(v, d) take the derivatives; on_var runs after the
// barrier, so it may write the next stage's spins.  The caller puts a barrier between
// on_var and the next clause phase.
template <typename T, int KMAX, bool EXACT, int S, typename FC, typename FV>
__device__ __forceinline__ void adj_rhs(const DevInstance& I, const AdjSmem<T>& A, T h, T knorm, FC&& on_clause,
                                        FV&& on_var) {
    const int tid = threadIdx.x, nt = blockDim.x, n = I.n;
    for (int m = tid; m < I.m; m += nt) {
        const T a = A.template input<S>(n + m, h);
        on_clause(n + m, wclause_fwd<T, KMAX, EXACT>(I, m, A.sy, A.cs, a, A.weight(m), knorm));
    }
    __syncthreads();
    for (int v = tid; v < n; v += nt) on_var(v, var_phase<T>(I, v, A.cs));
}
// Stage S < 6 of a step: K_S stored, the spins of stage S + 1 formed.
template <typename T, int KMAX, bool EXACT, int S>
__device__ __forceinline__ void adj_stage(const DevInstance& I, const AdjSmem<T>& A, T h_in, T h_next, T knorm) {
    T* const KS = A.V(S);
    adj_rhs<T, KMAX, EXACT, S>(I, A, h_in, knorm, [&](int e, T d) { KS[e] = d; },
                               [&](int v, T d) {
                                   KS[v] = d;
                                   A.sy[v] = A.template input<S + 1>(v, h_next);
                               });
    __syncthreads();
}

// Loads a public-layout vector (permuted to the internal order) into dst.
template <typename T>
__device__ __forceinline__ void load_public(const DevInstance& I, const T* src, T* dst) {
    for (int i = threadIdx.x; i < I.n; i += blockDim.x) dst[__ldg(I.iperm + i)] = src[i];
    for (int j = threadIdx.x; j < I.m; j += blockDim.x) dst[I.n + __ldg(I.icperm + j)] = src[I.n + j];
}

template <typename T>
__device__ __forceinline__ void store_public(const DevInstance& I, const T* src, double* dst) {
    for (int i = threadIdx.x; i < I.n; i += blockDim.x) dst[i] = (double)src[__ldg(I.iperm + i)];
    for (int j = threadIdx.x; j < I.m; j += blockDim.x) dst[I.n + j] = (double)src[I.n + __ldg(I.icperm + j)];
}

template <typename T>
__device__ __forceinline__ void load_weights(const DevInstance& I, const AdjointParams& P, int u, T* w) {
    if (w)
        for (int j = threadIdx.x; j < I.m; j += blockDim.x)
            w[__ldg(I.icperm + j)] = (T)P.weights[P.unit_wofs[u] + j];
}

// Block max of the error ratios (never negative), post-processed by one thread; two
// barriers.  FP32: an integer redux of the bit patterns, as in the lean solver.
template <typename F>
__device__ __forceinline__ double adj_max_then(float em, double* red, F&& fn) {
    uint32_t* const red_u = reinterpret_cast<uint32_t*>(red);
    const uint32_t v = __reduce_max_sync(0xffffffffu, __float_as_uint(em));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red_u[warp] = v;
    __syncthreads();
    if (warp == 0) {
        const uint32_t x = __reduce_max_sync(0xffffffffu, lane < (int)(blockDim.x >> 5) ? red_u[lane] : 0u);
        if (lane == 0) red[33] = fn((double)__uint_as_float(x));
    }
    __syncthreads();
    return red[33];
}
template <typename F>
__device__ __forceinline__ double adj_max_then(double em, double* red, F&& fn) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) em = fmax(em, __shfl_xor_sync(0xffffffffu, em, o));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red[warp] = em;
    __syncthreads();
    if (warp == 0) {
        double x = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
        if (lane == 0) red[33] = fn(x);
    }
    __syncthreads();
    return red[33];
}

// Adaptive forward pass to t_end recording the accepted step sizes and the checkpoints.
template <typename T, int KMAX, bool EXACT>
__global__ void __launch_bounds__(1024, 1) adj_forward_kernel(AdjointParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red_d[36];
    __shared__ int s_unit;
    __shared__ long long s_off;
    const int tid = threadIdx.x, nt = blockDim.x;
    while (true) {
        if (tid == 0) s_unit = atomicAdd(P.nsteps + P.num_units, 1);
        __syncthreads();
        const int u = s_unit;
        if (u >= P.num_units) break;
        const DevInstance I = P.inst[P.unit_inst[u]];
        const int n = I.n, E = n + I.m;
        AdjSmem<T> A;
        A.init(smem_raw, n, I.m, false, P.weights != nullptr);
        const T knorm = (T)ldexp(1.0, -I.k);
        load_public<T>(I, reinterpret_cast<const T*>(P.x0) + P.unit_state[u], A.X);
        load_weights<T>(I, P, u, A.w);
        for (int j = tid; j <= I.nslots; j += nt) A.cs[j] = T(0);
        if (tid == 0) A.sy[n] = T(-1);
        __syncthreads();
        for (int v = tid; v < n; v += nt) A.sy[v] = A.X[v];
        __syncthreads();
        double t = 0.0, hnext = 1e-9;
        int steps = 0, status = 0;
        double* hs = P.hs + (long long)u * P.max_steps;
        long long* off = P.ckpt_off + (long long)u * (P.max_steps + 1ll);
        // room for one checkpoint in the pool (one thread); -1 when it is full
        auto reserve = [&](int s) {
            const long long o = (long long)atomicAdd(P.ckpt_used, (unsigned long long)E);
            off[s] = s_off = o + E <= P.ckpt_cap ? o : -1;
        };
        while (t < P.t_end) {
            if (steps >= P.max_steps) { status = -1; break; }
            if (t + hnext > P.t_end) hnext = P.t_end - t;
            const double h0 = hnext;
            double h = hnext;
            adj_stage<T, KMAX, EXACT, 1>(I, A, T(0), (T)h, knorm);
            bool underflow = false;
            while (true) {
                const T hT = (T)h, h0T = (T)h0;
                adj_stage<T, KMAX, EXACT, 2>(I, A, hT, hT, knorm);
                adj_stage<T, KMAX, EXACT, 3>(I, A, hT, hT, knorm);
                adj_stage<T, KMAX, EXACT, 4>(I, A, hT, hT, knorm);
                adj_stage<T, KMAX, EXACT, 5>(I, A, hT, hT, knorm);
                T em = T(0);
                auto finish = [&](int e, T k6) {  // error ratio and the candidate state, in K2's place
                    const T x = A.X[e], k1 = A.V(1)[e], k3 = A.V(3)[e], k4 = A.V(4)[e], k5 = A.V(5)[e];
                    em = fmax(em, rk_err_ratio(x, k1, k3, k4, k5, k6, hT, h0T, false));
                    A.V(2)[e] = rk_new<T>(x, k1, k3, k4, k6, hT);
                };
                adj_rhs<T, KMAX, EXACT, 6>(I, A, hT, knorm, finish, finish);
                const double ermax = adj_max_then(em, red_d, [&](double emax) {
                    const double e = emax / P.eps;
                    double hn;
                    if (e <= 1.0)
                        hn = e > ck::ERRCON ? ck::SAFETY * h * pow(e, ck::PGROW) : 5.0 * h;
                    else
                        hn = fmax(ck::SAFETY * h * pow(e, ck::PSHRNK), ck::HFACTOR * h);
                    red_d[34] = hn;
                    if (e <= 1.0) {
                        hs[steps] = h;
                        reserve(steps);
                    }
                    return e;
                });
                const double hn = red_d[34];
                if (ermax <= 1.0) { hnext = hn; break; }
                h = hn;
                if (t + h == t) { underflow = true; break; }
                // the retry's stage-2 spins
                for (int v = tid; v < n; v += nt) A.sy[v] = A.template input<2>(v, (T)h);
                __syncthreads();
            }
            if (underflow) { status = -2; break; }
            steps++;
            t += h;
            T* ck = s_off >= 0 ? reinterpret_cast<T*>(P.ckpt) + s_off : nullptr;
            for (int e = tid; e < E; e += nt) {
                const T xn = A.V(2)[e];
                if (ck) ck[e] = A.X[e];
                A.X[e] = xn;
                if (e < n) A.sy[e] = xn;
            }
            __syncthreads();
        }
        if (tid == 0) {
            reserve(status ? 0 : steps);
            P.nsteps[u] = status ? status : steps;
        }
        __syncthreads();
        if (s_off >= 0) {
            T* ck = reinterpret_cast<T*>(P.ckpt) + s_off;
            for (int e = tid; e < E; e += nt) ck[e] = A.X[e];
        }
        __syncthreads();
    }
}

// The adjoint recursion backwards over the recorded steps.
template <typename T, int KMAX, bool EXACT>
__global__ void __launch_bounds__(1024, 1) adj_backward_kernel(AdjointParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red_d[36];
    __shared__ int s_unit;
    const int tid = threadIdx.x, nt = blockDim.x;
    while (true) {
        if (tid == 0) s_unit = atomicAdd(P.nsteps + P.num_units + 1, 1);
        __syncthreads();
        const int u = s_unit;
        if (u >= P.num_units) break;
        const int ns = P.nsteps[u];
        const DevInstance I = P.inst[P.unit_inst[u]];
        const int n = I.n, E = n + I.m;
        AdjSmem<T> A;
        A.init(smem_raw, n, I.m, true, P.weights != nullptr);
        const T knorm = (T)ldexp(1.0, -I.k);
        const double* hs = P.hs + (long long)u * P.max_steps;
        const long long* off = P.ckpt_off + (long long)u * (P.max_steps + 1ll);
        const T* pool = reinterpret_cast<const T*>(P.ckpt);
        const T* xT = pool + off[ns];
        load_weights<T>(I, P, u, A.w);
        for (int e = tid; e < E; e += nt) {
            const T x = xT[e];
            A.X[e] = x;
            if (e < n) A.sy[e] = x;
        }
        for (int j = tid; j <= I.nslots; j += nt) A.cs[j] = T(0);
        if (tid == 0) { A.sy[n] = T(-1); A.su[n] = T(0); }
        __syncthreads();
        // dL/dx(T) = (-ds/dt(x_T), w K^2), dL/dw = a K^2, L = sum w a K^2; the state and the
        // spins of the last step behind it
        double lsum = 0.0;
        const T* ck = ns > 0 ? pool + off[ns - 1] : xT;
        adj_rhs<T, KMAX, EXACT, 1>(
            I, A, T(0), knorm,
            [&](int e, T d) {
                const T a = A.X[e], K2 = a != T(0) ? d / a : T(0), w = A.weight(e - n);
                A.V(6)[e] = w * K2;
                A.gw[e - n] = a * K2;
                lsum += (double)(w * a * K2);
                A.X[e] = ck[e];
            },
            [&](int v, T d) {
                A.V(6)[v] = -d;
                A.sy[v] = A.X[v] = ck[v];
            });
        // loss = sum of the per-thread terms (warp shuffles, one slot per warp)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if ((tid & 31) == 0) red_d[tid >> 5] = lsum;
        __syncthreads();
        if (tid == 0) {
            double sacc = 0.0;
            for (int w = 0; w < (nt >> 5); w++) sacc += red_d[w];
            P.loss[u] = sacc;
        }
        // backward over the steps
        for (int s = ns - 1; s >= 0; s--) {
            const T h = (T)hs[s];
            ck = s > 0 ? pool + off[s - 1] : nullptr;
            adj_stage<T, KMAX, EXACT, 1>(I, A, h, h, knorm);
            adj_stage<T, KMAX, EXACT, 2>(I, A, h, h, knorm);
            adj_stage<T, KMAX, EXACT, 3>(I, A, h, h, knorm);
            adj_stage<T, KMAX, EXACT, 4>(I, A, h, h, knorm);
            // the stage inputs of an element, all from X, K1..K5: y_6 returned, y_2..y_5 into
            // K2..K5's places
            auto inputs = [&](int e, T k5) {
                const T x = A.X[e], k1 = A.V(1)[e], k2 = A.V(2)[e], k3 = A.V(3)[e], k4 = A.V(4)[e];
                A.V(2)[e] = stage_in<2, T>(x, k1, k2, k3, k4, k5, h);
                A.V(3)[e] = stage_in<3, T>(x, k1, k2, k3, k4, k5, h);
                A.V(4)[e] = stage_in<4, T>(x, k1, k2, k3, k4, k5, h);
                A.V(5)[e] = stage_in<5, T>(x, k1, k2, k3, k4, k5, h);
                return stage_in<6, T>(x, k1, k2, k3, k4, k5, h);
            };
            adj_rhs<T, KMAX, EXACT, 5>(I, A, h, knorm, [&](int e, T d) { A.V(5)[e] = d; },
                                       [&](int v, T d) {
                                           A.sy[v] = inputs(v, d);
                                           A.su[v] = A.template rho<6>(v, h);
                                       });
            __syncthreads();
            auto vjp = [&](auto stage) {
                constexpr int J = decltype(stage)::value;
                // sigma_J of element e: kept for the stages before it, or after stage 1 the sum
                // of all goes into lam (and the state of the step before takes X's place)
                auto keep = [&](int e, T sg) {
                    if constexpr (J >= 2) {
                        A.V(5 + J)[e] = sg;
                    } else {
                        T sum = A.V(11)[e];
#pragma unroll
                        for (int i = 5; i >= 2; i--) sum += A.V(5 + i)[e];
                        A.V(6)[e] += sum + sg;
                    }
                };
                for (int m = tid; m < I.m; m += nt) {
                    const int e = n + m;
                    T xp = T(0);
                    if constexpr (J == 1) if (ck) xp = ck[e];
                    const T a = J == 6 ? inputs(e, A.V(5)[e]) : A.V(J == 6 ? 5 : (J == 1 ? 0 : J))[e];
                    const T ua = A.template rho<J>(e, h);
                    T gw;
                    const T sg =
                        wclause_vjp<T, KMAX, EXACT>(I, m, A.sy, A.su, A.cs, a, ua, A.weight(m), knorm, gw);
                    A.gw[m] += gw;
                    keep(e, sg);
                    if constexpr (J == 1) if (ck) A.X[e] = xp;
                }
                __syncthreads();
                for (int v = tid; v < n; v += nt) {
                    T xp = T(0);
                    if constexpr (J == 1) if (ck) xp = ck[v];
                    keep(v, var_phase<T>(I, v, A.cs));
                    if constexpr (J >= 2) {
                        A.sy[v] = A.V(J == 2 ? 0 : J - 1)[v];
                        A.su[v] = A.template rho<J - 1>(v, h);
                    } else if (ck) {
                        A.sy[v] = A.X[v] = xp;
                    }
                }
                __syncthreads();
            };
            vjp(std::integral_constant<int, 6>{});
            vjp(std::integral_constant<int, 5>{});
            vjp(std::integral_constant<int, 4>{});
            vjp(std::integral_constant<int, 3>{});
            vjp(std::integral_constant<int, 2>{});
            vjp(std::integral_constant<int, 1>{});
        }
        __syncthreads();
        store_public<T>(I, A.V(6), P.grad_x0 + P.unit_state[u]);
        for (int j = tid; j < I.m; j += nt)
            P.grad_w[P.unit_wofs[u] + j] = (double)A.gw[__ldg(I.icperm + j)];
        __syncthreads();
    }
}

}  // namespace asb
