// tri_kernels.cuh -- residual / SSP-RK3 stage kernels of straight-sided
// triangles (physics mode), Euler and Navier-Stokes, templated on the
// arithmetic type like the quad kernels (double: FP64; float: the
// mixed-precision form with the per-element reference state).
//
// A triangle holds nt = (P+1)(P+2)/2 solution points in the first nt of its
// (P+1)^2 state slots and 3 (P+1) flux points in edges 0..2 of its trace rows
// (the layout the quads use, so faces between triangles and quads need no
// special case).  With the operators of tri_setup.cpp:
//   R_n = -(1/J) [ sum_k Dr_nk F~_k + Ds_nk G~_k + sum_q Phi_nq dF_q ],
//   dF_q = s_f F_common . n - (sum_k L_qk F~_k, sum_k L_qk G~_k) . n^_f,
// s_f = |edge| / |reference edge| (2, 2 sqrt 2, 2), n^_f the reference edge's
// unit outward normal.  Navier-Stokes: the corrected gradient
//   dU/dr = sum_k Dr_nk U_k + sum_q Phi_nq n^x_q dU_q,
//   dU/ds = sum_k Ds_nk U_k + sum_q Phi_nq n^y_q dU_q,  dU_q = (U_nbr - U_own)/2,
// chain rule with the constant metrics, and the quads' viscous law and
// common viscous flux.  The kernels visit the triangles through an element
// list; phases as the quad kernels (loads and fluxes, faces, divergence +
// correction + stage, traces and ghost rows).
#pragma once

#include "ns_kernels.cuh"

// 128-thread CTAs: more of them sit in different phases, and the last wave is
// finer (shear layer per step, 256 -> 128 threads: 384 x 384 P3 FP32 754 -> 734 us
// with 64 instead of 80 registers, 173 x 141 P2 FP64 221 -> 210 us).
#ifndef ZJ_TRI_THREADS
#define ZJ_TRI_THREADS 128
#endif
#ifndef ZJ_TRI_MIN_BLOCKS
#define ZJ_TRI_MIN_BLOCKS 4       // FP64 stage kernel (128 registers)
#endif
#ifndef ZJ_TRI32_MIN_BLOCKS
#define ZJ_TRI32_MIN_BLOCKS 8     // precision-form stage kernel (64 registers)
#endif

namespace zj {
namespace {

template <typename T> struct TriMinBlocks { static constexpr int stage = ZJ_TRI_MIN_BLOCKS; };
template <> struct TriMinBlocks<float> { static constexpr int stage = ZJ_TRI32_MIN_BLOCKS; };

// Shared layout.  Field tiles are [element][point][var], so a point is one or
// two 16-byte loads that the element's threads share; the operators' rows sit
// by thread: (Dr, Ds) pairs of a point's row, rows of L and of Phi, padded so
// that the rows of neighbouring threads fall on distinct banks.
// With scalar tiles and unpaired rows the products took 5 to 6 shared loads for
// 8 FMAs; the stage launch of 42 000 P3 triangles issued 51.7 M warp
// instructions in FP32 and now 36.7 M.
template <int P, typename T>
struct TriShape {
    static constexpr int N1 = P + 1;
    static constexpr int NT = (P + 1) * (P + 2) / 2;   // solution points
    static constexpr int NSP = N1 * N1;                // state slots per element
    static constexpr int NFT = 3 * N1;                 // flux points
    static constexpr int TPE = NT > NFT ? NT : NFT;
    static constexpr int EB = (ZJ_TRI_THREADS / TPE / EbDiv<T>::value) > 0 ? (ZJ_TRI_THREADS / TPE / EbDiv<T>::value) : 1;
    static constexpr int THREADS = EB * TPE;
    static constexpr int ES = 4 * NT + (sizeof(T) == 8 ? 2 : 4);    // element stride of a field tile
    static constexpr int DS = 4 * NFT + (sizeof(T) == 8 ? 2 : 4);   // and of the flux-point tile
    static constexpr int RD = 2 * NT + ((2 * NT) % 4 == 0 ? 2 : 4); // row strides: (Dr, Ds)
    static constexpr int RL = NT | 1, RF = NFT | 1;                 // L, Phi
    static constexpr int LO = NT * RD, PHI = LO + NFT * RL;
    static constexpr int NOPS = PHI + NT * RF;
    // packed operators (Dr, Ds, L, Phi, each row-major) into the rows above
    static __device__ __forceinline__ void fill(T* s, const T* ops) {
        for (int t = threadIdx.x; t < NT * NT; t += THREADS) {
            const int n = t / NT, k = t - n * NT;
            s[n * RD + 2 * k] = ops[t];
            s[n * RD + 2 * k + 1] = ops[NT * NT + t];
        }
        for (int t = threadIdx.x; t < NFT * NT; t += THREADS) {
            const int q = t / NT, k = t - q * NT;
            s[LO + q * RL + k] = ops[2 * NT * NT + t];
            const int n = t / NFT, p = t - n * NFT;
            s[PHI + n * RF + p] = ops[2 * NT * NT + NFT * NT + t];
        }
    }
};

// reference-edge unit outward normals and lengths
__device__ __forceinline__ double tri_nref_x(int f) { return f == 1 ? 0.70710678118654752440 : (f == 2 ? -1.0 : 0.0); }
__device__ __forceinline__ double tri_nref_y(int f) { return f == 0 ? -1.0 : (f == 1 ? 0.70710678118654752440 : 0.0); }
__device__ __forceinline__ double tri_ref_len(int f) { return f == 1 ? 2.82842712474619009760 : 2.0; }

// sum_k w[k] (point k of a field tile).
template <int NT, typename T>
__device__ __forceinline__ V4<T> tri_dot(const T* fld, const T* w) {
    V4<T> acc = v4_zero<T>();
#pragma unroll
    for (int k = 0; k < NT; ++k) acc = v4_fma(weight<T>(w[k]), v4_load(fld + 4 * k), acc);
    return acc;
}

// (Dr_k, Ds_k) of a row.
__device__ __forceinline__ void load_pair(const float* p, float& a, float& b) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    a = t.x; b = t.y;
}
__device__ __forceinline__ void load_pair(const double* p, double& a, double& b) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    a = t.x; b = t.y;
}

// Corrected reference gradient at solution point n from the state tile su and
// the face jumps du, chain rule with ji.  The corrections of an edge share its
// reference normal, so they are summed per edge first.
template <int P, typename T>
__device__ __forceinline__ void tri_gradient(const T* su, const T* du, const T* ops, int n, const T* ji, T* Qx,
                                             T* Qy) {
    using S = TriShape<P, T>;
    constexpr int NT = S::NT, N1 = S::N1;
    V4<T> dr = v4_zero<T>(), ds = v4_zero<T>();
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        T a, b;
        load_pair(ops + n * S::RD + 2 * k, a, b);
        const V4<T> u = v4_load(su + 4 * k);
        dr = v4_fma(weight<T>(a), u, dr);
        ds = v4_fma(weight<T>(b), u, ds);
    }
    const T* ph = ops + S::PHI + n * S::RF;
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        const V4<T> c = tri_dot<N1>(du + f * N1 * 4, ph + f * N1);
        if (f > 0) dr = v4_fma(weight<T>(T(tri_nref_x(f))), c, dr);
        if (f < 2) ds = v4_fma(weight<T>(T(tri_nref_y(f))), c, ds);
    }
    v4_get(v4_fma(weight<T>(ji[2]), ds, v4_mul(weight<T>(ji[0]), dr)), Qx);
    v4_get(v4_fma(weight<T>(ji[3]), ds, v4_mul(weight<T>(ji[1]), dr)), Qy);
}

// Element of thread group el in this CTA, or -1.
__device__ __forceinline__ long long tri_element(const int32_t* elist, long long n_list, int EB, int el) {
    const long long g = (long long)blockIdx.x * EB + el;
    return (g < n_list) ? (long long)elist[g] : -1;
}

// ---------------------------------------------------------------- traces --
template <int P, typename T>
__global__ void __launch_bounds__(TriShape<P, T>::THREADS)
k_tri_traces(const StageArgsT<T> a, const int32_t* __restrict__ elist, long long n_list) {
    using S = TriShape<P, T>;
    constexpr int N1 = S::N1, NT = S::NT, NSP = S::NSP, NFT = S::NFT, TPE = S::TPE, EB = S::EB, ES = S::ES;
    __shared__ __align__(16) T sOps[S::NOPS];
    __shared__ __align__(16) T sU[EB * ES];
    const int tid = threadIdx.x;
    S::fill(sOps, a.ops);
    const int el = tid / TPE, k = tid - el * TPE;
    const long long e = (el < EB) ? tri_element(elist, n_list, EB, el) : -1;
    const bool valid = e >= 0;
    constexpr bool kRef = UsesRef<T>::value;
    T ue[4] = {T(0), T(0), T(0), T(0)};
    if (kRef && valid) load_state(a.U + e * NSP * 4, ue);
    if (valid && k < NT) {
        double u[4];
        T w[4];
        stage_state(a, e * NSP + k, u, w);
        if constexpr (kRef) state_minus_ref(u, ue, w);
        store4(sU + el * ES + 4 * k, w);
    }
    __syncthreads();
    if (valid && k < NFT) {
        const int edge = k / N1, fp = k - edge * N1;
        T t[4];
        v4_get(tri_dot<NT>(sU + el * ES, sOps + S::LO + k * S::RL), t);
        if constexpr (kRef) {
#pragma unroll
            for (int v = 0; v < 4; ++v) t[v] += ue[v];
        }
        gstore4(a.Tout + (e * 4 * N1 + k) * 4, t);
        const EdgeRec r = a.edges[e * 4 + edge];
        if (r.flags & kEdgeBoundary) {
            T n[3];
            load_normal(a.enrm + e * 4 + edge, n);
            store_ghost<N1>(a, r, n[0], n[1], fp, t);
        }
    }
}

// ------------------------------------------------------- gradient (NS) --
template <int P, typename T>
__global__ void __launch_bounds__(TriShape<P, T>::THREADS)
k_tri_grad(const StageArgsT<T> a, const int32_t* __restrict__ elist, long long n_list) {
    using S = TriShape<P, T>;
    constexpr int N1 = S::N1, NT = S::NT, NSP = S::NSP, NFT = S::NFT, TPE = S::TPE, EB = S::EB;
    constexpr int ES = S::ES, DS = S::DS;
    __shared__ __align__(16) T sOps[S::NOPS];
    __shared__ __align__(16) T sU[EB * ES];    // the state, then dU/dy
    __shared__ __align__(16) T sDU[EB * DS];
    __shared__ __align__(16) T sQ[EB * ES];    // dU/dx
    const int tid = threadIdx.x;
    S::fill(sOps, a.ops);
    pdl_launch_dependents();
    pdl_wait();   // the state and traces come from the previous launches
    const int el = tid / TPE, k = tid - el * TPE;
    const long long e = (el < EB) ? tri_element(elist, n_list, EB, el) : -1;
    const bool valid = e >= 0;
    const bool is_sp = valid && k < NT, is_fp = valid && k < NFT;
    const int edge = k / N1, fp = k - edge * N1;
    constexpr bool kRef = UsesRef<T>::value;
    const T* Tin = after_wait(a.Tin);
    T ji[4];
    if (is_sp) {
        const long long idx = e * NSP + k;
        double ud[4];
        T u[4];
        stage_state(a, idx, ud, u);
        if constexpr (kRef) {
            T ue[4];
            load_state(a.U + e * NSP * 4, ue);
            state_minus_ref(ud, ue, u);
        }
        load4_nc(a.Jinv + idx * 4, ji);
        store4(sU + el * ES + 4 * k, u);
    }
    EdgeRec r{-1, 0, kEdgeOrphan, 0};
    T Ua[4];   // average state of the flux point
    if (is_fp) {
        r = a.edges[e * 4 + edge];
        T qn[4];
        load4_nc(Tin + (e * 4 * N1 + k) * 4, Ua);
        T d[4] = {T(0), T(0), T(0), T(0)};
        if (!(r.flags & kEdgeOrphan)) {
            load4_nc(Tin + (neighbour_row(r, a.n_elem) * N1 + (N1 - 1 - fp)) * 4, qn);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                d[v] = T(0.5) * (qn[v] - Ua[v]);
                Ua[v] = T(0.5) * (Ua[v] + qn[v]);
            }
        }
        store4(sDU + el * DS + k * 4, d);
    }
    __syncthreads();
    T Qx[4], Qy[4];
    if (is_sp) {
        tri_gradient<P>(sU + el * ES, sDU + el * DS, sOps, k, ji, Qx, Qy);
        store4(sQ + el * ES + 4 * k, Qx);
    }
    __syncthreads();   // the state tile is dead
    if (is_sp) store4(sU + el * ES + 4 * k, Qy);
    __syncthreads();
    if (is_fp) {
        T t[8];
        v4_get(tri_dot<NT>(sQ + el * ES, sOps + S::LO + k * S::RL), t);
        v4_get(tri_dot<NT>(sU + el * ES, sOps + S::LO + k * S::RL), t + 4);
        T n[3], f[4];
        load_normal(a.enrm + e * 4 + edge, n);
        viscous_share(a, r, n[0], n[1], Ua, t, f);
        gstore4(a.FVout + (e * 4 * N1 + k) * 4, f);
    }
}

// ----------------------------------------------------------------- stage --
template <int P, int RIEM, bool VISC, typename T>
__global__ void __launch_bounds__(TriShape<P, T>::THREADS, TriMinBlocks<T>::stage)
k_tri_stage(const StageArgsT<T> a, const int32_t* __restrict__ elist, long long n_list) {
    using S = TriShape<P, T>;
    constexpr int N1 = S::N1, NT = S::NT, NSP = S::NSP, NFT = S::NFT, TPE = S::TPE, EB = S::EB;
    constexpr int ES = S::ES, DS = S::DS;
    __shared__ __align__(16) T sOps[S::NOPS];
    __shared__ __align__(16) T sF[EB * ES];
    __shared__ __align__(16) T sG[EB * ES];
    __shared__ __align__(16) T sD[EB * DS];    // face jumps of U (NS), then flux differences
    __shared__ __align__(16) T sU[EB * ES];    // stage state (NS), then the new state
    __shared__ double sRed[32];
    const int tid = threadIdx.x;
    S::fill(sOps, a.ops);
    pdl_launch_dependents();
    pdl_wait();   // the state and traces come from the previous launches
    const int el = tid / TPE, k = tid - el * TPE;
    const long long e = (el < EB) ? tri_element(elist, n_list, EB, el) : -1;
    const bool valid = e >= 0;
    const bool is_sp = valid && k < NT, is_fp = valid && k < NFT;
    const int edge = k / N1, fp = k - edge * N1;
    const T g = T(a.gamma);
    constexpr bool kRef = UsesRef<T>::value;
    const T* Tin = after_wait(a.Tin);
    const T* FV = after_wait(a.FV);

    // ---- A1: loads; the stage state (NS) and face jumps into shared memory;
    // the common flux of the flux points
    T ue[4] = {T(0), T(0), T(0), T(0)};
    if (kRef && valid) load_state(a.U + e * NSP * 4, ue);
    EdgeRec r{-1, 0, kEdgeOrphan, 0};
    T nr[3] = {T(0), T(0), T(0)}, qo[4], qn[4] = {T(0), T(0), T(0), T(0)};
    T fv[4] = {T(0), T(0), T(0), T(0)};   // common normal viscous flux: both sides' shares
    if (is_fp) {
        r = a.edges[e * 4 + edge];
        load_normal(a.enrm + e * 4 + edge, nr);
        load4_nc(Tin + (e * 4 * N1 + k) * 4, qo);
        if constexpr (VISC) load4_nc(FV + (e * 4 * N1 + k) * 4, fv);
    }
    T u[4], ji[4], Jd = T(1);
    if (is_sp) {
        const long long idx = e * NSP + k;
        double ud[4];
        stage_state(a, idx, ud, u);
        load4_nc(a.Jinv + idx * 4, ji);
        Jd = ldg_any(a.J + idx);
        if (a.stage >= 2) prefetch_l2(a.U0 + idx * 4);
        if constexpr (VISC) {
            T w[4];
            if constexpr (kRef) state_minus_ref(ud, ue, w);
            else {
#pragma unroll
                for (int v = 0; v < 4; ++v) w[v] = u[v];
            }
            store4(sU + el * ES + 4 * k, w);
        }
    }
    const bool face = is_fp && !(r.flags & kEdgeOrphan);
    if (face) {
        load4_nc(Tin + (neighbour_row(r, a.n_elem) * N1 + (N1 - 1 - fp)) * 4, qn);
        if (VISC && !(r.flags & kEdgeBoundary)) {
            T fn[4];
            load4_nc(FV + (((long long)r.nbr * 4 + r.nbr_edge) * N1 + (N1 - 1 - fp)) * 4, fn);
#pragma unroll
            for (int v = 0; v < 4; ++v) fv[v] += fn[v];
        }
    }
    if constexpr (VISC) {
        if (is_fp) {
            T d[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) d[v] = face ? T(0.5) * (qn[v] - qo[v]) : T(0);
            store4(sD + el * DS + k * 4, d);
        }
    }
    T Fd[4] = {T(0), T(0), T(0), T(0)};
    if (face) {
        const bool right = (r.flags & kEdgeRight) != 0;
        T UL[4], UR[4], Fc[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) { UL[v] = right ? qn[v] : qo[v]; UR[v] = right ? qo[v] : qn[v]; }
        riemann<RIEM>(UL, UR, nr[0], nr[1], g, Fc);
        if constexpr (kRef) {
            T Fe[4];
            ref_flux_n(ue, g, nr[0], nr[1], Fe);
#pragma unroll
            for (int v = 0; v < 4; ++v) Fc[v] -= Fe[v];
        }
        const T sf = nr[2] * T(1.0 / tri_ref_len(edge));
        const T ss = right ? -sf : sf;
#pragma unroll
        for (int v = 0; v < 4; ++v) Fd[v] = ss * (Fc[v] - fv[v]);
    }
    if constexpr (VISC) __syncthreads();

    // ---- A2: transformed fluxes
    if (is_sp) {
        T F[4], G[4];
        euler_flux(u, g, F, G);
        if constexpr (kRef) {
            T Fe[4], Ge[4];
            euler_flux(ue, g, Fe, Ge);
#pragma unroll
            for (int v = 0; v < 4; ++v) { F[v] -= Fe[v]; G[v] -= Ge[v]; }
        }
        if constexpr (VISC) {
            T Qx[4], Qy[4], Fv[4], Gv[4];
            tri_gradient<P>(sU + el * ES, sD + el * DS, sOps, k, ji, Qx, Qy);
            viscous_flux_f(u, rcp_any(u[0]), Qx, Qy, g, inv_reynolds(a), T(a.kfac), Fv, Gv);
#pragma unroll
            for (int v = 0; v < 4; ++v) { F[v] -= Fv[v]; G[v] -= Gv[v]; }
        }
        T ft[4], gt[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            ft[v] = Jd * (ji[0] * F[v] + ji[1] * G[v]);
            gt[v] = Jd * (ji[2] * F[v] + ji[3] * G[v]);
        }
        store4(sF + el * ES + 4 * k, ft);
        store4(sG + el * ES + 4 * k, gt);
    }
    __syncthreads();

    // ---- B: flux differences at the faces (NS: the jumps were consumed in A2)
    if (is_fp) {
        if (face) {
            const T* Lr = sOps + S::LO + k * S::RL;
            V4<T> acc = v4(Fd);
            acc = v4_fma(weight<T>(T(-tri_nref_x(edge))), tri_dot<NT>(sF + el * ES, Lr), acc);
            acc = v4_fma(weight<T>(T(-tri_nref_y(edge))), tri_dot<NT>(sG + el * ES, Lr), acc);
            v4_get(acc, Fd);
        }
        store4(sD + el * DS + k * 4, Fd);
    }
    __syncthreads();

    // ---- C: divergence, correction, 1/J, stage update
    double rsq = 0.0;
    if (is_sp) {
        const long long idx = e * NSP + k;
        double u0[4];
        if (a.stage >= 2) gload4(a.U0 + idx * 4, u0);
        V4<T> div = tri_dot<NFT>(sD + el * DS, sOps + S::PHI + k * S::RF);
#pragma unroll
        for (int m = 0; m < NT; ++m) {
            T x, y;
            load_pair(sOps + k * S::RD + 2 * m, x, y);
            div = v4_fma(weight<T>(x), v4_load(sF + el * ES + 4 * m), div);
            div = v4_fma(weight<T>(y), v4_load(sG + el * ES + 4 * m), div);
        }
        const T iJ = rcp_any(Jd);
        T res[4];
        v4_get(div, res);
#pragma unroll
        for (int v = 0; v < 4; ++v) res[v] = -res[v] * iJ;
        if (a.stage == 0) {
            store_residual(a, idx, res, rsq);
        } else {
            double us[4];
            gload4(a.U + idx * 4, us);
            double uo[4];
            rk_update(a.stage, *a.dt, us, u0, res, uo);
            gstore4(a.Uout + idx * 4, uo);
            T un[4];
            if constexpr (kRef) state_minus_ref(uo, ue, un);
            else {
#pragma unroll
                for (int v = 0; v < 4; ++v) un[v] = T(uo[v]);
            }
            store4(sU + el * ES + 4 * k, un);
            if (a.stage == 3) {
#pragma unroll
                for (int v = 0; v < 4; ++v) rsq += double(res[v]) * double(res[v]);
            }
        }
    }
    if (a.stage == 0 || a.stage == 3) {
        const double bs = block_sum(rsq, sRed);
        if (tid == 0) a.partials[blockIdx.x] = bs;
    }
    if (a.stage == 0) return;
    __syncthreads();

    // ---- D: traces of the new state and ghost rows
    if (is_fp) {
        T t[4];
        v4_get(tri_dot<NT>(sU + el * ES, sOps + S::LO + k * S::RL), t);
        if constexpr (kRef) {
#pragma unroll
            for (int v = 0; v < 4; ++v) t[v] += ue[v];
        }
        gstore4(a.Tout + (e * 4 * N1 + k) * 4, t);
        if (r.flags & kEdgeBoundary) store_ghost<N1>(a, r, nr[0], nr[1], fp, t);
    }
}

template <int P, typename T>
cudaError_t tri_traces_t(const StageArgsT<T>& a, const int32_t* elist, long long n, cudaStream_t s) {
    using S = TriShape<P, T>;
    const long long grid = (n + S::EB - 1) / S::EB;
    if (grid <= 0) return cudaSuccess;
    k_tri_traces<P, T><<<(unsigned)grid, S::THREADS, 0, s>>>(a, elist, n);
    return cudaGetLastError();
}

// Triangles ask for the quads' split, also where their own kernels would want more
// for the CTAs of their launch bounds (inviscid, per SM: FP64 P5 121 KB against 93,
// FP32 P4 104 against 86 and P5 128 against 72). Six inviscid steps of the shear
// layer, this split against one that fits the triangles (Roe): FP32 P5 275 and 368 us
// at 60 x 57, 4222 and 4045 at 320 x 317; FP32 P4 296 and 399, 3037 and 3029; FP64 P5
// 413 and 450, 7185 and 6868: what large meshes would gain the others lose five times over.
template <int P, typename T>
cudaError_t tri_grad_t(const StageArgsT<T>& a, const int32_t* elist, long long n, cudaStream_t s) {
    using S = TriShape<P, T>;
    const long long grid = (n + S::EB - 1) / S::EB;
    if (grid <= 0) return cudaSuccess;
    static bool set = false;
    if (!set) { set_carveout(k_tri_grad<P, T>, ns_carveout<P, T>()); set = true; }   // the quads' split
    return launch_programmatic(k_tri_grad<P, T>, (unsigned)grid, S::THREADS, s, a, elist, n);
}

template <int P, int RIEM, bool VISC, typename T>
cudaError_t tri_stage_t(const StageArgsT<T>& a, const int32_t* elist, long long n, cudaStream_t s) {
    using S = TriShape<P, T>;
    const long long grid = (n + S::EB - 1) / S::EB;
    if (grid <= 0) return cudaSuccess;
    static bool set = false;
    if (!set) {   // the quads' split
        set_carveout(k_tri_stage<P, RIEM, VISC, T>, VISC ? ns_carveout<P, T>() : phys_carveout<P, T>());
        set = true;
    }
    return launch_programmatic(k_tri_stage<P, RIEM, VISC, T>, (unsigned)grid, S::THREADS, s, a, elist, n);
}

template <int P, bool VISC, typename T>
cudaError_t tri_stage_r(int riemann, const StageArgsT<T>& a, const int32_t* elist, long long n, cudaStream_t s) {
    switch (riemann) {
        case ZJ_RIEMANN_RUSANOV: return tri_stage_t<P, ZJ_RIEMANN_RUSANOV, VISC>(a, elist, n, s);
        case ZJ_RIEMANN_ROE: return tri_stage_t<P, ZJ_RIEMANN_ROE, VISC>(a, elist, n, s);
        case ZJ_RIEMANN_HLLC: return tri_stage_t<P, ZJ_RIEMANN_HLLC, VISC>(a, elist, n, s);
        default: return cudaErrorInvalidValue;
    }
}

template <typename T>
cudaError_t tri_dispatch(int what, int P, int riemann, bool visc, const StageArgsT<T>& a, const int32_t* elist,
                         long long n, cudaStream_t s) {
#define ZJ_TRI_CASE(PP)                                                                        \
    case PP:                                                                                   \
        if (what == 0) return tri_traces_t<PP>(a, elist, n, s);                                \
        if (what == 1) return tri_grad_t<PP>(a, elist, n, s);                                  \
        return visc ? tri_stage_r<PP, true>(riemann, a, elist, n, s)                           \
                    : tri_stage_r<PP, false>(riemann, a, elist, n, s);
    switch (P) {
        ZJ_TRI_CASE(1)
        ZJ_TRI_CASE(2)
        ZJ_TRI_CASE(3)
        ZJ_TRI_CASE(4)
        ZJ_TRI_CASE(5)
        default: return cudaErrorInvalidValue;
    }
#undef ZJ_TRI_CASE
}

template <int P>
int tri_grid_t(long long n) { return (int)((n + TriShape<P, double>::EB - 1) / TriShape<P, double>::EB); }

}  // namespace
}  // namespace zj
