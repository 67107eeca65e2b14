// ns_kernels.cuh -- Navier-Stokes residual and SSP-RK3 stages (physics mode,
// viscous on), templated on the arithmetic type T: double in ns_fp64.cu (the
// reference-parity path), float in ns_fp32.cu (the mixed-precision form; the
// state, the RK accumulation and the norm partials stay FP64).  Two launches
// per residual:
//
//  k_ns_grad_lines (float, double; k_ns_grad for dual numbers)
//              corrected gradient Q = grad U at the solution points, its
//              traces at the flux points and, from them, this element's share
//              of the faces' common viscous flux (written for both sides);
//  k_ns_stage  recomputes Q at the solution points, total flux F - F_v, the
//              common flux = Riemann(U_L, U_R) - (the two shares), FR
//              correction, stage update and traces of the new state.
//
// The common viscous flux F_v(avg U, (Q_L + Q_R)/2).n is linear in the
// gradient, so it is the sum of F_v(avg U, Q_L/2).n and F_v(avg U, Q_R/2).n.
// Each side evaluates its share where it has the gradient trace in registers
// and writes 4 values a flux point instead of the 8 of (dU/dx, dU/dy); the
// stage kernel adds the own and the neighbour's share (the same sum on both
// sides), with no viscous evaluation and no gradient data at its faces.
// Against exchanging the gradients (256 x 256, P3, serialised launches): stage
// 107 -> 86 us FP64 and 57 -> 54 us FP32, gradient 39 -> 46 and 25 -> 31 us;
// per step -10.5 % FP64, -4 % FP32 (P5 FP32: -2.5 %).
//
// Gradient: U^C = U^D + (U_c - U^D) g at the edges with the common solution
// U_c = (U_L + U_R)/2 (the ghost state on boundaries), the same VCJH
// correction functions as the flux, chain rule with the pointwise metrics:
//   dU/dxi  = D_xi U  + g_R'(xi) dU_1 + g_L'(xi) dU_3
//   dU/deta = D_eta U + g_L'(eta) dU_0 + g_R'(eta) dU_2,   dU_e = U_c - U_own
//   Q_x = xi_x dU/dxi + eta_x dU/deta,  Q_y = xi_y dU/dxi + eta_y dU/deta.
// Viscous flux: the reference's computeViscousFluxSPKernel law
// (kernels.cu:742-786); common viscous flux: average state and average
// gradients (BR2Scheme::commonFlux, navierstokes.hpp:177-204); boundaries
// copy the interior gradient (BoundaryCondition::ghostGradient) and walls
// impose their Neumann data on the common flux (wall_viscous_closure).
#pragma once

#include <cuda_runtime.h>

#include "zj_device.cuh"
#include "zj_kernels.h"
#include "zj_math.h"
#include "zj_physics.cuh"
#include "phys_kernels.cuh"

// Resident CTAs per SM the launch bounds ask for, counted in CTAs of 128
// threads (other CTA sizes scale them).
#ifndef ZJ_NS_MIN_BLOCKS
#define ZJ_NS_MIN_BLOCKS 4        // FP64 stage kernel (128 registers)
#endif
#ifndef ZJ_NS32_MIN_BLOCKS
#define ZJ_NS32_MIN_BLOCKS 8      // mixed-precision stage kernel (64 registers)
#endif
// Threads per CTA of the gradient kernel by lines (rounded down to whole
// elements): 64 spread a coarse mesh over more SMs and interleave more phases;
// against 128 per step 20 x 20 P3 FP32 -1.4 %, 64 x 64 and 256 x 256 FP64
// -0.6 and -0.8 %, P5 FP32 -0.5 %; 32 cost P5 4 %.
#ifndef ZJ_LINE_THREADS
#define ZJ_LINE_THREADS 64
#endif
#ifndef ZJ_NSL_MIN_BLOCKS
#define ZJ_NSL_MIN_BLOCKS 4       // FP64 gradient kernel by lines (128 registers; 24 B of spills at P5)
#endif
#ifndef ZJ_NSL32_MIN_BLOCKS
#define ZJ_NSL32_MIN_BLOCKS 8     // mixed-precision gradient kernel by lines (64 registers; 4 B of spills at P3)
#endif
#ifndef ZJ_NSL32_MIN_BLOCKS_HI
#define ZJ_NSL32_MIN_BLOCKS_HI 6  // the same from P4 up (80 registers; 28 B of spills at P5)
#endif

namespace zj {
namespace {

using namespace dev;
using namespace phys;

template <typename T, int P> struct NSMinBlocks;
constexpr int per_cta(int blocks128) { return blocks128 * 128 / kCtaThreads > 0 ? blocks128 * 128 / kCtaThreads : 1; }
template <int P> struct NSMinBlocks<double, P> {
    static constexpr int stage = per_cta(ZJ_NS_MIN_BLOCKS);
};
template <int P> struct NSMinBlocks<float, P> {
    static constexpr int stage = per_cta(ZJ_NS32_MIN_BLOCKS);
};
template <int P> struct NSMinBlocks<Dual, P> { static constexpr int stage = 1; };

// Corrected gradient at solution point (i, j) of one element: su is the
// element's state tile, du its face jumps U_c - U_own in the flux-point tile.
template <int P, typename T>
__device__ __forceinline__ void corrected_gradient(const T* su, const T* du, const Weight<T>* ops, int i,
                                                   int j, const T* ji, T* Qx, T* Qy) {
    using Op = OpTable<P + 1, T>;
    constexpr int N1 = P + 1, RP = Tiles<P, T>::RP;
    Weight<T> w[N1];
    load_weights<N1>(ops + i * N1, w);
    V4<T> dxi = line_dot<N1>(w, su + j * RP, 4, v4_zero<T>());
    dxi = v4_fma(ops[Op::GR + i], v4_load(du + face_slot<P, T>(1, 1, j)), dxi);
    dxi = v4_fma(ops[Op::GL + i], v4_load(du + face_slot<P, T>(1, 0, j)), dxi);
    load_weights<N1>(ops + j * N1, w);
    V4<T> deta = line_dot<N1>(w, su + 4 * i, RP, v4_zero<T>());
    deta = v4_fma(ops[Op::GL + j], v4_load(du + face_slot<P, T>(0, 0, i)), deta);
    deta = v4_fma(ops[Op::GR + j], v4_load(du + face_slot<P, T>(0, 1, i)), deta);
    v4_get(v4_fma(weight<T>(ji[2]), deta, v4_mul(weight<T>(ji[0]), dxi)), Qx);
    v4_get(v4_fma(weight<T>(ji[3]), deta, v4_mul(weight<T>(ji[1]), dxi)), Qy);
}

// A load of the stage kernel: in its place in FP32, the compiler's to place
// in FP64 and for dual numbers (see the load phase of k_ns_stage).
template <typename T>
__device__ __forceinline__ void load4_x(const T* p, T* v) {
    if constexpr (sizeof(T) == 4) load4_now(p, v);
    else load4_nc(p, v);
}

// Loads of a flux-point thread: edge record, normal, own trace; then the
// neighbour's coinciding trace point (interior) or the ghost row written with
// the trace (boundary).  Tin: the stage's traces, behind the wait.
template <typename T>
struct FacePoint {
    EdgeRec r;
    T nx, ny, len;
    T qo[4], qn[4];
};

template <int N1, typename T>
__device__ __forceinline__ void load_own_face(const StageArgsT<T>& a, const T* Tin, long long e, int edge, int fp,
                                              FacePoint<T>& f) {
    f.r = a.edges[e * 4 + edge];
    T n[3];
    load_normal(normal_rec<N1>(a, e, edge, fp), n);
    f.nx = n[0]; f.ny = n[1]; f.len = n[2];
    load4_x(Tin + (e * 4 * N1 + edge * N1 + fp) * 4, f.qo);
}

template <int N1, typename T>
__device__ __forceinline__ void load_neighbour_face(const StageArgsT<T>& a, const T* Tin, int fp, FacePoint<T>& f) {
    f.qn[0] = f.qo[0]; f.qn[1] = f.qo[1]; f.qn[2] = f.qo[2]; f.qn[3] = f.qo[3];
    if (!(f.r.flags & kEdgeOrphan)) load4_x(Tin + (neighbour_row(f.r, a.n_elem) * N1 + (N1 - 1 - fp)) * 4, f.qn);
}

// This element's share of the common normal viscous flux of a flux point: Ua
// the average state, t the own gradient trace, n the face normal.  Half of the
// flux where a neighbour adds the other half, all of it on a boundary (the
// ghost gradient is the interior one), with the walls' closure.
template <typename T>
__device__ __forceinline__ void viscous_share(const StageArgsT<T>& a, const EdgeRec& r, T nx, T ny,
                                              const T* Ua, const T* t, T* f) {
    T Fv[4], Gv[4];
    viscous_flux_f(Ua, rcp_any(Ua[0]), t, t + 4, T(a.gamma), inv_reynolds(a), T(a.kfac), Fv, Gv);
    const T w = has_neighbour_gradient(r) ? T(0.5) : T(1);
#pragma unroll
    for (int v = 0; v < 4; ++v) f[v] = w * (Fv[v] * nx + Gv[v] * ny);
    boundary_viscous_closure(r, a.bc, nx, ny, f);
}

// Gradient of the dual-number instantiation, a thread per point.
template <int P, typename T>
__global__ void __launch_bounds__(Shape<P, EbDiv<T>::value>::THREADS)
k_ns_grad(const StageArgsT<T> a) {
    using S = Shape<P, EbDiv<T>::value>;
    constexpr int N1 = S::N1, NSP = S::NSP, NFT = S::NFT, TPE = S::TPE, EB = S::EB;
    using Op = OpTable<P + 1, T>;
    constexpr int RP = Tiles<P, T>::RP, FP = Tiles<P, T>::FP, DP = Tiles<P, T>::DP;
    __shared__ __align__(16) Weight<T> sOps[Op::N];
    __shared__ __align__(16) T sU[EB * FP];
    __shared__ __align__(16) T sDU[EB * DP];
    __shared__ __align__(16) T sQx[EB * FP];
    __shared__ __align__(16) T sQy[EB * FP];

    const int tid = threadIdx.x;
    Op::fill(sOps, a.ops);
    pdl_launch_dependents();
    pdl_wait();   // the state and traces come from the previous stage
    const int el = tid / TPE, k = tid - el * TPE;
    bool valid;
    const long long e = block_element(a, EB, el, valid);
    const bool is_sp = valid && k < NSP, is_fp = valid && k < NFT;
    const FaceLane fl = lane_face<N1>(k);
    const int edge = fl.edge, fp = fl.fp, kf = edge * N1 + fp;
    int i, j;
    lane_point<N1>(k, i, j);

    T ji[4];
    if (is_sp) {
        const long long idx = e * NSP + j * N1 + i;
        T u[4];
        double ud[4];
        stage_state(a, idx, ud, u);
        load4_nc(a.Jinv + idx * 4, ji);
        store4(sU + el * FP + j * RP + 4 * i, u);
    }
    FacePoint<T> f;
    if (is_fp) {
        const T* Tin = after_wait(a.Tin);
        load_own_face<N1>(a, Tin, e, edge, fp, f);
        load_neighbour_face<N1>(a, Tin, fp, f);
        T d[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) d[v] = (f.r.flags & kEdgeOrphan) ? T(0) : T(0.5) * (f.qn[v] - f.qo[v]);
        store4(sDU + el * DP + face_slot<P, T>(fl.dir, fl.side, fl.line), d);
    }
    __syncthreads();
    if (is_sp) {
        T Qx[4], Qy[4];
        corrected_gradient<P>(sU + el * FP, sDU + el * DP, sOps, i, j, ji, Qx, Qy);
        store4(sQx + el * FP + j * RP + 4 * i, Qx);
        store4(sQy + el * FP + j * RP + 4 * i, Qy);
    }
    __syncthreads();
    if (is_fp) {
        T t[8];
        state_trace<P>(sQx + el * FP, sOps, fl, t);
        state_trace<P>(sQy + el * FP, sOps, fl, t + 4);
        T Ua[4], fv[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) Ua[v] = T(0.5) * (f.qo[v] + f.qn[v]);
        viscous_share(a, f.r, f.nx, f.ny, Ua, t, fv);
        gstore4(a.FVout + (e * NFT + kf) * 4, fv);
    }
}

// ---- gradient by lines (float and double)
//
// 2 N1 threads per element: one per row j (an xi-line of solution points
// (0..N1-1, j)) and one per column i (an eta-line (i, 0..N1-1)).  The CTA
// first stages its elements' states into shared memory with 16-byte cp.async
// copies (each 16-byte piece fetched once), while every line thread loads the
// traces at its line's two end points (its own and the neighbour's).  A line
// thread then takes the corrected derivative along its line in registers (row: dU/dxi with the jumps of edges 1 and 3; column:
// dU/deta with those of edges 0 and 2) and swaps derivatives with the
// crossing lines through one shared tile.  It forms Q = (xi_x dU/dxi + eta_x
// dU/deta, xi_y dU/dxi + eta_y dU/deta) at its N1 points and the traces of Q
// at its two end points (row j: edge 1 point j with l(+1), edge 3 point
// N1-1-j with l(-1); column i: edge 0 point i with l(-1), edge 2 point
// N1-1-i with l(+1)), and from them the element's viscous shares.
//
// Rows and columns run the same instruction stream (the role only selects
// strides, edges and weights) and fill separate warps at P3.  The derivative
// tile holds point (a = xi index, b = eta index) at a*(N1+1) + b; the staged
// rows are padded by 16 bytes; the element strides spread both access
// patterns over the banks.
template <int P, typename T>
struct LineShape {
    static constexpr int N1 = P + 1, NSP = N1 * N1, NFT = 4 * N1;
    static constexpr int EB = ZJ_LINE_THREADS / (2 * N1);   // elements per CTA
    static constexpr int THREADS = EB * 2 * N1;
    static constexpr int NOPS = N1 * N1 + 4 * N1;
    // derivative tile: [el][role][var][a*R + b]
    static constexpr int R = N1 + 1;
    static constexpr int VB = N1 * R;
    static constexpr int MOD = sizeof(T) == 8 ? 16 : 32;
    static constexpr int ES = 8 * VB + ((4 - (8 * VB) % MOD) + MOD) % MOD;
    // staged states (doubles): [el][b][a*4 + v], rows padded by 16 bytes, the
    // element stride 64 bytes past a multiple of 128
    static constexpr int RU = N1 * 4 + 2;
    static constexpr int EU = N1 * RU + ((8 - (N1 * RU) % 16) + 16) % 16;
    // dynamic shared memory layout (byte offsets, 16-byte aligned); the
    // metrics are read directly (one 16- or 32-byte load a point), which
    // measured faster than staging them with the states
    static constexpr size_t OFF_U = 0;
    static constexpr size_t OFF_D = OFF_U + sizeof(double) * EB * EU;
    static constexpr size_t OFF_OPS = OFF_D + ((sizeof(T) * EB * ES + 15) & ~size_t(15));
    static constexpr size_t SMEM = OFF_OPS + ((sizeof(T) * NOPS + 15) & ~size_t(15));
    static_assert(OFF_D % 16 == 0 && OFF_OPS % 16 == 0, "16-byte aligned regions");
    // A line thread holds a line's states and derivatives: twice the values
    // of a point thread, at half the threads per element.
    // (the counts are per 128 threads; other CTA sizes scale them)
    static constexpr int MIN_BLOCKS_128 =
        sizeof(T) == 8 ? ZJ_NSL_MIN_BLOCKS
                       : (P <= 3 ? ZJ_NSL32_MIN_BLOCKS : ZJ_NSL32_MIN_BLOCKS_HI);
    static constexpr int MIN_BLOCKS = MIN_BLOCKS_128 * 128 / ZJ_LINE_THREADS > 0 ? MIN_BLOCKS_128 * 128 / ZJ_LINE_THREADS : 1;
};

// 16-byte asynchronous global -> shared copy (cp.async, cached in L2 only),
// and the wait for all of this thread's copies.
__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int P, typename T>
__global__ void __launch_bounds__(LineShape<P, T>::THREADS, LineShape<P, T>::MIN_BLOCKS)
k_ns_grad_lines(const StageArgsT<T> a) {
    using L = LineShape<P, T>;
    constexpr int N1 = L::N1, NSP = L::NSP, NFT = L::NFT, EB = L::EB, R = L::R, VB = L::VB, ES = L::ES;
    constexpr int RU = L::RU, EU = L::EU;
    extern __shared__ __align__(16) unsigned char smem[];
    double* sU = reinterpret_cast<double*>(smem + L::OFF_U);
    T* sD = reinterpret_cast<T*>(smem + L::OFF_D);
    T* sOps = reinterpret_cast<T*>(smem + L::OFF_OPS);

    const int tid = threadIdx.x;
    for (int t = tid; t < L::NOPS; t += L::THREADS) sOps[t] = a.ops[t];
    pdl_launch_dependents();
    pdl_wait();   // the state and traces come from the previous stage
    for (int c = tid; c < EB * NSP * 2; c += L::THREADS) {
        const int el2 = c / (NSP * 2), r = c - el2 * NSP * 2, p = r >> 1, h = r & 1;
        bool v2;
        const long long e2 = block_element(a, EB, el2, v2);
        if (v2) cp_async16(sU + el2 * EU + (p / N1) * RU + (p % N1) * 4 + h * 2, a.U + (e2 * NSP + p) * 4 + h * 2);
    }
    cp_async_commit();

    const int role = tid / (EB * N1);            // 0: row (xi-line), 1: column (eta-line)
    const int rem = tid - role * EB * N1;
    const int el = rem / N1, line = rem - el * N1;
    bool valid;
    const long long e = block_element(a, EB, el, valid);
    // staged offset of the line's point m: row j -> (m, j), column i -> (i, m)
    const int ubase = role ? line * 4 : line * RU, ustride = role ? RU : 4;
    // derivative-tile offset of point m: (a, b) -> a*R + b
    const int tbase = role ? line * R : line, tstride = role ? 1 : R;
    const int eA = role ? 0 : 1, eB = role ? 2 : 3;
    const int fA = line, fB = N1 - 1 - line;
    constexpr bool kRef = UsesRef<T>::value;

    // jumps U_c - U_own = (U_nbr - U_own)/2 and average states at the line's
    // end points
    T dA[4], dB[4];
    T UaA[4], UaB[4];
    const T* Tin = after_wait(a.Tin);
    if (valid) {
#pragma unroll
        for (int s2 = 0; s2 < 2; ++s2) {
            const int ed = s2 ? eB : eA, fp = s2 ? fB : fA;
            const EdgeRec r = a.edges[e * 4 + ed];
            T qo[4], qn[4];
            load4_nc(Tin + (e * NFT + ed * N1 + fp) * 4, qo);
#pragma unroll
            for (int v = 0; v < 4; ++v) qn[v] = qo[v];
            if (!(r.flags & kEdgeOrphan)) load4_nc(Tin + (neighbour_row(r, a.n_elem) * N1 + (N1 - 1 - fp)) * 4, qn);
            T* d = s2 ? dB : dA;
            T* m = s2 ? UaB : UaA;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                d[v] = (r.flags & kEdgeOrphan) ? T(0) : T(0.5) * (qn[v] - qo[v]);
                m[v] = T(0.5) * (qo[v] + qn[v]);
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();   // staged states, operators

    T mine[N1][4];
    if (valid) {
        T u[N1][4];
        const double* su = sU + el * EU;
        T ue[4];
        if constexpr (kRef) {
            double d0[4];
            load4(su, d0);   // the element's first solution point
#pragma unroll
            for (int v = 0; v < 4; ++v) ue[v] = T(d0[v]);
        }
#pragma unroll
        for (int m = 0; m < N1; ++m) {
            double ud[4];
            load4(su + ubase + m * ustride, ud);
            if constexpr (kRef) {
                // D (U - U_e): the reference drops out of the derivative exactly
                state_minus_ref(ud, ue, u[m]);
            } else {
#pragma unroll
                for (int v = 0; v < 4; ++v) u[m][v] = T(ud[v]);
            }
        }
        // corrected derivative along the line: sum_k D[m][k] u_k, then
        // + g1(m) jump_A + g2(m) jump_B (rows: g_R, g_L; columns: g_L, g_R)
        const T* gL = sOps + N1 * N1 + 2 * N1;
        const T* gR = gL + N1;
        const T* g1 = role ? gL : gR;
        const T* g2 = role ? gR : gL;
#pragma unroll
        for (int m = 0; m < N1; ++m) {
            T Dm[N1];
            load_op_row<N1>(sOps, m, Dm);
            const T g1m = g1[m], g2m = g2[m];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                T acc = T(0);
#pragma unroll
                for (int k = 0; k < N1; ++k) acc = fma_any(Dm[k], u[k][v], acc);
                acc += g1m * dA[v] + g2m * dB[v];
                mine[m][v] = acc;
            }
        }
        T* sd = sD + el * ES + role * 4 * VB + tbase;
#pragma unroll
        for (int m = 0; m < N1; ++m)
#pragma unroll
            for (int v = 0; v < 4; ++v) sd[v * VB + m * tstride] = mine[m][v];
    }
    __syncthreads();
    if (!valid) return;

    // Q at the line's points and its traces at the two end points
    const T* WA = sOps + N1 * N1 + (role ? 0 : N1);   // row: l(+1) at edge 1; column: l(-1) at edge 0
    const T* WB = sOps + N1 * N1 + (role ? N1 : 0);   // row: l(-1) at edge 3; column: l(+1) at edge 2
    const T* so = sD + el * ES + (1 - role) * 4 * VB + tbase;
    T tA[8], tB[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) { tA[c] = T(0); tB[c] = T(0); }
#pragma unroll
    for (int m = 0; m < N1; ++m) {
        T ji[4];
        load4_nc(a.Jinv + (e * NSP + (role ? line + m * N1 : line * N1 + m)) * 4, ji);
        const T wa = WA[m], wb = WB[m];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const T other = so[v * VB + m * tstride];
            const T dxi = role ? other : mine[m][v];
            const T deta = role ? mine[m][v] : other;
            const T Qx = ji[0] * dxi + ji[2] * deta;
            const T Qy = ji[1] * dxi + ji[3] * deta;
            tA[v] = fma_any(wa, Qx, tA[v]);
            tA[4 + v] = fma_any(wa, Qy, tA[4 + v]);
            tB[v] = fma_any(wb, Qx, tB[v]);
            tB[4 + v] = fma_any(wb, Qy, tB[4 + v]);
        }
    }
    if constexpr (sizeof(T) == 8) {   // the adjoint's gradient traces (FP64 only), with the shares or alone
        if (a.GQ) {
            gstore8(a.GQ + (e * NFT + eA * N1 + fA) * 8, tA);
            gstore8(a.GQ + (e * NFT + eB * N1 + fB) * 8, tB);
        }
        if (!a.FVout) return;
    }
#pragma unroll
    for (int s2 = 0; s2 < 2; ++s2) {
        const int ed = s2 ? eB : eA, fp = s2 ? fB : fA;
        // (read again here: held from the jumps on, they cost more in
        // registers than the second L1 access)
        const EdgeRec r = a.edges[e * 4 + ed];
        T n[3], f[4];
        load_normal(normal_rec<N1>(a, e, ed, fp), n);
        viscous_share(a, r, n[0], n[1], s2 ? UaB : UaA, s2 ? tB : tA, f);
        gstore4(a.FVout + (e * NFT + ed * N1 + fp) * 4, f);
    }
}

template <int P, int RIEM, typename T>
__global__ void __launch_bounds__(Shape<P, EbDiv<T>::value>::THREADS, NSMinBlocks<T, P>::stage)
k_ns_stage(const StageArgsT<T> a) {
    using S = Shape<P, EbDiv<T>::value>;
    constexpr int N1 = S::N1, NSP = S::NSP, NFT = S::NFT, TPE = S::TPE, EB = S::EB;
    using Op = OpTable<P + 1, T>;
    constexpr int RP = Tiles<P, T>::RP, FP = Tiles<P, T>::FP, DP = Tiles<P, T>::DP;
    __shared__ __align__(16) Weight<T> sOps[Op::N];
    __shared__ __align__(16) T sF[EB * FP];
    __shared__ __align__(16) T sG[EB * FP];
    __shared__ __align__(16) T sD[EB * DP];   // face jumps of U, then flux differences
    __shared__ __align__(16) T sU[EB * FP];   // stage state, then the new state
    __shared__ double sRed[32];

    const int tid = threadIdx.x;
    Op::fill(sOps, a.ops);
    pdl_launch_dependents();
    pdl_wait();   // the viscous shares come from the gradient launch, the state from the previous stage
    const int el = tid / TPE, k = tid - el * TPE;
    bool valid;
    const long long e = block_element(a, EB, el, valid);
    const bool is_sp = valid && k < NSP, is_fp = valid && k < NFT;
    const T g = T(a.gamma);
    const FaceLane fl = lane_face<N1>(k);
    const int edge = fl.edge, fp = fl.fp, kf = edge * N1 + fp;
    int i, j;
    lane_point<N1>(k, i, j);
    const int ks = j * N1 + i;

    // ---- A1: loads, face jumps, stage state into shared memory; the common
    // flux of the flux points, which needs nothing else (a thread carries its
    // four values, not the traces they came from, through the volume phase)
    constexpr bool kRef = UsesRef<T>::value;
    T ue[4] = {T(0), T(0), T(0), T(0)};   // reference state (mixed form)
    T u[4], ji[4], Jd = T(1);
    T Fd[4] = {T(0), T(0), T(0), T(0)};
    const T* Tin = after_wait(a.Tin);
    const T* FV = after_wait(a.FV);
    FacePoint<T> f;
    f.r = EdgeRec{-1, 0, kEdgeOrphan, 0};
    T fo[4], fn[4] = {T(0), T(0), T(0), T(0)};
    double ud[4];
    auto load_point = [&] {
        const long long idx = e * NSP + ks;
        stage_state(a, idx, ud, u);
        load4_x(a.Jinv + idx * 4, ji);
        Jd = ldg_any(a.J + idx);
        if ((ks & 3) == 0 && a.stage >= 2) prefetch_l2(a.U0 + idx * 4);
    };
    auto store_point = [&] {
        T w[4];
        if constexpr (kRef) state_minus_ref(ud, ue, w);
        else {
#pragma unroll
            for (int v = 0; v < 4; ++v) w[v] = u[v];
        }
        store4(sU + el * FP + j * RP + 4 * i, w);
    };
    // FP32 issues every load before the first use, the edge record first (the
    // neighbour's rows hang on it): -6 % per step at 256 x 256, P3.  In FP64
    // that is 56 registers of data in flight and was slower; there the
    // solution point goes first and the face's loads are the compiler's to place.
    if constexpr (sizeof(T) == 4) {
        if (is_fp) {
            load_own_face<N1>(a, Tin, e, edge, fp, f);
            load4_now(FV + (e * NFT + kf) * 4, fo);
        }
        if (kRef && valid) load_state(a.U + e * NSP * 4, ue);
        if (is_sp) load_point();
        if (is_fp) {
            load_neighbour_face<N1>(a, Tin, fp, f);
            if (has_neighbour_gradient(f.r))
                load4_now(FV + (neighbour_row(f.r, a.n_elem) * N1 + (N1 - 1 - fp)) * 4, fn);
        }
        if (is_sp) store_point();
    } else {
        if (is_sp) {
            load_point();
            store_point();
        }
        if (is_fp) {
            load_own_face<N1>(a, Tin, e, edge, fp, f);
            load_neighbour_face<N1>(a, Tin, fp, f);
            load4_nc(FV + (e * NFT + kf) * 4, fo);
            if (has_neighbour_gradient(f.r))
                load4_nc(FV + (neighbour_row(f.r, a.n_elem) * N1 + (N1 - 1 - fp)) * 4, fn);
        }
    }
    const bool face = is_fp && !(f.r.flags & kEdgeOrphan);
    if (is_fp) {
        T d[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) d[v] = face ? T(0.5) * (f.qn[v] - f.qo[v]) : T(0);
        store4(sD + el * DP + face_slot<P, T>(fl.dir, fl.side, fl.line), d);
    }
    if (face) {
        // evaluated from the left element's side on both sides
        const bool right = (f.r.flags & kEdgeRight) != 0;
        T UL[4], UR[4], Fc[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) { UL[v] = right ? f.qn[v] : f.qo[v]; UR[v] = right ? f.qo[v] : f.qn[v]; }
        riemann<RIEM>(UL, UR, f.nx, f.ny, g, Fc);
        if constexpr (kRef) {
            T Fe[4];
            ref_flux_n(ue, g, f.nx, f.ny, Fe);
#pragma unroll
            for (int v = 0; v < 4; ++v) Fc[v] -= Fe[v];
        }
        const T ss = right ? T(-0.5) * f.len : T(0.5) * f.len;
#pragma unroll
        for (int v = 0; v < 4; ++v) Fd[v] = ss * (Fc[v] - (fo[v] + fn[v]));
    }
    __syncthreads();

    // ---- A2: gradient, total transformed fluxes
    if (is_sp) {
        T Qx[4], Qy[4], Fv[4], Gv[4];
        corrected_gradient<P>(sU + el * FP, sD + el * DP, sOps, i, j, ji, Qx, Qy);
        // one reciprocal density for the viscous and the Euler flux
        const T ir = rcp_any(u[0]);
        viscous_flux_f(u, ir, Qx, Qy, g, inv_reynolds(a), T(a.kfac), Fv, Gv);
        T F[4], G[4];
        euler_flux_ir(u, ir, g, F, G);
        if constexpr (kRef) {
            T Fe[4], Ge[4];
            euler_flux(ue, g, Fe, Ge);
#pragma unroll
            for (int v = 0; v < 4; ++v) { F[v] -= Fe[v]; G[v] -= Ge[v]; }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) { F[v] -= Fv[v]; G[v] -= Gv[v]; }
        store_fluxes<P>(sF + el * FP, sG + el * FP, i, j, Jd, ji, F, G);
    }
    __syncthreads();   // face jumps and the stage state in shared memory are dead now

    // ---- B: flux differences at the faces
    if (is_fp) {
        if (face) flux_difference<P>((fl.dir ? sF : sG) + el * FP, sOps, fl, Fd);
        store4(sD + el * DP + face_slot<P, T>(fl.dir, fl.side, fl.line), Fd);
    }
    __syncthreads();

    // ---- C: divergence, VCJH correction, 1/J, stage update
    double rsq = 0.0;
    if (is_sp) {
        const long long idx = e * NSP + ks;
        double u0[4];
        if (a.stage >= 2) gload4(a.U0 + idx * 4, u0);
        const T iJ = rcp_any(Jd);
        T res[4];
        divergence<P>(sF + el * FP, sG + el * FP, sD + el * DP, sOps, i, j, res);
#pragma unroll
        for (int v = 0; v < 4; ++v) res[v] = -res[v] * iJ;
        if (a.stage == 0) {
            store_residual(a, idx, res, rsq);
        } else {
            double us[4];
            if constexpr (sizeof(T) == 8) {
#pragma unroll
                for (int v = 0; v < 4; ++v) us[v] = double(u[v]);
            } else {
                gload4(a.U + idx * 4, us);
            }
            double uo[4];
            rk_update(a.stage, *a.dt, us, u0, res, uo);
            gstore4(a.Uout + idx * 4, uo);
            T un[4];
            if constexpr (kRef) state_minus_ref(uo, ue, un);
            else {
#pragma unroll
                for (int v = 0; v < 4; ++v) un[v] = T(uo[v]);
            }
            store4(sU + el * FP + j * RP + 4 * i, un);
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

    // ---- D: traces of the new state
    if (is_fp) {
        T t[4];
        state_trace<P>(sU + el * FP, sOps, fl, t);
        if constexpr (kRef) {
#pragma unroll
            for (int v = 0; v < 4; ++v) t[v] += ue[v];
        }
        gstore4(a.Tout + (e * NFT + kf) * 4, t);
        if (boundary_condition_edge(f.r)) store_ghost<N1>(a, f.r, f.nx, f.ny, fp, t);
    }
}

// One split for the gradient and the stage kernel.
template <int P, typename T>
constexpr int ns_carveout() {
    if constexpr (IsDual<T>::value) return 100;   // as phys_carveout
    else {
        const int st = carveout_bytes(NSMinBlocks<T, P>::stage, stage_smem<P, T>());
        const int gr = carveout_bytes(LineShape<P, T>::MIN_BLOCKS, LineShape<P, T>::SMEM);
        return carveout_percent(st > gr ? st : gr);
    }
}

template <int P, typename T>
cudaError_t ns_grad_t(const StageArgsT<T>& a, cudaStream_t s) {
    if constexpr (!IsDual<T>::value) {
        using L = LineShape<P, T>;
        const long long grid = ((a.elist ? a.n_list : a.n_elem) + L::EB - 1) / L::EB;
        if (grid <= 0) return cudaSuccess;
        static bool set = false;
        if (!set) {
            set_carveout(k_ns_grad_lines<P, T>, ns_carveout<P, T>());
            cudaFuncSetAttribute(k_ns_grad_lines<P, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM);
            set = true;
        }
        return launch_programmatic_smem(k_ns_grad_lines<P, T>, (unsigned)grid, L::THREADS, L::SMEM, s, a);
    } else {
        using S = Shape<P, EbDiv<T>::value>;
        const long long grid = ((a.elist ? a.n_list : a.n_elem) + S::EB - 1) / S::EB;
        if (grid <= 0) return cudaSuccess;
        static bool set = false;
        if (!set) { set_carveout(k_ns_grad<P, T>, ns_carveout<P, T>()); set = true; }
        return launch_programmatic(k_ns_grad<P, T>, (unsigned)grid, S::THREADS, s, a);
    }
}

template <int P, int RIEM, typename T>
cudaError_t ns_stage_t(const StageArgsT<T>& a, cudaStream_t s) {
    using S = Shape<P, EbDiv<T>::value>;
    const long long grid = ((a.elist ? a.n_list : a.n_elem) + S::EB - 1) / S::EB;
    if (grid <= 0) return cudaSuccess;
    static bool set = false;
    if (!set) { set_carveout(k_ns_stage<P, RIEM, T>, ns_carveout<P, T>()); set = true; }
    return launch_programmatic(k_ns_stage<P, RIEM, T>, (unsigned)grid, S::THREADS, s, a);
}

template <int P, typename T>
cudaError_t ns_stage_p(int riemann, const StageArgsT<T>& a, cudaStream_t s) {
    switch (riemann) {
        case ZJ_RIEMANN_RUSANOV: return ns_stage_t<P, ZJ_RIEMANN_RUSANOV>(a, s);
        case ZJ_RIEMANN_ROE: return ns_stage_t<P, ZJ_RIEMANN_ROE>(a, s);
        case ZJ_RIEMANN_HLLC: return ns_stage_t<P, ZJ_RIEMANN_HLLC>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

template <typename T>
cudaError_t ns_grad_dispatch(int P, const StageArgsT<T>& a, cudaStream_t s) {
    switch (P) {
        case 1: return ns_grad_t<1>(a, s);
        case 2: return ns_grad_t<2>(a, s);
        case 3: return ns_grad_t<3>(a, s);
        case 4: return ns_grad_t<4>(a, s);
        case 5: return ns_grad_t<5>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

template <typename T>
cudaError_t ns_stage_dispatch(int P, int riemann, const StageArgsT<T>& a, cudaStream_t s) {
    switch (P) {
        case 1: return ns_stage_p<1>(riemann, a, s);
        case 2: return ns_stage_p<2>(riemann, a, s);
        case 3: return ns_stage_p<3>(riemann, a, s);
        case 4: return ns_stage_p<4>(riemann, a, s);
        case 5: return ns_stage_p<5>(riemann, a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace
}  // namespace zj
