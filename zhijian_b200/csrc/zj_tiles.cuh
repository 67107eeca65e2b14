// zj_tiles.cuh -- shared-memory tiles of the quad kernels and the operator
// products over them: field tiles [row][col][var], the flux-point tile
// [dir][side][line][var], traces, flux differences and the corrected
// divergence.
#pragma once

#include "zj_device.cuh"
#include "zj_dual.cuh"

namespace zj {
namespace dev {

// Strides of the shared tiles, in values.  A field tile holds point (i, j) at
// j * RP + 4 i with its four variables; the rows are padded so that the points
// of a row and those of a column fall on distinct banks, the elements by RP's
// padding once more.  The flux-point tile is [dir][side][line][var]: the four
// loads of a solution point (its lines' ends) spread over the banks too.
template <int P, typename T>
struct Tiles {
    using S = Shape<P, EbDiv<T>::value>;
    static constexpr int N1 = S::N1;
    static constexpr int PAD = sizeof(T) == 4 ? 4 : (sizeof(T) == 8 ? 2 : 1);   // 16 bytes
    static constexpr int RP = 4 * N1 + PAD;
    static constexpr int FP = N1 * RP;
    static constexpr int DB = 4 * N1 + (sizeof(T) == 4 ? 0 : PAD);              // one (dir, side) block
    static constexpr int DP = 4 * DB + PAD * (sizeof(T) == 4 ? 4 : 1);
};

// Offset of a flux point in the [dir][side][line][var] tile.
template <int P, typename T>
__device__ __forceinline__ int face_slot(int dir, int side, int line) {
    return (dir * 2 + side) * Tiles<P, T>::DB + line * 4;
}

// Transformed fluxes F~ = J (xi_x F + xi_y G), G~ = J (eta_x F + eta_y G) of
// point (i, j) into the tiles.
template <int P, typename T>
__device__ __forceinline__ void store_fluxes(T* tF, T* tG, int i, int j, T Jd, const T* ji, const T* F,
                                             const T* G) {
    constexpr int RP = Tiles<P, T>::RP;
    T ft[4], gt[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        ft[v] = Jd * (ji[0] * F[v] + ji[1] * G[v]);
        gt[v] = Jd * (ji[2] * F[v] + ji[3] * G[v]);
    }
    store4(tF + j * RP + 4 * i, ft);
    store4(tG + j * RP + 4 * i, gt);
}

// The line of a tile that a flux point ends: first point and stride.
template <int P, typename T>
__device__ __forceinline__ const T* line_of(const T* tile, const FaceLane& f, int& stride) {
    constexpr int RP = Tiles<P, T>::RP;
    stride = f.dir ? 4 : RP;
    return tile + f.line * (f.dir ? RP : 4);
}

// Fd minus the outward extrapolated transformed flux of a flux point (tile:
// F~ for xi-lines, G~ for eta-lines; outward is -F~ at -1, +F~ at +1).
template <int P, typename T>
__device__ __forceinline__ void flux_difference(const T* tile, const Weight<T>* ops, const FaceLane& f, T* Fd) {
    using Op = OpTable<P + 1, T>;
    constexpr int N1 = P + 1;
    int stride;
    const T* p = line_of<P>(tile, f, stride);
    Weight<T> w[N1];
    load_weights<N1>(ops + (f.side ? Op::NLP : Op::LM), w);
    v4_get(line_dot<N1>(w, p, stride, v4(Fd)), Fd);
}

// Trace of a state tile at a flux point.
template <int P, typename T>
__device__ __forceinline__ void state_trace(const T* tile, const Weight<T>* ops, const FaceLane& f, T* t) {
    using Op = OpTable<P + 1, T>;
    constexpr int N1 = P + 1;
    int stride;
    const T* p = line_of<P>(tile, f, stride);
    Weight<T> w[N1];
    load_weights<N1>(ops + (f.side ? Op::LP : Op::LM), w);
    v4_get(line_dot<N1>(w, p, stride, v4_zero<T>()), t);
}

// acc + the VCJH corrections with the flux differences d at point (i, j).
template <int P, typename T>
__device__ __forceinline__ V4<T> correction(const T* d, const Weight<T>* ops, int i, int j, V4<T> acc) {
    using Op = OpTable<P + 1, T>;
    acc = v4_fma(ops[Op::GR + i], v4_load(d + face_slot<P, T>(1, 1, j)), acc);
    acc = v4_fma(ops[Op::NGL + i], v4_load(d + face_slot<P, T>(1, 0, j)), acc);
    acc = v4_fma(ops[Op::GR + j], v4_load(d + face_slot<P, T>(0, 1, i)), acc);
    return v4_fma(ops[Op::NGL + j], v4_load(d + face_slot<P, T>(0, 0, i)), acc);
}

// D_xi F~ + D_eta G~ + the corrections at point (i, j).
template <int P, typename T>
__device__ __forceinline__ void divergence(const T* tF, const T* tG, const T* d, const Weight<T>* ops, int i,
                                           int j, T* out) {
    constexpr int N1 = P + 1, RP = Tiles<P, T>::RP;
    Weight<T> w[N1];
    load_weights<N1>(ops + i * N1, w);
    V4<T> acc = line_dot<N1>(w, tF + j * RP, 4, v4_zero<T>());
    load_weights<N1>(ops + j * N1, w);
    acc = line_dot<N1>(w, tG + 4 * i, RP, acc);
    v4_get(correction<P>(d, ops, i, j, acc), out);
}

}  // namespace dev
}  // namespace zj
