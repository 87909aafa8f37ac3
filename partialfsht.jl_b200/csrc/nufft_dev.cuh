// Device helpers shared by the NUFFT's interpolation and spreading kernels (nufft.cu, nufft_mma.cu):
// the fine grids' element types, a bin's tile, a point's origin cell and its tap weights.
#pragma once
#include "es_horner_table.h"
#include "internal.cuh"

namespace pf {

// ---------------------------------------------------------------------------------------
// complex element of the fine grids: double2 in the FP64 form, float2 in the mixed form (whose
// mode columns, points and per-mode factors stay FP64)
// ---------------------------------------------------------------------------------------
template <class T> struct Cx;
template <> struct Cx<double> {
    using t = double2;
    __device__ static double2 make(double x, double y) { return make_double2(x, y); }
};
template <> struct Cx<float> {
    using t = float2;
    __device__ static float2 make(float x, float y) { return make_float2(x, y); }
};
template <class T> using cx = typename Cx<T>::t;

__device__ __forceinline__ int wrap(int i, int n) {
    int r = i % n;
    return r < 0 ? r + n : r;
}

// tile of a bin: the rows and columns its points' kernels reach,
// rows [br BR, br BR + BR + W - 1) x columns [bc BC, bc BC + BC + W - 1)
struct TileGeom {
    int tr0, tc0, TR, TC;
};
template <int W>
__device__ __forceinline__ TileGeom tile_geom(int bin, int nbc, int BR, int BC) {
    const int br = bin / nbc, bc = bin % nbc;
    return TileGeom{br * BR, bc * BC, BR + W - 1, BC + W - 1};
}

// origin cell of a point inside its bin's tile (the binning of bin_keys_kernel)
template <int W>
__device__ __forceinline__ void local_origin(double2 g, const TileGeom& tg, int nrows, int nf2,
                                             int row_wrap, int& r0, int& c0, double& v1,
                                             double& v2) {
    const int i10 = (int)ceil(g.x - 0.5 * W);
    const int i20 = (int)ceil(g.y - 0.5 * W);
    v1 = ((double)i10 - g.x) + (0.5 * W - 0.5);
    v2 = ((double)i20 - g.y) + (0.5 * W - 0.5);
    int r = i10, c = i20;
    if (row_wrap) r = wrap(r, nrows);
    c = wrap(c, nf2);
    r0 = r - tg.tr0;
    c0 = c - tg.tc0;
}

template <int W, class T> struct EsCoef;
template <int W> struct EsCoef<W, double> {
    __device__ static const double* get() { return EsHorner<W>::coef(); }
};
template <int W> struct EsCoef<W, float> {
    __device__ static const float* get() { return EsHorner<W>::coef_f(); }
};

// Weights of the mirrored taps a and W - 1 - a (a < W / 2) at offset v, u = v^2, in the grid's
// precision. Tap W - 1 - a is tap a reflected (v -> -v; the table holds the same coefficients
// with the odd powers negated), so with p_a(v) = E(v^2) + v O(v^2) the pair costs one even and
// one odd Horner chain in u: NC multiply-adds for two taps instead of 2 (NC - 1).
template <int W, class T>
__device__ __forceinline__ void es_pair(int a, T v, T u, T& ka, T& kb) {
    constexpr int NC = EsHorner<W>::NC;
    constexpr int NE = (NC + 1) / 2, NO = NC / 2;
    const T* cf = EsCoef<W, T>::get() + a * NC;
    T e = cf[2 * (NE - 1)];
#pragma unroll
    for (int i = NE - 2; i >= 0; --i) e = fma(e, u, cf[2 * i]);
    T o = cf[2 * (NO - 1) + 1];
#pragma unroll
    for (int i = NO - 2; i >= 0; --i) o = fma(o, u, cf[2 * i + 1]);
    ka = fma(v, o, e);
    kb = fma(-v, o, e);
}

// weight of the middle tap of an odd width (an even polynomial: its odd coefficients are 0)
template <int W, class T>
__device__ __forceinline__ T es_mid(T u) {
    constexpr int NC = EsHorner<W>::NC;
    constexpr int NE = (NC + 1) / 2;
    const T* cf = EsCoef<W, T>::get() + (W / 2) * NC;
    T e = cf[2 * (NE - 1)];
#pragma unroll
    for (int i = NE - 2; i >= 0; --i) e = fma(e, u, cf[2 * i]);
    return e;
}

// all W tap weights at offset v: mirrored pairs in FP64; one Horner chain per tap in FP32, where
// the spreading kernel measured faster that way (0.133 vs 0.142 ms at lmax 2048)
template <int W, class T>
__device__ __forceinline__ void es_weights(T v, T (&k)[W]) {
    if constexpr (sizeof(T) == 8) {
        const T u = v * v;
#pragma unroll
        for (int a = 0; a < W / 2; ++a) es_pair<W, T>(a, v, u, k[a], k[W - 1 - a]);
        if constexpr (W & 1) k[W / 2] = es_mid<W, T>(u);
    } else {
        constexpr int NC = EsHorner<W>::NC;
        const T* cf = EsCoef<W, T>::get();
#pragma unroll
        for (int a = 0; a < W; ++a) {
            T p = cf[a * NC + NC - 1];
#pragma unroll
            for (int q = NC - 2; q >= 0; --q) p = fma(p, v, cf[a * NC + q]);
            k[a] = p;
        }
    }
}

}  // namespace pf
