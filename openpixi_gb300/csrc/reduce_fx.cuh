// reduce_fx.cuh -- the squared magnetic field of a plane in FP64 with its group
// products in fixed point (fixed.cuh).  As in the update, a term whose links are
// not usable there, or lie within 2^-7 of the identity, is formed in FP64.
#pragma once
#include "fixed.cuh"
#include "observables.cuh"

namespace opx {
namespace fx {

// In FP64, calls as in leapfrog_fx.cuh (SU(2): the last product's three components and
// one factor for their squares)
template <int NC, typename I>
__device__ __noinline__ double plane_b2_f64(const double *__restrict__ U, const Lat &L, I s, I sj, I sk, int j, int k, double f) {
    using G = typename GroupOf<NC, double>::T;
    const LinkPlanes<G, double, I> Up{const_cast<double *>(U), (I)L.V};
    const auto P = G::mul_adj(G::mul_adj(G::mul(Up.load(j, s), Up.load(k, sj)), Up.load(j, sk)), Up.load(k, s));
    if constexpr (NC == 2) {
        return (P.e[1] * P.e[1] + P.e[2] * P.e[2] + P.e[3] * P.e[3]) * (4.0 * (f * f));
    } else {
        double b[G::NA];
        G::proj(P, b);
        return sqr<double, G::NA>(b) * (f * f);
    }
}

__device__ __forceinline__ double proj_square(const Q &A, const Q &B) {  // |proj(A B^dagger)|^2
    double b2 = 0.0;
#pragma unroll
    for (int a = 1; a < 4; a++) {
        Acc s = acc0v();
        qcomp<false, true>(s, A, B, a);
        const double v = (double)value(s);
        b2 = fma(v, v, b2);
    }
    return b2 * 0x1p-120;  // proj_a = 2 v 2^-61
}
// |B_d|^2 at site s (coordinates x) of the links U, in fixed point Uf
template <typename I>
__device__ __forceinline__ double plane_b2(const FxLinks<2, I> W, const double *__restrict__ U, const Lat &L, I s, const int *x,
                                           const Deltas<I> &D, int d) {
    const int j = d == 2 ? 0 : d + 1, k = d == 0 ? 2 : d - 1;
    const I sj = s + D.f(j), sk = s + D.f(k);
    const double f = LatR<double>::bfac(L, d);
    const Q Uj = W.load(j, s), Uk = W.load(k, s), A = W.load(k, sj), B = W.load(j, sk);
    if ((offdiag(Uj) | offdiag(Uk)) < WEAK_H || min(min(Uj.e[0].h, Uk.e[0].h), min(A.e[0].h, B.e[0].h)) == LINK_BAD)
        return plane_b2_f64<2, I>(U, L, s, sj, sk, j, k, f);
    return proj_square(qmul<false, true>(qmul<false, false>(Uj, A), B), Uk) * (f * f);
}
template <typename I>
__device__ __forceinline__ double plane_b2(const FxLinks<3, I> W, const double *__restrict__ U, const Lat &L, I s, const int *x,
                                           const Deltas<I> &D, int d) {
    const int j = d == 2 ? 0 : d + 1, k = d == 0 ? 2 : d - 1;
    const I sj = s + D.f(j), sk = s + D.f(k);
    const double f = LatR<double>::bfac(L, d);
    const FxEntries Uj = W.at(j, s), Uk = W.at(k, s), A = W.at(k, sj), B = W.at(j, sk);
    if ((offdiag(W.load(j, s)) | offdiag(W.load(k, s))) < WEAK_H ||
        min(min(Uj.mark(), Uk.mark()), min(A.mark(), B.mark())) == LINK_BAD)
        return plane_b2_f64<3, I>(U, L, s, sj, sk, j, k, f);
    i64 x9[9];
#pragma unroll
    for (int a = 0; a < 9; a++) x9[a] = 0;
#pragma unroll 1
    for (int r = 0; r < 3; r++) {
        const Row v = rmul<true>(rmul<false>(Uj.row(r), A), B);
        i64 re[3], im[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            Acc a = acc0v(), b = acc0v();
            rterm<true>(a, b, v, Uk, q);
            re[q] = value(a);
            im[q] = value(b);
        }
        proj_row(x9, r, re, im);
    }
    double b2 = (double)proj_eighth(x9);
    b2 = b2 * b2 * (4.0 / 3.0);
#pragma unroll
    for (int a = 0; a < 7; a++) {
        const double v = (double)x9[a];
        b2 = fma(v, v, b2);
    }
    return b2 * 0x1p-122 * (f * f);
}

}  // namespace fx
}  // namespace opx
