// reduce_fx.cuh -- the squared magnetic field of a plane in FP64 with its group
// products in fixed point (fixed.cuh).  As in the update, a term whose links are
// not usable there, or lie within 2^-7 of the identity, is formed in FP64.
#pragma once
#include "fixed.cuh"
#include "observables.cuh"

namespace opx {
namespace fx {

template <int NC>
__device__ __forceinline__ double plane_b2_f64(const double *__restrict__ U, const Lat &L, long s, const int *x, int d) {
    using G = typename GroupOf<NC, double>::T;
    const Nbr nb = neighbours(L, s, x);
    const LinkPlanes<G, double> Up{const_cast<double *>(U), L.V};
    const int j = d == 2 ? 0 : d + 1, k = d == 0 ? 2 : d - 1;
    const long pj = pick3(nb.fwd[0], nb.fwd[1], nb.fwd[2], j), pk = pick3(nb.fwd[0], nb.fwd[1], nb.fwd[2], k);
    auto P = G::mul_adj(G::mul_adj(G::mul(Up.load(j, s), Up.load(k, pj)), Up.load(j, pk)), Up.load(k, s));
    double b[G::NA];
    G::proj(P, b);
    const double f = LatR<double>::bfac(L, d);
#pragma unroll
    for (int a = 0; a < G::NA; a++) b[a] *= f;
    return sqr<double, G::NA>(b);
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
    const Q Uj = W.load(j, s), Uk = W.load(k, s), A = W.load(k, s + D.f(j)), B = W.load(j, s + D.f(k));
    if ((offdiag(Uj) | offdiag(Uk)) < WEAK_H || min(min(Uj.e[0].h, Uk.e[0].h), min(A.e[0].h, B.e[0].h)) == LINK_BAD)
        return plane_b2_f64<2>(U, L, (long)s, x, d);
    const double f = LatR<double>::bfac(L, d);
    return proj_square(qmul<false, true>(qmul<false, false>(Uj, A), B), Uk) * (f * f);
}
template <typename I>
__device__ __forceinline__ double plane_b2(const FxLinks<3, I> W, const double *__restrict__ U, const Lat &L, I s, const int *x,
                                           const Deltas<I> &D, int d) {
    const int j = d == 2 ? 0 : d + 1, k = d == 0 ? 2 : d - 1;
    const FxEntries Uj = W.at(j, s), Uk = W.at(k, s), A = W.at(k, s + D.f(j)), B = W.at(j, s + D.f(k));
    if ((offdiag(W.load(j, s)) | offdiag(W.load(k, s))) < WEAK_H ||
        min(min(Uj.mark(), Uk.mark()), min(A.mark(), B.mark())) == LINK_BAD)
        return plane_b2_f64<3>(U, L, (long)s, x, d);
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
    const double f = LatR<double>::bfac(L, d);
    return b2 * 0x1p-122 * (f * f);
}

}  // namespace fx
}  // namespace opx
