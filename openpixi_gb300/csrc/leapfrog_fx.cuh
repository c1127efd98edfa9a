// leapfrog_fx.cuh -- the FP64 leapfrog with its group products in fixed point
// (fixed.cuh), one link per thread: the equations of leapfrog.cuh,
//     E_i(x) += dt proj(U_i(x) S_i(x)) - g a_i dt J_i(x)
//     Unext_i(x) = exp(-i dt E_i(x)) U_i(x),
// E and the links read and written as doubles, the staples, the projection, the
// exponential and the product with it on the integer pipe.  The sums over the
// staple planes need one factor 1/a_j^2 (equal spacings).
//
// update_link returns false, having written nothing, where a link it needs is
// not usable in fixed point or where the link itself (SU(2): and the site's other
// two, whose nine entries together are hardly ever all small by chance) lies
// closer to the identity than 2^-7 in every entry (fixed.cuh: there the FP64
// product is the more exact one); the caller then makes the FP64 update.
//
// Bound: the issue slots of the integer pipes.  256 x 64^2 SU(2) 1.014 -> 0.291 ms
// a step, 128^3 2.014 -> 0.575, SU(3) 64^3 2.99 -> 0.492 ms (the FP64 pipe before);
// 32^3 0.041 -> 0.018 ms (0.014 with overlapped launches) and SU(3) 16^3 0.221 ->
// 0.027 ms, where a thread's serial chain counts: one link per thread is a third of
// it, and beats one site per thread with the forward staples of a plane sharing a
// product (21 instead of 24 products for a site) at every size tried (SU(2) 16^3
// 0.0123 against 0.0184 ms, 128^3 0.728 against 0.773, both before the asm
// multiply-adds).
// SU(3) by whole matrix products at 168 registers: 64^3 0.727 against 0.681 ms row
// by row at 128 (both before the multiply-adds were written in asm, 0.492).
#pragma once
#include "fixed.cuh"
#include "internal.h"
#include "leapfrog.cuh"

namespace opx {
namespace fx {

// Unext of one link from its new E where qexp / mexp refuses (a large or
// non-finite dt E): the FP64 exponential and product
template <int NC, typename I>
__device__ __forceinline__ void link_update_f64(const double *__restrict__ U, double *__restrict__ Un, const Lat &L, I s, int i,
                                             const double *e) {
    using G = typename GroupOf<NC, double>::T;
    double v[G::NA];
    for (int a = 0; a < G::NA; a++) v[a] = -L.dt * e[a];
    const LinkPlanes<G, double, I> Up{const_cast<double *>(U), (I)L.V}, Unp{Un, (I)L.V};
    Unp.store(i, s, G::mul(G::expi(v), Up.load(i, s)));
}

// SU(2): E and Unext of one link from its staple sum S (units of 2^-60, without 1/a^2)
template <bool HAS_J, typename I>
__device__ __forceinline__ void finish_link(const Q &Ui, const i64 *S, const double *__restrict__ U, double *__restrict__ E,
                                            const double *__restrict__ J, double *__restrict__ Unext, const Lat &L, I s, int i) {
    const AlgPlanes<3, double, I> Ep{E, (I)L.V}, Jp{const_cast<double *>(J), (I)L.V};
    const LinkPlanes<SU2<double>, double, I> Un{Unext, (I)L.V};
    const double kdt = L.dt * L.inva2[0] * 0x1p-58, kv = L.dt * -0x1p60;
    Q F;
#pragma unroll
    for (int c = 0; c < 4; c++) F.e[c] = quarter(S[c]);
    double e[3], t[3];
    Ep.load(i, s, e);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        // proj_a = 2 (U S)_a, the product in units of 2^-59
        Acc p = acc0v();
        qcomp<false, false>(p, Ui, F, 1 + a);
        e[a] = fma((double)value(p), kdt, e[a]);
    }
    if (HAS_J) {
        double jv[3];
        Jp.load_ro(i, s, jv);
        const double jf = LatR<double>::jfac(L, i);
#pragma unroll
        for (int a = 0; a < 3; a++) e[a] += jv[a] * jf;
    }
    Ep.store(i, s, e);
#pragma unroll
    for (int a = 0; a < 3; a++) t[a] = kv * e[a];
    Q X;
    if (qexp(t, X)) {
        Q2<double> V;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            Acc p = acc0v();
            qcomp<false, false>(p, X, Ui, c);
            V.e[c] = double_of(value(p));
        }
        Un.store(i, s, V);
    } else {
        link_update_f64<2, I>(U, Unext, L, s, i, e);
    }
}

// The FP64 update of one link (the staples in the order of update_site)
template <int NC, bool HAS_J, typename I>
__device__ __forceinline__ void update_link_f64(const double *__restrict__ U, double *__restrict__ E, const double *__restrict__ J,
                                             double *__restrict__ Unext, const Lat &L, I s, int i) {
    using G = typename GroupOf<NC, double>::T;
    using MM = typename G::M;
    constexpr int NA = G::NA;
    int x[3];
    site_coords<I>(L, s, x);
    const Deltas<I> D = deltas<I>(L, x);
    const LinkPlanes<G, double, I> Up{const_cast<double *>(U), (I)L.V}, Un{Unext, (I)L.V};
    const AlgPlanes<NA, double, I> Ep{E, (I)L.V}, Jp{const_cast<double *>(J), (I)L.V};
    const I pi = s + D.f(i);
    MM S = G::zero();
#pragma unroll 1
    for (int jj = 1; jj < 3; jj++) {
        const int j = i + jj >= 3 ? i + jj - 3 : i + jj;
        const I bj = D.b(j);
        MM F = G::mul_adj(G::mul_adj(Up.load(j, pi), Up.load(i, s + D.f(j))), Up.load(j, s));
        const MM C = G::mul(Up.load(i, s + bj), Up.load(j, pi + bj));
        G::add(F, G::adj_mul(C, Up.load(j, s + bj)));
        G::scale(F, LatR<double>::inva2(L, j));
        G::add(S, F);
    }
    const MM Ui = Up.load(i, s);
    double pr[NA], e[NA], v[NA];
    G::proj(G::mul(Ui, S), pr);
    Ep.load(i, s, e);
#pragma unroll
    for (int a = 0; a < NA; a++) e[a] += pr[a] * L.dt;
    if (HAS_J) {
        double jv[NA];
        Jp.load_ro(i, s, jv);
        const double jf = LatR<double>::jfac(L, i);
#pragma unroll
        for (int a = 0; a < NA; a++) e[a] += jv[a] * jf;
    }
    Ep.store(i, s, e);
#pragma unroll
    for (int a = 0; a < NA; a++) v[a] = -L.dt * e[a];
    Un.store(i, s, G::mul(G::expi(v), Ui));
}

// SU(2), one link
template <bool HAS_J, typename I>
__device__ __forceinline__ bool update_link(const FxLinks<2, I> W, const double *__restrict__ U, double *__restrict__ E,
                                            const double *__restrict__ J, double *__restrict__ Unext, const Lat &L, I s, int i) {
    const Q Ui = W.load(i, s);
    const int j1 = i == 2 ? 0 : i + 1, j2 = i == 0 ? 2 : i - 1;
    const Q Uj1 = W.load(j1, s), Uj2 = W.load(j2, s);
    if ((offdiag(Ui) | offdiag(Uj1) | offdiag(Uj2)) < WEAK_H) return false;
    int x[3];
    site_coords<I>(L, s, x);
    const Deltas<I> D = deltas<I>(L, x);
    int worst = min(min(Ui.e[0].h, Uj1.e[0].h), Uj2.e[0].h);
    auto load = [&](int d, I t) {
        const Q q = W.load(d, t);
        worst = min(worst, q.e[0].h);
        return q;
    };
    const I pi = s + D.f(i);
    i64 S[4] = {0, 0, 0, 0};
#pragma unroll
    for (int jj = 0; jj < 2; jj++) {
        const int j = jj ? j2 : j1;
        const I bj = D.b(j);
        qacc<false, true>(S, qmul<false, true>(load(j, pi), load(i, s + D.f(j))), jj ? Uj2 : Uj1);
        qacc<true, false>(S, qmul<false, false>(load(i, s + bj), load(j, pi + bj)), load(j, s + bj));
    }
    if (worst == LINK_BAD) return false;
    finish_link<HAS_J, I>(Ui, S, U, E, J, Unext, L, s, i);
    return true;
}

// SU(3), one link: the staple sum row by row, the loops over the row and the
// staple plane rolled
template <bool HAS_J, typename I>
__device__ __forceinline__ bool update_link(const FxLinks<3, I> W, const double *__restrict__ U, double *__restrict__ E,
                                            const double *__restrict__ J, double *__restrict__ Unext, const Lat &L, I s, int i) {
    int x[3];
    site_coords<I>(L, s, x);
    const Deltas<I> D = deltas<I>(L, x);
    const I pi = s + D.f(i);
    int worst = 0;
    auto see = [&](int d, I t) { worst = min(worst, __ldg(W.p + link_offset_t<I>(W.V, 18, d, 0, t)).y); };
    see(i, s);
#pragma unroll
    for (int jj = 1; jj < 3; jj++) {
        const int j = i + jj >= 3 ? i + jj - 3 : i + jj;
        const I bj = D.b(j);
        see(j, s);
        see(j, pi);
        see(i, s + D.f(j));
        see(i, s + bj);
        see(j, s + bj);
        see(j, pi + bj);
    }
    if (worst == LINK_BAD || offdiag(W.load(i, s)) < WEAK_H) return false;
    const AlgPlanes<8, double, I> Ep{E, (I)L.V}, Jp{const_cast<double *>(J), (I)L.V};
    const LinkPlanes<SU3<double>, double, I> Un{Unext, (I)L.V};
    const double kdt = L.dt * L.inva2[0] * 0x1p-58, kv = L.dt * -0x1p60;
    const FxEntries Ui = W.at(i, s);
    // U_i S, S's rows one by one: proj in units of 2^-58
    i64 x9[9];
#pragma unroll
    for (int a = 0; a < 9; a++) x9[a] = 0;
#pragma unroll 1
    for (int r = 0; r < 3; r++) {
        i64 S[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
        for (int jj = 1; jj < 3; jj++) {
            const int j = i + jj >= 3 ? i + jj - 3 : i + jj;
            const I bj = D.b(j);
            // U_j(x+i) U_i(x+j)^dagger U_j(x)^dagger
            racc<true>(S, rmul<true>(W.at(j, pi).row(r), W.at(i, s + D.f(j))), W.at(j, s));
            // U_j(x+i-j)^dagger U_i(x-j)^dagger U_j(x-j)
            racc<false>(S, rmul<true>(W.at(j, pi + bj).adj_row(r), W.at(i, s + bj)), W.at(j, s + bj));
        }
        Row F;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            F.r[q] = quarter(S[q]);
            F.i[q] = quarter(S[3 + q]);
        }
        // entry (p, q) of U_i S gains U_i(p, r) S(r, q)
#pragma unroll
        for (int p = 0; p < 3; p++) {
            Fx ur, ui;
            Ui(3 * p + r, ur, ui);
            i64 re[3], im[3];
#pragma unroll
            for (int q = 0; q < 3; q++) {
                Acc a{0, ONE30}, b{0, ONE30};
                mac(a, ur, F.r[q]);
                mac(a, neg(ui), F.i[q]);
                mac(b, ur, F.i[q]);
                mac(b, ui, F.r[q]);
                re[q] = a.a + (a.b >> 31);
                im[q] = b.a + (b.b >> 31);
            }
            proj_row(x9, p, re, im);
        }
    }
    double e[8], t[8];
    Ep.load(i, s, e);
#pragma unroll
    for (int a = 0; a < 7; a++) e[a] = fma((double)x9[a], kdt, e[a]);
    e[7] = fma((double)proj_eighth(x9), kdt * 1.15470053837925152902, e[7]);  // 2 / sqrt 3
    if (HAS_J) {
        double jv[8];
        Jp.load_ro(i, s, jv);
        const double jf = LatR<double>::jfac(L, i);
#pragma unroll
        for (int a = 0; a < 8; a++) e[a] += jv[a] * jf;
    }
    Ep.store(i, s, e);
#pragma unroll
    for (int a = 0; a < 7; a++) t[a] = kv * e[a];
    t[7] = kv * 0.57735026918962576451 * e[7];
    M X;
    if (mexp(t, X)) {
        M3<double> V;
#pragma unroll
        for (int r = 0; r < 3; r++) {
            Row v;
#pragma unroll
            for (int k = 0; k < 3; k++) { v.r[k] = X.r[3 * r + k]; v.i[k] = X.i[3 * r + k]; }
#pragma unroll
            for (int q = 0; q < 3; q++) {
                Acc a = acc0v(), b = acc0v();
                rterm<false>(a, b, v, Ui, q);
                V.r[3 * r + q] = double_of(value(a));
                V.i[3 * r + q] = double_of(value(b));
            }
        }
        Un.store(i, s, V);
    } else {
        link_update_f64<3, I>(U, Unext, L, s, i, e);
    }
    return true;
}

// One link per thread, the three links of 128 sites in three consecutive blocks
template <int NC> struct FxBounds { static constexpr int minb = 5; };
template <> struct FxBounds<3> { static constexpr int minb = 4; };
template <int NC, bool HAS_J, typename I>
__global__ void __launch_bounds__(128, FxBounds<NC>::minb)
k_update_links_fx(const int2 *__restrict__ Uf, const double *__restrict__ U, double *__restrict__ E,
                  const double *__restrict__ J, double *Unext, int2 *__restrict__ Unf,
                  const uint8_t *__restrict__ active, const __grid_constant__ Lat L, const unsigned *stop) {
    pdl_wait();
    if (stopped(stop)) return;
    const unsigned chunk = blockIdx.x / 3u;
    const int i = (int)(blockIdx.x - 3u * chunk);
    const I s = (I)chunk * (I)blockDim.x + (I)threadIdx.x;
    if (s >= (I)L.V) return;
    if (active && !active[s]) return;  // Cell.isActive gate (FastTYMSolver.java:51)
    if (!update_link<HAS_J, I>(FxLinks<NC, I>{Uf, (I)L.V}, U, E, J, Unext, L, s, i))
        update_link_f64<NC, HAS_J, I>(U, E, J, Unext, L, s, i);
    // the new link in fixed point, from the double that was stored
    fixed_link<NC, double, I>(Unext, Unf, (I)L.V, i, s);
}

}  // namespace fx
}  // namespace opx
