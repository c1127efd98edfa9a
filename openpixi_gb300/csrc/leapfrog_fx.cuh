// leapfrog_fx.cuh -- the FP64 leapfrog with its group products in fixed point
// (fixed.cuh), one link per thread: the equations of leapfrog.cuh,
//     E_i(x) += dt proj(U_i(x) S_i(x)) - g a_i dt J_i(x)
//     Unext_i(x) = exp(-i dt E_i(x)) U_i(x),
// E and the links read and written as doubles, the staples, the projection, the
// exponential and the product with it on the integer pipe.  The sums over the
// staple planes need one factor 1/a_j^2 (equal spacings).
//
// update_link returns false, having written nothing, where a link it needs is
// not usable in fixed point or where FP64 products are the more exact ones; the
// caller then makes the FP64 update.  The latter is a matter of each colour
// component: a product here is exact to 2^-61 of one, an FP64 product to 2^-53 of
// the component's own size, so a component that is small in all links of a
// stencil would lose its digits here.  A component (SU(3): an entry off the
// identity) counts as small where it is below 2^-14 in all three links of the site;
// all count as small where the site's links (SU(3): the link) are within 2^-7 of
// the identity.  Small components that are exactly zero in the whole stencil stay
// exactly zero here, so Abelian fields and vacuum keep the fixed-point form (the
// product with an exponential whose argument has such a component, below 2^-14
// but not zero, is FP64); any other small component is refused.  Components just
// above the line keep 14 digits.  The line is as low as that because one warp that takes
// the FP64 products by chance makes the whole grid wait (SU(3) 40^3 0.130 ms, with
// 2^-10 0.181): at a width of 0.05 it is one link in 10^7 (SU(2): 10^8).
//
// Bound: the issue slots of the integer pipes.  256 x 64^2 SU(2) 1.014 -> 0.286 ms
// a step, 128^3 2.014 -> 0.568, SU(3) 64^3 2.99 -> 0.477 ms (the FP64 pipe before);
// 32^3 0.041 -> 0.018 ms (0.0134 with overlapped launches) and SU(3) 16^3 0.221 ->
// 0.0246 ms, where a thread's serial chain counts: one link per thread is a third of
// it, and beats one site per thread with the forward staples of a plane sharing a
// product (21 instead of 24 products for a site) at every size tried (SU(2) 16^3
// 0.0123 against 0.0184 ms, 128^3 0.728 against 0.773, both before the asm
// multiply-adds).
// SU(3) by whole matrix products at 168 registers: 64^3 0.727 against 0.681 ms row
// by row at 128 (both before the multiply-adds were written in asm).
#pragma once
#include "fixed.cuh"
#include "internal.h"
#include "leapfrog.cuh"

namespace opx {
namespace fx {

// Unext of one link from its new E where qexp / mexp refuses (a large or
// non-finite dt E) or a component would lose digits: the FP64 exponential and product
template <int NC, typename I>
__device__ __noinline__ void link_update_f64(const double *__restrict__ U, double *__restrict__ Un, const Lat &L, I s, int i,
                                             const double *e) {
    using G = typename GroupOf<NC, double>::T;
    double v[G::NA];
    for (int a = 0; a < G::NA; a++) v[a] = -L.dt * e[a];
    const LinkPlanes<G, double, I> Up{const_cast<double *>(U), (I)L.V}, Unp{Un, (I)L.V};
    Unp.store(i, s, G::mul(G::expi(v), Up.load(i, s)));
}

// Bit a: component a + 1 of the three links of a site is small; WEAK: all where the
// links are within 2^-7 of the identity
template <bool WEAK = true> __device__ __forceinline__ int small_components(const Q &u0, const Q &u1, const Q &u2) {
    int m[3];
#pragma unroll
    for (int a = 0; a < 3; a++) m[a] = abs(u0.e[1 + a].h) | abs(u1.e[1 + a].h) | abs(u2.e[1 + a].h);
    const int all = m[0] | m[1] | m[2];
    const bool weak = WEAK && all < WEAK_H;
    if (min(min(m[0], m[1]), m[2]) >= SMALL_H && !weak) return 0;
    return weak ? 7 : (m[0] < SMALL_H ? 1 : 0) | (m[1] < SMALL_H ? 2 : 0) | (m[2] < SMALL_H ? 4 : 0);
}
// Whether the components of the mask are exactly zero in every link of the staples
// of the site's three links (own, one step forward or back, and diagonal: 24 links).
// From the doubles: the fixed-point form rounds what is below 2^-62 away
template <typename I>
__device__ __noinline__ bool zero_in_stencil(const double *U, const Lat &L, I s, int mask) {
    const LinkPlanes<SU2<double>, double, I> Up{const_cast<double *>(U), (I)L.V};
    auto zero = [&](int d, I t) {
        const Q2<double> q = Up.load(d, t);
        return (!(mask & 1) || is_zero(q.e[1])) && (!(mask & 2) || is_zero(q.e[2])) && (!(mask & 4) || is_zero(q.e[3]));
    };
    for (int d = 0; d < 3; d++)
        if (!zero(d, s)) return false;
    int x[3];
    site_coords<I>(L, s, x);
    const Deltas<I> D = deltas<I>(L, x);
#pragma unroll 1
    for (int j = 0; j < 3; j++) {
        const I mj = s + D.b(j);
        if (!zero(j, mj)) return false;
#pragma unroll 1
        for (int ii = 1; ii < 3; ii++) {
            const int i = j + ii >= 3 ? j + ii - 3 : j + ii;
            if (!zero(i, mj) || !zero(i, s + D.f(j)) || !zero(j, s + D.f(i) + D.b(j))) return false;
        }
    }
    return true;
}
// Whether a small component, zero in U, is to come out of exp(-i dt E) U with the
// digits that FP64 gives it
__device__ __forceinline__ bool tiny(double t) { return !is_zero(t) && exponent_of(t) < TINY_T; }
__device__ __forceinline__ bool tiny_component(int small, const double *t) {
    return small && (((small & 1) && tiny(t[0])) || ((small & 2) && tiny(t[1])) || ((small & 4) && tiny(t[2])));
}
// SU(3), small: a bit per entry (flag_bit).  H = -dt E^a lambda_a / 2 of the exponential:
// i H has t_0, t_3, t_5 in its off-diagonal imaginary parts, t_1, t_4, t_6 in the real
// ones, t_7 +- t_2 and -2 t_7 on the diagonal
__device__ __forceinline__ bool tiny_entry(unsigned small, const double *t) {
    if (!small) return false;
    bool refuse = false;
    auto see = [&](int c, int d, double h) {  // entries c and d of U, h of H
        const unsigned both = 1u << flag_bit(c) | 1u << flag_bit(d);
        refuse = refuse || ((small & both) == both && tiny(h));
    };
    see(10, 12, t[0]);
    see(1, 3, t[1]);
    see(11, 15, t[3]);
    see(2, 6, t[4]);
    see(14, 16, t[5]);
    see(5, 7, t[6]);
    see(9, 9, t[7] + t[2]);
    see(13, 13, t[7] - t[2]);
    see(17, 17, t[7]);
    return refuse;
}

// SU(2): E and Unext of one link from its staple sum S (units of 2^-60, without 1/a^2)
template <bool HAS_J, typename I>
__device__ __forceinline__ void finish_link(int small, const Q &Ui, const i64 *S, const double *__restrict__ U, double *__restrict__ E,
                                            const double *__restrict__ J, double *Unext, int2 *__restrict__ Unf,
                                            const Lat &L, I s, int i) {
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
    if (!tiny_component(small, t) && qexp(t, X)) {
        Q2<double> V;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            Acc p = acc0v();
            qcomp<false, false>(p, X, Ui, c);
            V.e[c] = double_of(value(p));
        }
        Un.store(i, s, V);
        if (Unf) write_fixed<2, I>(V.e, Unf, (I)L.V, i, s);
    } else {
        link_update_f64<2, I>(U, Unext, L, s, i, e);
        if (Unf) fixed_link<2, double, I>(Unext, Unf, (I)L.V, i, s);
    }
}

// The FP64 update of one link: the staples in the order of update_site, but every product
// of the sum added term by term and the one spacing factor applied to the projection:
// a tenth fewer FP64 operations a link, which is what a lattice of refused links waits
// for.  Calls: inlined, their code and registers were the integer path's too (SU(3): 304 B
// of spills at 128 registers, 4 now).  Lattices of width 0.005, ms a step, inlined products /
// this / k_update_grid: SU(2) 32^3 0.0456 / 0.0418 / 0.0411, 128^3 2.25 / 2.05 / 2.01 (the
// refusal and the fixed-point copy cost the rest), SU(3) 24^3 0.243 / 0.174 / 0.219, 40^3
// 0.746 / 0.531 / 0.845; SU(2) 128^3, half of it vacuum: 1.33 / 1.07 / 2.01.
// SU(2): S += A B, A = a or its adjoint, B likewise
template <bool CA, bool CB> __device__ __forceinline__ void qfma(double *S, const Q2<double> &a, const Q2<double> &b) {
    const double x1 = CA ? -a.e[1] : a.e[1], x2 = CA ? -a.e[2] : a.e[2], x3 = CA ? -a.e[3] : a.e[3];
    const double y1 = CB ? -b.e[1] : b.e[1], y2 = CB ? -b.e[2] : b.e[2], y3 = CB ? -b.e[3] : b.e[3];
    S[0] = fma(-x3, y3, fma(-x2, y2, fma(-x1, y1, fma(a.e[0], b.e[0], S[0]))));
    S[1] = fma(x3, y2, fma(-x2, y3, fma(x1, b.e[0], fma(a.e[0], y1, S[1]))));
    S[2] = fma(x1, y3, fma(-x3, y1, fma(x2, b.e[0], fma(a.e[0], y2, S[2]))));
    S[3] = fma(x2, y1, fma(-x1, y2, fma(x3, b.e[0], fma(a.e[0], y3, S[3]))));
}
// exp(i w_a sigma_a), w = k e: SU2::expi of 2 w without its halves
__device__ __forceinline__ Q2<double> expi_half(double k, const double *e) {
    const double w[3] = {k * e[0], k * e[1], k * e[2]}, m2 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
    if (!(m2 < 0.01)) {
        const double v[3] = {2.0 * w[0], 2.0 * w[1], 2.0 * w[2]};
        return SU2<double>::expi(v);
    }
    const double c = 1 + m2 * (-1.0 / 2 + m2 * (1.0 / 24 + m2 * (-1.0 / 720 + m2 * (1.0 / 40320 + m2 * (-1.0 / 3628800)))));
    const double h = 1 + m2 * (-1.0 / 6 + m2 * (1.0 / 120 + m2 * (-1.0 / 5040 + m2 * (1.0 / 362880 + m2 * (-1.0 / 39916800)))));
    return Q2<double>{{c, w[0] * h, w[1] * h, w[2] * h}};
}
template <bool HAS_J, typename I>
__device__ __noinline__ void update_link_f64(const LinkPlanes<SU2<double>, double, I> Up, double *__restrict__ E, const double *__restrict__ J,
                                             double *__restrict__ Unext, const Lat &L, I s, int i) {
    using G = SU2<double>;
    int x[3];
    site_coords<I>(L, s, x);
    const Deltas<I> D = deltas<I>(L, x);
    const LinkPlanes<G, double, I> Un{Unext, (I)L.V};
    const AlgPlanes<3, double, I> Ep{E, (I)L.V}, Jp{const_cast<double *>(J), (I)L.V};
    const I pi = s + D.f(i);
    Q2<double> S = G::zero();
#pragma unroll 1
    for (int jj = 1; jj < 3; jj++) {
        const int j = i + jj >= 3 ? i + jj - 3 : i + jj;
        const I bj = D.b(j);
        qfma<false, true>(S.e, G::mul_adj(Up.load(j, pi), Up.load(i, s + D.f(j))), Up.load(j, s));
        qfma<true, false>(S.e, G::mul(Up.load(i, s + bj), Up.load(j, pi + bj)), Up.load(j, s + bj));
    }
    const Q2<double> Ui = Up.load(i, s), P = G::mul(Ui, S);
    double e[3];
    Ep.load(i, s, e);
    const double k = 2.0 * (L.dt * L.inva2[0]);  // proj_a = 2 (U S)_a
#pragma unroll
    for (int a = 0; a < 3; a++) e[a] = fma(P.e[1 + a], k, e[a]);
    if (HAS_J) {
        double jv[3];
        Jp.load_ro(i, s, jv);
        const double jf = LatR<double>::jfac(L, i);
#pragma unroll
        for (int a = 0; a < 3; a++) e[a] += jv[a] * jf;
    }
    Ep.store(i, s, e);
    Un.store(i, s, G::mul(expi_half(-0.5 * L.dt, e), Ui));
}
// SU(3): row by row as the fixed-point form
struct RowD {
    double r[3], i[3];
};
struct EntriesD {
    const double *b;
    __device__ __forceinline__ double re(int c) const { return __ldg(b + 32 * c); }
    __device__ __forceinline__ double im(int c) const { return __ldg(b + 32 * (9 + c)); }
    __device__ __forceinline__ RowD row(int r) const { return RowD{{re(3 * r), re(3 * r + 1), re(3 * r + 2)}, {im(3 * r), im(3 * r + 1), im(3 * r + 2)}}; }
    __device__ __forceinline__ RowD adj_row(int r) const { return RowD{{re(r), re(3 + r), re(6 + r)}, {-im(r), -im(3 + r), -im(6 + r)}}; }
};
// S += v B or (CB) v B^dagger
template <bool CB> __device__ __forceinline__ void rfma(RowD &S, const RowD &v, const EntriesD &b) {
#pragma unroll
    for (int q = 0; q < 3; q++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int c = CB ? 3 * q + k : 3 * k + q;
            const double br = b.re(c), bi = CB ? -b.im(c) : b.im(c);
            S.r[q] = fma(-v.i[k], bi, fma(v.r[k], br, S.r[q]));
            S.i[q] = fma(v.i[k], br, fma(v.r[k], bi, S.i[q]));
        }
}
template <bool CB> __device__ __forceinline__ RowD rowmul(const RowD &v, const EntriesD &b) {
    RowD S{{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
    rfma<CB>(S, v, b);
    return S;
}
template <bool HAS_J, typename I>
__device__ __noinline__ void update_link_f64(const LinkPlanes<SU3<double>, double, I> Up, double *__restrict__ E, const double *__restrict__ J,
                                             double *__restrict__ Unext, const Lat &L, I s, int i) {
    using G = SU3<double>;
    int x[3];
    site_coords<I>(L, s, x);
    const Deltas<I> D = deltas<I>(L, x);
    const LinkPlanes<G, double, I> Un{Unext, (I)L.V};
    const AlgPlanes<8, double, I> Ep{E, (I)L.V}, Jp{const_cast<double *>(J), (I)L.V};
    const I pi = s + D.f(i);
    auto at = [&](int d, I t) { return EntriesD{Up.p + link_offset_t<I>(Up.V, 18, d, 0, t)}; };
    const EntriesD Ui = at(i, s);
    M3<double> P = G::zero();  // U_i S
#pragma unroll 1
    for (int r = 0; r < 3; r++) {
        RowD S{{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
#pragma unroll 1
        for (int jj = 1; jj < 3; jj++) {
            const int j = i + jj >= 3 ? i + jj - 3 : i + jj;
            const I bj = D.b(j);
            rfma<true>(S, rowmul<true>(at(j, pi).row(r), at(i, s + D.f(j))), at(j, s));
            rfma<false>(S, rowmul<true>(at(j, pi + bj).adj_row(r), at(i, s + bj)), at(j, s + bj));
        }
        // entry (p, q) gains U_i(p, r) S(r, q)
#pragma unroll
        for (int p = 0; p < 3; p++) {
            const double ur = Ui.re(3 * p + r), ui = Ui.im(3 * p + r);
#pragma unroll
            for (int q = 0; q < 3; q++) {
                P.r[3 * p + q] = fma(-ui, S.i[q], fma(ur, S.r[q], P.r[3 * p + q]));
                P.i[3 * p + q] = fma(ui, S.r[q], fma(ur, S.i[q], P.i[3 * p + q]));
            }
        }
    }
    double pr[8], e[8], v[8];
    G::proj(P, pr);
    Ep.load(i, s, e);
    const double k = L.dt * L.inva2[0];
#pragma unroll
    for (int a = 0; a < 8; a++) e[a] = fma(pr[a], k, e[a]);
    if (HAS_J) {
        double jv[8];
        Jp.load_ro(i, s, jv);
        const double jf = LatR<double>::jfac(L, i);
#pragma unroll
        for (int a = 0; a < 8; a++) e[a] += jv[a] * jf;
    }
    Ep.store(i, s, e);
#pragma unroll
    for (int a = 0; a < 8; a++) v[a] = -L.dt * e[a];
    Un.store(i, s, G::mul(G::expi(v), Up.load(i, s)));
}

// SU(2), one link
template <bool HAS_J, typename I>
__device__ __forceinline__ bool update_link(const FxLinks<2, I> W, const double *__restrict__ U, double *__restrict__ E,
                                            const double *__restrict__ J, double *Unext, int2 *__restrict__ Unf, const Lat &L, I s, int i) {
    const Q Ui = W.load(i, s);
    const int j1 = i == 2 ? 0 : i + 1, j2 = i == 0 ? 2 : i - 1;
    const Q Uj1 = W.load(j1, s), Uj2 = W.load(j2, s);
    const int small = small_components(Ui, Uj1, Uj2);
    if (small && !zero_in_stencil<I>(U, L, s, small)) return false;
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
    finish_link<HAS_J, I>(small, Ui, S, U, E, J, Unext, Unf, L, s, i);
    return true;
}

// SU(3), one link: the staple sum row by row, the loops over the row and the
// staple plane rolled
template <bool HAS_J, typename I>
__device__ __forceinline__ bool update_link(const FxLinks<3, I> W, const double *__restrict__ U, double *__restrict__ E,
                                            const double *__restrict__ J, double *Unext, int2 *__restrict__ Unf, const Lat &L, I s, int i) {
    int x[3];
    site_coords<I>(L, s, x);
    const Deltas<I> D = deltas<I>(L, x);
    const I pi = s + D.f(i);
    const int j1 = i == 2 ? 0 : i + 1, j2 = i == 0 ? 2 : i - 1;
    const unsigned own = W.flags(i, s), u1 = W.flags(j1, s), u2 = W.flags(j2, s);
    unsigned any = own | u1 | u2, every = own & u1 & u2;
    const unsigned small = own & LINK_WEAK ? SMALL_MASK : every & SMALL_MASK;
#pragma unroll
    for (int jj = 0; jj < 2; jj++) {
        const int j = jj ? j2 : j1;
        const I bj = D.b(j);
        const unsigned f[5] = {W.flags(j, pi), W.flags(i, s + D.f(j)), W.flags(i, s + bj), W.flags(j, s + bj), W.flags(j, pi + bj)};
#pragma unroll
        for (int k = 0; k < 5; k++) {
            any |= f[k];
            every &= f[k];
        }
    }
    if ((any & FLAG_BAD) || (small & ~(every >> ZERO_SHIFT))) return false;
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
    if (!tiny_entry(small, t) && mexp(t, X)) {
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
        if (Unf) {
            double u[18];
#pragma unroll
            for (int c = 0; c < 9; c++) { u[c] = V.r[c]; u[9 + c] = V.i[c]; }
            write_fixed<3, I>(u, Unf, (I)L.V, i, s);
        }
    } else {
        link_update_f64<3, I>(U, Unext, L, s, i, e);
        if (Unf) fixed_link<3, double, I>(Unext, Unf, (I)L.V, i, s);
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
    // the new link in fixed point too, from the doubles that are stored
    if (!update_link<HAS_J, I>(FxLinks<NC, I>{Uf, (I)L.V}, U, E, J, Unext, Unf, L, s, i)) {
        update_link_f64<HAS_J, I>(LinkPlanes<typename GroupOf<NC, double>::T, double, I>{const_cast<double *>(U), (I)L.V}, E, J, Unext, L, s, i);
        if (Unf) fixed_link<NC, double, I>(Unext, Unf, (I)L.V, i, s);
    }
}

}  // namespace fx
}  // namespace opx
