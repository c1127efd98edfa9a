// transport_fx.cuh -- the parallel transport U^dagger X U of an FP64 algebra
// element with its group products in fixed point (fixed.cuh), and the Gauss law's
// term of it.  The element is scaled by a power of two of its largest entry; the
// transport's error is then below 2^-59 of that entry.  Links that are not
// usable, or lie within 2^-7 of the identity, and elements that are zero,
// not finite or near the end of the exponent range take the FP64 products.
#pragma once
#include "fixed.cuh"

namespace opx {
namespace fx {

// Entries of U^dagger X U for X = x_a t_a, x below 2^(k - s) in magnitude, in
// units of 2^(k - 61): generator components
template <int NA> struct Scaled {
    i64 v[NA];
    double unit;
};
// x 2^(e_x - emax - lift) 2^61: the bits of fixed_of below a common exponent
__device__ __forceinline__ Fx fx_below(double x, int emax, int lift) {
    const i64 b = bits_of(x);
    const int e = (int)(b >> 52) & 0x7ff;
    const uint64_t m = (((uint64_t)b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 10;
    const unsigned r0 = (unsigned)(lift + emax - e), r = r0 < 63u ? r0 : 63u;
    const i64 g = (i64)(((m >> r) + 1) >> 1), s = b >> 63;
    return from_value((g ^ s) - s);
}
// x_a below 1/2 (lift 2): U^dagger X U, or (FWD) U X U^dagger, of a pure quaternion
template <bool FWD = false>
__device__ __forceinline__ void transport(const Q &U, const double *x, int emax, Scaled<3> &t) {
    Q X;
    X.e[0] = Fx{0, 0};
#pragma unroll
    for (int a = 0; a < 3; a++) X.e[1 + a] = fx_below(x[a], emax, 2);
    const Q A = qmul<false, FWD>(X, U);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        Acc s = acc0v();
        qcomp<!FWD, false>(s, U, A, 1 + a);
        t.v[a] = value(s);
    }
    t.unit = of_bits((i64)(emax - 59) << 52);  // 2^(emax - 1021 - 61)
}
template <bool FWD, class B> __device__ __forceinline__ Row start_row(const B &U, int r) {
    if constexpr (FWD) return U.row(r);
    else return U.adj_row(r);
}
// x_a below 1/4 (lift 3): with 2 X = x_a lambda_a, entries of U^dagger (2 X) U, or
// (FWD) U (2 X) U^dagger, row by row.  U: the link's entries
template <bool FWD = false, class B>
__device__ __forceinline__ void transport(const B &U, const double *x, int emax, Scaled<8> &t) {
    const Fx g2 = fx_below(x[2], emax, 3), g7 = fx_below(x[7] * 0.57735026918962576451, emax, 3);
    const Fx h0 = from_value(to_value(g2) + to_value(g7)), h1 = from_value(to_value(g7) - to_value(g2)), h2 = from_value(-2 * to_value(g7));
    const Fx ur = fx_below(x[0], emax, 3), vr = fx_below(x[3], emax, 3), wr = fx_below(x[5], emax, 3);
    const Fx ui = neg(fx_below(x[1], emax, 3)), vi = neg(fx_below(x[4], emax, 3)), wi = neg(fx_below(x[6], emax, 3));
    // the hermitian matrix's entries: upper 01, 02, 12 = u, v, w, the lower ones conjugate
    auto H = [&](int c, Fx &re, Fx &im) {
        const Fx zero{0, 0};
        switch (c) {
        case 0: re = h0; im = zero; break;
        case 1: re = ur; im = ui; break;
        case 2: re = vr; im = vi; break;
        case 3: re = ur; im = neg(ui); break;
        case 4: re = h1; im = zero; break;
        case 5: re = wr; im = wi; break;
        case 6: re = vr; im = neg(vi); break;
        case 7: re = wr; im = neg(wi); break;
        default: re = h2; im = zero; break;
        }
    };
    i64 w0 = 0, w1 = 0, w2 = 0;
#pragma unroll 1
    for (int r = 0; r < 3; r++) {
        // row r of the product, r = 0: entries 00, 01, 02; r = 1: 11, 12; r = 2: 22
        const Row v = rmul<false>(start_row<FWD>(U, r), H);
        i64 re[3], im[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            Acc a = acc0v(), b = acc0v();
            rterm<FWD>(a, b, v, U, q);
            re[q] = value(a);
            im[q] = value(b);
        }
        if (r == 0) {
            w0 = re[0];
            t.v[0] = re[1];
            t.v[1] = -im[1];
            t.v[3] = re[2];
            t.v[4] = -im[2];
        } else if (r == 1) {
            w1 = re[1];
            t.v[5] = re[2];
            t.v[6] = -im[2];
        } else {
            w2 = re[2];
        }
    }
    t.v[2] = (w0 - w1) >> 1;
    t.v[7] = ((w0 + w1) >> 1) - w2;  // x sqrt 3
    t.unit = of_bits((i64)(emax - 58) << 52);
}
__device__ __forceinline__ double component(const Scaled<3> &t, int a) { return (double)t.v[a]; }
__device__ __forceinline__ double component(const Scaled<8> &t, int a) {
    return a == 7 ? (double)t.v[7] * 0.57735026918962576451 : (double)t.v[a];
}

// The same in FP64 (calls, as in leapfrog_fx.cuh).  SU(2): with a pure quaternion X the first
// product has no scalar terms of X, and of the second three components are wanted: G::act without
// its products with zero and its halves (24 instead of 34 operations)
template <int NC, bool FWD, typename R>
__device__ __noinline__ void transport_f64(const R *__restrict__ U, const Lat &L, long s, int i, const double *x, double *t) {
    using G = typename GroupOf<NC, double>::T;
    using GR = typename GroupOf<NC, R>::T;
    const auto u = LinkPlanes<GR, R>{const_cast<R *>(U), L.V}.load(i, s);
    if constexpr (NC == 2) {
        const double q = FWD ? -1.0 : 1.0, u0 = (double)u.e[0], u1 = q * (double)u.e[1], u2 = q * (double)u.e[2], u3 = q * (double)u.e[3];
        // A = X V, t = V^dagger A, V = U or (FWD) its adjoint
        const double a0 = -(x[0] * u1 + x[1] * u2 + x[2] * u3), a1 = x[0] * u0 - x[1] * u3 + x[2] * u2;
        const double a2 = x[1] * u0 - x[2] * u1 + x[0] * u3, a3 = x[2] * u0 - x[0] * u2 + x[1] * u1;
        t[0] = u0 * a1 - u1 * a0 + u2 * a3 - u3 * a2;
        t[1] = u0 * a2 - u2 * a0 + u3 * a1 - u1 * a3;
        t[2] = u0 * a3 - u3 * a0 + u1 * a2 - u2 * a1;
    } else {
        typename G::M g;
#pragma unroll
        for (int c = 0; c < 9; c++) { g.r[c] = (double)u.r[c]; g.i[c] = (double)u.i[c]; }
        if constexpr (FWD) G::act(x, g, t);
        else G::act(x, G::adj(g), t);
    }
}

// Whether a link's transport is formed in fixed point
template <class T> __device__ __forceinline__ bool transportable(const T &u) { return first(u).h != LINK_BAD && offdiag(u) >= WEAK_H; }
// the entries of a link held in registers
struct HeldEntries {
    const M &m;
    __device__ __forceinline__ void operator()(int c, Fx &re, Fx &im) const {
        re = m.r[c];
        im = m.i[c];
    }
    __device__ __forceinline__ Row adj_row(int r) const {
        Row v;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const Fx re = r == 0 ? m.r[3 * k] : (r == 1 ? m.r[3 * k + 1] : m.r[3 * k + 2]);
            const Fx im = r == 0 ? m.i[3 * k] : (r == 1 ? m.i[3 * k + 1] : m.i[3 * k + 2]);
            v.r[k] = re;
            v.i[k] = neg(im);
        }
        return v;
    }
};

// r = x0 - U^dagger x U, or (FWD) x0 - U x U^dagger, U the link (i, s) of the array U and
// Uf the same in fixed point (SU(3): its entries), fixed: whether to use that
template <int NC, bool FWD, typename R, class T>
__device__ __forceinline__ void minus_transported(const T &Uf, bool fixed, const R *__restrict__ U, const Lat &L, long s, int i,
                                                  const double *x0, const double *x, double *r) {
    constexpr int NA = NC == 2 ? 3 : 8;
    int emax = 0;
#pragma unroll
    for (int a = 0; a < NA; a++) { const int e = exponent_of(x[a]); emax = e > emax ? e : emax; }
    if (fixed && emax >= 64 && emax < 0x7ff) {
        Scaled<NA> t;
        transport<FWD>(Uf, x, emax, t);
#pragma unroll
        for (int a = 0; a < NA; a++) r[a] = fma(-component(t, a), t.unit, x0[a]);
    } else {
        double t[NA];
        transport_f64<NC, FWD, R>(U, L, s, i, x, t);
#pragma unroll
        for (int a = 0; a < NA; a++) r[a] = x0[a] - t[a];
    }
}

// r = E_i(x) - U_i(x-i)^dagger E_i(x-i) U_i(x-i), sm = x - i, Ub = U_i(x-i) in
// fixed point (SU(3): its entries), fixed: whether to use it
template <int NC, typename I, class T>
__device__ __forceinline__ void gauss_term(const T &Ub, bool fixed, const double *__restrict__ U,
                                           const double *__restrict__ E, const Lat &L, I s, I sm, int i, double *r) {
    constexpr int NA = NC == 2 ? 3 : 8;
    const AlgPlanes<NA, double, I> Ep{const_cast<double *>(E), (I)L.V};
    double e0[NA], e1[NA];
    Ep.load_ro(i, s, e0);
    Ep.load_ro(i, sm, e1);
    minus_transported<NC, false, double>(Ub, fixed, U, L, (long)sm, i, e0, e1, r);
}

}  // namespace fx
}  // namespace opx
