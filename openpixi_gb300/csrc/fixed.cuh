// fixed.cuh -- SU(2) and SU(3) products of the FP64 form in 61-bit fixed point
// on the integer pipe.
//
// GB300 issues one FP64 multiply-add where it issues 32 of the integer
// 32 x 32 + 64 multiply-adds (measured per SM and clock: 1.96 DFMA, 64.8
// mad.wide.s32), so a product of 61-bit fixed-point numbers, three of the
// latter, costs a tenth of an FP64 multiply-add.  Group elements suit fixed
// point: their entries are bounded by one and a product of rows and columns of
// unit norm is bounded by one, so nothing overflows.
//
// A number is x = h 2^-30 + l 2^-61 with l in [-2^30, 2^30).  A sum of products
// is kept as a 2^-60 + b 2^-91: a collects the h h terms, b the h l terms; the
// l l terms (below 2^-62 each) are dropped.  Links converted from doubles are
// checked to be unitary within LINK_TOL (a link that is not, or that is not
// finite, carries the mark LINK_BAD in its first word), which bounds every sum:
//   |sum of h h| <= |row||column| 2^60 <= 1.02 2^60,
//   |sum of h l| <= 2 |row| (sqrt 6 2^30) 2^30 < 2^62.4.
// The error of a product is about 2^-61.5 (rms of the truncation of the operands, the dropped terms and
// the rounding of the result) against about 2^-53.8 m for the FP64 product of
// links whose entries off the identity are of size m: smaller for every m above
// 2^-7.7.  Callers take the FP64 arithmetic where the links are closer to
// the identity than WEAK_H (2^-7), so the fixed-point form is used only where
// it is the more exact one.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "group.cuh"
#include "lattice.cuh"

namespace opx {
namespace fx {

typedef long long i64;

struct Fx {
    int h, l;
};
struct Acc {
    i64 a, b;
};

constexpr int LINK_BAD = (int)0x80000000;     // h of a link's first entry when it is not usable here
constexpr float LINK_TOL = 1.0f / 256.0f;     // largest |U^dagger U - 1| entry of a usable link
constexpr int WEAK_H = 1 << 23;               // 2^-7 in units of 2^-30
constexpr int SMALL_H = 1 << 16;              // 2^-14: a small component in the update (leapfrog_fx.cuh)
constexpr int TINY_T = 1023 + 47;             // the exponent of 2^-14 in the exponential's argument, times 2^61
constexpr i64 HALF30 = 1LL << 29, ONE30 = 1LL << 30;

// the start of a sum that pack() ends (rounded, and offset for the split) and
// of one that value() ends (rounded)
OPX_HD OPX_INLINE Acc acc0() { return Acc{HALF30, HALF30}; }
OPX_HD OPX_INLINE Acc acc0v() { return Acc{0, HALF30}; }
// (asm: the compiler would turn a product with a negated factor into a product
// and a 64-bit subtraction, three instructions for one)
OPX_HD OPX_INLINE void mac(Acc &s, Fx x, Fx y) {
#ifdef __CUDA_ARCH__
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s.a) : "r"(x.h), "r"(y.h));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s.b) : "r"(x.h), "r"(y.l));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s.b) : "r"(x.l), "r"(y.h));
#else
    s.a += (i64)x.h * y.h;
    s.b += (i64)x.h * y.l;
    s.b += (i64)x.l * y.h;
#endif
}
OPX_HD OPX_INLINE Fx neg(Fx x) { return Fx{-x.h, -x.l}; }
// F + 2^30 (F in units of 2^-61) to (h, l)
OPX_HD OPX_INLINE Fx split(i64 f) {
    return Fx{(int)(f >> 31), (int)((unsigned)f & 0x7fffffffu) - (1 << 30)};
}
OPX_HD OPX_INLINE Fx pack(Acc s) { return split((i64)((uint64_t)s.a << 1) + (s.b >> 30)); }
OPX_HD OPX_INLINE i64 value(Acc s) { return (i64)((uint64_t)s.a << 1) + (s.b >> 30); }
OPX_HD OPX_INLINE Fx from_value(i64 f) { return split(f + ONE30); }
// back to units of 2^-61
OPX_HD OPX_INLINE i64 to_value(Fx x) { return ((i64)x.h << 31) + x.l; }

OPX_HD OPX_INLINE i64 bits_of(double x) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(x);
#else
    i64 b;
    memcpy(&b, &x, 8);
    return b;
#endif
}
OPX_HD OPX_INLINE double of_bits(i64 b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}
// x == 0 (an FP64 comparison would take the FP64 pipe)
OPX_HD OPX_INLINE bool is_zero(double x) { return (bits_of(x) << 1) == 0; }
OPX_HD OPX_INLINE int exponent_of(double x) { return (int)(bits_of(x) >> 52) & 0x7ff; }

// x 2^61 rounded to nearest (ties away), for |x| < 2 (fx_of: 2 - 2^-30); integer operations only
// (a double to integer conversion runs at the FP64 rate)
OPX_HD OPX_INLINE i64 fixed_of(double x) {
    const i64 b = bits_of(x);
    const int e = (int)(b >> 52) & 0x7ff;
    const uint64_t m = (((uint64_t)b & 0xfffffffffffffULL) | 0x10000000000000ULL) << 10;  // |x| = m 2^(e - 1085)
    const unsigned r0 = (unsigned)(1023 - e), r = r0 < 63u ? r0 : 63u;  // zero and subnormal x: 63; |x| >= 2 is the caller's to refuse
    const i64 g = (i64)(((m >> r) + 1) >> 1), s = b >> 63;
    return (g ^ s) - s;
}
OPX_HD OPX_INLINE Fx fx_of(double x) { return from_value(fixed_of(x)); }
// f 2^-61 (rounded to double once, by the conversion)
OPX_HD OPX_INLINE double double_of(i64 f) {
    const i64 b = bits_of((double)f);
    return of_bits(f != 0 ? b - (61LL << 52) : b);
}
// round to nearest integer of a double below 2^62 in magnitude
OPX_HD OPX_INLINE i64 round_of(double t) {
#ifdef __CUDA_ARCH__
    return __double2ll_rn(t);
#else
    return (i64)__builtin_llrint(t);
#endif
}
OPX_HD OPX_INLINE float approx(Fx x) { return (float)x.h * (1.0f / 1073741824.0f); }

OPX_HD OPX_INLINE int absor(int m, Fx x) { return m | (x.h ^ (x.h >> 31)); }

// The start of a sum at c (units of 2^-61), for pack()
OPX_HD OPX_INLINE Acc acc_at(i64 c) { return Acc{(c >> 1) + HALF30, ((c & 1) << 30) + HALF30}; }

// 2^61 / n! rounded, n <= 20
constexpr i64 fact_fx(int n) {
    uint64_t f = 1;
    for (int k = 2; k <= n; k++) f *= (uint64_t)k;
    return (i64)(((1ULL << 62) + f) / (2 * f));
}

// ------------------------------------------------------------------------ SU(2)
struct Q {
    Fx e[4];
};

// component c of A B, A = a or its adjoint, B likewise
template <bool CA, bool CB> OPX_HD OPX_INLINE void qterm(Acc &s, const Q &a, const Q &b, int i, int j, int sign) {
    const int sg = sign * (CA && i > 0 ? -1 : 1) * (CB && j > 0 ? -1 : 1);
    mac(s, sg > 0 ? a.e[i] : neg(a.e[i]), b.e[j]);
}
template <bool CA, bool CB> OPX_HD OPX_INLINE void qcomp(Acc &s, const Q &a, const Q &b, int c) {
    if (c == 0) {
        qterm<CA, CB>(s, a, b, 0, 0, 1);
        qterm<CA, CB>(s, a, b, 1, 1, -1);
        qterm<CA, CB>(s, a, b, 2, 2, -1);
        qterm<CA, CB>(s, a, b, 3, 3, -1);
    } else {
        const int d = c == 3 ? 1 : c + 1, f = c == 1 ? 3 : c - 1;  // (c, d, f) cyclic
        qterm<CA, CB>(s, a, b, 0, c, 1);
        qterm<CA, CB>(s, a, b, c, 0, 1);
        qterm<CA, CB>(s, a, b, d, f, -1);
        qterm<CA, CB>(s, a, b, f, d, 1);
    }
}
template <bool CA, bool CB> OPX_HD OPX_INLINE Q qmul(const Q &a, const Q &b) {
    Q r;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        Acc s = acc0();
        qcomp<CA, CB>(s, a, b, c);
        r.e[c] = pack(s);
    }
    return r;
}
// S += A B, S in units of 2^-60 (four unit terms stay below 2^62.1)
template <bool CA, bool CB> OPX_HD OPX_INLINE void qacc(i64 *S, const Q &a, const Q &b) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
        Acc s{S[c], ONE30};
        qcomp<CA, CB>(s, a, b, c);
        S[c] = s.a + (s.b >> 31);
    }
}
// A sum in units of 2^-60 as (h 2^-28 + l 2^-59): a product with it has units 2^-59
OPX_HD OPX_INLINE Fx quarter(i64 s60) { return from_value((s60 + 1) >> 1); }

// cos m and sin(m)/m of m^2 = m2 < 1/4 by their Taylor polynomials: six terms
// below 0.01 (the next one is below 2^-68), nine otherwise (below 2^-70)
OPX_HD OPX_INLINE void cos_sinc(Fx m2, Fx &c, Fx &s) {
    const bool small = m2.h < 10737418;  // 0.01
    Fx x{0, 0}, y{0, 0};
    if (!small) {
        x = from_value(fact_fx(16));
        y = from_value(fact_fx(17));
#pragma unroll
        for (int k = 7; k >= 6; k--) {
            Acc p = acc_at((k & 1) ? -fact_fx(2 * k) : fact_fx(2 * k)), q = acc_at((k & 1) ? -fact_fx(2 * k + 1) : fact_fx(2 * k + 1));
            mac(p, x, m2);
            mac(q, y, m2);
            x = pack(p);
            y = pack(q);
        }
    }
#pragma unroll
    for (int k = 5; k >= 0; k--) {
        Acc p = acc_at((k & 1) ? -fact_fx(2 * k) : fact_fx(2 * k)), q = acc_at((k & 1) ? -fact_fx(2 * k + 1) : fact_fx(2 * k + 1));
        mac(p, x, m2);
        mac(q, y, m2);
        x = pack(p);
        y = pack(q);
    }
    c = x;
    s = y;
}

// exp(i v_a sigma_a / 2) from t_a = (v_a / 2) 2^61 (not yet rounded); false
// where |v_a / 2| >= 1/2 (or is not finite) or m^2 = |v|^2 / 4 >= 1/4
OPX_HD OPX_INLINE bool qexp(const double *t, Q &X) {
    const int top = 1023 + 60;
    if (exponent_of(t[0]) >= top || exponent_of(t[1]) >= top || exponent_of(t[2]) >= top) return false;
    Fx w[3];
    Acc n = acc0();
#pragma unroll
    for (int a = 0; a < 3; a++) {
        w[a] = from_value(round_of(t[a]));
        mac(n, w[a], w[a]);
    }
    const Fx m2 = pack(n);
    if (m2.h >= (1 << 28)) return false;
    Fx c, s;
    cos_sinc(m2, c, s);
    X.e[0] = c;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        Acc p = acc0();
        mac(p, w[a], s);
        X.e[1 + a] = pack(p);
    }
    return true;
}

// ------------------------------------------------------------------------ SU(3)
struct M {
    Fx r[9], i[9];
};

// A row of a matrix.  The SU(3) kernels form products row by row, v -> v B, in a
// loop over the three rows, with B's entries read from the link arrays as they are
// used: a third of the code of whole matrix products (which overran the
// instruction cache and 168 registers).
struct Row {
    Fx r[3], i[3];
};
// component q of v B or (CB) v B^dagger; B(c) gives B's entry c = 3 row + column as (real, imaginary)
template <bool CB, class B> OPX_HD OPX_INLINE void rterm(Acc &re, Acc &im, const Row &v, const B &b, int q) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        Fx br, bi;
        b(CB ? 3 * q + k : 3 * k + q, br, bi);
        mac(re, v.r[k], br);
        mac(re, CB ? v.i[k] : neg(v.i[k]), bi);
        mac(im, CB ? neg(v.r[k]) : v.r[k], bi);
        mac(im, v.i[k], br);
    }
}
template <bool CB, class B> OPX_HD OPX_INLINE Row rmul(const Row &v, const B &b) {
    Row o;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        Acc re = acc0(), im = acc0();
        rterm<CB>(re, im, v, b, q);
        o.r[q] = pack(re);
        o.i[q] = pack(im);
    }
    return o;
}
// S += v B in units of 2^-60: S[q] real, S[3 + q] imaginary
template <bool CB, class B> OPX_HD OPX_INLINE void racc(i64 *S, const Row &v, const B &b) {
#pragma unroll
    for (int q = 0; q < 3; q++) {
        Acc re{S[q], ONE30}, im{S[3 + q], ONE30};
        rterm<CB>(re, im, v, b, q);
        S[q] = re.a + (re.b >> 31);
        S[3 + q] = im.a + (im.b >> 31);
    }
}
// Adds row r of a matrix (entries re, im in any one unit) to x_a = Im tr(lambda_a
// M), a < 7; x_7 collects the imaginary diagonal as its own three sums do: d0 + d1 in
// x_7, d2 in x_8
OPX_HD OPX_INLINE void proj_row(i64 *x, int r, const i64 *re, const i64 *im) {
    if (r == 0) {
        x[0] += im[1]; x[1] += re[1]; x[3] += im[2]; x[4] += re[2];
        x[2] += im[0]; x[7] += im[0];
    } else if (r == 1) {
        x[0] += im[0]; x[1] -= re[0]; x[5] += im[2]; x[6] += re[2];
        x[2] -= im[1]; x[7] += im[1];
    } else {
        x[3] += im[0]; x[4] -= re[0]; x[5] += im[1]; x[6] -= re[1];
        x[8] += im[2];
    }
}
// the eighth component times sqrt(3) / 2 (the halved sum stays in range)
OPX_HD OPX_INLINE i64 proj_eighth(const i64 *x) { return (x[7] >> 1) - x[8]; }

// exp(i H), H = v_a lambda_a / 2, from t_a = (v_a / 2) 2^61 (a < 7) and t_7 =
// (v_7 / (2 sqrt 3)) 2^61; false where an entry reaches 1/2 (or is not finite) or
// ||H||_F > 1.  H^3 = c1 H + c0 (Cayley-Hamilton), so the Taylor polynomial
// sum_k (i H)^k / k! by Horner's rule stays a quadratic q0 + q1 H + q2 H^2 in H
// with complex coefficients: one multiplication by H maps it to
// (c0 q2, q0 + c1 q2, q1).  As many terms as ||H||_F asks for: the first
// one left out is below 2^-63.
#ifdef __CUDACC__
static __constant__ i64 c_fact_fx[21] = {
    fact_fx(0), fact_fx(1), fact_fx(2), fact_fx(3), fact_fx(4), fact_fx(5), fact_fx(6), fact_fx(7), fact_fx(8), fact_fx(9), fact_fx(10),
    fact_fx(11), fact_fx(12), fact_fx(13), fact_fx(14), fact_fx(15), fact_fx(16), fact_fx(17), fact_fx(18), fact_fx(19), fact_fx(20)};
#endif
OPX_HD OPX_INLINE i64 fact_at(int k) {
#ifdef __CUDA_ARCH__
    return c_fact_fx[k];
#else
    return fact_fx(k);
#endif
}
OPX_HD OPX_INLINE bool mexp(const double *t, M &W) {
    int emax = 0;
#pragma unroll
    for (int a = 0; a < 8; a++) { const int e = exponent_of(t[a]); emax = e > emax ? e : emax; }
    if (emax >= 1023 + 59) return false;  // an entry |v_a / 2| >= 1/4: the norm below would pass 1 with the diagonal's sums
    const i64 g2 = round_of(t[2]), g7 = round_of(t[7]);
    const Fx d0 = from_value(g2 + g7), d1 = from_value(g7 - g2), d2 = from_value(-2 * g7);
    const Fx ur = from_value(round_of(t[0])), ui = neg(from_value(round_of(t[1])));
    const Fx vr = from_value(round_of(t[3])), vi = neg(from_value(round_of(t[4])));
    const Fx wr = from_value(round_of(t[5])), wi = neg(from_value(round_of(t[6])));
    Fx uu, vv, ww;
    { Acc s = acc0(); mac(s, ur, ur); mac(s, ui, ui); uu = pack(s); }
    { Acc s = acc0(); mac(s, vr, vr); mac(s, vi, vi); vv = pack(s); }
    { Acc s = acc0(); mac(s, wr, wr); mac(s, wi, wi); ww = pack(s); }
    // H^2: real diagonal; off-diagonal 01, 02, 12
    Fx q00, q11, q22, q01r, q01i, q02r, q02i, q12r, q12i;
    { Acc s = acc_at(to_value(uu) + to_value(vv)); mac(s, d0, d0); q00 = pack(s); }
    { Acc s = acc_at(to_value(uu) + to_value(ww)); mac(s, d1, d1); q11 = pack(s); }
    { Acc s = acc_at(to_value(vv) + to_value(ww)); mac(s, d2, d2); q22 = pack(s); }
    const i64 tr = to_value(q00) + to_value(q11) + to_value(q22);  // tr H^2 = ||H||_F^2
    if (tr > (1LL << 61)) return false;
    const Fx c1 = from_value((tr + 1) >> 1);
    // d_a + d_b = -d_c
    const Fx n0 = neg(d0), n1 = neg(d1), n2 = neg(d2);
    { Acc s = acc0(); mac(s, ur, n2); mac(s, vr, wr); mac(s, vi, wi); q01r = pack(s); }
    { Acc s = acc0(); mac(s, ui, n2); mac(s, vi, wr); mac(s, neg(vr), wi); q01i = pack(s); }
    { Acc s = acc0(); mac(s, vr, n1); mac(s, ur, wr); mac(s, neg(ui), wi); q02r = pack(s); }
    { Acc s = acc0(); mac(s, vi, n1); mac(s, ur, wi); mac(s, ui, wr); q02i = pack(s); }
    { Acc s = acc0(); mac(s, wr, n0); mac(s, ur, vr); mac(s, ui, vi); q12r = pack(s); }
    { Acc s = acc0(); mac(s, wi, n0); mac(s, ur, vi); mac(s, neg(ui), vr); q12i = pack(s); }
    // det H = tr H^3 / 3 = (H^2 H)_00-row expansion: d0 (d1 d2 - ww) - d1 vv - d2 uu + 2 Re(u w conj v)
    Fx c0;
    {
        Acc s = acc_at(-to_value(ww));
        mac(s, d1, d2);
        const Fx k0 = pack(s);
        Acc p = acc0();
        mac(p, wr, vr); mac(p, wi, vi);
        const Fx k1 = pack(p);
        Acc q = acc0();
        mac(q, wr, vi); mac(q, neg(wi), vr);
        const Fx k2 = pack(q);
        Acc z = acc0();
        mac(z, d0, k0);
        mac(z, n1, vv);
        mac(z, n2, uu);
        mac(z, ur, k1); mac(z, ur, k1);
        mac(z, ui, k2); mac(z, ui, k2);
        c0 = pack(z);
    }
    // terms: ||H||_F <= 1/8, 3/8, 1
    int K = tr <= (1LL << 55) ? 12 : (tr <= (9LL << 55) ? 16 : 20);
    Fx q0r{0, 0}, q0i{0, 0}, q1r{0, 0}, q1i{0, 0}, q2r{0, 0}, q2i{0, 0};
    q0r = from_value(fact_at(K));  // K is a multiple of four: i^K = 1
#pragma unroll 1
    for (; K > 0; K -= 4) {
#pragma unroll
        for (int u = 1; u <= 4; u++) {
            // i^(K - u): -i, -1, i, 1
            const i64 f = fact_at(K - u);
            Acc ar = acc_at(u == 2 ? -f : (u == 4 ? f : 0)), ai = acc_at(u == 1 ? -f : (u == 3 ? f : 0));
            mac(ar, c0, q2r);
            mac(ai, c0, q2i);
            Acc br = acc_at(to_value(q0r)), bi = acc_at(to_value(q0i));
            mac(br, c1, q2r);
            mac(bi, c1, q2i);
            q2r = q1r; q2i = q1i;
            q1r = pack(br); q1i = pack(bi);
            q0r = pack(ar); q0i = pack(ai);
        }
    }
    auto diag = [&](int k, Fx d, Fx q) {
        Acc r = acc_at(to_value(q0r)), i = acc_at(to_value(q0i));
        mac(r, q1r, d); mac(r, q2r, q);
        mac(i, q1i, d); mac(i, q2i, q);
        W.r[k] = pack(r);
        W.i[k] = pack(i);
    };
    diag(0, d0, q00);
    diag(4, d1, q11);
    diag(8, d2, q22);
    auto off = [&](int k, int kt, Fx hr, Fx hi, Fx qr, Fx qi) {
        Acc a = acc0(), b = acc0(), c = acc0(), d = acc0();
        mac(a, q1r, hr); mac(a, q2r, qr); b = a;
        mac(a, neg(q1i), hi); mac(a, neg(q2i), qi);   // Re upper
        mac(b, q1i, hi); mac(b, q2i, qi);             // Re lower
        mac(c, q1i, hr); mac(c, q2i, qr); d = c;
        mac(c, q1r, hi); mac(c, q2r, qi);             // Im upper
        mac(d, neg(q1r), hi); mac(d, neg(q2r), qi);   // Im lower
        W.r[k] = pack(a); W.i[k] = pack(c);
        W.r[kt] = pack(b); W.i[kt] = pack(d);
    };
    off(1, 3, ur, ui, q01r, q01i);
    off(2, 6, vr, vi, q02r, q02i);
    off(5, 7, wr, wi, q12r, q12i);
    return true;
}

// ------------------------------------------------------------------------ links from doubles
// Whether a link's entries (all below 2 in magnitude) form a unitary matrix to LINK_TOL
OPX_HD OPX_INLINE bool usable(const Q &q) {
    float n = 0.f;
#pragma unroll
    for (int c = 0; c < 4; c++) n += approx(q.e[c]) * approx(q.e[c]);
    return fabsf(n - 1.f) <= LINK_TOL;
}
OPX_HD OPX_INLINE bool usable(const M &m) {
    float dev = 0.f;
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
        for (int q = 0; q <= p; q++) {
            float re = p == q ? -1.f : 0.f, im = 0.f;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float ar = approx(m.r[3 * k + p]), ai = approx(m.i[3 * k + p]), br = approx(m.r[3 * k + q]), bi = approx(m.i[3 * k + q]);
                re += ar * br + ai * bi;
                im += ar * bi - ai * br;
            }
            dev = fmaxf(dev, fmaxf(fabsf(re), fabsf(im)));
        }
    return dev <= LINK_TOL;
}

template <int NC> struct LinkOf;
template <> struct LinkOf<2> {
    typedef Q T;
    static constexpr int NG = 4;
};
template <> struct LinkOf<3> {
    typedef M T;
    static constexpr int NG = 18;
};
OPX_HD OPX_INLINE Fx &entry(Q &q, int c) { return q.e[c]; }
OPX_HD OPX_INLINE Fx &entry(M &m, int c) { return c < 9 ? m.r[c] : m.i[c - 9]; }
OPX_HD OPX_INLINE Fx first(const Q &q) { return q.e[0]; }
OPX_HD OPX_INLINE Fx first(const M &m) { return m.r[0]; }

// A link's entries in fixed point; where the link is not usable its first
// entry's h is LINK_BAD (a usable one's is at least -1.01 2^30)
template <int NC> OPX_HD OPX_INLINE typename LinkOf<NC>::T link_of(const double *u) {
    typename LinkOf<NC>::T m;
    bool ok = true;
#pragma unroll
    for (int c = 0; c < LinkOf<NC>::NG; c++) {
        ok = ok && exponent_of(u[c]) <= 1023;
        entry(m, c) = fx_of(u[c]);
    }
    if (!(ok && usable(m))) entry(m, 0).h = LINK_BAD;
    return m;
}

// The largest entry off the identity (a bound within a factor of two, units of 2^-30; zero for
// the identity): below WEAK_H, the link lies within 2^-7 of it
OPX_HD OPX_INLINE int offdiag(const Q &q) { return absor(absor(absor(0, q.e[1]), q.e[2]), q.e[3]); }
OPX_HD OPX_INLINE int offdiag(const M &m) {
    int o = absor(absor(absor(0, m.i[0]), m.i[4]), m.i[8]);
#pragma unroll
    for (int k = 0; k < 9; k++)
        if (k != 0 && k != 4 && k != 8) o = absor(absor(o, m.r[k]), m.i[k]);
    return o;
}

#ifdef __CUDACC__
// Fixed-point links in global memory: the layout of the FP64 links, an entry's
// eight bytes holding (l, h).  SU(3) links have a word of flags each behind them,
// [3][sites padded to 32]: what the update asks of every link of a stencil before it
// forms a product (45 loads a thread from the entries themselves).  A bit per entry
// off the identity (flag_bit): below 2^-14, and (ZERO_SHIFT) exactly zero as a double.
constexpr unsigned SMALL_MASK = 0x7fff, LINK_WEAK = 1u << 30, FLAG_BAD = 1u << 31;
constexpr int ZERO_SHIFT = 15;
// entries 1, 2, 3, 5, 6, 7 (real), 9 .. 17 (imaginary) to bits 0 .. 14
__host__ __device__ constexpr int flag_bit(int c) { return c >= 9 ? c - 3 : (c > 4 ? c - 2 : c - 1); }
// bytes of an array of fixed-point links
__host__ __device__ inline size_t fixed_links_bytes(long V, int ng) {
    return (size_t)link_elems(V, ng) * 8 + (ng == 18 ? (size_t)link_blocks(V) * 32 * 3 * sizeof(unsigned) : 0);
}
template <int NC, typename I> struct FxLinks;
template <typename I> struct FxLinks<2, I> {
    const int2 *p;
    I V;
    __device__ __forceinline__ Q load(int d, I s) const {
        const int4 *b = reinterpret_cast<const int4 *>(p + link_offset_t<I>(V, 4, d, 0, s));
        const int4 x = __ldg(b), y = __ldg(b + 1);
        return Q{{{x.y, x.x}, {x.w, x.z}, {y.y, y.x}, {y.w, y.z}}};
    }
};
// the entries of one link in memory
struct FxEntries {
    const int2 *b;
    __device__ __forceinline__ Fx at(int c) const {
        const int2 x = __ldg(b + 32 * c);
        return Fx{x.y, x.x};
    }
    __device__ __forceinline__ void operator()(int c, Fx &re, Fx &im) const {
        re = at(c);
        im = at(9 + c);
    }
    // row r, and row r of the adjoint
    __device__ __forceinline__ Row row(int r) const {
        Row v;
#pragma unroll
        for (int k = 0; k < 3; k++) (*this)(3 * r + k, v.r[k], v.i[k]);
        return v;
    }
    __device__ __forceinline__ Row adj_row(int r) const {
        Row v;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            (*this)(3 * k + r, v.r[k], v.i[k]);
            v.i[k] = neg(v.i[k]);
        }
        return v;
    }
    __device__ __forceinline__ int mark() const { return __ldg(b).y; }  // h of the first entry: LINK_BAD or not
};
template <typename I> struct FxLinks<3, I> {
    const int2 *p;
    I V;
    __device__ __forceinline__ unsigned flags(int d, I s) const {
        const I n = ((V + 31) >> 5) << 5;
        return __ldg(reinterpret_cast<const unsigned *>(p + 54 * n) + ((I)d * n + s));
    }
    __device__ __forceinline__ FxEntries at(int d, I s) const { return FxEntries{p + link_offset_t<I>(V, 18, d, 0, s)}; }
    __device__ __forceinline__ M load(int d, I s) const {
        const int2 *b = p + link_offset_t<I>(V, 18, d, 0, s);
        M m;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const int2 x = __ldg(b + k * 32), y = __ldg(b + (9 + k) * 32);
            m.r[k] = Fx{x.y, x.x};
            m.i[k] = Fx{y.y, y.x};
        }
        return m;
    }
};

// The entries u of link (d, s) in fixed point into out
template <int NC, typename I>
__device__ __forceinline__ void write_fixed(const double *u, int2 *out, I V, int d, I s) {
    constexpr int NG = LinkOf<NC>::NG;
    const I o = link_offset_t<I>(V, NG, d, 0, s);
    auto m = link_of<NC>(u);
    if constexpr (NC == 2) {
        int4 *q = reinterpret_cast<int4 *>(out + o);
        q[0] = make_int4(m.e[0].l, m.e[0].h, m.e[1].l, m.e[1].h);
        q[1] = make_int4(m.e[2].l, m.e[2].h, m.e[3].l, m.e[3].h);
    } else {
#pragma unroll
        for (int c = 0; c < NG; c++) {
            const Fx x = entry(m, c);
            out[o + 32 * c] = make_int2(x.l, x.h);
        }
        unsigned flags = entry(m, 0).h == LINK_BAD ? FLAG_BAD : 0u;
        int all = 0, least = SMALL_H;
#pragma unroll
        for (int c = 1; c < NG; c++) {
            if (c == 4 || c == 8) continue;
            const int h = abs(entry(m, c).h);
            all |= h;
            least = min(least, h);
        }
        if (all < WEAK_H) flags |= LINK_WEAK;
        if (least < SMALL_H) {  // hardly ever
#pragma unroll
            for (int c = 1; c < NG; c++) {
                if (c == 4 || c == 8) continue;
                const unsigned bit = 1u << flag_bit(c);
                if (abs(entry(m, c).h) < SMALL_H) flags |= is_zero(u[c]) ? bit | bit << ZERO_SHIFT : bit;
            }
        }
        const I n = ((V + 31) >> 5) << 5;
        reinterpret_cast<unsigned *>(out + 54 * n)[(I)d * n + s] = flags;
    }
}
// Link (d, s) of U (double, or float: widened) in fixed point into out
template <int NC, typename R, typename I>
__device__ __forceinline__ void fixed_link(const R *U, int2 *out, I V, int d, I s) {
    constexpr int NG = LinkOf<NC>::NG;
    double u[NG];
    const I o = link_offset_t<I>(V, NG, d, 0, s);
    if constexpr (NC == 2 && sizeof(R) == 8) {
        const double2 *b = reinterpret_cast<const double2 *>(U + o);
        const double2 x = b[0], y = b[1];
        u[0] = x.x; u[1] = x.y; u[2] = y.x; u[3] = y.y;
    } else if constexpr (NC == 2) {
        const float4 x = *reinterpret_cast<const float4 *>(U + o);
        u[0] = x.x; u[1] = x.y; u[2] = x.z; u[3] = x.w;
    } else {
#pragma unroll
        for (int c = 0; c < NG; c++) u[c] = (double)U[o + 32 * c];
    }
    write_fixed<NC, I>(u, out, V, d, s);
}

// One link per thread (blockIdx.y its direction)
template <int NC, typename R>
__global__ void __launch_bounds__(128) k_fixed_links(const R *__restrict__ U, int2 *__restrict__ out, Lat L) {
    const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < L.V) fixed_link<NC, R, long>(U, out, L.V, (int)blockIdx.y, s);
}
#endif

}  // namespace fx
}  // namespace opx
