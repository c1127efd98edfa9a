// Host check of the fixed-point group arithmetic (fixed.cuh) against long
// double: conversions at the edges of their range, the products with each
// operand plain or adjoint, the staple sums, the projection and the exponentials.
//
// Bound of one product's entry: operands off by at most 2^-62 each (a row and a
// column of up to six reals of norm one: 2 sqrt 6 2^-62), the dropped low
// products (6 2^-62), the shifts and the rounding (3 2^-61): below 2^-58.
#include <cmath>
#include <cstdio>
#include <complex>

#include "../openpixi_gb300/csrc/fixed.cuh"

using namespace opx;
typedef long double Wide;
typedef std::complex<Wide> C;

static unsigned long long rng = 0x9E3779B97F4A7C15ULL;
static double uni() {
    rng = rng * 6364136223846793005ULL + 1442695040888963407ULL;
    return (double)(rng >> 11) / 9007199254740992.0 * 2 - 1;
}
static int bad = 0;
static void need(bool ok, const char *what, double a = 0, double b = 0) {
    if (!ok) { bad++; std::printf("wrong: %s %.17g %.17g\n", what, a, b); }
}
static Wide val(fx::i64 f) { return std::ldexp((Wide)f, -61); }
static Wide val(fx::Fx x) { return std::ldexp((Wide)x.h, -30) + std::ldexp((Wide)x.l, -61); }

template <int N> struct Mat { C m[N][N]; };
template <int N> static Mat<N> mul(const Mat<N> &a, const Mat<N> &b) {
    Mat<N> c;
    for (int i = 0; i < N; i++)
        for (int j = 0; j < N; j++) { c.m[i][j] = 0; for (int k = 0; k < N; k++) c.m[i][j] += a.m[i][k] * b.m[k][j]; }
    return c;
}
template <int N> static Mat<N> adj(const Mat<N> &a) {
    Mat<N> c;
    for (int i = 0; i < N; i++) for (int j = 0; j < N; j++) c.m[i][j] = std::conj(a.m[j][i]);
    return c;
}
static Mat<2> of(const Wide *e) { return {{{C(e[0], e[3]), C(e[2], e[1])}, {C(-e[2], e[1]), C(e[0], -e[3])}}}; }
static Mat<3> of3(const double *u) { Mat<3> m; for (int k = 0; k < 9; k++) m.m[k / 3][k % 3] = C(u[k], u[9 + k]); return m; }
// exp(i H) by its series in long double
template <int N> static Mat<N> expi(const Mat<N> &H) {
    Mat<N> r = {}, t = {};
    for (int i = 0; i < N; i++) r.m[i][i] = t.m[i][i] = 1;
    for (int k = 1; k < 40; k++) {
        t = mul(t, H);
        for (int i = 0; i < N; i++) for (int j = 0; j < N; j++) { t.m[i][j] *= C(0, 1) / (Wide)k; r.m[i][j] += t.m[i][j]; }
    }
    return r;
}
template <typename T> static Mat<3> herm(const T *x) {
    const Wide r = 1 / std::sqrt((Wide)3);
    Mat<3> h;
    h.m[0][0] = ((Wide)x[2] + r * x[7]) / (Wide)2; h.m[1][1] = (r * x[7] - (Wide)x[2]) / (Wide)2; h.m[2][2] = -r * x[7];
    h.m[0][1] = C(x[0], -x[1]) / (Wide)2; h.m[0][2] = C(x[3], -x[4]) / (Wide)2; h.m[1][2] = C(x[5], -x[6]) / (Wide)2;
    h.m[1][0] = std::conj(h.m[0][1]); h.m[2][0] = std::conj(h.m[0][2]); h.m[2][1] = std::conj(h.m[1][2]);
    return h;
}

static const Wide TOL = std::ldexp((Wide)1, -58);

static void su2(double w) {
    double e[2][4];
    for (auto &q : e) {
        double n = 0;
        q[0] = 1;
        for (int c = 1; c < 4; c++) q[c] = w * uni();
        for (int c = 0; c < 4; c++) n += q[c] * q[c];
        for (int c = 0; c < 4; c++) q[c] /= std::sqrt(n);
    }
    const fx::Q a = fx::link_of<2>(e[0]), b = fx::link_of<2>(e[1]);
    need(a.e[0].h != fx::LINK_BAD && b.e[0].h != fx::LINK_BAD, "a unitary link is usable");
    Wide u[4], v[4];
    for (int c = 0; c < 4; c++) { u[c] = e[0][c]; v[c] = e[1][c]; need(std::fabs(val(a.e[c]) - u[c]) <= std::ldexp((Wide)1, -62), "conversion", e[0][c]); }
    const Mat<2> A = of(u), B = of(v);
    auto cmp = [&](const fx::Q &q, const Mat<2> &M, const char *what) {
        const Wide r[4] = {M.m[0][0].real(), M.m[0][1].imag(), M.m[0][1].real(), M.m[0][0].imag()};
        for (int c = 0; c < 4; c++) need(std::fabs(val(q.e[c]) - r[c]) < TOL, what, (double)val(q.e[c]), (double)r[c]);
    };
    cmp(fx::qmul<false, false>(a, b), mul(A, B), "a b");
    cmp(fx::qmul<true, false>(a, b), mul(adj(A), B), "a* b");
    cmp(fx::qmul<false, true>(a, b), mul(A, adj(B)), "a b*");
    cmp(fx::qmul<true, true>(a, b), mul(adj(A), adj(B)), "a* b*");
    fx::i64 S[4] = {0, 0, 0, 0};
    for (int k = 0; k < 4; k++) fx::qacc<false, true>(S, a, b);
    const Mat<2> P = mul(A, adj(B));
    for (int c = 0; c < 4; c++) {
        const Wide r[4] = {P.m[0][0].real(), P.m[0][1].imag(), P.m[0][1].real(), P.m[0][0].imag()};
        need(std::fabs(std::ldexp((Wide)S[c], -60) - 4 * r[c]) < 4 * TOL, "sum of four");
        need(std::fabs(4 * val(fx::quarter(S[c])) - 4 * r[c]) < 5 * TOL, "quarter");
    }
    double x[3], t[3];
    for (int k = 0; k < 3; k++) { x[k] = w * uni(); t[k] = std::ldexp(x[k] / 2, 61); }
    fx::Q X;
    const Wide m2 = ((Wide)x[0] * x[0] + (Wide)x[1] * x[1] + (Wide)x[2] * x[2]) / 4;
    const bool ok = fx::qexp(t, X);
    need(ok == (m2 < 0.25 && std::fabs(x[0]) < 1 && std::fabs(x[1]) < 1 && std::fabs(x[2]) < 1) || std::fabs(m2 - 0.25) < 1e-8, "range of the exponential", (double)m2);
    if (ok) {
        const Wide m = std::sqrt(m2), s = m > 0 ? std::sin(m) / m : 1, r[4] = {std::cos(m), s * x[0] / 2, s * x[1] / 2, s * x[2] / 2};
        for (int c = 0; c < 4; c++) need(std::fabs(val(X.e[c]) - r[c]) < TOL, "exp", (double)val(X.e[c]), (double)r[c]);
    }
}

static void su3(double w) {
    double u[2][18], x[8], t[8];
    Mat<3> A[2];
    for (int k = 0; k < 2; k++) {
        for (double &c : x) c = w * uni();
        const Mat<3> E = expi(herm(x));
        for (int c = 0; c < 9; c++) { u[k][c] = (double)E.m[c / 3][c % 3].real(); u[k][9 + c] = (double)E.m[c / 3][c % 3].imag(); }
        A[k] = of3(u[k]);
    }
    const fx::M a = fx::link_of<3>(u[0]), b = fx::link_of<3>(u[1]);
    need(a.r[0].h != fx::LINK_BAD && b.r[0].h != fx::LINK_BAD, "a unitary matrix is usable");
    auto cmp = [&](const fx::M &f, const Mat<3> &M, const char *what) {
        for (int k = 0; k < 9; k++) {
            need(std::fabs(val(f.r[k]) - M.m[k / 3][k % 3].real()) < TOL, what, (double)val(f.r[k]), (double)M.m[k / 3][k % 3].real());
            need(std::fabs(val(f.i[k]) - M.m[k / 3][k % 3].imag()) < TOL, what, (double)val(f.i[k]), (double)M.m[k / 3][k % 3].imag());
        }
    };
    // products row by row: row r of A or (dag) A^dagger times B or B^dagger
    auto entries = [](const fx::M &m) { return [&m](int k, fx::Fx &re, fx::Fx &im) { re = m.r[k]; im = m.i[k]; }; };
    auto row = [](const fx::M &m, int r, bool dag) {
        fx::Row v;
        for (int k = 0; k < 3; k++) {
            const int x = dag ? 3 * k + r : 3 * r + k;
            v.r[k] = m.r[x];
            v.i[k] = dag ? fx::neg(m.i[x]) : m.i[x];
        }
        return v;
    };
    fx::M c, d, f;
    fx::i64 S[18] = {};
    for (int r = 0; r < 3; r++) {
        const fx::Row ab = fx::rmul<false>(row(a, r, false), entries(b)), db = fx::rmul<false>(row(a, r, true), entries(b)),
                      bd = fx::rmul<true>(row(a, r, false), entries(b));
        for (int q = 0; q < 3; q++) {
            c.r[3 * r + q] = ab.r[q]; c.i[3 * r + q] = ab.i[q];
            d.r[3 * r + q] = db.r[q]; d.i[3 * r + q] = db.i[q];
            f.r[3 * r + q] = bd.r[q]; f.i[3 * r + q] = bd.i[q];
        }
        fx::i64 T[6] = {};
        for (int k = 0; k < 4; k++) { if (k & 1) fx::racc<false>(T, row(a, r, true), entries(b)); else fx::racc<true>(T, row(a, r, false), entries(b)); }
        for (int q = 0; q < 3; q++) { S[3 * r + q] = T[q]; S[9 + 3 * r + q] = T[3 + q]; }
    }
    cmp(c, mul(A[0], A[1]), "A B");
    cmp(d, mul(adj(A[0]), A[1]), "A* B");
    cmp(f, mul(A[0], adj(A[1])), "A B*");
    const Mat<3> P = mul(adj(A[0]), A[1]), Q = mul(A[0], adj(A[1]));
    for (int k = 0; k < 9; k++) {
        const C r = (Wide)2 * (P.m[k / 3][k % 3] + Q.m[k / 3][k % 3]);
        need(std::fabs(std::ldexp((Wide)S[k], -60) - r.real()) < 4 * TOL && std::fabs(std::ldexp((Wide)S[9 + k], -60) - r.imag()) < 4 * TOL, "sum of four matrices");
        fx::entry(c, k) = fx::quarter(S[k]);
        fx::entry(c, 9 + k) = fx::quarter(S[9 + k]);
    }
    // proj of A times the quarter of that sum
    fx::i64 p[9] = {};
    for (int r = 0; r < 3; r++) {
        const fx::Row v = row(a, r, false);
        fx::i64 re[3], im[3];
        for (int q = 0; q < 3; q++) {
            fx::Acc x = fx::acc0v(), y = fx::acc0v();
            fx::rterm<false>(x, y, v, entries(c), q);
            re[q] = fx::value(x);
            im[q] = fx::value(y);
        }
        fx::proj_row(p, r, re, im);
    }
    p[7] = fx::proj_eighth(p);
    Mat<3> R = {};
    for (int i = 0; i < 3; i++) for (int j = 0; j < 3; j++) R.m[i][j] = (P.m[i][j] + Q.m[i][j]) / (Wide)2;
    R = mul(A[0], R);
    const Wide pr[8] = {R.m[0][1].imag() + R.m[1][0].imag(), R.m[0][1].real() - R.m[1][0].real(), R.m[0][0].imag() - R.m[1][1].imag(),
                      R.m[0][2].imag() + R.m[2][0].imag(), R.m[0][2].real() - R.m[2][0].real(), R.m[1][2].imag() + R.m[2][1].imag(),
                      R.m[1][2].real() - R.m[2][1].real(), (R.m[0][0].imag() + R.m[1][1].imag()) / 2 - R.m[2][2].imag()};
    for (int k = 0; k < 8; k++) need(std::fabs(val(p[k]) - pr[k]) < 8 * TOL, "proj", (double)val(p[k]), (double)pr[k]);
    Wide n2 = 0, top = 0;
    for (int k = 0; k < 8; k++) {
        x[k] = w * uni();
        t[k] = std::ldexp(x[k] / 2, 61);
        n2 += (Wide)x[k] * x[k] / 2;
        if (k == 7) t[k] /= std::sqrt(3.0);
        top = std::fmax(top, std::fabs(t[k]));
    }
    const bool ok = fx::mexp(t, c);
    need(ok == (n2 <= 1 && top < std::ldexp((Wide)1, 59)) || std::fabs(n2 - 1) < 1e-8, "range of the matrix exponential", (double)n2);
    // the matrix that t stands for (t_7 is a rounded double)
    Wide y[8];
    for (int k = 0; k < 8; k++) y[k] = std::ldexp((Wide)t[k], -60) * (k == 7 ? std::sqrt((Wide)3) : (Wide)1);
    if (ok) cmp(c, expi(herm(y)), "matrix exp");
}

int main() {
    // conversions: exact where the double has no bit below 2^-61, half-away rounding, zero, subnormal
    const double exact[] = {0.0, -0.0, 1.0, -1.0, 0.5, 1.99, -1.99, std::ldexp(1.0, -61), -std::ldexp(3.0, -61), 1.0 / 3, -0.7};
    for (double d : exact) need(val(fx::fixed_of(d)) == (Wide)d && val(fx::fx_of(d)) == (Wide)d, "exact conversion", d);
    need(fx::fixed_of(std::ldexp(1.0, -62)) == 1 && fx::fixed_of(-std::ldexp(1.0, -62)) == -1 && fx::fixed_of(std::ldexp(0.999, -62)) == 0, "rounding");
    need(fx::fixed_of(5e-324) == 0 && fx::fixed_of(1e-300) == 0, "tiny");
    for (double d : {1.0, -0.3, 1e-3, std::ldexp(1.0, -61)}) need(fx::double_of(fx::fixed_of(d)) == d || std::fabs(d) < 1e-2, "back to double", d);
    need(fx::double_of(0) == 0.0, "zero back");
    // links that are not usable: not unitary, too large, not finite
    const double nan = std::nan(""), inf = HUGE_VAL;
    for (double d : {1.01, 2.0, 1e9, nan, inf, -inf, 0.0}) {
        const double q[4] = {d, 0, 0, 0};
        double m[18] = {d, 0, 0, 0, 1, 0, 0, 0, 1};
        need(fx::link_of<2>(q).e[0].h == fx::LINK_BAD, "quaternion refused", d);
        need(fx::link_of<3>(m).r[0].h == fx::LINK_BAD, "matrix refused", d);
    }
    const double one[4] = {1, 0, 0, 0}, skew[18] = {1, 0.01, 0, 0, 1, 0, 0, 0, 1};
    need(fx::link_of<2>(one).e[0].h == 1 << 30 && fx::offdiag(fx::link_of<2>(one)) == 0, "identity");
    need(fx::link_of<3>(skew).r[0].h == fx::LINK_BAD, "rows that are not orthogonal");
    for (int k = 0; k < 20000; k++) { su2(0.01 + 0.3 * (k % 8)); }
    for (int k = 0; k < 3000; k++) { su3(0.01 + 0.15 * (k % 8)); }
    su2(0.0);
    su3(0.0);
    if (bad) return 1;
    std::printf("ok\n");
    return 0;
}
