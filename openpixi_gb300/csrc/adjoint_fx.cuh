// adjoint_fx.cuh -- the reverse step of the SU(2) leapfrog with its staples and
// gather products on the integer pipe (fixed.cuh).
//
// The cotangent of a staple sum is Sbar_i(x) = U_i(x)^* M_i(x) with the pure quaternion
// M_i = (0, 2 dt Ebar_i), so what the gather needs of each link is three numbers,
// not four, and its twelve terms share factors.  For link (y, k) and another
// direction i, z = y - i, T = U_k(y+i) U_i(y+k)^*, V = U_k(z) U_i(z+k):
//   Wbar_k(y) += [-c_k M_i(y) U_i(y) - c_i U_i(y) M_k(y+i)] T + c_k U_i(y) T M_i(y+k)
//              + U_i(z)^* { [c_k M_i(z) - c_i M_k(z)] V - c_k U_k(z) M_i(z+k) U_i(z+k) }
// (ten products, half of them with a zero scalar part, for the twelve of the terms taken one by
// one; no unitarity is assumed).  The M that a thread reads are scaled by one
// power of two; equal spacings, so the c are one factor at the end.
#pragma once
#include "leapfrog_fx.cuh"
#include "transport_fx.cuh"

namespace opx {
namespace fx {

typedef SU2<double> G2d;
typedef Q2<double> Qd;

// (0, m) q and q (0, m), the products of SU2GroupElement.mult
__device__ __forceinline__ Qd left_mul(const double *m, const Qd &q) {
    return Qd{{-(m[0] * q.e[1] + m[1] * q.e[2] + m[2] * q.e[3]), m[0] * q.e[0] - m[1] * q.e[3] + m[2] * q.e[2],
               m[1] * q.e[0] - m[2] * q.e[1] + m[0] * q.e[3], m[2] * q.e[0] - m[0] * q.e[2] + m[1] * q.e[1]}};
}
__device__ __forceinline__ Qd right_mul(const Qd &q, const double *m) {
    return Qd{{-(m[0] * q.e[1] + m[1] * q.e[2] + m[2] * q.e[3]), m[0] * q.e[0] + m[1] * q.e[3] - m[2] * q.e[2],
               m[1] * q.e[0] + m[2] * q.e[1] - m[0] * q.e[3], m[2] * q.e[0] + m[0] * q.e[2] - m[1] * q.e[1]}};
}

// The staple sum S_i(s) (with 1/a_j^2) of the links W, in doubles; false where the update
// would refuse the link (leapfrog_fx.cuh)
template <typename I>
__device__ __forceinline__ bool staple_sum_fx(const FxLinks<2, I> W, const double *__restrict__ U, const Lat &L, I s, const Deltas<I> &D, int i, Qd &S) {
    const Q Ui = W.load(i, s);
    const int j1 = i == 2 ? 0 : i + 1, j2 = i == 0 ? 2 : i - 1;
    const Q Uj1 = W.load(j1, s), Uj2 = W.load(j2, s);
    const int small = small_components(Ui, Uj1, Uj2);
    if (small && !zero_in_stencil<I>(U, L, s, small)) return false;
    int worst = min(min(Ui.e[0].h, Uj1.e[0].h), Uj2.e[0].h);
    auto load = [&](int d, I t) {
        const Q q = W.load(d, t);
        worst = min(worst, q.e[0].h);
        return q;
    };
    const I pi = s + D.f(i);
    i64 F[4] = {0, 0, 0, 0};
#pragma unroll
    for (int jj = 0; jj < 2; jj++) {
        const int j = jj ? j2 : j1;
        const I bj = D.b(j);
        qacc<false, true>(F, qmul<false, true>(load(j, pi), load(i, s + D.f(j))), jj ? Uj2 : Uj1);
        qacc<true, false>(F, qmul<false, false>(load(i, s + bj), load(j, pi + bj)), load(j, s + bj));
    }
    const double c = L.inva2[0] * 0x1p-60;
#pragma unroll
    for (int a = 0; a < 4; a++) S.e[a] = (double)F[a] * c;
    return worst != LINK_BAD;
}

// C += A B or (CA) A^* B, the components of a running sum
template <bool CA> __device__ __forceinline__ void qadd(Acc *s, const Q &a, const Q &b) {
#pragma unroll
    for (int c = 0; c < 4; c++) qcomp<CA, false>(s[c], a, b, c);
}
__device__ __forceinline__ Q qpack(Acc *s) {
    Q q;
#pragma unroll
    for (int c = 0; c < 4; c++) q.e[c] = pack(s[c]);
    return q;
}
// a pure quaternion from three scaled numbers (units 2^-61)
__device__ __forceinline__ Q pure_of(const i64 *m) { return Q{{Fx{0, 0}, from_value(m[0]), from_value(m[1]), from_value(m[2])}}; }

// Pass 2 of the reverse step: Wbar_k(y) from Uown and the staples that the link
// enters, one link per thread.  FP64 pipe bound before (64^3 0.60 ms), the
// integer pipes' issue slots now (0.069 ms).
template <typename I>
__global__ void __launch_bounds__(128, 4)
k_adj_gather_fx(const int2 *__restrict__ Wf, const double *__restrict__ Wd, const double *__restrict__ Mv,
                const double *__restrict__ Uown, const __grid_constant__ Lat L, int fixed, double *__restrict__ Wbar_prev) {
    const unsigned chunk = blockIdx.x / 3u;
    const int k = (int)(blockIdx.x - 3u * chunk);
    const I y = (I)chunk * (I)blockDim.x + (I)threadIdx.x;
    if (y >= (I)L.V) return;
    int x[3];
    site_coords<I>(L, y, x);
    const Deltas<I> D = deltas<I>(L, x);
    const FxLinks<2, I> W{Wf, (I)L.V};
    const AlgPlanes<3, double, I> Mp{const_cast<double *>(Mv), (I)L.V};
    const LinkPlanes<G2d, double, I> Wp{const_cast<double *>(Wd), (I)L.V}, UO{const_cast<double *>(Uown), (I)L.V}, OUT{Wbar_prev, (I)L.V};
    const I ypk = y + D.f(k);
    Qd out = UO.load(k, y);
    // the largest exponent of the M that enter, and their components that are not all zero
    int emax = 0, worst = 0;
    unsigned some[3] = {0u, 0u, 0u};
    auto see = [&](int d, I s) {
        double m[3];
        Mp.load_ro(d, s, m);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int e = exponent_of(m[a]);
            emax = e > emax ? e : emax;
            some[a] |= (unsigned)__double2loint(m[a]) | ((unsigned)__double2hiint(m[a]) << 1);
        }
    };
#pragma unroll
    for (int ii = 1; ii < 3; ii++) {
        const int i = k + ii >= 3 ? k + ii - 3 : k + ii;
        const I z = y + D.b(i);
        see(i, y);
        see(k, y + D.f(i));
        see(i, ypk);
        see(i, z);
        see(k, z);
        see(i, z + D.f(k));
    }
    if (!(some[0] | some[1] | some[2])) {
        OUT.store(k, y, out);
        return;
    }
    bool ok = fixed && emax >= 64 && emax < 0x7ff;
    if (ok) {
        // a component that is small in the links keeps its digits only if it is zero in all (as in
        // the update; links near the identity lose none: M itself is of order one)
        const int small = small_components<false>(W.load(0, y), W.load(1, y), W.load(2, y));
        if (small) {
            const int nonzero = (some[0] ? 1 : 0) | (some[1] ? 2 : 0) | (some[2] ? 4 : 0);
            if ((small & nonzero) || !zero_in_stencil<I>(Wd, L, y, small)) ok = false;
        }
    }
    if (ok) {
        auto mval = [&](int d, I s, i64 *v) {  // below 1/4 in units of 2^-61
            double m[3];
            Mp.load_ro(d, s, m);
#pragma unroll
            for (int a = 0; a < 3; a++) v[a] = to_value(fx_below(m[a], emax, 3));
        };
        auto load = [&](int d, I t) {
            const Q q = W.load(d, t);
            worst = min(worst, q.e[0].h);
            return q;
        };
        i64 sum[4] = {0, 0, 0, 0};  // units of 2^-60
#pragma unroll 1
        for (int ii = 1; ii < 3; ii++) {
            const int i = k + ii >= 3 ? k + ii - 3 : k + ii;
            const I z = y + D.b(i), ypi = y + D.f(i), zpk = z + D.f(k);
            i64 a[3], b[3];
            {
                const Q T = qmul<false, true>(load(k, ypi), load(i, ypk)), Ui = load(i, y);
                // -M_i(y) U_i(y) - U_i(y) M_k(y+i)
                mval(i, y, a);
                mval(k, ypi, b);
#pragma unroll
                for (int c = 0; c < 3; c++) { a[c] = -a[c]; b[c] = -b[c]; }
                Acc X[4] = {acc0(), acc0(), acc0(), acc0()};
                qadd<false>(X, pure_of(a), Ui);
                qadd<false>(X, Ui, pure_of(b));
                qacc<false, false>(sum, qpack(X), T);
                mval(i, ypk, a);
                qacc<false, false>(sum, qmul<false, false>(Ui, T), pure_of(a));
            }
            {
                const Q Uk = load(k, z), Ui = load(i, zpk);
                mval(i, z, a);
                mval(k, z, b);
#pragma unroll
                for (int c = 0; c < 3; c++) a[c] -= b[c];
                Acc X[4] = {acc0(), acc0(), acc0(), acc0()};
                qadd<false>(X, pure_of(a), qmul<false, false>(Uk, Ui));
                mval(i, zpk, b);
#pragma unroll
                for (int c = 0; c < 3; c++) b[c] = -b[c];
                qadd<false>(X, qmul<false, false>(Uk, pure_of(b)), Ui);
                qacc<true, false>(sum, load(i, z), qpack(X));
            }
        }
        ok = worst != LINK_BAD;
        if (ok) {
            const double u = of_bits((i64)(emax - 57) << 52) * L.inva2[0];
#pragma unroll
            for (int c = 0; c < 4; c++) out.e[c] = fma((double)sum[c], u, out.e[c]);
        }
    }
    if (!ok) {
#pragma unroll 1
        for (int ii = 1; ii < 3; ii++) {
            const int i = k + ii >= 3 ? k + ii - 3 : k + ii;
            const I z = y + D.b(i), ypi = y + D.f(i), zpk = z + D.f(k);
            const double ck = LatR<double>::inva2(L, k), ci = LatR<double>::inva2(L, i);
            double a[3], b[3];
            const Qd T = G2d::mul_adj(Wp.load(k, ypi), Wp.load(i, ypk)), Ui = Wp.load(i, y);
            Mp.load_ro(i, y, a);
            Mp.load_ro(k, ypi, b);
#pragma unroll
            for (int c = 0; c < 3; c++) { a[c] *= -ck; b[c] *= -ci; }
            Qd X = left_mul(a, Ui);
            G2d::add(X, right_mul(Ui, b));
            G2d::add(out, G2d::mul(X, T));
            Mp.load_ro(i, ypk, a);
#pragma unroll
            for (int c = 0; c < 3; c++) a[c] *= ck;
            G2d::add(out, right_mul(G2d::mul(Ui, T), a));
            const Qd Uk = Wp.load(k, z), Uz = Wp.load(i, zpk);
            Mp.load_ro(i, z, a);
            Mp.load_ro(k, z, b);
#pragma unroll
            for (int c = 0; c < 3; c++) a[c] = ck * a[c] - ci * b[c];
            X = left_mul(a, G2d::mul(Uk, Uz));
            Mp.load_ro(i, zpk, b);
#pragma unroll
            for (int c = 0; c < 3; c++) b[c] *= -ck;
            G2d::add(X, G2d::mul(right_mul(Uk, b), Uz));
            G2d::add(out, G2d::adj_mul(Wp.load(i, z), X));
        }
    }
    OUT.store(k, y, out);
}

}  // namespace fx
}  // namespace opx
