// ic_kernels.cu -- seeded synthetic initial conditions on the device.
//
// The reference has no Gauss-projecting initializer; the synthetic benchmark
// lattices need one.  Links U_i(x) = exp(i A_i^a(x) t_a) with A ~ N(0, sigma_a^2)
// per generator component, E_i^a(x) ~ N(0, sigma_e^2), then E is projected onto
// Gauss's law (Grid.getGaussConstraint, Grid.java:944-968) by conjugate
// gradients on the covariant Laplacian:
//     div(divT mu) = rho - div E,   E <- E + divT mu,
// (div E)(x)   = sum_i c_i [E_i(x) - Ad(U_i(x-i)^dagger) E_i(x-i)],
// (divT l)_i(x) = c_i [l(x) - Ad(U_i(x)) l(x+i)],  c_i = 1/(a_i g a_i),
// divT being the adjoint of div.  Everything here runs in FP64; an FP32 handle
// receives the rounded result.  The random numbers use the same counter-based
// recipe as the CPU oracle (splitmix64 finaliser, Box-Muller), so both sides
// draw the same A and E.
#include <algorithm>

#include "cg_loop.h"
#include "internal.h"
#include "ksum.cuh"
#include "observables.cuh"
#include "transport_fx.cuh"

namespace opx {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}
__device__ __forceinline__ double unif(uint64_t seed, uint64_t ctr) {
    uint64_t h = mix64(seed ^ mix64(ctr));
    return ((double)(h >> 11) + 0.5) * (1.0 / 9007199254740992.0);
}
__device__ __forceinline__ double normal(uint64_t seed, uint64_t ctr) {
    double u1 = unif(seed, 2 * ctr), u2 = unif(seed, 2 * ctr + 1);
    return sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
}

template <int NC>
__global__ void k_init_random(double *__restrict__ U, double *__restrict__ E, Lat L, uint64_t seed, double sa,
                              double se) {
    using G = typename GroupOf<NC, double>::T;
    constexpr int NA = G::NA;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;  // t = s*3 + d
    if (t >= L.V * 3) return;
    const long s = t / 3;
    const int d = (int)(t - s * 3);
    double A[NA], e[NA];
    const uint64_t baseA = 0ull << 40, baseE = 1ull << 40;
#pragma unroll
    for (int a = 0; a < NA; a++) {
        A[a] = sa * normal(seed, baseA + (uint64_t)(t * NA + a));
        e[a] = se * normal(seed, baseE + (uint64_t)(t * NA + a));
    }
    const LinkPlanes<G, double> Up{U, L.V};
    const AlgPlanes<NA, double> Ep{E, L.V};
    Up.store(d, s, G::expi(A));
    Ep.store(d, s, e);
}

template <int NC>
__global__ void k_div(const double *__restrict__ U, const double *__restrict__ El, Lat L, double *__restrict__ out) {
    using G = typename GroupOf<NC, double>::T;
    constexpr int NA = G::NA;
    const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= L.V) return;
    const LinkPlanes<G, double> Up{const_cast<double *>(U), L.V};
    const AlgPlanes<NA, double> Ep{const_cast<double *>(El), L.V};
    int x[3];
    site_coords(L, s, x);
    const Nbr nb = neighbours(L, s, x);
    double acc[NA];
#pragma unroll
    for (int a = 0; a < NA; a++) acc[a] = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double ci = 1.0 / (L.a[i] * L.g * L.a[i]);
        double e0[NA], e1[NA], t[NA];
        Ep.load_ro(i, s, e0);
        Ep.load_ro(i, nb.bwd[i], e1);
        G::act(e1, G::adj(Up.load(i, nb.bwd[i])), t);
#pragma unroll
        for (int a = 0; a < NA; a++) acc[a] += ci * (e0[a] - t[a]);
    }
    const AlgPlanes<NA, double> Op{out, L.V};
    Op.store(0, s, acc);
}

template <int NC>
__global__ void k_divT(const double *__restrict__ U, const double *__restrict__ l, Lat L, double *__restrict__ out,
                       int accumulate) {
    using G = typename GroupOf<NC, double>::T;
    constexpr int NA = G::NA;
    const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= L.V) return;
    const LinkPlanes<G, double> Up{const_cast<double *>(U), L.V};
    const AlgPlanes<NA, double> Lp{const_cast<double *>(l), L.V};
    const AlgPlanes<NA, double> Op{out, L.V};
    int x[3];
    site_coords(L, s, x);
    const Nbr nb = neighbours(L, s, x);
    double l0[NA];
    Lp.load_ro(0, s, l0);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double ci = 1.0 / (L.a[i] * L.g * L.a[i]);
        double l1[NA], t[NA], o[NA];
        Lp.load_ro(0, nb.fwd[i], l1);
        G::act(l1, Up.load(i, s), t);
        if (accumulate) Op.load(i, s, o);
#pragma unroll
        for (int a = 0; a < NA; a++) o[a] = (accumulate ? o[a] : 0.0) + ci * (l0[a] - t[a]);
        Op.store(i, s, o);
    }
}

__global__ void k_to_float(const double *__restrict__ src, float *__restrict__ dst, long n) {
    const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) dst[k] = (float)src[k];
}
int ic_init_random(Ctx &c, uint64_t seed, double sigma_a, double sigma_e) {
    const long V = c.L.V;
    const size_t nU = (size_t)link_elems(V, c.ng), nE = (size_t)V * 3 * c.na;
    double *U64 = nullptr, *E64 = nullptr;
    const bool f32 = c.prec == OPX_F32;
    if (f32) {
        if (dev_malloc(c, &U64, nU * 8) != cudaSuccess || dev_malloc(c, &E64, nE * 8) != cudaSuccess) {
            cudaFree(U64);
            c.err = "opx_init_random: cannot allocate FP64 scratch";
            return OPX_ERR_NOMEM;
        }
    } else {
        U64 = (double *)c.U;
        E64 = (double *)c.E;
    }
    const int B = 256;
    if (c.nc == 2) k_init_random<2><<<grid_for(V * 3, B), B, 0, c.stream>>>(U64, E64, c.L, seed, sigma_a, sigma_e);
    else k_init_random<3><<<grid_for(V * 3, B), B, 0, c.stream>>>(U64, E64, c.L, seed, sigma_a, sigma_e);
    c.launches++;
    if (f32) {
        k_to_float<<<grid_for((long)nU, B), B, 0, c.stream>>>(U64, (float *)c.U, (long)nU);
        k_to_float<<<grid_for((long)nE, B), B, 0, c.stream>>>(E64, (float *)c.E, (long)nE);
        c.launches += 2;
        cudaStreamSynchronize(c.stream);
        cudaFree(U64);
        cudaFree(E64);
    }
    return OPX_OK;
}

// div and divT on FP64 fields with the FP64 links U64 (NA components per site)
void ic_div(Ctx &c, const double *U64, const double *El, double *o) {
    if (c.nc == 2) k_div<2><<<grid_for(c.L.V, 128), 128, 0, c.stream>>>(U64, El, c.L, o);
    else k_div<3><<<grid_for(c.L.V, 128), 128, 0, c.stream>>>(U64, El, c.L, o);
    c.launches++;
}
void ic_divT(Ctx &c, const double *U64, const double *l, double *o, int acc) {
    if (c.nc == 2) k_divT<2><<<grid_for(c.L.V, 128), 128, 0, c.stream>>>(U64, l, c.L, o, acc);
    else k_divT<3><<<grid_for(c.L.V, 128), 128, 0, c.stream>>>(U64, l, c.L, o, acc);
    c.launches++;
}

// ---- conjugate gradients on K = div divT ----
// One iteration is three launches without a word from the host: the direction
// p = r + beta p, its gradient t_i = p - Ad(U_i) p(x+i) with the sum of c_i^2 t_i^2
// (= p K p, divT being the transpose of div), and r -= alpha div(c^2 t), mu += alpha p
// with the sum of r^2.  The last block of a sum forms the next scalar; once done is
// set the launches that follow return at once, and the host looks at it eight
// iterations behind.  Transports in fixed point (transport_fx.cuh).
// 64^3 SU(3): 1.6 -> 0.26 ms an iteration (0.38 ms of it were two one-thread sums of
// 608 partials, 1.2 ms the FP64 pipe, the rest host round trips).
struct CgState {
    double rr, pAp, alpha, beta, stop;
    int done, it, maxit, pad;
};
static_assert(sizeof(CgState) <= 64, "two states fit the handle's sixteen pinned doubles");

// The block's sum of v (its warps' in order) to part[block]; the last block to finish
// returns true on every thread with the total of all blocks
__device__ __forceinline__ bool grid_sum(double v, double *part, unsigned *count, double &total) {
    __shared__ double ws[3];
    __shared__ bool last;
    __shared__ double tot;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0) ws[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = (ws[0] + ws[1]) + ws[2];
        part[2 * blockIdx.x + 1] = 0.0;
        __threadfence();
        last = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    if (w == 0) {
        const double t = warp_sum_pairs(part, (int)gridDim.x, 2);
        if (lane == 0) {
            tot = t;
            *count = 0u;
        }
    }
    __syncthreads();
    total = tot;
    return true;
}

// p = r + beta p
__global__ void __launch_bounds__(256) k_cg_direction(const CgState *st, const double *__restrict__ r, double *__restrict__ p, long n) {
    if (st->done) return;
    const double b = st->beta;
    for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) p[k] = fma(b, p[k], r[k]);
}

// Three warps share 32 sites, warp i of them taking link i (as the BulkQuantities
// pass).  FINAL: E_i += c_i t_i to Eout (the handle's E) and, in FP64, to t.
template <int NC, typename R, bool FINAL>
__global__ void __launch_bounds__(96, 4)
    k_cg_gradient(CgState *st, const int2 *__restrict__ Uf, const R *__restrict__ U, const double *__restrict__ p,
                  const __grid_constant__ Lat L, int fixed, double *__restrict__ t, R *__restrict__ Eout, double *__restrict__ part,
                  unsigned *__restrict__ count) {
    constexpr int NA = NC == 2 ? 3 : 8;
    if (!FINAL && st->done) return;
    const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
    const double ci = LatR<double>::gfac(L, i);
    const AlgPlanes<NA, double> Pp{const_cast<double *>(p), L.V}, Tp{t, L.V};
    KSum acc{0.0, 0.0};
    double sum = 0.0;
    int run = 0;
    for (long g = blockIdx.x; g < (L.V + 31) >> 5; g += gridDim.x) {
        const long s = g * 32 + lane;
        if (s < L.V) {
            int x[3];
            site_coords<long>(L, s, x);
            const Deltas<long> D = deltas<long>(L, x);
            double l0[NA], l1[NA], r[NA];
            Pp.load_ro(0, s, l0);
            Pp.load_ro(0, s + D.f(i), l1);
            const fx::FxLinks<NC, long> W{Uf, L.V};
            const auto u = W.load(i, s);
            const bool fx_ok = fixed && fx::transportable(u);
            if constexpr (NC == 2) fx::minus_transported<NC, true, R>(u, fx_ok, U, L, s, i, l0, l1, r);
            else fx::minus_transported<NC, true, R>(W.at(i, s), fx_ok, U, L, s, i, l0, l1, r);
            if (FINAL) {
#pragma unroll
                for (int a = 0; a < NA; a++) {
                    const long o = ((long)i * NA + a) * L.V + s;
                    r[a] = fma(ci, r[a], (double)Eout[o]);
                    Eout[o] = (R)r[a];
                }
            } else {
                sum += sqr<double, NA>(r);
            }
            Tp.store(i, s, r);
        }
        if ((++run & 31) == 0) { two_sum_add(acc, sum); sum = 0.0; }
    }
    if (FINAL) return;
    double total;
    if (grid_sum(((acc.s + sum) + acc.c) * (ci * ci), part, count, total) && threadIdx.x == 0) {
        st->pAp = total;
        if (total > 0.0) st->alpha = st->rr / total;
        else st->done = 1;
    }
}

// d = sum_i w_i (t_i(x) - Ad(U_i(x-i)^dagger) t_i(x-i)):
//   CG_STEP   r -= alpha d, mu += alpha p (w = c^2), the sum of r^2
//   CG_BEGIN  r = p = rho - d, mu = 0 (t = E, w = c), the sum of r^2
//   CG_END    the sum of (rho - d)^2 alone
enum { CG_STEP, CG_BEGIN, CG_END };
template <int NC, typename R, typename RT, int MODE>
__global__ void __launch_bounds__(96, 4)
    k_cg_divergence(CgState *st, const int2 *__restrict__ Uf, const R *__restrict__ U, const RT *__restrict__ t,
                    const R *__restrict__ rho, const __grid_constant__ Lat L, int fixed, double *__restrict__ r,
                    double *__restrict__ p, double *__restrict__ mu, double *__restrict__ part, unsigned *__restrict__ count) {
    constexpr int NA = NC == 2 ? 3 : 8;
    __shared__ double gt[2][3][NA][32];
    if (MODE == CG_STEP && st->done) return;
    const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
    const double alpha = MODE == CG_STEP ? st->alpha : 0.0;
    const AlgPlanes<NA, RT> Tp{const_cast<RT *>(t), L.V};
    KSum acc{0.0, 0.0};
    double sum = 0.0;
    int run = 0;
    for (long g = blockIdx.x; g < (L.V + 31) >> 5; g += gridDim.x) {
        const long s = g * 32 + lane;
        if (s < L.V) {
            int x[3];
            site_coords<long>(L, s, x);
            const Deltas<long> D = deltas<long>(L, x);
            const long sm = s + D.b(i);
            RT a0[NA], a1[NA];
            double e0[NA], e1[NA], d[NA];
            Tp.load_ro(i, s, a0);
            Tp.load_ro(i, sm, a1);
#pragma unroll
            for (int a = 0; a < NA; a++) { e0[a] = (double)a0[a]; e1[a] = (double)a1[a]; }
            const fx::FxLinks<NC, long> W{Uf, L.V};
            const auto u = W.load(i, sm);
            const bool fx_ok = fixed && fx::transportable(u);
            if constexpr (NC == 2) fx::minus_transported<NC, false, R>(u, fx_ok, U, L, sm, i, e0, e1, d);
            else fx::minus_transported<NC, false, R>(W.at(i, sm), fx_ok, U, L, sm, i, e0, e1, d);
#pragma unroll
            for (int a = 0; a < NA; a++) gt[run & 1][i][a][lane] = d[a];
        }
        __syncthreads();
        if (s < L.V) {
#pragma unroll
            for (int a = 0; a < NA; a++) {
                if (a % 3 != i) continue;
                double d = 0.0;
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const double c = LatR<double>::gfac(L, j);
                    d = fma(gt[run & 1][j][a][lane], MODE == CG_STEP ? c * c : c, d);
                }
                const long o = (long)a * L.V + s;
                double v;
                if (MODE == CG_STEP) {
                    v = fma(-alpha, d, r[o]);
                    r[o] = v;
                    mu[o] = fma(alpha, p[o], mu[o]);
                } else {
                    v = (rho ? (double)rho[o] : 0.0) - d;
                    if (MODE == CG_BEGIN) {
                        r[o] = v;
                        p[o] = v;
                        mu[o] = 0.0;
                    }
                }
                sum = fma(v, v, sum);
            }
        }
        if ((++run & 31) == 0) { two_sum_add(acc, sum); sum = 0.0; }
    }
    double total;
    if (grid_sum((acc.s + sum) + acc.c, part, count, total) && threadIdx.x == 0) {
        if (MODE == CG_STEP) {
            st->beta = total / st->rr;
            st->rr = total;
            st->it++;
            if (!(total > st->stop) || st->it >= st->maxit) st->done = 1;
        } else if (MODE == CG_BEGIN) {
            st->rr = total;
            st->beta = 0.0;
            if (!(total > st->stop) || st->maxit <= 0) st->done = 1;
        } else {
            st->pAp = total;
        }
    }
}

// r = p = b, mu = 0, the sum of b^2; stop = (stop |b|)^2
__global__ void __launch_bounds__(96) k_cg_start(CgState *st, const double *__restrict__ b, long n, double *__restrict__ r, double *__restrict__ p,
                                                 double *__restrict__ mu, double *__restrict__ part, unsigned *__restrict__ count) {
    KSum acc{0.0, 0.0};
    for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
        const double v = b[k];
        r[k] = v;
        p[k] = v;
        mu[k] = 0.0;
        two_sum_add(acc, v * v);
    }
    double total;
    if (grid_sum(acc.s + acc.c, part, count, total) && threadIdx.x == 0) {
        st->rr = total;
        st->beta = 0.0;
        st->stop = st->stop * st->stop * total;
        if (!(total > st->stop) || !(total > 0.0) || st->maxit <= 0) st->done = 1;
    }
}

namespace {

// The solver's buffers (one allocation) and launches for the links U of type R
template <int NC, typename R> struct Cg {
    Ctx &c;
    const R *U;
    const int2 *Uf = nullptr;
    char *arena = nullptr;
    double *r = nullptr, *p = nullptr, *mu = nullptr, *t = nullptr, *part = nullptr;
    CgState *st = nullptr;
    unsigned *count = nullptr;
    int blocks = 1, fixed = 1, maxit = 0;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    static constexpr int MAX_BLOCKS = 4 * 152;  // resident at once

    Cg(Ctx &c_, const R *U_) : c(c_), U(U_) {}
    ~Cg() {
        for (cudaEvent_t e : ev) if (e) cudaEventDestroy(e);
        if (arena) cudaFree(arena);
    }
    // mu_out: where the solution goes (null: a buffer of its own)
    bool begin(double *mu_out, double stop, int maxit_) {
        maxit = maxit_;
        const long V = c.L.V, ns = V * c.na;
        // With the handle's own fixed-point links the arena has none; without room for it
        // these are given back, and without room for its own an FP64 solve goes without:
        // the FP64 products of every link, Uf the doubles, which nothing then looks at (an FP32
        // solve keeps its array, an FP64 one's size, in any case)
        bool own = sizeof(R) == 8 && (const void *)U == c.U && c.fixed_kernel;
        size_t links = 0;
        auto take_arena = [&]() {
            links = own || (sizeof(R) == 8 && !fixed) ? 0 : fx::fixed_links_bytes(V, c.ng);
            const size_t n = sizeof(double) * (size_t)(2 * ns + (mu_out ? 0 : ns) + 3 * ns) + links + sizeof(double) * 2 * MAX_BLOCKS + 512;
            if (cudaMalloc((void **)&arena, n) == cudaSuccess) return true;
            cudaGetLastError();
            arena = nullptr;
            return false;
        };
        fixed = c.fp64_only ? 0 : 1;
        if (!take_arena()) {
            const bool given = drop_fixed_links(c);
            own = false;
            if (!(given && take_arena()) && sizeof(R) == 8) {
                fixed = 0;
                take_arena();
            }
        }
        if (!arena || cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        char *q = arena;
        auto take = [&](size_t bytes) { char *x = q; q += (bytes + 15) & ~size_t(15); return x; };
        int2 *f = (int2 *)take(links);
        r = (double *)take(8 * ns);
        p = (double *)take(8 * ns);
        mu = mu_out ? mu_out : (double *)take(8 * ns);
        t = (double *)take(24 * ns);
        part = (double *)take(16 * MAX_BLOCKS);
        st = (CgState *)take(sizeof(CgState));
        count = (unsigned *)take(sizeof(unsigned));
        if (own) {
            ensure_fixed_links(c, true, false);
            Uf = (const int2 *)c.fx_U;
        } else if (!links) {
            Uf = (const int2 *)U;
        } else {
            fx::k_fixed_links<NC, R><<<dim3(grid_for(V, 128), 3), 128, 0, c.stream>>>(U, f, c.L);
            c.launches++;
            Uf = f;
        }
        blocks = (int)std::min<long>((V + 31) / 32, MAX_BLOCKS);
        CgState *h = (CgState *)c.red_host;
        *h = CgState{0.0, 0.0, 0.0, 0.0, stop, 0, 0, maxit, 0};
        cudaMemcpyAsync(st, h, sizeof(CgState), cudaMemcpyHostToDevice, c.stream);
        cudaMemsetAsync(count, 0, sizeof(unsigned), c.stream);
        cudaStreamSynchronize(c.stream);  // the pinned state is free again
        return true;
    }
    // iterations until done; the first error of the runtime
    cudaError_t iterate() {
        constexpr int STEPS = 8;
        CgState *h = (CgState *)c.red_host;
        const long ns = c.L.V * c.na;
        cudaError_t err = cudaSuccess;
        auto queue = [&](long k) {
            for (int j = 0; j < STEPS; j++) {
                k_cg_direction<<<std::min(grid_for(ns, 256), 8 * 152), 256, 0, c.stream>>>(st, r, p, ns);
                k_cg_gradient<NC, R, false><<<blocks, 96, 0, c.stream>>>(st, Uf, U, p, c.L, fixed, t, nullptr, part, count);
                k_cg_divergence<NC, R, double, CG_STEP><<<blocks, 96, 0, c.stream>>>(st, Uf, U, t, nullptr, c.L, fixed, r, p, mu, part, count);
            }
            c.launches += 3 * STEPS;
            cudaMemcpyAsync((char *)h + 64 * (k & 1), st, sizeof(CgState), cudaMemcpyDeviceToHost, c.stream);
            cudaEventRecord(ev[k & 1], c.stream);
            return (err = cudaGetLastError()) == cudaSuccess;
        };
        auto look = [&](long k) {
            if ((err = cudaEventSynchronize(ev[k & 1])) != cudaSuccess) return CG_FAILED;
            return ((const CgState *)((const char *)h + 64 * (k & 1)))->done ? CG_DONE : CG_GOES_ON;
        };
        cg_batches(std::max<long>(1, ((long)maxit + STEPS - 1) / STEPS), queue, look);
        return err;
    }
    CgState read() {
        CgState *h = (CgState *)c.red_host;
        cudaStreamSynchronize(c.stream);
        cudaMemcpyAsync(h, st, sizeof(CgState), cudaMemcpyDeviceToHost, c.stream);
        cudaStreamSynchronize(c.stream);
        return *h;
    }
};

template <int NC, typename R> int project_t(Ctx &c, double tol, int maxit, int *iters, double *final_g2) {
    const double V = (double)c.L.V;
    Cg<NC, R> cg(c, (const R *)c.U);
    if (!cg.begin(nullptr, tol * 1e-4 * V, maxit)) { c.err = "opx_gauss_project: out of device memory"; return OPX_ERR_NOMEM; }
    const R *rho = c.rho_nonzero ? (const R *)c.rho : nullptr;
    k_cg_divergence<NC, R, R, CG_BEGIN><<<cg.blocks, 96, 0, c.stream>>>(cg.st, cg.Uf, cg.U, (const R *)c.E, rho, c.L, cg.fixed, cg.r, cg.p, cg.mu,
                                                                        cg.part, cg.count);
    cudaError_t e = cg.iterate();
    const CgState s = cg.read();
    if (e != cudaSuccess) { c.err = std::string("opx_gauss_project: ") + cudaGetErrorString(e); return OPX_ERR_CUDA; }
    // E <- E + divT mu, and the residual recomputed from the projected field
    k_cg_gradient<NC, R, true><<<cg.blocks, 96, 0, c.stream>>>(cg.st, cg.Uf, cg.U, cg.mu, c.L, cg.fixed, cg.t, (R *)c.E, cg.part, cg.count);
    k_cg_divergence<NC, R, double, CG_END><<<cg.blocks, 96, 0, c.stream>>>(cg.st, cg.Uf, cg.U, cg.t, rho, c.L, cg.fixed, nullptr, nullptr, nullptr,
                                                                           cg.part, cg.count);
    c.launches += 3;
    const double g2 = cg.read().pAp / V;
    e = cudaGetLastError();
    if (iters) *iters = s.it;
    if (final_g2) *final_g2 = g2;
    if (e != cudaSuccess) { c.err = std::string("opx_gauss_project: ") + cudaGetErrorString(e); return OPX_ERR_CUDA; }
    return OPX_OK;
}

template <int NC> int solve_t(Ctx &c, const double *U64, const double *b, double *x, double tol_rel, int maxit, int *iters) {
    Cg<NC, double> cg(c, U64);
    if (!cg.begin(x, tol_rel, maxit)) { c.err = "covariant Laplacian solve: out of device memory"; return OPX_ERR_NOMEM; }
    k_cg_start<<<cg.blocks, 96, 0, c.stream>>>(cg.st, b, c.L.V * c.na, cg.r, cg.p, cg.mu, cg.part, cg.count);
    c.launches++;
    cudaError_t e = cg.iterate();
    const CgState s = cg.read();
    if (e == cudaSuccess) e = cudaGetLastError();
    if (iters) *iters = s.it;
    if (e != cudaSuccess) { c.err = std::string("covariant Laplacian solve: ") + cudaGetErrorString(e); return OPX_ERR_CUDA; }
    if (s.rr > s.stop && s.rr > 0) { c.err = "covariant Laplacian solve: no convergence"; return OPX_ERR_NUMERIC; }
    return OPX_OK;
}

}  // namespace

// x = K^+ b for the covariant Laplacian K = div divT of the links U64, by
// conjugate gradients from x = 0 until |r| <= tol_rel |b| (b in the range of
// div, so the iterates stay orthogonal to K's null space).
int ic_covariant_solve(Ctx &c, const double *U64, const double *b, double *x, double tol_rel, int maxit,
                       int *iters) {
    return c.nc == 2 ? solve_t<2>(c, U64, b, x, tol_rel, maxit, iters) : solve_t<3>(c, U64, b, x, tol_rel, maxit, iters);
}

int ic_gauss_project(Ctx &c, double tol, int maxit, int *iters, double *final_g2) {
    if (c.nc == 2) return c.prec == OPX_F64 ? project_t<2, double>(c, tol, maxit, iters, final_g2) : project_t<2, float>(c, tol, maxit, iters, final_g2);
    return c.prec == OPX_F64 ? project_t<3, double>(c, tol, maxit, iters, final_g2) : project_t<3, float>(c, tol, maxit, iters, final_g2);
}

}  // namespace opx
