"""The error of FP64 runs against the same run in extended precision (numpy's long
double: 64 or 113 bits): with the group products in fixed point no larger than with
every product in FP64, for links, E and the BulkQuantities rows.

Both forms round the stored links and E to doubles every step; the comparison is of
the two root-mean-square errors of the same run, with 5 % and, for the rows (the
mean of seven columns of the size of half a unit in the last place), 2^-53 left for
chance."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu

C, W = np.clongdouble, np.longdouble


def generators(nc):
    if nc == 2:
        m = [[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]]
    else:
        m = [[[0, 1, 0], [1, 0, 0], [0, 0, 0]], [[0, -1j, 0], [1j, 0, 0], [0, 0, 0]], [[1, 0, 0], [0, -1, 0], [0, 0, 0]],
             [[0, 0, 1], [0, 0, 0], [1, 0, 0]], [[0, 0, -1j], [0, 0, 0], [1j, 0, 0]], [[0, 0, 0], [0, 0, 1], [0, 1, 0]],
             [[0, 0, 0], [0, 0, -1j], [0, 1j, 0]], [[1, 0, 0], [0, 1, 0], [0, 0, -2]]]
    t = np.array(m, C)
    if nc == 3:
        t[7] /= np.sqrt(W(3))
    return t / 2


def mul(a, b):
    o = a[:, 0:1] * b[0:1]
    for k in range(1, a.shape[1]):
        o = o + a[:, k:k + 1] * b[k:k + 1]
    return o


def adj(a):
    return np.conj(np.swapaxes(a, 0, 1))


def herm(x, t):
    return sum(t[a][(...,) + (None,) * 3] * x[a][None, None] for a in range(len(t)))


def expi(h):
    one = np.eye(h.shape[0], dtype=C).reshape(h.shape[:2] + (1,) * 3)
    o = one + C(1j) * h / 26
    for k in range(25, 0, -1):
        o = one + mul(C(1j) * h / k, o)
    return o


def roll(x, d, o):
    return np.roll(x, -o, axis=x.ndim - 3 + d)


def trace(m, t):
    n = m.shape[0]
    return np.stack([2 * sum(t[a][i, j] * m[j, i] for i in range(n) for j in range(n) if t[a][i, j] != 0) for a in range(len(t))])


def force(U, i, t):
    S = 0
    for j in range(3):
        if j != i:
            S = S + mul(mul(roll(U[j], i, 1), adj(roll(U[i], j, 1))), adj(U[j]))
            Uj = roll(U[j], j, -1)
            S = S + mul(adj(mul(roll(U[i], j, -1), roll(Uj, i, 1))), Uj)
    return trace(mul(U[i], S), t).imag


def links_step(U, E, dt, t):
    return [mul(expi(herm(-dt * E[i], t)), U[i]) for i in range(3)]


def plaquette(U, j, k):
    return mul(mul(mul(U[j], roll(U[k], j, 1)), adj(roll(U[j], k, 1))), adj(U[k]))


def row(U, Un, E, t):
    V = U[0][0, 0].size
    sq = lambda x: (x * x).sum()  # noqa: E731
    b2 = [sq(trace(plaquette(u, (d + 1) % 3, (d + 2) % 3), t).imag) for u in (U, Un) for d in range(3)]
    act = lambda x, u: trace(mul(mul(adj(u), herm(x, t)), u), t).real  # noqa: E731
    G = sum(E[i] - roll(act(E[i], U[i]), i, -1) for i in range(3))
    return np.array([sq(E[d]) / V for d in range(3)] + [(b2[d] + b2[3 + d]) / V / 2 for d in range(3)] + [sq(G) / V], W)


def as_links(U):
    o = []
    for u in U:
        u = u.reshape(u.shape[0], u.shape[1], -1)
        if u.shape[0] == 2:
            o.append(np.stack([u[0, 0].real, u[0, 1].imag, u[0, 1].real, u[0, 0].imag]))
        else:
            m = u.reshape(9, -1)
            o.append(np.concatenate([m.real, m.imag]))
    return np.ascontiguousarray(np.stack(o).transpose(2, 0, 1))


def as_gen(E):
    return np.ascontiguousarray(np.stack([e.reshape(e.shape[0], -1) for e in E]).transpose(2, 0, 1))


def rms(a, b):
    d = a.reshape(b.shape).astype(W) - b
    return float(np.sqrt((d * d).sum() / (b * b).sum()))


@pytest.mark.parametrize("nc,dims,sigma,steps,seed", [(3, (6, 5, 7), 0.2, 6, 1), (3, (6, 5, 7), 0.1, 3, 2), (2, (7, 6, 8), 0.1, 12, 3),
                                                      (2, (7, 6, 8), 0.5, 6, 4)])
def test_error_is_no_larger_than_fp64_products(native, monkeypatch, nc, dims, sigma, steps, seed):
    if np.finfo(W).nmant < 63:
        pytest.skip("long double is not wider than double here")
    t = generators(nc)
    rng = np.random.default_rng(seed)
    U, E = [], []
    for _ in range(3):
        U.append(expi(herm(rng.normal(0, sigma, (len(t),) + dims).astype(W), t)).astype(np.complex128))
        E.append(rng.normal(0, sigma, (len(t),) + dims))
    got = []
    for only in (True, False):
        if only:
            monkeypatch.setenv("OPX_FP64_ONLY", "1")
        else:
            monkeypatch.delenv("OPX_FP64_ONLY")
        h = opx.Handle(nc, dims, a=1.0, dt=0.05, g=1.0, precision=N.OPX_F64)
        h.upload(N.FIELD_U, as_links(U))
        h.upload(N.FIELD_E, as_gen(E), layout=N.LAYOUT_GEN)
        h.initialize()
        rows = [list(o.e2) + list(o.b2) + [o.gauss] for o in h.step_measured(steps)]
        got.append((h.download(N.FIELD_UNEXT), h.download(N.FIELD_E, layout=N.LAYOUT_GEN), np.array(rows)))
    dt = W(0.05)
    U, E = [u.astype(C) for u in U], [e.astype(W) for e in E]
    Un, rows = links_step(U, E, dt, t), []
    for _ in range(steps):
        U = Un
        E = [E[i] + dt * force(U, i, t) for i in range(3)]
        Un = links_step(U, E, dt, t)
        rows.append(row(U, Un, E, t))
    want = (as_links(Un), as_gen(E), np.stack(rows))
    (u0, e0, r0), (u1, e1, r1) = ([rms(x, y) for x, y in zip(g, want)] for g in got)
    print(f"SU({nc}) {dims} links {u0:.3e} -> {u1:.3e}  E {e0:.3e} -> {e1:.3e}  rows {r0:.3e} -> {r1:.3e}")
    assert u1 <= 1.05 * u0 and e1 <= 1.05 * e0
    assert r1 <= r0 + 2.0 ** -53
