"""FP64 steps of fields whose colour components are of very different size: the small
ones keep their relative accuracy, as products in FP64 keep it.

One component (SU(2): of the algebra; SU(3): a few of the eight) is of order 0.1, the
others of size eps.  A small component of a product of FP64 numbers is a sum of terms
each proportional to small factors, rounded to 2^-53 of themselves, so two FP64 forms of
three steps differ by some tens of such roundings of its largest value; 2^-40 of it
bounds what a form in another arithmetic may differ by: 1e-12 (the small components
are then right to about 12 digits whatever their size)."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu

RTOL = 1e-12
DIMS = (7, 6, 9)


def lambdas(nc):
    if nc == 2:
        m = [[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]]
    else:
        r = 1 / np.sqrt(3.0)
        m = [[[0, 1, 0], [1, 0, 0], [0, 0, 0]], [[0, -1j, 0], [1j, 0, 0], [0, 0, 0]], [[1, 0, 0], [0, -1, 0], [0, 0, 0]],
             [[0, 0, 1], [0, 0, 0], [1, 0, 0]], [[0, 0, -1j], [0, 0, 0], [1j, 0, 0]], [[0, 0, 0], [0, 0, 1], [0, 1, 0]],
             [[0, 0, 0], [0, 0, -1j], [0, 1j, 0]], [[r, 0, 0], [0, r, 0], [0, 0, -2 * r]]]
    return np.array(m, complex) / 2


def links(nc, A):
    """exp(i A^a t_a) to first order in the small components' commutators: a Taylor
    polynomial, whose small entries come out to relative accuracy."""
    t = lambdas(nc)
    h = np.einsum("vda,aij->vdij", A, t)
    one = np.eye(nc)
    u = one + 1j * h / 20
    for k in range(19, 0, -1):
        u = one + 1j * np.einsum("vdij,vdjk->vdik", h, u) / k
    if nc == 2:
        return np.stack([u[..., 0, 0].real, u[..., 0, 1].imag, u[..., 0, 1].real, u[..., 0, 0].imag], -1)
    m = u.reshape(u.shape[:2] + (9,))
    return np.concatenate([m.real, m.imag], -1)


def run(monkeypatch, nc, U, E, steps, only):
    if only:
        monkeypatch.setenv("OPX_FP64_ONLY", "1")
    else:
        monkeypatch.delenv("OPX_FP64_ONLY", raising=False)
    h = opx.Handle(nc, DIMS, precision=N.OPX_F64, dt=0.05)
    h.upload(N.FIELD_U, U)
    h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
    h.initialize()
    h.step(steps)
    return h.download(N.FIELD_UNEXT), h.download(N.FIELD_E, layout=N.LAYOUT_GEN)


def close(x, y, groups):
    for g in groups:
        top = np.abs(x[..., g]).max()
        assert np.abs(x[..., g] - y[..., g]).max() <= RTOL * top, (g, top, np.abs(x[..., g] - y[..., g]).max())


EPS = [1e-3, 1e-5, 1e-8, 1e-12, 1e-18, 1e-30]
# the large components, the small ones, and the link entries that hold the small ones
FORMS = [(2, [2], [0, 1], [1, 2]), (2, [0], [1, 2], [2, 3]),
         (3, [2], [0, 1, 3, 4, 5, 6], [1, 2, 3, 5, 6, 7, 10, 11, 12, 14, 15, 16]),
         (3, [0], [3, 4, 5, 6], [2, 5, 6, 7, 11, 14, 15, 16]),
         (3, [0, 1, 2], [3, 4, 5, 6], [2, 5, 6, 7, 11, 14, 15, 16])]


@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("form", range(len(FORMS)))
def test_small_components_of_links_and_fields(native, monkeypatch, form, eps):
    nc, big, small, entries = FORMS[form]
    rng = np.random.default_rng(form)
    V, na = int(np.prod(DIMS)), 3 if nc == 2 else 8
    A, E = (np.zeros((V, 3, na)) for _ in range(2))
    for X in (A, E):
        X[..., big] = rng.normal(0, 0.15, (V, 3, len(big)))
        X[..., small] = rng.normal(0, eps, (V, 3, len(small)))
    U = links(nc, A)
    (ua, ea), (ub, eb) = (run(monkeypatch, nc, U, E, 3, only) for only in (True, False))
    close(ea, eb, [big, small])
    close(ua, ub, [entries])


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("eps", EPS)
def test_small_fields_in_other_directions(native, monkeypatch, nc, eps):
    """Strong links in direction 2 only, one colour; the other links are exactly 1 and
    their E of size eps in the other colours."""
    rng = np.random.default_rng(11)
    V, na = int(np.prod(DIMS)), 3 if nc == 2 else 8
    A, E = (np.zeros((V, 3, na)) for _ in range(2))
    A[:, 2, 2] = rng.normal(0, 0.2, V)
    E[:, :2] = rng.normal(0, eps, (V, 2, na))
    E[:, 2, 2] = rng.normal(0, 0.2, V)
    U = links(nc, A)
    (ua, ea), (ub, eb) = (run(monkeypatch, nc, U, E, 3, only) for only in (True, False))
    close(ea[:, :2], eb[:, :2], [[0, 1]])
    off = [1, 2] if nc == 2 else [1, 2, 3, 5, 6, 7, 10, 11, 12, 14, 15, 16]
    close(ua[:, :2], ub[:, :2], [off])


@pytest.mark.parametrize("nc", [2, 3])
def test_vacuum_and_abelian_fields_stay_exact(native, monkeypatch, nc):
    """Components that are exactly zero everywhere stay so; links of exactly 1 without
    fields do not change."""
    rng = np.random.default_rng(12)
    V, na = int(np.prod(DIMS)), 3 if nc == 2 else 8
    A, E = (np.zeros((V, 3, na)) for _ in range(2))
    A[..., 2] = rng.normal(0, 0.2, (V, 3))
    E[..., 2] = rng.normal(0, 0.2, (V, 3))
    half = V // 2
    A[:half] = 0
    E[:half] = 0
    U = links(nc, A)
    (ua, ea), (ub, eb) = (run(monkeypatch, nc, U, E, 2, only) for only in (True, False))
    others = [a for a in range(na) if a != 2]
    assert not eb[..., others].any()
    off = [1, 2] if nc == 2 else [1, 2, 3, 5, 6, 7, 10, 11, 12, 14, 15, 16, 17]
    assert not ub[..., off].any()
    close(ea, eb, [[2]])
    # sites whose stencil is vacuum over both steps: planes 0 .. of the first half, away from its edges
    far = np.arange(V).reshape(DIMS)[2:DIMS[0] // 2 - 2].ravel()
    assert np.array_equal(ua[far], ub[far]) and np.array_equal(ea[far], eb[far])


@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("form", [0, 1])
def test_gradient_in_small_components(native, monkeypatch, form, eps):
    """The gradient with respect to E is of the size of the field in each component (its
    sums come in no fixed order: some tens of roundings more)."""
    nc, big, small, _ = FORMS[form]
    rng = np.random.default_rng(20 + form)
    V = int(np.prod(DIMS))
    A, E = (np.zeros((V, 3, 3)) for _ in range(2))
    for X in (A, E):
        X[..., big] = rng.normal(0, 0.15, (V, 3, len(big)))
        X[..., small] = rng.normal(0, eps, (V, 3, len(small)))
    out = []
    for only in (True, False):
        if only:
            monkeypatch.setenv("OPX_FP64_ONLY", "1")
        else:
            monkeypatch.delenv("OPX_FP64_ONLY")
        h = opx.Handle(nc, DIMS, precision=N.OPX_F64, dt=0.05)
        h.upload(N.FIELD_U, links(nc, A))
        h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
        out.append(h.energy_gradient(6, 4, (2, 1, 3), (4, 4, 6))[1].reshape(V, 3, 3))
    close(out[0], out[1], [big, small])
