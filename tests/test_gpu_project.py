"""opx_gauss_project (conjugate gradients, three launches an iteration, transports
in fixed point) against the same solve with every product in FP64
(OPX_FP64_ONLY=1 at creation).

Both iterate until mean r^2 <= 1e-4 tol; what is left of E's error is of the size of
that residual over the smallest eigenvalue of the covariant Laplacian, far below
the 1e-9 of the largest E held here (tol = 1e-24); an FP32 handle rounds the
result once (one unit in the last place: 2^-23)."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("prec", [N.OPX_F64, N.OPX_F32])
@pytest.mark.parametrize("dims,a,rho", [((4, 4, 4), 1.0, False), ((7, 5, 9), 1.0, True), ((6, 4, 33), (1.0, 0.5, 2.0), False),
                                        ((16, 16, 16), 0.5, True), ((40, 30, 25), 1.0, False)])
def test_projection_matches_fp64(native, monkeypatch, nc, prec, dims, a, rho):
    out = []
    for only in ("1", None):
        if only:
            monkeypatch.setenv("OPX_FP64_ONLY", only)
        else:
            monkeypatch.delenv("OPX_FP64_ONLY")
        h = opx.Handle(nc, dims, a=a, dt=0.05, precision=prec)
        h.init_random(7, 0.2, 0.2)
        if rho:
            h.upload(N.FIELD_RHO, np.random.default_rng(1).normal(0, 0.1, (h.V, h.ngen)), layout=N.LAYOUT_GEN)
        it, g2 = h.gauss_project(1e-24)
        assert g2 <= 1e-24
        out.append((it, h.download(N.FIELD_E, layout=N.LAYOUT_GEN)))
    (ia, ea), (ib, eb) = out
    assert abs(ia - ib) <= 1
    tol = 1e-9 if prec == N.OPX_F64 else 2.0 ** -23
    assert np.abs(ea - eb).max() <= tol * np.abs(ea).max()


def test_no_iterations_and_zero_field(native):
    h = opx.Handle(3, (5, 4, 6), dt=0.05)
    h.init_random(3, 0.2, 0.2)
    e = h.download(N.FIELD_E)
    it, g2 = h.gauss_project(1e-24, maxit=0)
    assert it == 0 and g2 > 1e-4 and np.array_equal(h.download(N.FIELD_E), e)
    h.upload(N.FIELD_E, np.zeros_like(e))
    it, g2 = h.gauss_project(1e-24)
    assert it == 0 and g2 == 0.0 and not h.download(N.FIELD_E).any()
