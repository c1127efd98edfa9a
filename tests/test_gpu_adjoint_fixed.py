"""The adjoint gradient with its staples and gather products in fixed point against
the same sweep in FP64 (OPX_FP64_ONLY=1 at creation): every step rounds its
cotangents to doubles, so ten steps differ by some 1e-15 of the largest entry; 1e-13
is held.  Boxes that leave most cotangents zero at first, weak links, unequal
spacings and odd sizes go through the other branches."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,a,sigma,ckpt", [((6, 6, 6), 1.0, 0.2, 3), ((5, 7, 3), 1.0, 0.1, 4), ((12, 10, 9), 0.5, 0.01, 10),
                                               ((8, 4, 6), (1.0, 0.5, 1.0), 0.2, 3), ((9, 9, 9), 1.0, 1e-5, 2), ((1, 2, 3), 1.0, 0.3, 1)])
@pytest.mark.parametrize("kind,wrt", [(N.OBJ_ENERGY, N.WRT_E), (N.OBJ_ANISOTROPY, N.WRT_E), (N.OBJ_ENERGY, N.WRT_RHO)])
def test_gradient_matches_fp64(native, monkeypatch, dims, a, sigma, ckpt, kind, wrt):
    out = []
    for only in ("1", None):
        if only:
            monkeypatch.setenv("OPX_FP64_ONLY", only)
        else:
            monkeypatch.delenv("OPX_FP64_ONLY")
        h = opx.Handle(2, dims, a=a, dt=0.05, precision=N.OPX_F64)
        h.init_random(11, sigma, 0.2)
        if wrt == N.WRT_RHO:
            if min(dims) < 4 or sigma < 0.05:
                pytest.skip("the Laplacian of these links is nearly singular")
            h.gauss_project(1e-26)
        U, E = h.download(N.FIELD_U), h.download(N.FIELD_E)
        hi = tuple(max(0, d // 2) for d in dims)
        out.append(h.objective_gradient(10, ckpt, kind, 0, lo=(0, 0, 0), hi=hi, wrt=wrt))
        assert np.array_equal(h.download(N.FIELD_U), U) and np.array_equal(h.download(N.FIELD_E), E)
    (Ja, ga), (Jb, gb) = out
    assert abs(Ja - Jb) <= 1e-13 * abs(Ja)
    # the solve for rho amplifies what enters it by its condition number
    assert np.abs(ga - gb).max() <= (1e-13 if wrt == N.WRT_E else 1e-9) * np.abs(ga).max()
