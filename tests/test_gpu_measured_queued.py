"""opx_step_measured outside the fused form: the steps and reductions are queued
without the host in between; rows, fields, step count and the state after a
non-finite row are those of opx_step(ctx, 1) + opx_reduce per step, bit for bit."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu


def vec(o):
    return np.array(list(o.e2) + list(o.b2) + [o.px, o.py, o.pz, o.gauss, o.rho2, o.e2_total, o.b2_total])


def twins(nc, dims, prec, reunit=0, J=None, active=None, evaluate=None):
    out = []
    for _ in range(2):
        h = opx.Handle(nc, dims, dt=0.05, precision=prec, reunit_every=reunit)
        h.init_random(3, 0.2, 0.2)
        if J is not None:
            h.upload(N.FIELD_J, J, layout=N.LAYOUT_GEN)
        if active is not None:
            h.set_active(active)
        if evaluate is not None:
            h.set_evaluatable(evaluate)
        h.initialize()
        out.append(h)
    return out


def same_state(a, b):
    assert a.steps_done == b.steps_done
    for f in (N.FIELD_U, N.FIELD_UNEXT, N.FIELD_E):
        assert np.array_equal(a.download(f), b.download(f), equal_nan=True), f


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("prec,reunit", [(N.OPX_F64, 0), (N.OPX_F32, 2)])
@pytest.mark.parametrize("masks", [False, True])
@pytest.mark.parametrize("dims,n", [((1, 2, 3), 3), ((9, 6, 5), 6), ((16, 16, 16), 2), ((24, 20, 30), 3)])
def test_rows_are_step_and_reduce(native, nc, prec, reunit, masks, dims, n):
    rng = np.random.default_rng(2)
    V = int(np.prod(dims))
    # a current keeps SU(3) FP32 out of its fused form
    kw = dict(J=rng.normal(0, 0.05, (V, 3, 3 if nc == 2 else 8)))
    if masks:
        kw.update(active=(rng.random(V) < 0.8).astype(np.uint8), evaluate=(rng.random(V) < 0.7).astype(np.uint8))
    a, b = twins(nc, dims, prec, reunit, **kw)
    rows = a.step_measured(n)
    for k in range(n):
        b.step(1)
        assert np.array_equal(vec(rows[k]), vec(b.reduce())), k
    same_state(a, b)
    a.step(1), b.step(1)
    assert np.array_equal(vec(a.reduce()), vec(b.reduce()))
    if nc == 2:
        assert np.array_equal(a.projected_energy(1), b.projected_energy(1))


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("top", [0.9, 2.5, 3.5, 4.5])
def test_stops_at_the_first_non_finite_row(native, nc, top):
    """A constant current on one link raises its E by a constant a step until E^2 overflows."""
    dims = (6, 5, 7)
    J = np.zeros((210, 3, 3 if nc == 2 else 8))
    J[17, 1, 0] = -1.3e154 / top / 0.05
    a, b = twins(nc, dims, N.OPX_F64, J=J)
    good = 0
    with pytest.raises(opx.OpixiError) as want:
        for _ in range(8):
            b.step(1)
            b.reduce()
            good += 1
    with pytest.raises(opx.OpixiError) as got:
        a.step_measured(8)
    assert got.value.code == want.value.code == N.OPX_ERR_NUMERIC
    assert a.steps_done == good + 1
    same_state(a, b)
    # usable afterwards
    z = np.zeros_like(J)
    for h in (a, b):
        h.upload(N.FIELD_J, z, layout=N.LAYOUT_GEN)
        h.init_random(4, 0.1, 0.1)
        h.initialize()
    ra = a.step_measured(3)
    for k in range(3):
        b.step(1)
        assert np.array_equal(vec(ra[k]), vec(b.reduce()))
