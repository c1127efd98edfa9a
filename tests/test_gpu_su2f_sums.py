"""The sums of the SU(2) FP32 BulkQuantities pass against exact sums of the same
per-site values, the values spread over many orders of magnitude, and every
column of a large lattice against the FP64 pass on its own scale."""
import math

import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu

DIMS = (144, 136, 132)
# the sites of one thread when 4 blocks of 128 threads are resident on each of 152 SMs:
# every 77824th of a lattice that is larger than that
STRIDE = 4 * 152 * 128


def handle(dims, prec, U, E, rho=None):
    h = opx.Handle(2, dims, a=1.0, dt=0.05, g=1.0, precision=prec)
    h.upload(N.FIELD_U, U)
    h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
    if rho is not None:
        h.upload(N.FIELD_RHO, rho, layout=N.LAYOUT_GEN)
    h.initialize()
    return h


def identity(V):
    U = np.zeros((V, 3, 4))
    U[..., 0] = 1.0
    return U


@pytest.mark.parametrize("decades", [0, 4, 7, 10, 16])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_localised_values_keep_fp64_sums(native, decades, seed):
    """E nonzero at the sites of one thread only, its squares over `decades` orders.

    One component per link, so that a site's value is float32(e * e) exactly; the sum
    has 34 terms >= 0: a FP64 sum's 34 roundings of 2^-53, the lattice mean's and
    the unit factor's are below 1e-15 with the correct sum's ordering left free."""
    rng = np.random.default_rng(seed)
    V = int(np.prod(DIMS))
    at = np.arange(100 + seed, V, STRIDE)
    E = np.zeros((V, 3, 3))
    for i in range(3):
        E[at, i, i] = (rng.uniform(1, 2, len(at)) * 10.0 ** (-rng.uniform(0, decades, len(at)) / 2)).astype(np.float32)
    o = handle(DIMS, N.OPX_F32, identity(V), E).reduce()
    e = E[at][:, range(3), range(3)].astype(np.float32)
    want = np.array([math.fsum((e[:, i] * e[:, i]).astype(np.float64).tolist()) / V for i in range(3)])
    assert np.abs(np.array(list(o.e2)) / want - 1).max() <= 1e-15


def test_small_among_large_and_zero(native):
    """A run whose first value is 2^100 times the others, and subnormal squares."""
    V = int(np.prod(DIMS))
    at = np.arange(7, V, STRIDE)
    E = np.zeros((V, 3, 3))
    E[at, 0, 0] = np.float32(3.3e-16)
    E[at[0], 0, 0] = np.float32(1.7e14)
    E[at, 1, 1] = np.float32(1.1e-19)
    E[at, 2, 2] = np.float32(1.3e-22)
    E[at[-1], 2, 2] = np.float32(0.7)
    o = handle(DIMS, N.OPX_F32, identity(V), E).reduce()
    e = E[at][:, range(3), range(3)].astype(np.float32)
    want = np.array([math.fsum((e[:, i] * e[:, i]).astype(np.float64).tolist()) / V for i in range(3)])
    assert np.abs(np.array(list(o.e2)) / want - 1).max() <= 1e-15


@pytest.mark.parametrize("dims", [(9, 7, 5), (64, 40, 31), (144, 136, 132)])
def test_every_column_on_its_own_scale(native, dims):
    """Unit links and E of order one: below 20 roundings of 2^-24 a component, twice
    that in its square, and a sum of squares is off by no more than its terms: 2.4e-6
    of each column.  rho^2 is a square of the input: 3 roundings, 2e-7."""
    rng = np.random.default_rng(21)
    V = int(np.prod(dims))
    q = rng.normal(size=(V, 3, 4))
    q = (q / np.linalg.norm(q, axis=-1, keepdims=True)).astype(np.float32).astype(np.float64)
    E = rng.normal(size=(V, 3, 3)).astype(np.float32).astype(np.float64)
    rho = rng.normal(size=(V, 3)).astype(np.float32).astype(np.float64)
    a, b = (handle(dims, p, q, E, rho).reduce() for p in (N.OPX_F32, N.OPX_F64))
    for x, y, tol in [(u, v, 2.4e-6) for u, v in zip(list(a.e2) + list(a.b2) + [a.gauss], list(b.e2) + list(b.b2) + [b.gauss])] + \
            [(a.rho2 ** 2, b.rho2 ** 2, 2e-7)]:
        assert abs(x - y) <= tol * abs(y)
