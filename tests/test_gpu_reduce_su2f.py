"""BulkQuantities of SU(2) FP32 fields (runs of exact FP32 pairs per thread, 32 sites
a warp): against the FP64 reduction of the same fields, exactly summable values
against their integer sum, and values whose FP32 runs would overflow."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu

# one site; 31 / 32 / 33 sites; a ragged lattice of a few groups; a little more than one
# pass of every resident warp (77824 sites); more than a run of 32 per thread
DIMS = [(1, 1, 1), (31, 1, 1), (8, 2, 2), (3, 11, 1), (9, 7, 5), (64, 40, 31), (144, 136, 132)]


def columns(o):
    return np.array(list(o.e2) + list(o.b2) + [o.gauss, o.rho2])


def handle(dims, prec, U, E, rho=None, mask=None):
    h = opx.Handle(2, dims, a=1.0, dt=0.05, g=1.0, precision=prec)
    h.upload(N.FIELD_U, U)
    h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
    if rho is not None:
        h.upload(N.FIELD_RHO, rho, layout=N.LAYOUT_GEN)
    if mask is not None:
        h.set_evaluatable(mask)
    h.initialize()
    return h


def links(rng, V):
    q = rng.normal(size=(V, 3, 4))
    q /= np.linalg.norm(q, axis=-1, keepdims=True)
    return q.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("dims", DIMS)
def test_against_fp64(native, dims, masked):
    # a plaquette component is three products of unit quaternions, a transported
    # component two: below 20 roundings of 2^-24 of a quantity of order one, 2.4e-6 of
    # the squares' sums (random links and E: the sums are of order one a site too)
    rng = np.random.default_rng(11)
    V = int(np.prod(dims))
    U = links(rng, V)
    E = rng.normal(size=(V, 3, 3)).astype(np.float32).astype(np.float64)
    rho = rng.normal(size=(V, 3)).astype(np.float32).astype(np.float64)
    mask = (rng.random(V) < 0.7).astype(np.uint8) if masked else None
    a, b = (handle(dims, p, U, E, rho, mask) for p in (N.OPX_F32, N.OPX_F64))
    x, y = columns(a.reduce()), columns(b.reduce())
    scale = max(y.max(), 1e-30)
    assert np.abs(x - y).max() <= 1e-5 * scale


@pytest.mark.parametrize("dims", DIMS)
def test_sum_is_exact(native, dims):
    # E = k / 2048 with k < 2048: every site's square fits FP32 and the sum FP64, so
    # only the one rounding of each stage of the sum (thread, warp, block, lattice) is left
    rng = np.random.default_rng(12)
    V = int(np.prod(dims))
    k = rng.integers(0, 2048, size=(V, 3, 3))
    U = np.zeros((V, 3, 4))
    U[..., 0] = 1.0
    o = handle(dims, N.OPX_F32, U, k / 2048.0).reduce()
    want = (k.astype(np.int64) ** 2).sum(axis=(0, 2)) / 2.0**22 / V
    assert np.abs(np.array(list(o.e2)) / want - 1).max() <= 8 * 2.0**-52


@pytest.mark.parametrize("dims", DIMS)
def test_large_values(native, dims):
    # squares of 1e38: a run of them is beyond FP32, their sum is not beyond FP64
    V = int(np.prod(dims))
    U = np.zeros((V, 3, 4))
    U[..., 0] = 1.0
    E = np.zeros((V, 3, 3))
    E[:, 1, 2] = 1e19
    E[::7, 0, 0] = 0.5
    o = handle(dims, N.OPX_F32, U, E).reduce()
    assert np.isclose(o.e2[1], float(np.float32(1e19)) ** 2, rtol=1e-6, atol=0)
    assert np.isclose(o.e2[0], 0.25 * len(range(0, V, 7)) / V, rtol=1e-6, atol=0)
    assert o.e2[2] == 0.0
