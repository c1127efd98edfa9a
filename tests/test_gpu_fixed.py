"""The FP64 leapfrog with its group products in fixed point against the same
handle with every product in FP64 (OPX_FP64_ONLY=1 at creation).

Both round every step's links and E to doubles and differ otherwise by the
rounding of a few products of unit matrices (2^-53 each at most), which three
steps add up: 1e-14 of the largest entry bounds it with room.  Inputs that the
fixed-point form refuses (links off unitarity or not finite, links within 2^-7
of the identity, dt E beyond its exponential) go through the FP64 products
site by site, so they are held to the same bound, non-finite values in the
same places.
"""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu

RTOL = 1e-14


def pair(monkeypatch, nc, dims, **kw):
    monkeypatch.setenv("OPX_FP64_ONLY", "1")
    a = opx.Handle(nc, dims, precision=N.OPX_F64, **kw)
    monkeypatch.delenv("OPX_FP64_ONLY")
    return a, opx.Handle(nc, dims, precision=N.OPX_F64, **kw)


def seed_fields(h, sigma, sigma_e, seed=5):
    h.init_random(seed, sigma, sigma_e)
    return h.download(N.FIELD_U), h.download(N.FIELD_E, layout=N.LAYOUT_GEN)


def load(hs, U, E, J=None, active=None):
    for h in hs:
        h.upload(N.FIELD_U, U)
        h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
        if J is not None:
            h.upload(N.FIELD_J, J, layout=N.LAYOUT_GEN)
        if active is not None:
            h.set_active(active)
        h.initialize()


def same(a, b):
    for f in (N.FIELD_U, N.FIELD_UNEXT, N.FIELD_E):
        x, y = a.download(f), b.download(f)
        fine = np.isfinite(x)
        assert np.array_equal(fine, np.isfinite(y)), f
        if fine.any():
            assert np.abs(x[fine] - y[fine]).max() <= RTOL * max(np.abs(x[fine]).max(), 1e-300), f


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 3, 5), (8, 4, 4), (7, 9, 11), (3, 2, 65), (16, 16, 16)])
@pytest.mark.parametrize("sigma", [1e-5, 0.01, 0.15, 1.0])
def test_steps_match(native, monkeypatch, nc, dims, sigma):
    a, b = pair(monkeypatch, nc, dims, dt=0.05)
    load((a, b), *seed_fields(a, sigma, sigma))
    a.step(3), b.step(3)
    same(a, b)


@pytest.mark.parametrize("nc", [2, 3])
def test_current_mask_and_long_offsets(native, monkeypatch, nc):
    dims = (6, 5, 12)
    rng = np.random.default_rng(3)
    V = int(np.prod(dims))
    a, b = pair(monkeypatch, nc, dims, dt=0.1, a=0.5, g=2.0)
    monkeypatch.setenv("OPX_LONG_OFFSETS", "1")
    c = opx.Handle(nc, dims, precision=N.OPX_F64, dt=0.1, a=0.5, g=2.0)
    monkeypatch.delenv("OPX_LONG_OFFSETS")
    U, E = seed_fields(a, 0.2, 0.2)
    load((a, b, c), U, E, J=rng.normal(0, 0.1, E.shape), active=(rng.random(V) < 0.7).astype(np.uint8))
    for h in (a, b, c):
        h.step(3)
    same(a, b)
    for f in (N.FIELD_U, N.FIELD_UNEXT, N.FIELD_E):
        assert np.array_equal(b.download(f), c.download(f)), f


@pytest.mark.parametrize("nc", [2, 3])
def test_links_it_refuses(native, monkeypatch, nc):
    """Strong, weak and identity links side by side, links scaled off unitarity,
    and single links that are not finite."""
    dims = (8, 6, 10)
    a, b = pair(monkeypatch, nc, dims, dt=0.05)
    U, E = seed_fields(a, 0.2, 0.1)
    W, _ = seed_fields(a, 1e-7, 0.1)
    U, W = U.reshape(dims + U.shape[1:]), W.reshape(dims + W.shape[1:])
    U[2:4] = W[2:4]
    ident = np.zeros(U.shape[-1])
    ident[[0] if nc == 2 else [0, 4, 8]] = 1.0
    U[4:6] = ident
    U[6, 1] *= 1.3
    U[6, 3] *= 1.0 + 1e-6
    load((a, b), U.reshape(-1, 3, U.shape[-1]), E)
    a.step(2), b.step(2)
    same(a, b)
    U[0, 0, 0, 1, 0] = np.nan
    U[7, 5, 9, 2, 1] = np.inf
    load((a, b), U.reshape(-1, 3, U.shape[-1]), E)
    a.step(1), b.step(1)
    same(a, b)


@pytest.mark.parametrize("nc", [2, 3])
def test_exponentials_it_refuses(native, monkeypatch, nc):
    """dt E across the range of the fixed-point exponential and beyond, and not finite."""
    dims = (6, 6, 6)
    a, b = pair(monkeypatch, nc, dims, dt=0.5)
    U, E = seed_fields(a, 0.2, 0.1)
    E *= 10.0 ** np.linspace(-9, 2, len(E))[:, None, None]
    load((a, b), U, E)
    a.step(1), b.step(1)
    same(a, b)
    E[17, 1, 0] = np.nan
    E[40, 2, 2] = -np.inf
    load((a, b), U, E)
    a.step(1), b.step(1)
    same(a, b)


@pytest.mark.parametrize("nc", [2, 3])
def test_unequal_spacings_stay_in_fp64(native, monkeypatch, nc):
    a, b = pair(monkeypatch, nc, (6, 4, 8), dt=0.05, a=(1.0, 0.5, 1.0))
    load((a, b), *seed_fields(a, 0.2, 0.2))
    a.step(2), b.step(2)
    for f in (N.FIELD_U, N.FIELD_UNEXT, N.FIELD_E):
        assert np.array_equal(a.download(f), b.download(f)), f
