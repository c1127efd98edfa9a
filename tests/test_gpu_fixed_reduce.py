"""BulkQuantities, ProjectedEnergyDensity and the Gauss law of the FP64 form with
its products in fixed point, column by column against the handle that keeps every
product in FP64 (OPX_FP64_ONLY=1 at creation), and opx_reduce_noalloc against
opx_reduce on both kinds of handle.

A plaquette's component is three products of unit matrices, a transported
component two: their rounding is below 30 roundings of 2^-53 of order one (links and
E of width 0.2 to 0.5, components of order 0.1 to 1), and a column sums squares:
1e-13 of it bounds the difference."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu

RTOL = 1e-13


def columns(o):
    return np.array(list(o.e2) + list(o.b2) + [o.gauss, o.rho2])


def fields(nc, dims, sigma, seed):
    rng = np.random.default_rng(seed)
    h = opx.Handle(nc, dims, precision=N.OPX_F64, dt=0.05)
    h.init_random(seed, sigma, sigma)
    U, E = h.download(N.FIELD_U), h.download(N.FIELD_E, layout=N.LAYOUT_GEN)
    h.close()
    return rng, U, E


def pair(monkeypatch, nc, dims, U, E, rho=None, mask=None):
    out = []
    for only in (True, False):
        if only:
            monkeypatch.setenv("OPX_FP64_ONLY", "1")
        else:
            monkeypatch.delenv("OPX_FP64_ONLY", raising=False)
        h = opx.Handle(nc, dims, precision=N.OPX_F64, dt=0.05)
        h.upload(N.FIELD_U, U)
        h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
        if rho is not None:
            h.upload(N.FIELD_RHO, rho, layout=N.LAYOUT_GEN)
        if mask is not None:
            h.set_evaluatable(mask)
        h.initialize()
        out.append(h)
    return out


def agree(a, b):
    x, y = columns(a.reduce()), columns(b.reduce())
    assert np.abs(x - y).max() <= RTOL * np.abs(x).max(), (x, y)
    assert (np.abs(x - y) <= RTOL * np.abs(x)).all(), (x, y)
    for d in range(3):
        p, q = a.projected_energy(d), b.projected_energy(d)
        assert np.abs(p - q).max() <= RTOL * np.abs(p).max(), d


# a ragged lattice of many blocks' second rounds; one whose warps pass 32 rounds (the
# fold into the compensated sums: three warps a group, 912 groups SU(2), 608 SU(3))
@pytest.mark.parametrize("nc,dims", [(2, (51, 47, 45)), (3, (51, 47, 45)), (2, (128, 96, 80)), (3, (96, 90, 76))])
@pytest.mark.parametrize("masked", [False, True])
def test_large_lattices(native, monkeypatch, nc, dims, masked):
    rng, U, E = fields(nc, dims, 0.3, 3)
    V = len(U)
    kw = dict(rho=rng.normal(0, 0.2, (V, E.shape[-1])), mask=(rng.random(V) < 0.7).astype(np.uint8)) if masked else {}
    agree(*pair(monkeypatch, nc, dims, U, E, **kw))


@pytest.mark.parametrize("nc", [2, 3])
def test_links_that_are_refused(native, monkeypatch, nc):
    """Strong, weak, identity and off-unitary links side by side (FP64 products a term)."""
    dims = (12, 10, 14)
    rng, U, E = fields(nc, dims, 0.2, 5)
    _, W, _ = fields(nc, dims, 1e-4, 6)
    U, W = U.reshape(dims + U.shape[1:]), W.reshape(dims + W.shape[1:])
    U[2:4] = W[2:4]
    ident = np.zeros(U.shape[-1])
    ident[[0] if nc == 2 else [0, 4, 8]] = 1.0
    U[5:7] = ident
    U[8, 1] *= 1.3
    U[9, 3] *= 1.0 + 1e-6
    agree(*pair(monkeypatch, nc, dims, U.reshape(-1, 3, U.shape[-1]), E, rho=rng.normal(0, 0.2, (len(E), E.shape[-1]))))


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("only", [False, True])
def test_noalloc_follows_the_environment(native, monkeypatch, nc, only):
    """After a Gauss projection G^2 is rounding alone, so the two calls agree in that
    column only where they form the same products (1e-12: the order of the sums)."""
    import ctypes as C

    torch = pytest.importorskip("torch")
    from test_zz_no_alloc import as_vec, link_blocks, planes
    dims = (10, 6, 8)
    if only:
        monkeypatch.setenv("OPX_FP64_ONLY", "1")
    else:
        monkeypatch.delenv("OPX_FP64_ONLY", raising=False)
    h = opx.Handle(nc, dims, dt=0.05, precision=N.OPX_F64)
    h.init_random(31, 0.3, 0.3)
    h.gauss_project(1e-26)
    h.initialize()
    ref = as_vec(h.reduce())
    dev = torch.device("cuda", 0)
    U, Un = (torch.from_numpy(link_blocks(h.download(f))).to(dev) for f in (N.FIELD_U, N.FIELD_UNEXT))
    E = torch.from_numpy(planes(h.download(N.FIELD_E, layout=N.LAYOUT_GEN), 3)).to(dev)
    out = torch.full((13,), float("nan"), dtype=torch.float64, device=dev)
    rc = native.opx_reduce_noalloc(nc, N.OPX_F64, (C.c_int * 3)(*dims), (C.c_double * 3)(1.0, 1.0, 1.0), 1.0,
                                   C.c_void_p(U.data_ptr()), C.c_void_p(Un.data_ptr()), C.c_void_p(E.data_ptr()), None, None,
                                   C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    assert rc == N.OPX_OK
    torch.cuda.synchronize(dev)
    assert np.allclose(out.cpu().numpy(), ref, rtol=1e-12, atol=1e-300)


@pytest.mark.parametrize("nc", [2, 3])
def test_batch_follows_the_environment(native, monkeypatch, nc):
    """The FP64 batch reduction forms its Gauss terms as opx_reduce of a handle made
    under the same environment does."""
    dims = (10, 6, 8)
    rng, U, E = fields(nc, dims, 0.3, 9)
    for only in (True, False):
        if only:
            monkeypatch.setenv("OPX_FP64_ONLY", "1")
        else:
            monkeypatch.delenv("OPX_FP64_ONLY", raising=False)
        h = opx.Handle(nc, dims, dt=0.05, precision=N.OPX_F64)
        h.upload(N.FIELD_U, U)
        h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
        h.gauss_project(1e-26)
        b = opx.Batch(nc, [dims], dt=0.05, precision=N.OPX_F64)
        b.upload(0, N.FIELD_U, U)
        b.upload(0, N.FIELD_E, h.download(N.FIELD_E, layout=N.LAYOUT_GEN), layout=N.LAYOUT_GEN)
        h.initialize()
        b.initialize()
        x, y = h.reduce(), b.reduce()[0]
        assert np.isclose(x.gauss, y.gauss, rtol=1e-12, atol=0), only
