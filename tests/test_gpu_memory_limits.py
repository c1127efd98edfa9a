"""Calls that fit in the device's memory without the optional fixed-point copies of the
FP64 links still run when those copies do not fit beside them: the gradient's stored
steps, and what a handle allocates after its creation.

A filler takes the device's memory but for the amount under test.  Kernels are loaded
(a first call) before that."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Filler:
    """Device memory but for `free` bytes and 12 MB at most (torch takes whole segments of
    at least 10 MB)."""

    def __init__(self, torch, free):
        torch.cuda.empty_cache()
        torch.cuda.synchronize()
        self.torch, self.blocks = torch, []
        while torch.cuda.mem_get_info()[0] - free >= 12 * MB:
            n = min(torch.cuda.mem_get_info()[0] - free, 16 << 30)
            self.blocks.append(torch.empty(int(n) // (2 * MB) * (2 * MB), dtype=torch.uint8, device="cuda"))

    def release(self):
        self.blocks = []
        self.torch.cuda.empty_cache()


def handle(nc, dims, sigma=0.1, prec=N.OPX_F64, **kw):
    h = opx.Handle(nc, dims, dt=0.05, precision=prec, **kw)
    h.init_random(3, sigma, sigma)
    return h


N_GRAD, STEPS = 64, 24
V = N_GRAD ** 3
LINKS, FIELDS = 96 * V, 72 * V  # bytes of one FP64 copy of the links and of E


# with every step's fixed-point links 264 B a site and step, without 168 B: two margins
# between the sum of either form's other buffers and the next form's
@pytest.mark.parametrize("spare", [10, 4])
def test_gradient_without_room_for_fixed_links(native, spare):
    torch = pytest.importorskip("torch")
    h = handle(2, (N_GRAD,) * 3)
    J0, g0 = h.energy_gradient(STEPS, STEPS)
    # checkpoint, cotangents, two of each field in flight, and `spare` arrays of links
    need = (STEPS + 1) * (LINKS + FIELDS) + 2 * (LINKS + FIELDS) + 6 * LINKS + 3 * FIELDS + spare * LINKS // 2
    fill = Filler(torch, need)
    try:
        J, g = h.energy_gradient(STEPS, STEPS)
    finally:
        fill.release()
    # the same products, or FP64 ones where not even one more copy fits
    assert abs(J - J0) <= 1e-13 * abs(J0)
    assert np.abs(g - g0).max() <= 1e-12 * np.abs(g0).max()


@pytest.mark.parametrize("kw", [dict(a=(1.0, 0.5, 1.0)), dict(prec=N.OPX_F32)])
def test_gradient_reserves_what_it_uses(native, kw):
    """Unequal spacings use no fixed-point links, an FP32 handle none of its own."""
    torch = pytest.importorskip("torch")
    h = handle(2, (N_GRAD,) * 3, **kw)
    h.energy_gradient(STEPS, STEPS)
    need = (STEPS + 1) * (LINKS + FIELDS) + 2 * (LINKS + FIELDS) + 6 * LINKS + 3 * FIELDS
    if "prec" in kw:
        need += 2 * LINKS
    fill = Filler(torch, need)
    try:
        h.energy_gradient(STEPS, STEPS)
    finally:
        fill.release()


@pytest.mark.parametrize("nc", [2, 3])
def test_handle_gives_its_fixed_links_back(native, nc):
    """What is allocated after creation finds the memory of the fixed-point links."""
    torch = pytest.importorskip("torch")
    dims = (64, 64, 64)
    v = 64 ** 3
    ng, na = (4, 3) if nc == 2 else (18, 8)
    warm, h, ref = (handle(nc, dims) for _ in range(3))
    for x in (warm, h, ref):
        x.initialize()
    E = h.download(N.FIELD_E, layout=N.LAYOUT_GEN)
    ref.step(3)
    warm.set_field_solver(N.SOLVER_IMPLICIT, 1, 0.5)
    warm.step(1)
    warm.gauss_project(1e-20)
    warm.close()
    h.step(2)
    # the projection's arena is six site vectors, less than the two copies of the links
    arena = 6 * 8 * na * v
    fill = Filler(torch, arena // 2)
    try:
        h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
        it, g2 = h.gauss_project(1e-20)
        assert g2 <= 1e-20
        h.upload(N.FIELD_E, E, layout=N.LAYOUT_GEN)
        h.step(1)
        h.reduce()
    finally:
        fill.release()
    h.upload(N.FIELD_U, ref.download(N.FIELD_U))
    h.upload(N.FIELD_UNEXT, ref.download(N.FIELD_UNEXT))
    h.upload(N.FIELD_E, ref.download(N.FIELD_E, layout=N.LAYOUT_GEN), layout=N.LAYOUT_GEN)
    h.step(2), ref.step(2)
    for f in (N.FIELD_UNEXT, N.FIELD_E):
        x, y = h.download(f), ref.download(f)
        assert np.abs(x - y).max() <= 1e-14 * np.abs(y).max()
    a, b = h.reduce(), ref.reduce()
    assert abs(a.e2_total + a.b2_total - b.e2_total - b.b2_total) <= 1e-13 * (b.e2_total + b.b2_total)


def test_batch_gives_its_staging_back(native):
    """Autotune's copy of the fields finds the memory of the transfers' staging buffer."""
    torch = pytest.importorskip("torch")
    dims = (64, 64, 64)
    v = 64 ** 3
    b = opx.Batch(3, [dims], dt=0.05)
    b.init_random([3], 0.1, 0.1)
    b.initialize()
    b.autotune(steps=1)
    store, staging = v * (2 * 3 * 18 + 3 * 8) * 4, v * 3 * 18 * 8
    U = b.download(0, N.FIELD_U)  # pageable: takes the staging buffer
    fill = Filler(torch, store - staging // 2)
    try:
        b.autotune(steps=1)
    finally:
        fill.release()
    assert np.array_equal(b.download(0, N.FIELD_U), U)


@pytest.mark.parametrize("prec", [N.OPX_F32, N.OPX_F64])
def test_charge_direction_without_room_for_fixed_links(native, prec):
    """The covariant solve of a charge direction: six site vectors beside the run's own
    buffers (three of links, two of E, two site vectors)."""
    torch = pytest.importorskip("torch")
    n = 96
    v = n ** 3
    h = handle(2, (n,) * 3, prec=prec)
    drho = np.random.default_rng(5).normal(0, 0.1, (v, 3))
    J0 = h.objective_value(2, drho=drho, h=0.5)
    need = (3 * 96 + 2 * 72 + (2 + 6) * 24) * v + 4 * MB
    if prec == N.OPX_F64:
        need -= 2 * 96 * v  # the handle's own
    fill = Filler(torch, need)
    try:
        J = h.objective_value(2, drho=drho, h=0.5)
    finally:
        fill.release()
    # conjugate gradients to 1e-13 of the right side, either way
    assert abs(J - J0) <= 1e-9 * abs(J0)


def test_implicit_solver_tries_its_buffers_again(native):
    """Without room for all of its buffers a step is refused, every time, and works once
    there is room."""
    torch = pytest.importorskip("torch")
    dims = (64, 64, 64)
    h, ref = (handle(3, dims, prec=N.OPX_F32) for _ in range(2))
    for x in (h, ref):
        x.initialize()
        x.step(1)
        x.set_field_solver(N.SOLVER_IMPLICIT, 2, 0.5)
    ref.step(1)
    links = 64 ** 3 * 3 * 18 * 4  # room for one of the two copies of the links
    fill = Filler(torch, links + links // 4)
    try:
        for _ in range(2):
            with pytest.raises(opx.OpixiError) as e:
                h.update_grid()
            assert e.value.code == N.OPX_ERR_NOMEM
    finally:
        fill.release()
    h.store_fields()
    h.update_grid()
    for f in (N.FIELD_UNEXT, N.FIELD_E):
        assert np.array_equal(h.download(f), ref.download(f))
