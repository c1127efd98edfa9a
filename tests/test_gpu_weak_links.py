"""FP64 lattices that the fixed-point form refuses (links near the identity) take no
longer than with every product in FP64 from the start (OPX_FP64_ONLY=1 at creation):
the device time of a step, the least of several runs in turn, 6 % left for what the
runs differ by and for the refusal itself (measured: 2 % at most)."""
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,n", [(2, 32), (2, 64), (2, 96), (3, 24), (3, 32)])
def test_refused_links_cost_no_more_than_fp64(native, monkeypatch, nc, n):
    both = []
    for only in (True, False):
        if only:
            monkeypatch.setenv("OPX_FP64_ONLY", "1")
        else:
            monkeypatch.delenv("OPX_FP64_ONLY")
        h = opx.Handle(nc, (n,) * 3, dt=0.05, precision=N.OPX_F64)
        h.init_random(5, 0.005, 0.005)
        h.initialize()
        h.time_steps(5)
        both.append(h)
    times = [[h.time_steps(10) for h in both] for _ in range(6)]
    fp64, here = (min(t[k] for t in times) for k in (0, 1))
    assert here <= 1.06 * fp64, (here / 10, fp64 / 10)
