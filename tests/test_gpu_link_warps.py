"""SU(3) FP32: the one-link-per-warp form of the leapfrog (up to 10^6 sites) and the
one-site-pair-per-thread form share their arithmetic, so a plain step on either
side of the line gives the fields of the measured step (always the latter form)
bit for bit."""
import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 1, 11), (2, 4, 8), (5, 13, 1), (4, 4, 12), (31, 9, 7), (100, 100, 100), (101, 100, 100)])
def test_forms_agree(native, dims):
    hs = []
    for measured in (False, True):
        h = opx.Handle(3, dims, dt=0.05, precision=N.OPX_F32, reunit_every=2)
        h.init_random(5, 0.2, 0.2)
        h.initialize()
        if measured:
            h.step_measured(3)
        else:
            h.step(3)
        hs.append(h)
    for f in (N.FIELD_U, N.FIELD_UNEXT, N.FIELD_E):
        assert np.array_equal(hs[0].download(f), hs[1].download(f)), f
