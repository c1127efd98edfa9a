"""Page-locked host buffers that begin off the eight-byte grid go through the staging copy
like pageable ones, in the handle's and the batch's transfers."""
import ctypes as C

import numpy as np
import pytest

import openpixi_gb300 as opx
from openpixi_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,prec", [(2, N.OPX_F32), (2, N.OPX_F64), (3, N.OPX_F32), (3, N.OPX_F64)])
@pytest.mark.parametrize("offset", [1, 4])
def test_buffers_off_the_grid(native, nc, prec, offset):
    dims = (5, 4, 7)
    src = opx.Handle(nc, dims, precision=prec)
    src.init_random(3, 0.2, 0.2)
    h = opx.Handle(nc, dims, precision=prec)
    b = opx.Batch(nc, [dims], dt=0.05, precision=prec)
    for field, layout in ((N.FIELD_U, N.LAYOUT_REF), (N.FIELD_E, N.LAYOUT_GEN), (N.FIELD_E, N.LAYOUT_REF)):
        want = src.download(field, layout=layout)
        pin = opx.PinnedArray(want.nbytes + 8, dtype=np.uint8)
        pin.array[offset:offset + want.nbytes] = np.frombuffer(want.tobytes(), np.uint8)
        p = C.cast(C.c_void_p(pin.p + offset), C.POINTER(C.c_double))
        assert native.opx_upload(h.h, field, p, want.size, layout) == N.OPX_OK
        assert native.opx_batch_upload(b.h, 0, field, p, want.size, layout) == N.OPX_OK
        src.upload(field, want, layout=layout)  # pageable (the hermitian layout's conversion rounds)
        want = src.download(field, layout=layout)
        assert np.array_equal(h.download(field, layout=layout), want)
        assert np.array_equal(b.download(0, field, layout=layout), want)
        for get in (lambda: native.opx_download(h.h, field, p, want.size, layout),
                    lambda: native.opx_batch_download(b.h, 0, field, p, want.size, layout)):
            pin.array[:] = 0
            assert get() == N.OPX_OK
            assert pin.array[offset:offset + want.nbytes].tobytes() == want.tobytes()
        pin.free()
