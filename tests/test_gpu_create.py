"""How many allocations a context's creation makes: each takes up to half a
millisecond, which a caller with many frame sizes pays again and again."""
import ctypes

import pytest

from test_gpu_faults import small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,most", [(7, 28), (5, 28), (6, 30)])
def test_allocations_of_a_context(rihvr, mode, most):
    # device and pinned host allocations; 28 (30 in mode 6) carry the volumes, the tables and the
    # pinned blocks, with the planes of the hologram's spectra together in one of them
    L = rihvr.load_library()
    p = small(rihvr)
    p.mode = mode
    if mode == 5:
        p.regularization_TV_param = 0.0
    out = ctypes.c_void_p()
    try:
        for n in range(60):
            L.rihvr_debug_fail_allocations_after(n)
            rc = L.rihvr_create(ctypes.byref(p), 64, 64, ctypes.byref(out))
            if rc == rihvr.OK:
                break
    finally:
        L.rihvr_debug_fail_allocations_after(-1)
    assert rc == rihvr.OK
    L.rihvr_destroy(out)
    assert n <= most
