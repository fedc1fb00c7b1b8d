"""The segmentation's threshold as one comparison of the raw values: values on
both sides of the reference's q > min_intensity max q / 256, where the square of
the rounded square root decides, against the oracle bit for bit; and inputs whose
q is NaN, negative zero or infinite."""
import numpy as np
import pytest

import oracle as O
from test_segment import as_rows, same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mi,top", [(1.0, 256.0), (3.0, 71.3), (0.0, 5.0), (1.0, 1e-38), (255.0, 2.0)])
def test_values_around_the_threshold(rihvr, mi, top):
    q = np.float32(np.sqrt(np.float32(top))) ** 2
    thr = np.float32(mi * float(q) / 256.0)
    I = np.zeros((4, 16, 40), np.float32)
    I[3, 2, 2] = top
    v = thr
    for _ in range(20):
        v = np.nextafter(v, np.float32(0), dtype=np.float32)
    vals = []
    for _ in range(40):
        vals.append(v)
        v = np.nextafter(v, np.float32(np.inf), dtype=np.float32)
    I[1, 8, :] = vals  # touching voxels of one row: which of them are on shows in the objects
    I[1, 2, ::2] = vals[::2]
    I[1, 12, 20] = top
    got, info = rihvr.segment_intensity(I, rihvr.segment_params(min_intensity=mi, close_size=0, min_area=1))
    ref, (rmax, rthr) = O.segment(I, mi, 0, 1, 1)
    assert info["max_intensity"] == rmax and info["threshold"] == rthr
    same_bits(as_rows(got), as_rows(ref))


def test_special_values(rihvr):
    sp = rihvr.segment_params(min_intensity=1.0, close_size=0, min_area=1)
    I = np.zeros((2, 8, 36), np.float32)
    I[0, 3, 5] = 4.0
    I[1, 6, 35] = -0.0
    got, info = rihvr.segment_intensity(I, sp)
    assert len(got) == 1 and info["max_intensity"] == 4.0
    for bad in (np.float32(np.nan), np.float32(-1.0)):
        J = I.copy()
        J[1, 1, 1] = bad
        got, info = rihvr.segment_intensity(J, sp)
        assert len(got) == 0 and np.isnan(info["max_intensity"])
    J = I.copy()
    J[1, 1, 1] = np.inf
    got, info = rihvr.segment_intensity(J, sp)
    assert len(got) == 0 and np.isinf(info["max_intensity"])
