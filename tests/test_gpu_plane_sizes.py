"""The line FFTs of plane sides without a register-resident split (radices 2
to 16 in registers, two to four stages) and the register-resident column passes
on planes of another width, at the sizes where they can go wrong: every radix,
prime squares, the smallest and largest sides, widths that do not fill a block
of columns or are narrower than one, evenly and unevenly spaced planes.
Against the FP64 oracle through the C ABI.

Tolerance: an FP32 transform of n points rounds about sqrt(log2 n) times at
6e-8 (below 4e-7 here), the transfer function adds 5e-7 and, by recurrence or
Horner's scheme, its rotation's rounding once a plane (below 1e-6); 1e-5 leaves
a factor of five."""
import numpy as np
import pytest

import oracle as O
from test_gpu_sizes import make, oparams, rel

pytestmark = pytest.mark.gpu
TOL = 1e-5

# (W, H): rows by W, columns by H
SIZES = [
    # two stages
    (16, 16), (18, 20), (24, 28), (30, 36), (42, 50), (98, 60), (90, 72), (112, 126),
    # three and four
    (162, 196), (450, 168), (250, 686), (480, 270), (1080, 96), (1200, 240), (1458, 16), (4096, 16), (16, 4096),
    (4050, 18), (16, 2058),
    # 24 elements a thread in the rows, in the columns
    (2592, 16), (3430, 20), (16, 4050), (18, 2430), (20, 3024),
    # register-resident columns at other widths, wider and narrower than a block of them
    (18, 1024), (100, 512), (20, 256), (140, 128), (16, 768), (90, 384), (24, 640), (1000, 64), (64, 1000),
    (50, 2304),
]


@pytest.mark.parametrize("dz", [40.0, 0.1])
@pytest.mark.parametrize("W,H", SIZES)
def test_operators_match_oracle(rihvr, W, H, dz):
    nz = 3 if W * H < 200_000 else 2
    p = make(rihvr, nz, plane_stepsize=dz)
    rng = np.random.default_rng(W * 5 + H)
    vol = (0.05 * (rng.standard_normal((nz, H, W)) + 1j * rng.standard_normal((nz, H, W)))).astype(np.complex64)
    r = rng.standard_normal((H, W)).astype(np.float32)
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        d = s.forward(vol)
        g = s.adjoint(r)
    op = oparams(rihvr, p, W, H)
    assert rel(d, O.forward(op, vol.astype(np.complex128))) < TOL
    assert rel(g, O.adjoint(op, r.astype(np.float64))) < TOL


def test_recurrence_on_rectangular_planes(rihvr):
    """Enough planes a block that the adjoint takes the recurrence untuned, on
    a plane wider than its columns' side."""
    W, H, nz = 1080, 64, 160
    p = make(rihvr, nz, plane_stepsize=2.0)
    r = np.random.default_rng(3).standard_normal((H, W)).astype(np.float32)
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        assert s.tuning()["adj_recurrence"] == 2
        g = s.adjoint(r)
    ref = O.adjoint(oparams(rihvr, p, W, H), r.astype(np.float64))
    assert rel(g, ref) < TOL
