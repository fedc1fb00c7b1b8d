"""The measured hologram's spectrum is made in FP64 and rounded once: it enters
every iteration's residual alike, so its error does not average out."""
import numpy as np
import pytest

from test_gpu_sizes import make

pytestmark = pytest.mark.gpu


# sides that two lines of FP64 fit shared memory for, and not; every radix
@pytest.mark.parametrize("W,H", [(16, 16), (18, 14 * 16), (2880, 16), (16, 2916), (4096, 32), (30, 4096),
                                 (3430, 50), (2304, 2304)])
def test_residual_of_nothing(rihvr, W, H):
    # x = 0: the residual's norm, from the spectrum, is the hologram's
    p = make(rihvr, 1)
    b = np.random.default_rng(W * H).standard_normal((H, W)).astype(np.float32)
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        s.setHologram(b)
        f = s.calcObjectiveFunction()[0]
    ref = 0.5 * float((b.astype(np.float64) ** 2).sum())
    assert abs(f - ref) < 1.2e-7 * ref  # two roundings of 2^-24 at most in each |B|^2
