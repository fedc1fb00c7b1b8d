"""The 3-D total-variation prox (mode 6: 7-point stencil steps, up to three a
pass) and the prox of mode 5 at the edges of their tiles: widths and heights
below, at and just above a tile with its halo, one plane and a few, every split
of the step count over passes, each storage type.  Against the FP64 oracle.

Tolerance: a stencil step rounds its few sums at 6e-8 and contracts, so the
prox itself stays near 1e-7 a step; its input carries the adjoint's 1e-6.  2e-5
for FP32, the rounding of the stored result for FP16 (5e-4)."""
import numpy as np
import pytest

import oracle as O
from test_gpu_sizes import make, oparams, rel

pytestmark = pytest.mark.gpu


def prox(rihvr, W, H, nz, mode, n_tv, storage=0, record=1):
    p = make(rihvr, nz, mode=mode, num_tv_iterations=n_tv, storage=storage, record_objective=record,
             regularization_TV_param=0.0 if mode == 5 else 0.02)
    rng = np.random.default_rng(W * 3 + H * 5 + nz * 7 + n_tv)
    x = (0.05 * (rng.standard_normal((nz, H, W)) + 1j * rng.standard_normal((nz, H, W)))).astype(np.complex64)
    if storage == 2:  # the storage's own rounding of x is not what is tested
        x = (x.real.astype(np.float16).astype(np.float32) + 1j * x.imag.astype(np.float16).astype(np.float32)).astype(
            np.complex64)
    r = rng.standard_normal((H, W)).astype(np.float32)
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        out, sums = s.prox_step(x, r, 0.3)
    ref, rsums = O.prox_from(oparams(rihvr, p, W, H), x.astype(np.complex128), x.astype(np.complex128),
                             r.astype(np.float64), 0.3)
    return out, sums, ref, rsums


@pytest.mark.parametrize("W,H,nz,n_tv", [(56, 24, 3, 3), (60, 28, 4, 2), (64, 30, 5, 1), (60, 54, 1, 5),
                                         (112, 56, 7, 7), (16, 16, 2, 4), (120, 28, 33, 6), (48, 80, 2, 0),
                                         (126, 54, 2, 8), (18, 100, 40, 10)])
def test_tv3d_matches_oracle(rihvr, W, H, nz, n_tv):
    out, sums, ref, rsums = prox(rihvr, W, H, nz, 6, n_tv)
    assert rel(out, ref) < 2e-5
    for k in range(2):
        assert abs(sums[k] - rsums[k]) < 1e-4 * max(abs(rsums[k]), 1e-3 * abs(rsums[1]))


@pytest.mark.parametrize("mode", [5, 6])
@pytest.mark.parametrize("record", [0, 1])
def test_fp16_storage(rihvr, mode, record):
    out, _, ref, _ = prox(rihvr, 96, 30, 5, mode, 5, storage=2, record=record)
    assert rel(out, ref) < 1e-3


@pytest.mark.parametrize("W,H,nz", [(16, 16, 1), (18, 16, 3), (48, 80, 2), (96, 64, 3), (640, 512, 2)])
def test_l1_matches_oracle(rihvr, W, H, nz):
    out, sums, ref, rsums = prox(rihvr, W, H, nz, 5, 5)
    assert rel(out, ref) < 2e-5
    for k in range(2):
        assert abs(sums[k] - rsums[k]) < 1e-4 * abs(rsums[k])
