"""The forward operator's Horner sums turn the last plane of a z-chunk of n + 1
planes n times by a rotation held in FP32; its drift must not reach the result n
times over.

Tolerance for a volume with one plane: the passes' own error (5e-7 at most at
these sizes) and the drift.  The components of the rotation round by 2^-25 and
sincospi errs by up to an ulp, 2^-25 a step together (rms); the sum is anchored in
the middle of the chunk, which leaves n / 2 steps: n 2^-26.  Anchored at the first
plane, with a rotation whose phase was rounded to FP32 (2 pi 2^-26 / sqrt 3, rms), the
last plane of 60 was 3e-6 off."""
import numpy as np
import pytest

import numpy_ref
from test_gpu_sizes import make, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,nz,form", [(64, 64, 960, "horner_tma"), (64, 64, 960, "horner_onebuf"),
                                         (64, 64, 960, "horner"), (128, 128, 600, "horner_tma"),
                                         (384, 384, 150, "horner_tma"), (96, 64, 900, "horner_tma"),
                                         (512, 512, 96, "horner"), (32, 32, 100, "horner_tma")])
def test_ends_of_a_chunk(rihvr, monkeypatch, W, H, nz, form):
    monkeypatch.setenv("RIHVR_FWD_COL", form)
    p = make(rihvr, nz)
    rng = np.random.default_rng(W + nz)
    plane = (rng.standard_normal((H, W)) + 1j * rng.standard_normal((H, W))).astype(np.complex64)
    c = numpy_ref.phase_coeff(H, W, float(np.float32(p.resolution)), float(np.float32(p.wavelength)))
    z = rihvr.plane_list(p)
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        per = -(-nz // s.tuning()["fwd_chunks"])  # planes a chunk
        for k in (0, per // 2, per - 1):
            vol = np.zeros((nz, H, W), np.complex64)
            vol[k] = plane
            ref = np.fft.ifft2(np.exp(1j * z[k] * c) * np.fft.fft2(plane.astype(np.complex128))).real
            assert rel(s.forward(vol), ref) < 5e-7 + (per - 1) * 2.0 ** -26, k
