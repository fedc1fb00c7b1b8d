"""The hologram's side of an iteration in the frequency domain, seen from
outside: the estimate and the residual that a run leaves agree with the volume
it leaves, in square, rectangular and odd-factor planes and through every way of
running it; a checkpoint of the version before the spectrum was saved resumes;
and the operators give the same bits on host memory, on device memory in place
and on device memory they must not use in place.

Tolerance of the estimate: two FP32 transforms of the same volume, one summed
over planes before and one after the momentum step: 1e-5 (see
test_gpu_plane_sizes.py)."""
import ctypes
import struct

import numpy as np
import pytest

from test_gpu_sizes import make, rel

pytestmark = pytest.mark.gpu


def hologram(W, H, seed):
    rng = np.random.default_rng(seed)
    b = 0.1 * rng.standard_normal((H, W)).astype(np.float32)
    b[H // 3:H // 3 + 4, W // 4:W // 4 + 3] -= 0.5
    return b


def check(s, b):
    est, res, X = s.getEstimate(), s.getResidual(), s.getVolume()
    assert np.array_equal(res, est - b)
    fx = s.iterations()["f_resid_x"][-1]
    assert abs(0.5 * float((res.astype(np.float64) ** 2).sum()) - fx) < 1e-5 * fx
    assert rel(s.forward(X), est) < 1e-5


@pytest.mark.parametrize("W,H,nz,mode", [(64, 64, 5, 7), (96, 64, 3, 7), (16, 18, 2, 5), (50, 1024, 2, 7),
                                         (384, 384, 17, 7), (126, 60, 4, 6)])
def test_estimate_and_residual_after_a_run(rihvr, W, H, nz, mode):
    b = hologram(W, H, W + H)
    p = make(rihvr, nz, mode=mode)
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        s.setHologram(b)
        assert np.array_equal(s.getResidual(), -b) and not s.getEstimate().any()
        s.iterate(1)   # eager
        check(s, b)
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        s.setHologram(b)
        s.iterate(6)   # graphs
        check(s, b)


def test_initial_volume_sets_the_holograms(rihvr):
    W, H, nz = 96, 48, 3
    b = hologram(W, H, 5)
    rng = np.random.default_rng(6)
    x0 = (0.1 * (rng.standard_normal((nz, H, W)) + 1j * rng.standard_normal((nz, H, W)))).astype(np.complex64)
    with rihvr.SparseCompressiveHolo(make(rihvr, nz), W, H) as s:
        s.setHologram(b)
        s.setInitialVolume(x0)
        est, res = s.getEstimate(), s.getResidual()
        assert np.array_equal(res, est - b)
        assert rel(s.forward(x0), est) < 1e-5


def test_checkpoint_of_the_version_before(rihvr, tmp_path):
    """A version 2 file ends before the spectrum that version 3 appends (one
    complex plane) and resumes from the saved holograms: the same solve up to
    FP32 rounding."""
    W, H, nz = 64, 48, 4
    b = hologram(W, H, 9)
    p = make(rihvr, nz)
    path, old = str(tmp_path / "s3"), str(tmp_path / "s2")
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        s.setHologram(b)
        s.iterate(4)
        s.saveState(path)
    data = bytearray(open(path, "rb").read())
    assert struct.unpack_from("<i", data, 8) == (3,)
    struct.pack_into("<i", data, 8, 2)
    open(old, "wb").write(data[:-8 * W * H])
    got = []
    for f in (path, old):
        with rihvr.SparseCompressiveHolo(p, W, H) as s:
            s.loadState(f)
            s.iterate(3)
            check(s, b)
            got.append((s.getVolume(), s.iterations()))
    assert rel(got[1][0], got[0][0]) < 1e-5
    assert np.array_equal(got[0][1]["backtracks"], got[1][1]["backtracks"])
    open(old, "wb").write(data[:-8 * W * H - 8])
    with rihvr.SparseCompressiveHolo(p, W, H) as s:
        with pytest.raises(rihvr.RihvrError) as e:
            s.loadState(old)
        assert e.value.code == rihvr.ERR_INVALID_FILE


def test_operators_in_place_and_not(rihvr):
    import torch

    W, H, nz = 80, 64, 3
    rng = np.random.default_rng(11)
    vol = (rng.standard_normal((nz, H, W)) + 1j * rng.standard_normal((nz, H, W))).astype(np.complex64)
    r = rng.standard_normal((H, W)).astype(np.float32)
    n = 2 * nz * H * W
    with rihvr.SparseCompressiveHolo(make(rihvr, nz), W, H) as s:
        d, g = s.forward(vol), s.adjoint(r)
        L = rihvr.load_library()
        rd, out = torch.from_numpy(r).cuda(), torch.empty((H, W), device="cuda")
        for shift in (0, 1):  # floats: complex-aligned (in place) and not
            buf = torch.zeros(n + 2, device="cuda")
            buf[shift:shift + n] = torch.from_numpy(vol.view(np.float32).ravel()).cuda()
            torch.cuda.synchronize()
            ptr = ctypes.c_void_p(buf.data_ptr() + 4 * shift)
            assert L.rihvr_forward(s._h, ptr, ctypes.c_void_p(out.data_ptr()), 1) == 0
            assert np.array_equal(out.cpu().numpy(), d)
            assert np.array_equal(buf[shift:shift + n].cpu().numpy(), vol.view(np.float32).ravel())
            buf.zero_()
            torch.cuda.synchronize()
            assert L.rihvr_adjoint(s._h, ctypes.c_void_p(rd.data_ptr()), ptr, 1) == 0
            got = buf.cpu().numpy()
            assert np.array_equal(got[shift:shift + n], g.view(np.float32).ravel())
            assert not got[:shift].any() and not got[shift + n:].any()
        # the volume that volume_device() views lies where the passes work
        s.setHologram(r)
        s.iterate(2)
        X = s.getVolume()
        view = s.volume_device()
        assert L.rihvr_forward(s._h, ctypes.c_void_p(view.data_ptr()), ctypes.c_void_p(out.data_ptr()), 1) == 0
        assert np.array_equal(out.cpu().numpy(), s.forward(X))
