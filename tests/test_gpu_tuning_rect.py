"""What rihvr_tuning reports on rectangular planes is what runs: forcing the
reported variant leaves every bit of the operators as it is, and tuning keeps to
the variants that such planes have.  The planes are evenly spaced."""
import numpy as np
import pytest

from test_gpu_sizes import make, rel

pytestmark = pytest.mark.gpu

ADJ = ("direct", "recurrence", "recurrence_hoisted", "recurrence_table")
FWD = ("direct", "horner", "horner_onebuf", "horner_tma")


def operators(rihvr, W, H, nz):
    rng = np.random.default_rng(W + H)
    x = (rng.standard_normal((nz, H, W)) + 1j * rng.standard_normal((nz, H, W))).astype(np.complex64)
    r = rng.standard_normal((H, W)).astype(np.float32)
    with rihvr.SparseCompressiveHolo(make(rihvr, nz), W, H) as s:
        return s.tuning(), s.forward(x), s.adjoint(r)


# narrower than a block of columns (no TMA map, so the direct passes), as wide, and wide; the last
# two have planes enough for the recurrence untuned
@pytest.mark.parametrize("W,H,nz", [(16, 64, 6), (30, 64, 6), (32, 64, 6), (96, 64, 6), (64, 128, 9), (48, 1024, 5),
                                    (16, 64, 4800), (96, 64, 1600)])
def test_reported_variant_runs(rihvr, monkeypatch, W, H, nz):
    t, f, g = operators(rihvr, W, H, nz)
    if W < 32 and H == 64:
        assert (t["adj_recurrence"], t["fwd_horner"]) == (0, 0)
    monkeypatch.setenv("RIHVR_ADJ_COL", ADJ[t["adj_recurrence"]])
    monkeypatch.setenv("RIHVR_FWD_COL", FWD[t["fwd_horner"]])
    _, f1, g1 = operators(rihvr, W, H, nz)
    assert np.array_equal(f, f1) and np.array_equal(g, g1)


@pytest.mark.parametrize("W,H", [(96, 64), (16, 64), (48, 384)])
def test_tuned_rectangle(rihvr, W, H):
    nz = 24
    rng = np.random.default_rng(5)
    b = rng.standard_normal((H, W)).astype(np.float32)
    x = {}
    for tune in (0, 1):
        with rihvr.SparseCompressiveHolo(make(rihvr, nz), W, H) as s:
            s.setHologram(b)
            if tune:
                s.autotune()
            t = s.tuning()
            assert t["adj_recurrence"] in (0, 2, 3) and t["fwd_horner"] in (0, 3)
            if W < 32:
                assert t["adj_recurrence"] == 0 and t["fwd_horner"] == 0
            s.iterate(6)
            x[tune] = s.getVolume()
    assert rel(x[1], x[0]) < 1e-4  # as the square planes' tuning test
