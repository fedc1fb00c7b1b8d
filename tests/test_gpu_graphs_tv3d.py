"""Graphs of the 3-D TV solve (mode 6): not built for a first run that is too
short to win their building back, built once a context has run for longer, and
the same bits either way."""
import numpy as np
import pytest

from test_gpu_graphs import CONTROL_KERNELS

pytestmark = pytest.mark.gpu


def solver(rihvr, synthmod, cache_dir, most, side=64, nz=5):
    cfg = synthmod.small_config(W=side, H=side, Nz=nz, seed=47)
    _, b = synthmod.make_hologram(cfg, cache_dir=cache_dir)
    s = rihvr.SparseCompressiveHolo(rihvr.params_from_config(cfg, mode=6, max_backtracks=most), side, side)
    s.setHologram(b)
    return s


def launches(s, n):
    before = s.launch_count()
    s.iterate(n)
    return s.launch_count() - before


def test_short_first_runs_are_eager(rihvr, synthmod, cache_dir):
    # every context's first iteration is eager; a device-decided one has its control kernels more
    with solver(rihvr, synthmod, cache_dir, 0) as s:
        one = launches(s, 1)
        assert [launches(s, 1) for _ in range(14)] == [one] * 14
        assert launches(s, 1) == one + CONTROL_KERNELS  # the sixteenth: graphs from here on
        per = launches(s, 2) - launches(s, 1)
    with solver(rihvr, synthmod, cache_dir, 0) as s:
        assert launches(s, 3) == one + 2 * (per - CONTROL_KERNELS)
    with solver(rihvr, synthmod, cache_dir, 0) as s:
        assert launches(s, 20) == one + 19 * per


@pytest.mark.parametrize("runs", [(1,) * 18, (13, 6), (18,)])
def test_same_bits_eagerly_and_by_graphs(rihvr, synthmod, cache_dir, runs):
    out = {}
    for eager in (True, False):
        with solver(rihvr, synthmod, cache_dir, 2) as s:
            s.set_profiling(eager)
            for n in runs:
                s.iterate(n)
            out[eager] = (s.iterations(), s.getVolume())
    (le, xe), (lg, xg) = out[True], out[False]
    assert np.array_equal(xe, xg)
    for k in ("f_x", "f_prox", "lim", "ratio", "beta", "backtracks", "restarted", "t"):
        assert np.array_equal(le[k], lg[k]), k
