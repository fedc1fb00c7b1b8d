"""The segmentation's workspace where its spare room for the later steps does not
fit memory: the same objects from allocations of their own, and a context's kept
workspace that does not ask for the room again (every ask would free and make its
first allocation anew)."""
import pytest

from test_gpu_segment_threads import volume

pytestmark = pytest.mark.gpu


def test_standalone_without_spare_room(rihvr):
    L = rihvr.load_library()
    v, sp = volume(3), rihvr.segment_params(close_size=2, min_intensity=20.0)
    whole = rihvr.segment_intensity(v, sp)[0]
    try:
        L.rihvr_debug_fail_allocations_after(0)
        got = rihvr.segment_intensity(v, sp)[0]
        assert L.rihvr_debug_fail_allocations_after(-1) == -1  # the failure was met
    finally:
        L.rihvr_debug_fail_allocations_after(-1)
    assert len(got) > 0 and got.tobytes() == whole.tobytes()


def test_out_of_memory_is_reported(rihvr):
    # the second allocation of the smaller workspace, the list of voxels, fails too
    L = rihvr.load_library()
    v, sp = volume(3), rihvr.segment_params(close_size=2, min_intensity=20.0)
    v[:] = 1.0  # more voxels on than the spare room holds
    try:
        L.rihvr_debug_fail_allocations_after(1)
        with pytest.raises(rihvr.RihvrError) as e:
            rihvr.segment_intensity(v, sp)
        assert e.value.code == rihvr.ERR_OUT_OF_MEMORY
    finally:
        L.rihvr_debug_fail_allocations_after(-1)


def test_kept_workspace_asks_once(rihvr, synthmod, cache_dir):
    L = rihvr.load_library()
    cfg = synthmod.small_config(W=96, H=96, Nz=12, seed=5)
    _, b = synthmod.make_hologram(cfg, cache_dir=cache_dir)
    sp = rihvr.segment_params(close_size=1, min_intensity=20.0)
    with rihvr.SparseCompressiveHolo(rihvr.params_from_config(cfg), 96, 96) as s:
        s.setHologram(b)
        s.iterate(6)
        try:
            L.rihvr_debug_fail_allocations_after(0)
            first = s.segment(sp)[0]
            assert L.rihvr_debug_fail_allocations_after(-1) == -1
            L.rihvr_debug_fail_allocations_after(0)
            again = [s.segment(sp)[0] for _ in range(3)]
            assert L.rihvr_debug_fail_allocations_after(-1) == 0  # nothing was allocated
        finally:
            L.rihvr_debug_fail_allocations_after(-1)
    with rihvr.SparseCompressiveHolo(rihvr.params_from_config(cfg), 96, 96) as s:
        s.setHologram(b)
        s.iterate(6)
        whole = s.segment(sp)[0]
    assert len(whole) > 0
    for got in [first] + again:
        assert got.tobytes() == whole.tobytes()
