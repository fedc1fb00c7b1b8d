"""The z-walking inference convolutions at their edges: fewer planes than the
slices' lag or the ring, z-ranges of one block and several, rows that leave the
last y-tile ragged (4, 3 and 2 rows a tile by layer), more than one x-tile.  The
MMAs add every output's taps in the per-tile kernel's order, so the prediction
is bit-equal to the one without them."""
import os
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_unet_tc import _PREDICT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 4, 512), (8, 20, 512), (12, 8, 1024), (68, 16, 512)])
def test_z_walking_equals_per_tile(tmp_path, shape):
    from conftest import PKG_NAME, ROOT

    script = tmp_path / "predict.py"
    script.write_text(_PREDICT)
    out = []
    for value in ("1", "0"):
        f = tmp_path / f"{value}.npy"
        r = subprocess.run([sys.executable, str(script), ROOT, PKG_NAME, *map(str, shape), str(f)],
                           env=dict(os.environ, RIHVR_UNET_ZWALK=value), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        out.append(np.load(f))
    assert np.all(np.isfinite(out[0]))
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
