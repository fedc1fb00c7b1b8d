"""The 3-D total-variation prox (mode 6) on planes whose finish pass takes more
blocks than any other pass of the context: its block sums have to fit.

Tolerance as in test_gpu_prox_edges.py: 2e-5 for FP32."""
import pytest

from test_gpu_prox_edges import prox
from test_gpu_sizes import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,nz", [(588, 3360, 1), (900, 2240, 1), (648, 2268, 2), (16, 4096, 3)])
def test_tall_planes(rihvr, W, H, nz):
    out, sums, ref, rsums = prox(rihvr, W, H, nz, 6, 2)
    assert rel(out, ref) < 2e-5
    for k in range(2):
        assert abs(sums[k] - rsums[k]) < 1e-4 * max(abs(rsums[k]), 1e-3 * abs(rsums[1]))
