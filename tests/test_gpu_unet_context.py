"""The network's convolutions ask for more than 48 KB of shared memory, which is
granted per device context: a network works in a context other than the one
that the process's first network ran in (a second GPU's, or this GPU's next
one, as here, in a process of its own)."""
import subprocess
import sys

import conftest
import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes, importlib, sys
sys.path.insert(0, %(root)r)
rihvr = importlib.import_module(%(name)r)
lib = rihvr.load_library()
rt = ctypes.CDLL("libcudart.so.12")
D, H, W = %(shape)r
n = D * H * W * 8
first = None
for turn in range(2):
    net, a, b = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    assert lib.rihvr_unet_create(D, H, W, 3, ctypes.byref(net)) == 0
    for p in (a, b):
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(n)) == 0
    host = (ctypes.c_float * (n // 4))(*[0.001 * (i %% 97) for i in range(n // 4)])
    assert rt.cudaMemcpy(a, host, ctypes.c_size_t(n), 1) == 0
    rc = lib.rihvr_unet_predict(net, a, b)
    assert rc == 0, rc
    loss = ctypes.c_double()
    rc = lib.rihvr_unet_gradients(net, a, a, None, ctypes.byref(loss))
    assert rc == 0, rc
    assert rt.cudaMemcpy(host, b, ctypes.c_size_t(n), 2) == 0
    out = list(host)
    norm = sum(v * v for v in out) ** 0.5
    assert 0 < norm < float("inf")
    # one rounding of the input's scale (a sum in any order) may turn single BF16 roundings
    assert first is None or sum((v - w) ** 2 for v, w in zip(out, first)) ** 0.5 < 1e-3 * norm
    first = out
    for p in (a, b):
        rt.cudaFree(p)
    lib.rihvr_unet_destroy(net)
    assert rt.cudaDeviceReset() == 0
print("both contexts")
"""


# widths that reach the z-walking form at every level, the per-tile forms, and neither
@pytest.mark.parametrize("shape", [(4, 8, 512), (4, 8, 128), (8, 8, 32)])
def test_second_context(shape):
    code = PROGRAM % {"root": conftest.ROOT, "name": conftest.PKG_NAME, "shape": shape}
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "both contexts" in r.stdout, r.stdout + r.stderr
