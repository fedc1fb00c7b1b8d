"""The weight gradient's kernel alone, where its blocks walk several bricks: large
and small bricks, ragged in x, y and z, every number of output channels, against
FP64 sums of the same BF16-rounded operands.

Tolerance: a chain of 16 tensor-core steps truncates its sum by at most 2^-23 of
it a step (1.9e-6), the sums of up to 600 blocks meet in any order by FP32 atomic
adds (sqrt(600) 2^-24 = 1.5e-6); 5e-6 of the gradient's norm."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

# rihvr::unet::conv3_wgrad(X, Cin, dY, Cout, dW, D, H, W, stream)
SYMBOL = "_ZN5rihvr4unet11conv3_wgradEPKfiS2_iPfiiiP11CUstream_st"


def wgrad(rihvr, X, dY):
    import torch

    D, H, W, cin = X.shape
    cout = dY.shape[-1]
    dW = torch.zeros((cout, 27, cin), device="cuda")
    torch.cuda.synchronize()
    fn = getattr(rihvr.load_library(), SYMBOL)
    fn.restype = ctypes.c_int
    vp = ctypes.c_void_p
    rc = fn(vp(X.data_ptr()), cin, vp(dY.data_ptr()), cout, vp(dW.data_ptr()), D, H, W, vp(None))
    assert rc == 0
    torch.cuda.synchronize()
    return dW


def reference(X, dY):
    import torch

    D, H, W, cin = X.shape
    Xp = torch.nn.functional.pad(X.bfloat16().double(), (0, 0, 1, 1, 1, 1, 1, 1))
    Y = dY.bfloat16().double().reshape(-1, dY.shape[-1]).T
    taps = [Xp[k // 9:k // 9 + D, k // 3 % 3:k // 3 % 3 + H, k % 3:k % 3 + W].reshape(-1, cin) for k in range(27)]
    return torch.stack([Y @ t for t in taps], 1)


# (D, H, W), Cin, Cout
@pytest.mark.parametrize("shape,cin,cout", [
    ((32, 128, 128), 16, 16),   # large bricks, whole: 512 for 296 blocks
    ((30, 125, 131), 16, 16),   # ragged: 640
    ((18, 66, 130), 96, 32),    # six slices: 225 for 49
    ((19, 67, 97), 48, 16),
    ((15, 61, 125), 16, 16),    # small bricks: 1024 for 592
    ((9, 45, 67), 32, 32),      # 300 for 296
    ((7, 30, 35), 64, 64),      # two small bricks a block, an odd one left
    ((32, 32, 32), 32, 64),
    ((3, 5, 7), 16, 32),
])
def test_weight_gradient(rihvr, shape, cin, cout):
    import torch

    g = torch.Generator(device="cuda").manual_seed(sum(shape) + cin + cout)
    X = torch.relu(torch.randn(shape + (cin,), generator=g, device="cuda"))
    dY = torch.randn(shape + (cout,), generator=g, device="cuda") * 0.01 + 0.002
    got, ref = wgrad(rihvr, X, dY).double(), reference(X, dY)
    assert torch.linalg.vector_norm(got - ref) < 5e-6 * torch.linalg.vector_norm(ref)
