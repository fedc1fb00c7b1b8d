"""The U-Net's weight gradient over bricks of voxels: a volume large enough for
the large bricks in its wide layers and ragged in x, y and z, against the FP64
reference with BF16-rounded operands, at the tolerances of test_gpu_unet.py (the
operands' rounding is emulated, so what is left is the FP32 accumulation and the
rounding of values that differ in their last FP32 bits)."""
import numpy as np
import pytest

import unet_ref as U
from test_gpu_unet import rel, sample

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 36, 132), (4, 4, 4)])
def test_gradients_match_reference(rihvr, shape):
    params = U.init_params(5).astype(np.float32)
    xbp, xstar = sample(4, shape)
    with rihvr.UNet(*shape) as net:
        net.set_params(params)
        loss, grad = net.gradients(xbp, xstar)
    U.emulate_bf16(True)
    try:
        rloss, rgrad = U.loss_and_grad(params.astype(np.float64), xbp.astype(np.complex128),
                                       xstar.astype(np.complex128))
    finally:
        U.emulate_bf16(False)
    assert abs(loss - rloss) / rloss < 2e-3
    off = 0
    for i, (cin, cout, _) in enumerate(U.LAYERS):
        m = cout * 27 * cin + cout
        assert rel(grad[off:off + m], rgrad[off:off + m]) < 1e-2, i
        off += m
    assert rel(grad[off:], rgrad[off:]) < 1e-2
