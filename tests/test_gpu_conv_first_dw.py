"""Weight and bias gradient of 3 x 3 layers with one to four input channels (exact fp32 on CUDA cores) against the oracle, at the edges
of the kernel's variants: filters below, at and above 8 / 16 / 32 / 64, strides 1 and 2, one to four values per copy, odd outputs,
images that share a tile, one unit altogether."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import cpu_oracle as co

pytestmark = pytest.mark.gpu

#         N  C  H   W   F  s  pad
SHAPES = [(1, 1, 2, 2, 1, 1, 1), (5, 1, 28, 28, 8, 1, 1), (3, 3, 32, 32, 64, 1, 1), (2, 4, 9, 11, 65, 1, 1), (7, 2, 6, 10, 16, 1, 1),
          (33, 1, 4, 4, 33, 1, 1), (2, 3, 16, 14, 32, 2, 1), (3, 1, 64, 64, 32, 2, 1), (2, 4, 13, 7, 9, 2, 0), (1, 3, 20, 8, 130, 1, 2)]


@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_short_patch_weight_gradient(shape, act):
    import engine_np as E
    from ml_framework_b200 import capi
    L = capi.load()
    capi.check(L.seera_init(capi.default_device()))
    capi.check(L.seera_set_precision(3))
    N, C, H, W, F, s, pad = shape
    OH, OW = (H + 2 * pad - 3) // s + 1, (W + 2 * pad - 3) // s + 1
    rs = np.random.RandomState(sum(shape) + act)
    X, Wt, b = (rs.standard_normal(q).astype(np.float32) for q in ((N, C, H, W), (F, C, 3, 3), (F,)))
    for pooled in ([False, True] if OH % 2 == 0 and OW % 2 == 0 else [False]):
        if pooled:
            gp = rs.standard_normal((N, F, OH // 2, OW // 2)).astype(np.float32)
            y, _, _, dW, db = E.conv2d_layer_roundtrip(X, Wt, b, s, s, pad, pad, act, gp=gp, need_dx=False)
            _, mask = co.maxpool2d_forward(y, 2, 2, 2, 2, 0, 0)
            dy = co.maxpool2d_backward(gp, mask, N, F, OH, OW, 2, 2, 2, 2, 0, 0)
        else:
            dy = rs.standard_normal((N, F, OH, OW)).astype(np.float32)
            y, _, _, dW, db = E.conv2d_layer_roundtrip(X, Wt, b, s, s, pad, pad, act, g=dy, need_dx=False)
        y = y.astype(np.float64)
        dz = (dy * [1.0, (y > 0), y * (1 - y)][act]).astype(np.float32)
        _, rW = co.conv2d_backward(dz, X, Wt, s, s, pad, pad)
        assert rel_l2(dW, rW) < 3e-6
        assert rel_l2(db, dz.astype(np.float64).sum(axis=(0, 2, 3))) < 3e-6
    assert L.seera_tc_device_status() == 0
    capi.check(L.seera_set_precision(0))
