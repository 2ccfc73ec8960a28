"""3 x 3 convolutions of little work (exact fp32 on CUDA cores): forward, forward with its 2x2 max-pool, and both gradients, at full
resolution and through the pool, against the oracle."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import cpu_oracle as co

pytestmark = pytest.mark.gpu

#         N  C   H   W   F   pad
SHAPES = [(1, 8, 14, 14, 16, 1), (64, 8, 14, 14, 16, 1), (2, 13, 5, 7, 5, 0), (3, 8, 9, 6, 64, 1), (1, 9, 1, 1, 1, 1), (2, 10, 4, 500, 3, 2),
          (1, 16, 12, 380, 8, 1), (7, 32, 6, 6, 16, 1)]            # bands of one window row


def activated(z, act):
    return [z, np.maximum(z, 0), 1 / (1 + np.exp(-z.astype(np.float64)))][act].astype(np.float32)


def slope(y, act):
    return [np.ones_like(y), (y > 0).astype(np.float32), y * (1 - y)][act]


@pytest.mark.parametrize("mode", [2, 3, 4])
@pytest.mark.parametrize("shape", SHAPES)
def test_small_convolution(shape, mode):
    from ml_framework_b200 import capi, seera_cuda as sc
    sc.init(0)
    sc.set_precision(mode)
    N, C, H, W, F, pad = shape
    act = (sum(shape) + mode) % 3
    OH, OW = H + 2 * pad - 2, W + 2 * pad - 2
    rs = np.random.RandomState(sum(shape))
    x, w, b, g = (rs.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (F, C, 3, 3), (F,), (N, F, OH, OW)))
    w /= np.float32(3 * np.sqrt(C))
    xd, wd, bd, gd = (sc.to_device_f32(a.ravel()) for a in (x, w, b, g))
    yd, dx, dw, db = (sc.cuda_malloc_f32(a.size) for a in (g, x, w, b))
    back = lambda p, a: sc.to_host_f32(p, a.shape)      # noqa: E731
    sc.conv2d_bias_act_fwd(xd, wd, bd, yd, N, C, H, W, F, 3, 3, pad, pad, 1, 1, act)
    z = co.conv2d_forward(x, w, 1, 1, pad, pad) + b.reshape(1, F, 1, 1)
    y = back(yd, g)
    assert rel_l2(y, activated(z, act)) < 2e-6

    def gradients(dz):
        rx, rw = co.conv2d_backward(dz, x, w, 1, 1, pad, pad)
        assert rel_l2(back(dx, x), rx) < 2e-6 and rel_l2(back(dw, w), rw) < 2e-6
        return dz.astype(np.float64).sum((0, 2, 3))
    sc.conv2d_act_bwd(wd, xd, yd, gd, 0, 0, 0, dx, dw, db, N, C, H, W, F, 3, 3, 1, 1, pad, pad, act, 0)
    assert rel_l2(back(db, b), gradients(g * slope(y, act))) < 1e-5
    sc.cuda_conv2d_bwd(wd, xd, gd, dx, dw, N, C, H, W, F, 3, 3, 1, 1, pad, pad)
    gradients(g)
    assert sc.conv2d_pool_fusable(N, C, H, W, F, 3, 3, 1, 1, pad, pad) or OH % 2 or OW % 2 or F % 8
    if sc.conv2d_pool_fusable(N, C, H, W, F, 3, 3, 1, 1, pad, pad):
        half = (N, F, OH // 2, OW // 2)
        pooled, mask = sc.cuda_malloc_f32(g.size // 4), sc.cuda_malloc_i32(g.size // 4)
        sc.conv2d_bias_act_pool_fwd_s(xd, wd, bd, pooled, mask, N, C, H, W, F, 3, 3, pad, pad, 1, 1, act, 0, False)
        want, want_mask = co.maxpool2d_forward(y, 2, 2, 2, 2, 0, 0)
        yp, m = sc.to_host_f32(pooled, half), sc.to_host_i32(mask, half)
        assert rel_l2(yp, want) < 2e-6 and (m == want_mask.reshape(half)).mean() > 0.99
        gp = rs.standard_normal(half).astype(np.float32)
        gpd = sc.to_device_f32(gp.ravel())
        sc.conv2d_act_bwd(wd, xd, 0, 0, gpd, mask, pooled, dx, dw, db, N, C, H, W, F, 3, 3, 1, 1, pad, pad, act, 0)
        dz = np.zeros(g.shape, np.float32)
        n, f, i, j = np.indices(half)
        dz[n, f, 2 * i + m // 2, 2 * j + m % 2] = gp * slope(yp, act)
        assert rel_l2(back(db, b), gradients(dz)) < 1e-5
        for p in (pooled, gpd):
            sc.cuda_free(p)
        sc.cuda_free(mask)
    for p in (xd, wd, bd, gd, yd, dx, dw, db):
        sc.cuda_free(p)
    sc.set_precision(0)
    assert capi.load().seera_tc_device_status() == 0


#         N  C  H   W   F  pad stride
DIRECT = [(1, 1, 3, 3, 1, 0, 1), (3, 3, 9, 11, 7, 1, 1), (40, 3, 32, 32, 32, 1, 1), (64, 1, 64, 62, 32, 1, 2), (2, 4, 17, 13, 24, 2, 2),
          (1, 2, 5, 900, 16, 1, 2), (30, 1, 63, 65, 48, 0, 1), (5, 3, 6, 1300, 8, 2, 1)]


@pytest.mark.parametrize("mode", [3, 4])
@pytest.mark.parametrize("shape", DIRECT)
def test_forward_of_a_layer_with_few_channels(shape, mode):
    from ml_framework_b200 import capi, seera_cuda as sc
    sc.init(0)
    sc.set_precision(mode)
    N, C, H, W, F, pad, st = shape
    act = sum(shape) % 3
    OH, OW = (H + 2 * pad - 3) // st + 1, (W + 2 * pad - 3) // st + 1
    rs = np.random.RandomState(sum(shape))
    x, w, b = (rs.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (F, C, 3, 3), (F,)))
    xd, wd, bd = (sc.to_device_f32(a.ravel()) for a in (x, w, b))
    yd = sc.cuda_malloc_f32(N * F * OH * OW)
    want = activated(co.conv2d_forward(x, w, st, st, pad, pad) + b.reshape(1, F, 1, 1), act)
    w2d = sc.to_device_f32(rs.standard_normal(5 * F * 25).astype(np.float32))
    outs = [sc.cuda_malloc_f32(N * 5 * OH * OW) for _ in range(2)]
    for copies in (True, False):
        hx, hw, hy = sc.conv2d_bias_act_fwd_k(xd, wd, bd, yd, N, C, H, W, F, 3, 3, pad, pad, st, st, act, 0, copies)
        # (copies of a number of filters that is no multiple of 8 are the tensor-core kernel's)
        assert rel_l2(sc.to_host_f32(yd, want.shape), want) < (2e-5 if copies and F % 8 else 2e-6) and not hx and not hw
        if hy:                      # what a convolution makes of the copies is what it makes of the output itself
            for o, given in zip(outs, (hy, 0)):
                sc.shadow_free(sc.conv2d_bias_act_fwd_s(yd, w2d, 0, o, N, F, OH, OW, 5, 5, 5, 2, 2, 1, 1, 0, given))
            assert np.array_equal(*(sc.to_host_f32(o, (N, 5, OH, OW)) for o in outs))
            sc.shadow_free(hy)
        assert bool(hy) == copies or F % 8
    for p in (xd, wd, bd, yd, w2d, *outs):
        sc.cuda_free(p)
    sc.set_precision(0)
    assert capi.load().seera_tc_device_status() == 0
