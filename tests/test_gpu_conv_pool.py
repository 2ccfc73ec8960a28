"""3 x 3 convolution + bias + activation + 2x2 max-pool of a layer with few input channels (exact fp32 on CUDA cores) against the
oracle, at the edges of its variants: 8 or 16 filters per warp, one or several bands per image, one buffer, images too wide to stage."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from oracle import cpu_oracle as co

pytestmark = pytest.mark.gpu

#         N  C  H   W    F  pad
SHAPES = [(1, 1, 2, 2, 8, 1), (5, 1, 28, 28, 8, 1), (3, 3, 32, 32, 64, 1), (2, 2, 30, 18, 24, 0), (9, 7, 6, 10, 16, 2),
          (1, 3, 70, 90, 16, 1),          # several bands, the last one partial
          (2, 3, 6, 900, 8, 1),           # one window row per band, one buffer
          (1, 7, 4, 1500, 16, 1),         # not staged
          # on the tensor cores: one to three channels, a ragged last tile, filters in one chunk of 16s or several of 64, images across tiles
          (77, 3, 32, 32, 64, 1), (18, 1, 70, 62, 32, 1), (19, 2, 66, 66, 48, 0), (13, 3, 60, 54, 128, 2), (2401, 1, 6, 10, 64, 0),
          (701, 2, 18, 18, 32, 1)]        # several tiles per CTA


@pytest.mark.parametrize("mode,act", [(3, 1), (4, 1), (1, 2), (3, 0)])
@pytest.mark.parametrize("shape", SHAPES)
def test_convolution_with_the_pool_folded_in(shape, mode, act):
    from ml_framework_b200 import capi
    L = capi.load()
    capi.check(L.seera_init(capi.default_device()))
    capi.check(L.seera_set_precision(mode))
    N, C, H, W, F, pad = shape
    OH, OW = H + 2 * pad - 2, W + 2 * pad - 2
    rs = np.random.RandomState(sum(shape) + act)
    X, Wt, b = (rs.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (F, C, 3, 3), (F,)))
    up = lambda a: L.seera_to_device(np.ascontiguousarray(a).ctypes.data_as(ctypes.c_void_p), a.nbytes)      # noqa: E731

    def down(p, s, dt=np.float32):
        a = np.empty(s, dt)
        capi.check(L.seera_to_host(a.ctypes.data_as(ctypes.c_void_p), p, a.nbytes))
        return a
    shp = (N, F, OH // 2, OW // 2)
    dev = [up(X), up(Wt), up(b), L.seera_cuda_malloc(4 * int(np.prod(shp))), L.seera_cuda_malloc(4 * int(np.prod(shp)))]
    xd, wd, bd, p, m = dev
    assert L.seera_conv2d_pool_fusable(N, C, H, W, F, 3, 3, 1, 1, pad, pad) == 1
    keep, copies = ctypes.c_void_p(), ctypes.c_void_p()
    capi.check(L.seera_conv2d_bias_act_pool_fwd_s(xd, wd, bd, p, m, N, C, H, W, F, 3, 3, pad, pad, 1, 1, act, None, ctypes.byref(keep),
                                                  ctypes.byref(copies)))
    z = co.conv2d_forward(X, Wt, 1, 1, pad, pad) + b.reshape(1, F, 1, 1)
    y = (np.maximum(z, 0) if act == 1 else 1 / (1 + np.exp(-z)) if act == 2 else z).astype(np.float32)
    want, want_mask = co.maxpool2d_forward(y, 2, 2, 2, 2, 0, 0)
    got, mask = down(p, shp), down(m, shp, np.int32)
    assert rel_l2(got, want) < 2e-6
    assert (mask == want_mask.reshape(shp)).mean() > 0.999          # ties within rounding may pick another position
    assert np.all(mask[got == 0] == 0) if act == 1 else True        # a window without a positive entry: the first of its zeros
    # the channels-last copies feed the next convolution: the same result as from the pooled values themselves
    W2 = rs.standard_normal((5, F, 1, 1)).astype(np.float32)
    w2, out = up(W2), [L.seera_cuda_malloc(4 * N * 5 * shp[2] * shp[3]) for _ in range(2)]
    for o, given in zip(out, (copies, None)):
        k = ctypes.c_void_p()
        capi.check(L.seera_conv2d_bias_act_fwd_s(p, w2, None, o, N, F, shp[2], shp[3], 5, 1, 1, 0, 0, 1, 1, 0, given, ctypes.byref(k)))
        L.seera_shadow_free(k)
    assert np.array_equal(down(out[0], (N, 5) + shp[2:]), down(out[1], (N, 5) + shp[2:]))
    L.seera_shadow_free(copies)
    L.seera_shadow_free(keep)
    for d in dev + [w2] + out:
        L.seera_cuda_free(d)
    assert L.seera_tc_device_status() == 0
    capi.check(L.seera_set_precision(0))


@pytest.mark.parametrize("act", [1, 0, 2])
@pytest.mark.parametrize("where", ["input", "filters", "both"])
@pytest.mark.parametrize("shape", [(75, 3, 32, 32, 64, 1), (19, 2, 66, 66, 48, 0), (19, 1, 70, 62, 128, 2)])
def test_infinities_and_nans_give_what_the_fp32_kernel_gives(shape, where, act):
    """The tensor-core form in batches that fill the chip, the fp32 kernel on slices of them.  Windows that see such a value are the fp32
    kernel's to the bit, with their index and their copies; no other window notices."""
    from ml_framework_b200 import capi
    L = capi.load()
    capi.check(L.seera_init(capi.default_device()))
    capi.check(L.seera_set_precision(3))
    N, C, H, W, F, pad = shape
    OH, OW = H + 2 * pad - 2, W + 2 * pad - 2
    rs = np.random.RandomState(7)
    X, Wt, b = (rs.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (F, C, 3, 3), (F,)))
    touched = np.zeros((N, 1, OH // 2, OW // 2), bool)
    if where != "filters":
        for v in (np.inf, -np.inf, np.nan, 3.402e38, -3.39e38, 3.37e38, 0.0):
            for _ in range(6):
                n, c, h, w = (rs.randint(k) for k in (N, C, H, W))
                h, w = [(h, w), (0, 0), (H - 1, W - 1)][rs.randint(3)]
                X[n, c, h, w] = v
        for n, c, h, w in np.argwhere(~(np.abs(X) <= 3.38e38)):                  # the windows whose 4 x 4 patch holds it
            touched[n, 0, max(0, (h + pad - 2) // 2):(h + pad) // 2 + 1, max(0, (w + pad - 2) // 2):(w + pad) // 2 + 1] = True
    if where != "input":
        Wt[3, 0, 1, 1], Wt[F - 1, C - 1, 0, 2], Wt[F // 2, 0, 2, 2] = np.inf, np.nan, -3.4e38
        touched[:] = True
    up = lambda a: L.seera_to_device(np.ascontiguousarray(a).ctypes.data_as(ctypes.c_void_p), a.nbytes)      # noqa: E731

    def run(x):
        shp = (len(x), F, OH // 2, OW // 2)
        dev = [up(x), up(Wt), up(b), L.seera_cuda_malloc(4 * int(np.prod(shp))), L.seera_cuda_malloc(4 * int(np.prod(shp)))]
        keep, copies = ctypes.c_void_p(), ctypes.c_void_p()
        capi.check(L.seera_conv2d_bias_act_pool_fwd_s(*dev, len(x), C, H, W, F, 3, 3, pad, pad, 1, 1, act, None, ctypes.byref(keep),
                                                      ctypes.byref(copies)))
        w2, o = up(np.eye(F, dtype=np.float32)[:5].reshape(5, F, 1, 1)), L.seera_cuda_malloc(4 * len(x) * 5 * shp[2] * shp[3])
        k = ctypes.c_void_p()
        capi.check(L.seera_conv2d_bias_act_fwd_s(dev[3], w2, None, o, len(x), F, shp[2], shp[3], 5, 1, 1, 0, 0, 1, 1, 0, copies, ctypes.byref(k)))
        out = []
        for p, s, dt in ((dev[3], shp, np.float32), (dev[4], shp, np.int32), (o, (len(x), 5) + shp[2:], np.float32)):
            a = np.empty(s, dt)
            capi.check(L.seera_to_host(a.ctypes.data_as(ctypes.c_void_p), p, a.nbytes))
            out.append(a)
        for h in (k, keep, copies):
            L.seera_shadow_free(h)
        for d in dev + [w2, o]:
            L.seera_cuda_free(d)
        return out
    got = run(X)
    parts = [run(X[i:i + 4]) for i in range(0, N, 4)]
    want = [np.concatenate(p) for p in zip(*parts)]
    t = np.broadcast_to(touched, got[0].shape)
    assert t.any() and np.array_equal(got[0][t], want[0][t], equal_nan=True) and np.array_equal(got[1][t], want[1][t])
    assert np.array_equal(got[2][t[:, :5]], want[2][t[:, :5]], equal_nan=True)
    if not t.all():
        small = ~t & (np.abs(want[0]) < 1e30)
        assert np.allclose(got[0][small], want[0][small], rtol=1e-4, atol=2e-5)
        # the product of two leading copies, each within 2^-9 of its value, may overflow in the last 2^-8 below the largest number
        last = (np.abs(want[0]) > 3.4028e38 / (1 + 2.0 ** -8)) & (np.abs(got[0]) == np.inf)
        bad = ~t & ~last & ~np.isclose(got[0], want[0], rtol=1e-4, atol=2e-5)
        assert not bad.any(), (np.argwhere(bad)[:10], got[0][bad][:20], want[0][bad][:20])
        assert (got[1][~t] == want[1][~t]).mean() > 0.999
    assert L.seera_tc_device_status() == 0
    capi.check(L.seera_set_precision(0))
