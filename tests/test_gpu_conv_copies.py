"""Operand copies handed from call to call: the forward's filters to the data gradient, an output's channels-last copies to the
convolution that reads it, and the transposed convolution's backward in one call, against the oracle."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import cpu_oracle as co

pytestmark = pytest.mark.gpu


@pytest.fixture
def sc():
    from ml_framework_b200 import capi, seera_cuda as sc
    sc.init(0)
    sc.set_precision(3)
    yield sc
    sc.set_precision(0)
    assert capi.load().seera_tc_device_status() == 0


def activated(z, act):
    return [z, np.maximum(z, 0), 1 / (1 + np.exp(-z.astype(np.float64)))][act].astype(np.float32)


def slope(y, act):
    return [np.ones_like(y), (y > 0).astype(np.float32), y * (1 - y)][act]


#         N  C  H  W   F  R  S  pad stride
CONVS = [(1, 8, 5, 6, 8, 1, 1, 0, 1), (3, 70, 4, 4, 40, 3, 3, 1, 1), (2, 72, 9, 7, 66, 3, 3, 1, 1), (3, 17, 12, 13, 130, 3, 3, 0, 1), (2, 64, 11, 9, 40, 5, 3, 2, 1),
         (2, 24, 12, 12, 33, 3, 3, 1, 2),        # strided: no filters kept
         (4, 3, 20, 16, 24, 3, 3, 1, 1), (2, 1, 12, 15, 17, 5, 5, 2, 1)]        # short patches: the copies of y by the first-layer kernel


@pytest.mark.parametrize("mode,tol", [(3, 1e-5), (4, 1e-5), (1, 1e-2)])
@pytest.mark.parametrize("shape", CONVS)
def test_convolution_with_everything_kept(sc, shape, mode, tol):
    sc.set_precision(mode)
    N, C, H, W, F, R, S, pad, st = shape
    act = sum(shape) % 3
    OH, OW = (H + 2 * pad - R) // st + 1, (W + 2 * pad - S) // st + 1
    rs = np.random.RandomState(sum(shape))
    x, w, b, g = (rs.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (F, C, R, S), (F,), (N, F, OH, OW)))
    w /= np.float32(np.sqrt(C * R * S))
    xd, wd, bd, gd = (sc.to_device_f32(a.ravel()) for a in (x, w, b, g))
    yd, dx, dw, db = (sc.cuda_malloc_f32(a.size) for a in (g, x, w, b))
    hx, hw, hy = sc.conv2d_bias_act_fwd_k(xd, wd, bd, yd, N, C, H, W, F, R, S, pad, pad, st, st, act, 0, True)
    y = activated(co.conv2d_forward(x, w, st, st, pad, pad) + b.reshape(1, F, 1, 1), act)
    assert rel_l2(sc.to_host_f32(yd, y.shape), y) < tol
    # the copies of y are what a convolution would have made of y
    w2 = rs.standard_normal((5, F, 5, 5)).astype(np.float32)
    w2d, outs = sc.to_device_f32(w2.ravel()), [sc.cuda_malloc_f32(N * 5 * OH * OW) for _ in range(2)]
    assert hy
    for o, given in zip(outs, (hy, 0)):
        k = sc.conv2d_bias_act_fwd_s(yd, w2d, 0, o, N, F, OH, OW, 5, 5, 5, 2, 2, 1, 1, 0, given)
        assert bool(k) != bool(given)
        sc.shadow_free(k)
    assert np.array_equal(*(sc.to_host_f32(o, (N, 5, OH, OW)) for o in outs))
    sc.conv2d_act_bwd_k(wd, xd, yd, gd, 0, 0, 0, dx, dw, db, N, C, H, W, F, R, S, st, st, pad, pad, act, hx, hw)
    assert bool(hw) == (C * R * S > 64 and st == 1)
    dz = g * slope(sc.to_host_f32(yd, y.shape), act)
    rx, rw = co.conv2d_backward(dz, x, w, st, st, pad, pad)
    assert rel_l2(sc.to_host_f32(dx, x.shape), rx) < tol and rel_l2(sc.to_host_f32(dw, w.shape), rw) < (1e-3 if mode == 4 else tol)      # one fp16 product there
    assert rel_l2(sc.to_host_f32(db, b.shape), dz.astype(np.float64).sum((0, 2, 3))) < max(tol, 1e-5)
    for h in (hx, hy):
        sc.shadow_free(h)
    sc.rows_free(hw)
    for p in (xd, wd, bd, gd, yd, dx, dw, db, w2d, *outs):
        sc.cuda_free(p)


#           N  Ci  H  W  Co K  s  pad
CONVTS = [(1, 16, 4, 5, 16, 3, 1, 1), (2, 40, 7, 6, 33, 3, 2, 1), (3, 66, 5, 9, 20, 4, 2, 1), (2, 8, 6, 6, 3, 3, 1, 1), (1, 8, 3, 3, 9, 1, 3, 0)]


@pytest.mark.parametrize("mode,tol", [(3, 1e-5), (4, 1e-5), (0, 3e-6)])
@pytest.mark.parametrize("shape", CONVTS)
def test_transposed_convolution_backward_in_one_call(sc, shape, mode, tol):
    sc.set_precision(mode)
    N, Ci, H, W, Co, K, st, pad = shape
    act = sum(shape) % 3
    Ho, Wo = (H - 1) * st - 2 * pad + K, (W - 1) * st - 2 * pad + K
    rs = np.random.RandomState(sum(shape))
    x, w, b, g = (rs.standard_normal(s).astype(np.float32) for s in ((N, Ci, H, W), (Ci, Co, K, K), (Co,), (N, Co, Ho, Wo)))
    w /= np.float32(np.sqrt(Ci * K * K))
    xd, wd, bd, gd = (sc.to_device_f32(a.ravel()) for a in (x, w, b, g))
    yd, dx, dw, db = (sc.cuda_malloc_f32(a.size) for a in (g, x, w, b))
    h = sc.conv2DTranspose_bias_act_fwd_k(xd, wd, bd, yd, N, Ci, H, W, Co, K, K, st, st, pad, pad, act, 0)
    y = activated(co.conv_transpose2d_forward(x, w, st, st, pad, pad) + b.reshape(1, Co, 1, 1), act)
    assert rel_l2(sc.to_host_f32(yd, y.shape), y) < tol
    dz = g * slope(sc.to_host_f32(yd, y.shape), act)
    rx, rw = co.conv_transpose2d_backward(dz, x, w, st, st, pad, pad)
    for keep, want_dx in ((h, True), (0, True), (h, False)):
        sc.conv2DTranspose_act_bwd_k(wd, xd, yd, gd, dx if want_dx else 0, dw, db, N, Ci, H, W, Co, K, K, st, st, pad, pad, act, keep)
        assert rel_l2(sc.to_host_f32(dx, x.shape), rx) < tol and rel_l2(sc.to_host_f32(dw, w.shape), rw) < (1e-3 if mode == 4 else tol)      # one fp16 product there
        assert rel_l2(sc.to_host_f32(db, b.shape), dz.astype(np.float64).sum((0, 2, 3))) < 1e-5
    assert np.array_equal(sc.to_host_f32(gd, g.shape), g)
    if h:
        sc.shadow_free(h)
    for p in (xd, wd, bd, gd, yd, dx, dw, db):
        sc.cuda_free(p)
