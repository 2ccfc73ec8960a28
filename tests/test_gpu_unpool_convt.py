"""2x2 unpooling + 3 x 3 transposed convolution onto one channel as one operation on the low-resolution tensor, against the oracle's
separate steps; and the front end's use of it."""
import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from oracle import cpu_oracle as co

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1), (2, 3, 5, 7), (3, 32, 8, 32), (1, 33, 9, 33), (2, 70, 3, 65), (5, 4, 16, 31)]      # N, C, H, W


@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_unpool_and_transposed_convolution(shape, act):
    from ml_framework_b200 import capi, seera_cuda as sc
    sc.init(0)
    sc.set_precision(3)
    N, C, H, W = shape
    assert sc.unpool2_convT_fusable(N, C, H, W, 1, 3, 3, 1, 1, 1, 1) and not sc.unpool2_convT_fusable(N, C, H, W, 2, 3, 3, 1, 1, 1, 1)
    rs = np.random.RandomState(sum(shape) + act)
    x, w, b = (rs.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (C, 1, 3, 3), (1,)))
    w /= np.float32(3 * np.sqrt(C))
    g = rs.standard_normal((N, 1, 2 * H, 2 * W)).astype(np.float32)
    d = [sc.to_device_f32(a.ravel()) for a in (x, w, b, g)]
    y, dx, dw, db = (sc.cuda_malloc_f32(n) for n in (g.size, x.size, w.size, 1))
    sc.unpool2_convT_bias_act_fwd(d[0], d[1], d[2], y, N, C, H, W, act)
    sc.unpool2_convT_act_bwd(d[1], d[0], y, d[3], dx, dw, db, N, C, H, W, act)
    up = co.unpooling_forward(x, 2, 2)
    z = co.conv_transpose2d_forward(up, w, 1, 1, 1, 1).astype(np.float64) + b
    want = [z, np.maximum(z, 0), 1 / (1 + np.exp(-z))][act]
    got = sc.to_host_f32(y, g.shape)
    assert rel_l2(got, want) < 3e-6
    yy = got.astype(np.float64)
    dz = (g * [1.0, (yy > 0), yy * (1 - yy)][act]).astype(np.float32)
    rX, rW = co.conv_transpose2d_backward(dz, up, w, 1, 1, 1, 1)
    assert rel_l2(sc.to_host_f32(dw, w.shape), rW) < 3e-6
    assert rel_l2(sc.to_host_f32(dx, x.shape), co.unpooling_backward(rX, N, C, H, W, 2, 2)) < 3e-6
    assert rel_l2(sc.to_host_f32(db, (1,)), dz.astype(np.float64).sum()) < 1e-5
    for p in d + [y, dx, dw, db]:
        sc.cuda_free(p)
    sc.set_precision(0)
    assert capi.load().seera_tc_device_status() == 0


def test_the_unpooled_output_is_there_for_whoever_reads_it(monkeypatch):
    from ml_framework_b200 import seera as S, seera_cuda as sc
    sc.init(0)
    sc.set_precision(3)
    rs = np.random.RandomState(5)
    X = rs.uniform(0, 1, (3, 1, 8, 8)).astype(np.float32)
    got = []
    for lazy in (True, False):
        monkeypatch.setattr(S, "_LAZY_UNPOOL", lazy)
        np.random.seed(3)
        model = S.Sequential([S.Input((1, 8, 8)), S.Conv2D(6, 1, (3, 3), "relu", stride=1, zero_padding=1), S.Unpool2D_Nearest((2, 2)),
                              S.ConvTranspose2D(1, 6, (3, 3), "sigmoid", stride=1, zero_padding=1)])
        pred = model.forward(X)
        S.autograd4nn(S.Loss().mse(pred, S.Tensor(np.zeros((3, 1, 16, 16), np.float32), is_leaf=True)))
        assert (model.model[2].outputs.value._ptr is None) == lazy
        grads = [t.grad.to_host_f32() for t in model.parameters()]
        got.append((pred.to_numpy(), model.model[2].outputs.to_numpy(), grads))
    assert np.array_equal(got[0][1], got[1][1])
    assert rel_l2(got[0][0], got[1][0]) < 1e-5
    for a, b in zip(got[0][2], got[1][2]):
        assert rel_l2(a, b) < 1e-4
    sc.set_precision(0)


def test_an_unpooling_left_out_of_a_recorded_step_is_read_as_of_the_last_replay():
    from ml_framework_b200 import seera as S, seera_cuda as sc, train, workloads as wl
    sc.init(0)
    work = wl.WORKLOADS["c4"]()
    tr = train.Trainer(work, seed=2, precision=train.policy_for(work))
    X, Y = work.batch(4, 1)
    x, y = S.Tensor(X, is_leaf=True), S.Tensor(Y, is_leaf=True)
    for _ in range(2):
        tr.step(x, y)
    tr.capture(x, y)
    layers = [(l, l.inpobj.outputs) for l in tr.model.model if isinstance(l, S.Unpool2D_Nearest)]
    assert layers
    for replay in range(3):
        sc.upload_f32(x.value.main_ptr, work.batch(4, 10 + replay)[0])
        tr.replay()
        for l, low in layers:
            a = low.value.to_host_f32()
            assert np.array_equal(l.outputs.to_numpy(), a.repeat(2, axis=2).repeat(2, axis=3))
    tr.release_graph()
    sc.set_precision(0)


def test_a_softmax_of_a_recorded_forward_is_read_as_of_the_last_replay():
    from ml_framework_b200 import seera as S, seera_cuda as sc, train, workloads as wl
    sc.init(0)
    sc.set_precision(3)
    work = wl.WORKLOADS["c1"]()
    model = train.build_model(work, work.params(1))
    x = S.Tensor(work.batch(5, 1)[0], is_leaf=True)
    model.predict(x)
    sc.graph_begin()
    out = model.predict(x)
    g = sc.graph_end()
    for replay in range(3):
        X = work.batch(5, 20 + replay)[0]
        sc.upload_f32(x.value.main_ptr, X)
        sc.graph_launch(g)
        got = out.to_numpy()
        assert np.array_equal(got, model.predict(X).to_numpy())
    sc.graph_destroy(g)
    sc.set_precision(0)
