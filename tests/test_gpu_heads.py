"""Classifier heads: dense products of few output columns (exact fp32) and the softmax cross-entropy, at the edges of their variants."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture
def sc():
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    sc.set_precision(3)
    yield sc
    sc.set_precision(0)


#         rows  K    N
SHAPES = [(1, 1, 1), (3, 5, 7), (64, 784, 10), (593, 256, 16), (1000, 1024, 10), (1185, 1030, 10), (2500, 1500, 3), (601, 1026, 13), (1300, 2050, 16)]


@pytest.mark.parametrize("shape", SHAPES)
def test_products_of_few_columns(sc, shape):
    M, K, N = shape
    rs = np.random.RandomState(sum(shape))
    a, b, g, bias = (rs.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N), (M, N), (N,)))
    ad, bd, gd, biasd = (sc.to_device_f32(t.ravel()) for t in (a, b, g, bias))
    cd, da, db = (sc.cuda_malloc_f32(t.size) for t in (g, a, b))
    sc.matmul_bias_act_fwd(ad, bd, biasd, cd, M, N, K, 1)
    a64, b64, g64 = (t.astype(np.float64) for t in (a, b, g))
    assert rel_l2(sc.to_host_f32(cd, (M, N)), np.maximum(a64 @ b64 + bias, 0)) < 2e-6
    sc.cuda_matmul_bwd(ad, bd, gd, da, db, M, N, K, 1)
    assert rel_l2(sc.to_host_f32(da, (M, K)), g64 @ b64.T) < 2e-6 and rel_l2(sc.to_host_f32(db, (K, N)), a64.T @ g64) < 2e-6
    for p in (ad, bd, gd, biasd, cd, da, db):
        sc.cuda_free(p)


@pytest.mark.parametrize("shape", [(1, 1), (1, 10), (64, 10), (4097, 10), (5000, 16), (37, 17), (300, 32), (33, 33), (9, 128), (7, 129)])
def test_softmax_cross_entropy(sc, shape):
    N, C = shape
    rs = np.random.RandomState(N + C)
    z, y = (rs.standard_normal(shape) * 3).astype(np.float32), np.eye(C, dtype=np.float32)[rs.randint(0, C, N)]
    zd, yd = sc.to_device_f32(z.ravel()), sc.to_device_f32(y.ravel())
    p, rows, loss, dz = (sc.cuda_malloc_f32(k) for k in (N * C, N, 1, N * C))
    eps = 1e-7
    for _ in range(2):                          # the finish counter starts from zero again
        sc.softmax_cce_fwd_bwd(zd, yd, p, rows, loss, dz, N, C, eps, 1.0 / N)
    e = np.exp(z.astype(np.float64) - z.max(1, keepdims=True))
    want = e / e.sum(1, keepdims=True)
    clipped = np.clip(want, eps, 1 - eps)
    per_row = -(y * np.log(clipped)).sum(1)
    g = np.where((want >= eps) & (want <= 1 - eps), -y / clipped / N, 0)
    assert rel_l2(sc.to_host_f32(p, shape), want) < 1e-6
    assert np.allclose(sc.to_host_f32(rows, (N,)), per_row, rtol=2e-5, atol=2e-7)
    assert np.allclose(sc.to_host_f32(loss, (1,)), per_row.mean(), rtol=2e-5, atol=2e-7)
    assert np.abs(sc.to_host_f32(dz, shape) - want * (g - (g * want).sum(1, keepdims=True))).max() < 2e-6 / N
    for q in (zd, yd, p, rows, loss, dz):
        sc.cuda_free(q)


def test_the_predictions_are_there_for_whoever_reads_them(sc):
    from ml_framework_b200 import seera as S
    rs = np.random.RandomState(1)
    x, y = rs.standard_normal((6, 5)).astype(np.float32), np.eye(3, dtype=np.float32)[[0, 1, 2, 0, 1, 2]]
    model = S.Sequential([S.Input((5,)), S.Dense(5, 3, "softmax")])
    before = model.forward(x).to_numpy()        # read before any loss
    pred = model.forward(x)
    S.Loss().categorical_cross_entropy(pred, S.Tensor(y, is_leaf=True))
    assert np.allclose(pred.to_numpy(), before, rtol=1e-6) and np.allclose(before.sum(1), 1, rtol=1e-5)


#  rows: one, odd, both sizes of the kernel of few rows, the other one;  K: within a slice of the weights, over one
@pytest.mark.parametrize("shape", [(1, 7, 1), (5, 40, 2), (37, 784, 10), (601, 96, 16), (1185, 1500, 3), (1187, 2100, 13), (1300, 64, 16)])
def test_a_head_gives_its_probabilities_with_its_logits(sc, shape):
    """The bits of the softmax launch, infinite and undefined logits among them."""
    M, K, N = shape
    rs = np.random.RandomState(sum(shape))
    a, b, bias = (rs.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N), (N,)))
    a[M // 2, 0], a[M - 1, K // 2] = np.inf, np.nan
    ad, bd, biasd = (sc.to_device_f32(t.ravel()) for t in (a, b, bias))
    c, p, alone, q = (sc.cuda_malloc_f32(M * N + 1) for _ in range(4))
    for out in (c, p, alone, q):
        sc.upload_f32(out, np.full(M * N + 1, 7, np.float32))
    before = sc.launch_count()
    assert sc.matmul_softmax_fwd(ad, bd, biasd, c, p, M, N, K)
    assert sc.launch_count() == before + 1
    sc.matmul_bias_act_fwd(ad, bd, biasd, alone, M, N, K, 0)
    sc.cuda_softmax_fwd(alone, q, M, N)
    bits = [sc.to_host_f32(t, (M * N + 1,)).view(np.int32) for t in (c, alone, p, q)]
    assert np.array_equal(bits[0], bits[1]) and np.array_equal(bits[2], bits[3])
    sc.set_precision(0)
    assert not sc.matmul_softmax_fwd(ad, bd, biasd, c, p, M, N, K)
    for t in (ad, bd, biasd, c, p, alone, q):
        sc.cuda_free(t)


@pytest.mark.parametrize("classes,predicted", [(10, 1), (40, None)])
def test_the_loss_of_a_prediction_takes_one_launch(sc, classes, predicted):
    from ml_framework_b200 import seera as S
    rs = np.random.RandomState(classes)
    model, lossf = S.Sequential([S.Input((50,)), S.Dense(50, classes, "softmax")]), S.Loss().categorical_cross_entropy
    x = S.Tensor(rs.standard_normal((64, 50)).astype(np.float32), is_leaf=True)
    y = S.Tensor(np.eye(classes, dtype=np.float32)[rs.randint(0, classes, 64)], is_leaf=True)
    for _ in range(3):                          # the first pass, and batched ones
        counts = [sc.launch_count()]
        pred = model.predict(x)
        counts.append(sc.launch_count())
        loss = lossf(pred, y)
        counts.append(sc.launch_count())
        assert predicted is None or counts[1] - counts[0] == predicted
        assert counts[2] - counts[1] == 1
        values = pred.to_numpy()
        assert np.array_equal(values, model.predict(x).to_numpy()) and loss.item() > 0


def test_losses_on_two_streams_finish_each_by_itself():
    """On the library's stream, on a caller's, and recorded and replayed on the caller's: more launches than there ever were counters."""
    import torch
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    sc.set_precision(3)
    N, C, n = 60000, 10, 500000
    rs = np.random.RandomState(4)
    z, y = rs.standard_normal((N, C)).astype(np.float32), np.eye(C, dtype=np.float32)[rs.randint(0, C, N)]
    a, b = rs.standard_normal(n).astype(np.float32), rs.standard_normal(n).astype(np.float32)
    dz, dy, da, db = (sc.to_device_f32(v) for v in (z, y, a, b))
    lp = z.astype(np.float64) - np.log(np.exp(z.astype(np.float64)).sum(1, keepdims=True))
    want = (-(y * lp).sum(1).mean(), ((a.astype(np.float64) - b) ** 2).mean())
    side = torch.cuda.Stream()

    def buffers():
        return ([sc.cuda_malloc_f32(k) for k in (N * C, N, 1, N * C)], [sc.cuda_malloc_f32(k) for k in (sc.mse_partials(n), 1, n)])

    def losses(bufs):
        (p, rows, loss, grad), (part, mse, dp) = bufs
        sc.softmax_cce_fwd_bwd(dz, dy, p, rows, loss, grad, N, C, 1e-7, 1.0 / N)
        sc.mse_fwd_bwd(da, db, part, mse, dp, n, 1.0 / n)
    own, theirs, recorded = buffers(), buffers(), [buffers() for _ in range(2)]
    sc.stream_synchronize()
    graphs = []
    for bufs in recorded:
        sc.graph_begin()
        losses(bufs)
        graphs.append(sc.graph_end())
    try:
        for rep in range(100):
            sc.set_stream(side.cuda_stream)
            losses(theirs)
            sc.graph_launch(graphs[0])
            sc.set_stream(0)
            losses(own)
            sc.graph_launch(graphs[1])
            if rep % 10 == 9:
                torch.cuda.synchronize()
                for bufs in [own, theirs] + recorded:
                    got = [float(sc.to_host_f32(q, (1,))[0]) for q in (bufs[0][2], bufs[1][1])]
                    assert np.allclose(got, want, rtol=1e-5), got
                    sc.cuda_memset(bufs[0][2], 0, 4)
                    sc.cuda_memset(bufs[1][1], 0, 4)
                torch.cuda.synchronize()
    finally:
        sc.set_stream(0)
        torch.cuda.synchronize()
        for g in graphs:
            sc.graph_destroy(g)
        for bufs in [own, theirs] + recorded:
            for q in bufs[0] + bufs[1]:
                sc.cuda_free(q)
        for q in (dz, dy, da, db):
            sc.cuda_free(q)
        sc.set_precision(0)


def test_more_recorded_losses_than_counters():
    """Beyond the counters that recordings hold a launch brings a word of its own; a destroyed recording gives its counters back.  The same
    for callers' streams."""
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    sc.set_precision(3)
    n = 5000
    a, b = np.linspace(-1, 1, n, dtype=np.float32), np.linspace(1, 3, n, dtype=np.float32)
    da, db = sc.to_device_f32(a), sc.to_device_f32(b)
    part, dp = sc.cuda_malloc_f32(sc.mse_partials(n)), sc.cuda_malloc_f32(n)
    want = float(((a.astype(np.float64) - b) ** 2).mean())
    for rep in range(3):
        out = [sc.cuda_zeros_f(1) for _ in range(300)]
        sc.graph_begin()
        for q in out:
            sc.mse_fwd_bwd(da, db, part, q, dp, n, 1.0 / n)
        g = sc.graph_end()
        for _ in range(2):
            sc.graph_launch(g)
        assert np.allclose([float(sc.to_host_f32(q, (1,))[0]) for q in out], want, rtol=1e-5)
        sc.graph_destroy(g)
        for q in out:
            sc.cuda_free(q)
    import torch
    streams = [torch.cuda.Stream() for _ in range(32)]       # (torch has 32 a device and deals them out in turn)
    loss = sc.cuda_zeros_f(1)
    for rep in range(3):
        for st in streams:
            sc.set_stream(st.cuda_stream)
            sc.cuda_memset(loss, 0, 4)
            sc.mse_fwd_bwd(da, db, part, loss, dp, n, 1.0 / n)
            assert np.allclose(sc.to_host_f32(loss, (1,)), want, rtol=1e-5)
    sc.set_stream(0)
    for q in (da, db, part, dp, loss):
        sc.cuda_free(q)
    sc.set_precision(0)


@pytest.mark.parametrize("entry", ["convolution", "dense", "update"])
def test_a_loss_gradient_that_was_written_since_has_a_factor_of_its_own(sc, entry):
    """In the fp16 modes: scaled in place by a power of two that leaves fp16's range, at the address that the loss launch knew."""
    N, C, H, F = 2, 16, 8, 32
    rs = np.random.RandomState(2)
    p, y = (rs.standard_normal(N * F * H * H).astype(np.float32) for _ in range(2))
    x, w = rs.standard_normal((N, C, H, H)).astype(np.float32), rs.standard_normal((F, C, 3, 3)).astype(np.float32)
    d = [sc.to_device_f32(a.ravel()) for a in (p, y, x, w)]
    part, loss, dp, dx, dw = (sc.cuda_malloc_f32(n) for n in (sc.mse_partials(p.size), 1, p.size, max(x.size, p.size), max(w.size, F * F)))
    sc.set_precision(4)
    for factor in (1.0, 2.0 ** 20, 2.0 ** -30):
        sc.mse_fwd_bwd(d[0], d[1], part, loss, dp, p.size, 1.0 / p.size)
        sc.cuda_scaler_multiply_f(dp, factor, p.size)
        g = sc.to_host_f32(dp, (p.size,)).astype(np.float64)
        if entry == "dense":                                 # [N H H, F] @ [F, F]: dB = A^T g
            M = N * H * H
            sc.cuda_matmul_bwd(d[0], d[3], dp, dx, dw, M, F, F, 1)
            got, want = sc.to_host_f32(dw, (F, F)), p.reshape(M, F).T.astype(np.float64) @ g.reshape(M, F)
        else:
            if entry == "update":
                sc.grad_scale_update(dp, p.size)
            sc.cuda_conv2d_bwd(d[3], d[2], dp, dx, dw, N, C, H, H, F, 3, 3, 1, 1, 1, 1)
            import torch
            got = sc.to_host_f32(dw, w.shape)
            want = torch.nn.grad.conv2d_weight(torch.from_numpy(x).double(), w.shape, torch.from_numpy(g.reshape(N, F, H, H)), padding=1).numpy()
        assert rel_l2(got, want) < 1e-3, factor              # weight gradients of this mode: one fp16 copy of each operand
    for q in d + [part, loss, dp, dx, dw]:
        sc.cuda_free(q)


def test_a_launch_of_both_gradients_is_booked_as_such(sc):
    """Neither under the data gradients nor under the weight gradients: of a classifier head, of a small convolution, of an unpooled image."""
    M, K, N = 600, 96, 10
    images, C, F, H = 8, 8, 16, 14
    a, b, g = (sc.cuda_zeros_f(n) for n in (M * K, K * N, M * N))
    x, w, dy = (sc.cuda_zeros_f(n) for n in (images * C * H * H, F * C * 9, images * F * H * H))
    low = images * C * H * H                             # an unpooled layer's input, twice the height and width in its output
    u, du, yu, gu = (sc.cuda_zeros_f(n) for n in (low, low, 4 * images * H * H, 4 * images * H * H))
    wu, dwu, dbu = (sc.cuda_zeros_f(n) for n in (C * 9, C * 9, 1))
    out = {n: sc.cuda_zeros_f(n) for n in {M * K, K * N, images * C * H * H, F * C * 9}}
    sc.profile_enable(1)
    try:
        sc.cuda_matmul_bwd(a, b, g, out[M * K], out[K * N], M, N, K, 1)
        sc.cuda_conv2d_bwd(w, x, dy, out[images * C * H * H], out[F * C * 9], images, C, H, H, F, 3, 3, 1, 1, 1, 1)
        sc.unpool2_convT_act_bwd(wu, u, yu, gu, du, dwu, dbu, images, C, H, H, 2)
        table, kinds = sc.profile_report(), sc.profile_read_kinds()
    finally:
        sc.profile_enable(0)
    assert {tag: (kind, n, work) for tag, kind, n, _, work in table if kind != 3} == {
        "cuda_matmul_bwd(dA+dB)": (4, 1, 4 * M * N * K), "conv2d_small_bwd(dX+dW)": (4, 1, 4 * images * H * H * F * C * 9),
        "unpool2_convT_bwd(dX+dW)": (4, 1, 16 * images * H * H * C * 9)}
    assert [k[0] for k in kinds] == [0, 0, 0]
    for p in (a, b, g, x, w, dy, u, du, yu, gu, wu, dwu, dbu, *out.values()):
        sc.cuda_free(p)
