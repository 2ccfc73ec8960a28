"""Batches of launches (seera_batch_begin / _end) and the kept page-locked blocks: what they hand to the device is what the same
calls, made one by one, would have."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sc():
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    yield sc
    sc.set_precision(0)
    assert sc.tc_device_status() == 0


def _chain(sc, n, k, reader=False):
    """k in-place additions after a fill; `reader`: a read-back in the middle."""
    p = sc.cuda_ones_f(n)
    for i in range(k):
        sc.cuda_scaler_add_f(p, float(i + 1), n)
        if reader and i == k // 2:
            mid = float(sc.to_host_f32(p, (n,))[0])
            assert mid == 1 + sum(range(1, i + 2))
    return p


@pytest.mark.parametrize("n,k", [(1, 1), (1000, 7), (4096, 64)])
def test_a_batch_runs_its_launches_in_order(sc, n, k):
    want = 1 + sum(range(1, k + 1))
    for rep in range(4):                                     # the executable graph is built, then updated with other addresses
        sc.batch_begin(17)
        p = _chain(sc, n, k)
        sc.batch_end()
        assert np.all(sc.to_host_f32(p, (n,)) == want)
        if rep % 2:
            sc.cuda_free(p)


def test_a_read_inside_a_batch_sees_what_came_before_it(sc):
    for _ in range(3):
        sc.batch_begin(18)
        sc.batch_begin(19)                                   # nested: the outer one counts
        p = _chain(sc, 100, 6, reader=True)
        sc.batch_end()
        sc.batch_end()
        assert np.all(sc.to_host_f32(p, (100,)) == 22)


def test_a_tag_may_bring_other_launches(sc):
    x = sc.to_device_f32(np.linspace(-1, 1, 256, dtype=np.float32))
    for k in range(6):
        o, g = sc.cuda_malloc_f32(256), sc.cuda_malloc_f32(256)
        sc.batch_begin(20)
        (sc.cuda_relu_fwd if k % 2 else sc.cuda_abs_fwd)(x, o, g, 256)
        sc.cuda_scaler_multiply_f(o, 2.0, 256)
        sc.batch_end()
        h = np.linspace(-1, 1, 256, dtype=np.float32)
        assert np.array_equal(sc.to_host_f32(o, (256,)), 2 * (np.maximum(h, 0) if k % 2 else np.abs(h)))
    with pytest.raises(RuntimeError):
        sc.batch_end()                                       # none is open
    from ml_framework_b200 import capi
    capi.load().seera_clear_status()


@pytest.mark.parametrize("name,n", [("c1", 5), ("c2", 33), ("c4", 3)])
def test_batched_steps_equal_launches_one_by_one(sc, name, n, monkeypatch):
    from ml_framework_b200 import seera as S, train, workloads as wl
    work = wl.WORKLOADS[name]()
    X, Y = work.batch(n, 5)
    got = []
    for batched in (True, False):
        if not batched:
            monkeypatch.setattr(S, "_batch_begin", None)
        tr = train.Trainer(work, seed=5, precision=train.policy_for(work))
        x, y = S.Tensor(X, is_leaf=True), S.Tensor(Y, is_leaf=True)
        losses = [float(tr.step(x, y).value.to_host_f32()[0]) for _ in range(5)]
        pred = tr.model.predict(X).to_numpy()
        got.append((losses, pred, [p for p in tr.host_params() if p is not None]))
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
    for a, b in zip(got[0][2], got[1][2]):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("nbytes", [1, 4096, 5000, (1 << 20) + 1])
def test_page_locked_blocks_are_used_again_only_when_their_copies_have_passed(sc, nbytes):
    n = max(1, nbytes // 4)
    d = sc.cuda_zeros_f(n)
    sc.stream_synchronize()
    for k in range(4):
        p = sc.host_alloc_pinned(4 * n)
        sc.host_view(p, 4 * n).view(np.float32)[:] = k
        if k % 2:
            sc.stream_delay(300)
        sc.upload_from_host_ptr(d, p, 4 * n)
        sc.host_free_pinned(p)                               # the upload may still be reading it
        q = sc.host_alloc_pinned(4 * n)
        sc.host_view(q, 4 * n).view(np.float32)[:] = -1
        assert np.all(sc.to_host_f32(d, (n,)) == k)
        sc.host_free_pinned(q)
    sc.cuda_free(d)


@pytest.mark.parametrize("labels", [False, True])
def test_a_recorded_fit_equals_an_eager_one(monkeypatch, labels):
    """Ragged last batches between replays, BatchNorm's running statistics, history, weights and what the layers hold afterwards."""
    from ml_framework_b200 import seera as S, seera_cuda as sc
    sc.init(0)
    sc.set_precision(3)
    rs = np.random.RandomState(4)
    X, lab = rs.standard_normal((75, 1, 8, 8)).astype(np.float32), rs.randint(0, 5, 75).astype(np.int32)
    runs = []
    for first in (10 ** 9, 1):
        monkeypatch.setattr(S, "_RECORD_FROM", first)
        np.random.seed(2)
        m = S.Sequential([S.Input((1, 8, 8)), S.Conv2D(8, 1, (3, 3), "relu", stride=1, zero_padding=1), S.BatchNorm2d(8),
                          S.MaxPool2D((2, 2), stride=2), S.Flatten(), S.Dense(128, 5, activation="softmax")])
        opt = S.Adam(m, lr=1e-2)
        h = m.fit(X, lab if labels else np.eye(5, dtype=np.float32)[lab], opt, S.Loss().categorical_cross_entropy, Epochs=3, batch_size=16,
                  Loss_interval=100, num_classes=5 if labels else None)
        bn = m.model[2]
        runs.append([h, opt.t, bn._rm.to_host_f32(), bn._rv.to_host_f32(), m.model[-1].outputs.to_numpy(),
                     *(t.to_numpy() for t in m.parameters()), *(t.grad.to_host_f32() for t in m.parameters())])
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
    sc.set_precision(0)


def test_recordings_made_from_one_another():
    """A recording destroyed leaves its executable to the next of as many launches: other operators, addresses and optimizer scalars."""
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    n = 1000
    rs = np.random.RandomState(0)
    host = [rs.standard_normal(n).astype(np.float32) for _ in range(3)]
    for round_ in range(8):
        d = [sc.to_device_f32(a) for a in host]
        out, vel = sc.cuda_malloc_f32(n), sc.cuda_zeros_f(n)
        other = round_ % 3
        sc.graph_begin()
        (sc.cuda_elemadd, sc.cuda_elemmult, sc.cuda_elemadd)[other](d[0], d[1], out, n)
        sc.cuda_sgd_step(d[2], out, vel, n, 0.1, 0.0, 1.0)
        if other == 2:
            sc.cuda_elemadd(d[0], d[0], out, n)
        g = sc.graph_end()
        w = host[2].copy()
        base = host[0] * host[1] if other == 1 else host[0] + host[1]
        for lr in (0.5, 0.25):
            sc.graph_set_scalars(g, [lr, 0.0, 1.0])
            sc.graph_launch(g)
            w = w - np.float32(lr) * base
        assert np.allclose(sc.to_host_f32(d[2], (n,)), w, rtol=1e-6, atol=1e-6)
        sc.graph_destroy(g)
        if round_ == 5:
            sc.pool_trim()
        for p in d + [out, vel]:
            sc.cuda_free(p)


@pytest.mark.parametrize("n0,n1,shift", [(1, 0, 0), (0, 5, 0), (3, 17, 1), (4096, 10, 0), (1000003, 640, 2), (70, 2000000, 4)])
def test_three_copies_in_one_launch(n0, n1, shift):
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    rs = np.random.RandomState(n0 + n1)
    a, b = (rs.standard_normal(n + shift).astype(np.float32) for n in (n0, n1))
    src = [sc.to_device_f32(t) for t in (np.append(a, 0.0).astype(np.float32), np.append(b, 0.0).astype(np.float32))]
    dst, last = [sc.cuda_zeros_f(n + 1) for n in (n0, n1)], sc.cuda_zeros_f(2)
    sc.copy_three(dst[0], src[0] + 4 * shift, n0, dst[1], src[1] + 4 * shift, n1, last, src[0], 1)
    for d, t, n in ((dst[0], a, n0), (dst[1], b, n1)):
        got = sc.to_host_f32(d, (n + 1,))
        assert np.array_equal(got[:n], t[shift:]) and got[n] == 0
    assert np.array_equal(sc.to_host_f32(last, (2,)), [np.append(a, 0.0).astype(np.float32)[0], 0])
    for p in src + dst + [last]:
        sc.cuda_free(p)


@pytest.mark.parametrize("transposed", [False, True])
def test_gradient_entries_submitted_as_one_batch(transposed):
    """The first call of a shape launches one by one, later ones as a batch: the same bits, other addresses, other operands, no data gradient."""
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    for mode in (1, 3, 4):
        sc.set_precision(mode)
        N, C, H, W, F = 3, 20, 9, 11, 24
        call = sc.cuda_conv2DTranspose_bwd if transposed else sc.cuda_conv2d_bwd
        got = []
        for k in range(5):
            rs = np.random.RandomState(7 + k % 2)
            ci, co = (C, F)
            x, g = (rs.standard_normal((N, c, H, W)).astype(np.float32) for c in (ci, co))
            w = rs.standard_normal((C, F, 3, 3) if transposed else (F, C, 3, 3)).astype(np.float32)
            hold = sc.cuda_malloc_f32(1000 * (k + 1))                    # other addresses than the call before
            d = [sc.to_device_f32(a.ravel()) for a in (w, x, g)]
            dx, dw = sc.cuda_malloc_f32(x.size), sc.cuda_malloc_f32(w.size)
            call(d[0], d[1], d[2], dx if k < 4 else 0, dw, N, C, H, W, F, 3, 3, 1, 1, 1, 1)
            got.append((sc.to_host_f32(dx, x.shape) if k < 4 else None, sc.to_host_f32(dw, w.shape)))
            for p in d + [dx, dw, hold]:
                sc.cuda_free(p)
        assert np.array_equal(got[0][0], got[2][0]) and np.array_equal(got[1][0], got[3][0])
        assert all(np.array_equal(got[k][1], got[k + 2][1]) for k in range(3)) and not np.array_equal(got[0][1], got[1][1])
    sc.set_precision(0)


def test_more_rows_of_kernels_than_are_kept(sc):
    """64 rows have an executable from their second time on, the rest is launched call by call: kernels (some of them clusters), fills and
    copies, at other addresses each time."""
    n, m = 1000, 256
    rs = np.random.RandomState(3)
    a, b = (rs.standard_normal((m, m)).astype(np.float32) for _ in range(2))
    da, db, dc = sc.to_device_f32(a), sc.to_device_f32(b), sc.cuda_malloc_f32(m * m)
    sc.set_precision(1)
    sc.pool_trim()
    try:
        for pair in (0, 1):
            sc.set_option("pair_tiles", pair)
            sc.cuda_matmul(da, db, dc, m, m, m, 1)
            want = sc.to_host_f32(dc, (m, m))
            hold = []
            for rep in range(4):
                for tag in range(40):
                    p, q = sc.cuda_ones_f(n), sc.cuda_malloc_f32(n)
                    sc.cuda_memset(dc, 255, 4 * m * m)
                    sc.batch_begin((1000 << 8) + tag)
                    sc.cuda_memset(q, rep, 4 * n)
                    sc.cuda_scaler_add_f(p, float(tag + rep), n)
                    sc.cuda_memcopy_devicetodevice(q, p, n // 2 + rep)
                    sc.cuda_scaler_multiply_f(q, 2.0, n)
                    sc.cuda_matmul(da, db, dc, m, m, m, 1)
                    sc.batch_end()
                    got, fill = sc.to_host_f32(q, (n,)), np.frombuffer(bytes([rep] * 4), np.float32)[0]
                    assert np.all(got[:n // 2 + rep] == 2 * (tag + rep + 1)) and np.all(got[n // 2 + rep:] == 2 * fill)
                    assert np.array_equal(sc.to_host_f32(dc, (m, m)), want)
                    hold.append(p)                           # the next one gets another address
                    sc.cuda_free(q)
                assert sc.batches_kept() == (0 if rep == 0 else 40) if not pair else sc.batches_kept() == (40 if rep == 0 else 64)
            for p in hold:
                sc.cuda_free(p)
    finally:
        sc.set_option("pair_tiles", 0)
        sc.set_precision(0)
        for p in (da, db, dc):
            sc.cuda_free(p)


def test_predictions_over_more_sizes_than_executables_are_kept(sc, monkeypatch):
    """A server's batches: no size waits for another's executable.  The time allows a quarter over launches made one by one."""
    import time
    from ml_framework_b200 import seera as S, train, workloads as wl
    sc.set_precision(3)
    work = wl.WORKLOADS["c1"]()
    model = train.build_model(work, work.params(1))
    xs = [S.Tensor(work.batch(n, n)[0], is_leaf=True) for n in range(1, 121)]
    took, got = [], []
    for batched in (False, True):
        monkeypatch.setattr(S, "_batch_begin", sc.batch_begin if batched else None)
        best = 1e9
        for rep in range(12):
            sc.stream_synchronize()
            t = time.perf_counter()
            out = [model.predict(x) for x in xs]
            sc.stream_synchronize()
            if rep:
                best = min(best, time.perf_counter() - t)
        took.append(best)
        got.append([o.to_numpy() for o in out])
    assert all(np.array_equal(a, b) for a, b in zip(*got))
    assert sc.batches_kept() <= 64
    assert took[1] <= 1.25 * took[0], took
    sc.set_precision(0)


def test_trimming_gives_back_the_executables_of_batches(sc):
    for rep in range(3):
        p = sc.cuda_ones_f(100)
        for k in (2, 3, 2, 3):
            sc.batch_begin(21)
            for i in range(k):
                sc.cuda_scaler_add_f(p, 1.0, 100)
            sc.batch_end()
        assert sc.batches_kept() >= 2
        sc.pool_trim()                                       # the last batch may still be running
        assert sc.batches_kept() == 0
        assert np.all(sc.to_host_f32(p, (100,)) == 11)
        sc.cuda_free(p)


def _device_now(ptr):
    """The first value at an address once the device has nothing left to do, past the library."""
    import ctypes
    cu, v = ctypes.CDLL("libcuda.so.1"), np.empty(1, np.float32)
    assert cu.cuCtxSynchronize() == 0
    assert cu.cuMemcpyDtoH_v2(v.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(ptr), ctypes.c_size_t(4)) == 0
    return float(v[0])


def test_a_batch_that_grows_the_pool_goes_on_launch_by_launch(sc):
    """The device works through what came before while the driver looks for memory; blocks at hand leave the batch together."""
    n = (37 << 20) // 4
    sc.pool_trim()
    for rep in range(2):
        p = sc.cuda_ones_f(100)
        sc.batch_begin(22)
        sc.cuda_scaler_add_f(p, 1.0, 100)
        assert _device_now(p) == 1
        q = sc.cuda_malloc_f32(n)                            # from the driver the first time, from the pool the second
        assert _device_now(p) == (2 if rep == 0 else 1)
        sc.cuda_memset(q, 0, 4 * n)
        sc.cuda_scaler_add_f(p, 1.0, 100)
        sc.batch_end()
        assert np.all(sc.to_host_f32(p, (100,)) == 3) and not sc.to_host_f32(q, (n,)).any()
        sc.cuda_free(p)
        sc.cuda_free(q)


def test_another_thread_may_synchronise_the_device_during_a_batch(sc):
    import threading
    import torch
    x = torch.ones(1000, device="cuda")
    for rep in range(3):
        p, seen = sc.cuda_ones_f(100), []

        def other():
            torch.cuda.synchronize()
            seen.append(float((2 * x).sum()))
        sc.batch_begin(25)
        sc.cuda_scaler_add_f(p, 1.0, 100)
        t = threading.Thread(target=other)
        t.start()
        t.join()
        sc.cuda_scaler_multiply_f(p, 3.0, 100)
        sc.batch_end()
        assert seen == [2000.0] and np.all(sc.to_host_f32(p, (100,)) == 6)
        sc.cuda_free(p)


@pytest.mark.parametrize("k,parts", [(11, 1), (12, 2), (40, 2)])
def test_an_idle_device_gets_a_long_inner_batch_at_its_end(sc, k, parts):
    for rep in range(3):
        p = sc.cuda_ones_f(100)
        sc.stream_synchronize()
        sc.batch_begin(23)
        for inner in range(2):
            sc.batch_begin(24)
            for i in range(k):
                sc.cuda_scaler_add_f(p, 1.0, 100)
            sc.batch_end()
            assert _device_now(p) == (1 + k if parts > 1 else 1)
        sc.cuda_scaler_multiply_f(p, 2.0, 100)
        sc.batch_end()
        assert np.all(sc.to_host_f32(p, (100,)) == 2 * (1 + 2 * k))
        sc.cuda_free(p)


def test_launches_of_one_kernel_with_less_and_less_shared_memory(sc):
    """The limit on dynamic shared memory belongs to the kernel: a later launch's does not take it from one that is held back."""
    rs = np.random.RandomState(6)
    sc.set_precision(2)
    N, C, H, W = 2, 4, 20, 20
    x = sc.to_device_f32(rs.standard_normal(N * C * H * W).astype(np.float32))
    ws = [(F, sc.to_device_f32(rs.standard_normal(F * C * 9).astype(np.float32)), sc.cuda_malloc_f32(N * F * H * W)) for F in (304, 208, 64)]
    got = []
    for batched in (False, True, True, True):
        if batched:
            sc.batch_begin(26)
        for F, w, y in ws:
            sc.cuda_conv2d_fwd(x, w, y, N, C, H, W, F, 3, 3, 1, 1, 1, 1)
        if batched:
            sc.batch_end()
        got.append([sc.to_host_f32(y, (N, F, H, W)) for F, w, y in ws])
        for F, w, y in ws:
            sc.cuda_memset(y, 0, 4 * N * F * H * W)
    for g in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(g, got[0]))
    for F, w, y in ws:
        sc.cuda_free(w)
        sc.cuda_free(y)
    sc.cuda_free(x)
    sc.set_precision(0)


def test_a_recording_keeps_its_update_apart_from_the_spares(sc):
    """As many launches and updates as a destroyed recording had, the update elsewhere: its scalars go to the update."""
    n = 1000
    rs = np.random.RandomState(1)
    a, b, w = (rs.standard_normal(n).astype(np.float32) for _ in range(3))
    for first in (True, False, True, False):
        da, db, dw = (sc.to_device_f32(x) for x in (a, b, w))
        out, vel = sc.cuda_malloc_f32(n), sc.cuda_zeros_f(n)
        sc.graph_begin()
        if first:
            sc.cuda_elemadd(da, db, out, n)
        sc.cuda_sgd_step(dw, da, vel, n, 0.1, 0.0, 1.0)
        if not first:
            sc.cuda_elemadd(da, db, out, n)
        g = sc.graph_end()
        sc.graph_set_scalars(g, [0.5, 0.0, 1.0])
        sc.graph_launch(g)
        assert np.array_equal(sc.to_host_f32(out, (n,)), a + b)
        assert np.allclose(sc.to_host_f32(dw, (n,)), w - 0.5 * a, rtol=1e-6, atol=1e-6)
        sc.graph_destroy(g)
        for p in (da, db, dw, out, vel):
            sc.cuda_free(p)


def test_a_recorded_update_that_cannot_be_found_again_is_an_error(sc):
    """It would keep the scalars of the step it was recorded in."""
    n = 100
    d = [sc.cuda_ones_f(n) for _ in range(4)]
    for lost in (True, False):
        sc.set_option("graph_test_lose_update", int(lost))
        sc.graph_begin()
        try:
            if lost:
                with pytest.raises(RuntimeError, match="scalars"):
                    sc.cuda_sgd_step(d[0], d[1], d[2], n, 0.5, 0.0, 1.0)
            else:
                sc.cuda_sgd_step(d[0], d[1], d[2], n, 0.5, 0.0, 1.0)
        finally:
            g = sc.graph_end()
        if lost:
            with pytest.raises(RuntimeError, match="scalars"):
                sc.graph_set_scalars(g, [0.25, 0.0, 1.0])
        else:
            sc.graph_set_scalars(g, [0.25, 0.0, 1.0])
            sc.graph_launch(g)
            assert np.all(sc.to_host_f32(d[0], (n,)) == 0.75)
        sc.graph_destroy(g)
    sc.clear_status()
    for p in d:
        sc.cuda_free(p)


def test_batches_of_two_threads(sc):
    """Each thread's are its own: what one has ended is on the device whatever the other has open, and all calls keep their order."""
    import threading
    p, q = sc.cuda_ones_f(100), sc.cuda_ones_f(100)
    sc.stream_synchronize()
    turn, log = [threading.Event() for _ in range(6)], []

    def other():
        turn[0].wait(10)
        sc.cuda_scaler_multiply_f(p, 10.0, 100)              # between the two of the first thread's batch, which goes on call by call
        log.append(_device_now(p))
        turn[1].set()
        turn[2].wait(10)
        sc.batch_begin(31)
        sc.cuda_scaler_add_f(q, 1.0, 100)
        turn[3].set()
        turn[4].wait(10)
        sc.cuda_scaler_multiply_f(q, 2.0, 100)
        sc.batch_end()
        turn[5].set()
    t = threading.Thread(target=other)
    t.start()
    sc.batch_begin(30)
    sc.cuda_scaler_add_f(p, 1.0, 100)
    assert _device_now(p) == 1
    turn[0].set()
    turn[1].wait(10)
    assert log == [20]
    sc.cuda_scaler_add_f(p, 1.0, 100)
    turn[2].set()
    turn[3].wait(10)
    sc.batch_end()
    assert _device_now(p) == 21 and _device_now(q) == 1      # the other's is still open
    turn[4].set()
    turn[5].wait(10)
    t.join()
    assert _device_now(q) == 4
    with pytest.raises(RuntimeError):
        sc.batch_end()
    sc.clear_status()
    for x in (p, q):
        sc.cuda_free(x)
