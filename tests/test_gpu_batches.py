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
