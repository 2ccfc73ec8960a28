"""Branches of the bandwidth-bound passes that their general tests do not reach: whole planes of batch normalisation by size, broadcast axes
that merge or take 16-byte pieces."""
import numpy as np
import pytest

import test_gpu_ops as ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(200, 9, 2, 2), (33, 7, 4, 4), (5, 40, 32, 32), (3, 2, 36, 36), (130, 3, 8, 8), (700, 40)])
def test_batchnorm_planes(shape):
    ops.test_batchnorm_forward_and_backward(shape)


@pytest.mark.parametrize("a,b", [((1, 1, 1000, 1024), (1, 1, 1, 1024)), ((1, 1, 129, 64), (1, 1, 129, 1)), ((3, 5, 7, 8), (1, 5, 1, 1)), ((1, 1, 1, 12), (6, 1, 5, 12)),
                                 ((4, 1, 3, 16), (4, 6, 1, 16)), ((2, 3, 4, 5), (2, 3, 4, 5)), ((1, 1, 1, 1), (1, 1, 1, 1)), ((1, 1, 1, 1), (2, 2, 2, 4))])
@pytest.mark.parametrize("shift", [0, 1])                    # an operand that is not 16-byte aligned
def test_broadcast_axes(a, b, shift):
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    rs = np.random.RandomState(sum(a) + sum(b))
    x, y = rs.standard_normal(a).astype(np.float32), rs.standard_normal(b).astype(np.float32)
    p, q = sc.to_device_f32(np.concatenate([np.zeros(shift, np.float32), x.ravel()])), sc.to_device_f32(y.ravel())
    want = x + y
    o = sc.cuda_malloc_f32(want.size)
    for f, ref in ((sc.broadcast_add_4d, want), (sc.broadcast_mul_4d, x * y)):
        f(p + 4 * shift, q, o, *a, *b)
        assert np.array_equal(sc.to_host_f32(o, ref.shape), ref)
        f(q, p + 4 * shift, o, *b, *a)
        assert np.array_equal(sc.to_host_f32(o, ref.shape), ref)
    for t in (p, q, o):
        sc.cuda_free(t)


@pytest.mark.parametrize("M,K,N,shift", [(64, 784, 10, 0), (8, 33, 3, 0), (700, 1024, 10, 0), (700, 1024, 10, 1), (513, 1026, 16, 0), (1, 5, 1, 0), (300, 2050, 7, 0)])
def test_both_gradients_of_a_narrow_product(M, K, N, shift):
    """One launch for dA and dB; every pairing of their widths (16-byte rows of dA, 8-byte rows of A or not)."""
    from conftest import rel_l2
    from ml_framework_b200 import seera_cuda as sc
    sc.init(0)
    sc.set_precision(3)
    rs = np.random.RandomState(M + K + N)
    a, b, g = (rs.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N), (M, N)))
    ad, bd, gd = sc.to_device_f32(np.concatenate([np.zeros(shift, np.float32), a.ravel()])), sc.to_device_f32(b.ravel()), sc.to_device_f32(g.ravel())
    da, db = sc.cuda_malloc_f32(M * K), sc.cuda_malloc_f32(K * N)
    sc.cuda_matmul_bwd(ad + 4 * shift, bd, gd, da, db, M, N, K, 1)
    assert rel_l2(sc.to_host_f32(da, (M, K)), g.astype(np.float64) @ b.T) < 1e-6
    assert rel_l2(sc.to_host_f32(db, (K, N)), a.T.astype(np.float64) @ g) < 2e-6            # 32-bit sums over up to 700 rows
    for p in (ad, bd, gd, da, db):
        sc.cuda_free(p)
    sc.set_precision(0)


def test_axes_of_a_reduction():
    """What is kept of a shape per axis does not take an axis for another: arrays count as they stand, a float is refused."""
    import torch

    from ml_framework_b200.cuTen import cuten
    x = np.arange(24, dtype=np.float32).reshape(2, 3, 4)
    c, axis, t = cuten(x), np.array(1), torch.tensor(1)
    for dim in (1, np.int64(1), axis, t, -2, True):
        assert np.array_equal(c.sum(dim).to_host_f32(), x.sum(1))
    axis[...], t[...] = 0, 0
    for dim in (axis, t):
        assert np.array_equal(c.sum(dim).to_host_f32(), x.sum(0))
    with pytest.raises(TypeError):
        c.sum(1.0)
    with pytest.raises(ValueError):
        c.sum(3)
