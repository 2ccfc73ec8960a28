"""Tiles of the TMA-fed products where they can go wrong: accumulator widths with the operand copies of B joined, ragged edges, every
activation of the epilogues, windows of a pooled epilogue without one maximum.  Against float64."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

#: bf16x3 leaves 2^-17 of a product out, bf16x6 and fp16x3 2^-22 or less; their sums run in 32 bits (see test_gpu_tensorcore.py).
TOL = {1: 1e-2, 2: 2e-5, 3: 4e-6, 4: 1e-5}


@pytest.fixture
def sc():
    from ml_framework_b200 import capi, seera_cuda as sc
    sc.init(0)
    sc.set_option("skinny_gemm", 0)
    yield sc
    sc.set_option("skinny_gemm", 1)
    sc.set_precision(0)
    assert capi.load().seera_tc_device_status() == 0


def activated(z, act):
    return [z, np.maximum(z, 0), 1 / (1 + np.exp(-z)), np.tanh(z)][act]


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("M,N,K", [(127, 17, 65), (129, 64, 192), (260, 65, 640), (33, 96, 130), (300, 131, 72), (128, 257, 448),
                                   (200, 33, 4100), (1, 300, 2304), (700, 130, 1000)])       # few tiles: clusters of every size share them
def test_widths_and_edges(sc, mode, M, N, K):
    sc.set_precision(mode)
    rs = np.random.RandomState(M + N + K)
    a, w, b = (rs.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N), (N,)))
    g = (rs.standard_normal((M, N)) / 8).astype(np.float32)
    act = (M + mode) % 4
    w /= np.float32(np.sqrt(K))
    ad, wd, bd, gd = (sc.to_device_f32(t.ravel()) for t in (a, w, b, g))
    y, da, dw = (sc.cuda_malloc_f32(n) for n in (M * N, M * K, K * N))
    sc.matmul_bias_act_fwd(ad, wd, bd, y, M, N, K, act)
    ref = activated(a.astype(np.float64) @ w + b, act)
    assert rel_l2(sc.to_host_f32(y, (M, N)), ref) < TOL[mode]
    sc.cuda_matmul_bwd(ad, wd, gd, da, dw, M, N, K, 1)
    assert rel_l2(sc.to_host_f32(da, (M, K)), g.astype(np.float64) @ w.T) < TOL[mode]
    assert rel_l2(sc.to_host_f32(dw, (K, N)), a.T.astype(np.float64) @ g) < (1e-3 if mode == 4 else TOL[mode])      # one fp16 product there
    for p in (ad, wd, bd, gd, y, da, dw):
        sc.cuda_free(p)


@pytest.mark.parametrize("act", [0, 1, 2, 3])
@pytest.mark.parametrize("N,C,H,F", [(3, 16, 16, 40), (5, 72, 8, 33), (9, 24, 4, 130)])
def test_pooled_epilogue(sc, act, N, C, H, F):
    """The pool of the same layer's own output, bit for bit: values, and the first of equal maxima."""
    sc.set_precision(3)
    rs = np.random.RandomState(N + C + F + act)
    x = rs.standard_normal((N, C, H, H)).astype(np.float32)
    w = (rs.standard_normal((F, C, 3, 3)) / np.sqrt(9 * C)).astype(np.float32)
    b = rs.standard_normal(F).astype(np.float32)
    w[1], b[1] = 0, -0.5                                     # all equal
    b[2] = np.inf
    xd, wd, bd = (sc.to_device_f32(t.ravel()) for t in (x, w, b))
    n = N * F * H * H // 4
    out, mask, y = sc.cuda_malloc_f32(n), sc.cuda_malloc_i32(n), sc.cuda_malloc_f32(4 * n)
    assert sc.conv2d_pool_fusable(N, C, H, H, F, 3, 3, 1, 1, 1, 1)
    sc.shadow_free(sc.conv2d_bias_act_pool_fwd_s(xd, wd, bd, out, mask, N, C, H, H, F, 3, 3, 1, 1, 1, 1, act, 0, False)[0])
    sc.shadow_free(sc.conv2d_bias_act_fwd_s(xd, wd, bd, y, N, C, H, H, F, 3, 3, 1, 1, 1, 1, act, 0))
    full = sc.to_host_f32(y, (N, F, H // 2, 2, H // 2, 2)).transpose(0, 1, 2, 4, 3, 5).reshape(N, F, H // 2, H // 2, 4)
    assert np.array_equal(sc.to_host_f32(out, full.shape[:-1]), full.max(-1))
    assert np.array_equal(sc.to_host_i32(mask, full.shape[:-1]), full.argmax(-1))
    for p in (xd, wd, bd, out, mask, y):
        sc.cuda_free(p)


@pytest.mark.parametrize("mode", [1, 3, 4])
@pytest.mark.parametrize("N,C,H,W,F,K,st,pad", [(3, 33, 9, 12, 40, 3, 2, 1),        # odd height: phases of different sizes
                                                (2, 32, 16, 17, 72, 4, 2, 1), (3, 40, 10, 10, 24, 5, 3, 2),        # nine phases
                                                (40, 32, 16, 16, 64, 3, 2, 1),      # tiles for every CTA, each warp half in turn
                                                (2, 130, 8, 8, 70, 2, 2, 0), (2, 20, 12, 12, 16, 4, 4, 0)])          # sixteen
def test_phases_of_a_strided_data_gradient(sc, mode, N, C, H, W, F, K, st, pad):
    """Against float64; pixels that no window reaches are zero; a NaN stays with the pixels whose windows hold it."""
    import torch
    sc.set_precision(mode)
    rs = np.random.RandomState(N + C + H + F)
    OH, OW = (H + 2 * pad - K) // st + 1, (W + 2 * pad - K) // st + 1
    w = (rs.standard_normal((F, C, K, K)) / np.sqrt(F * K)).astype(np.float32)
    dy = rs.standard_normal((N, F, OH, OW)).astype(np.float32)
    x, dx, dw = sc.to_device_f32(np.zeros(N * C * H * W, np.float32)), sc.cuda_malloc_f32(N * C * H * W), sc.cuda_malloc_f32(w.size)
    wd = sc.to_device_f32(w.ravel())
    for bad in (False, True):
        if bad:
            if mode == 4:
                break                                    # its conversion saturates
            dy[0, 3, OH // 2, OW // 2] = np.nan
        g = sc.to_device_f32(dy.ravel())
        sc.cuda_conv2d_bwd(wd, x, g, dx, dw, N, C, H, W, F, K, K, st, st, pad, pad)
        ref = torch.nn.grad.conv2d_input((N, C, H, W), torch.from_numpy(w).double(), torch.from_numpy(dy).double(), st, pad).numpy()
        got, ok = sc.to_host_f32(dx, ref.shape), ~np.isnan(ref)
        assert np.array_equal(np.isnan(got), ~ok)
        assert rel_l2(got[ok], ref[ok]) < TOL[mode]
        assert not got[ref == 0].any()
        sc.cuda_free(g)
    for p in (x, dx, dw, wd):
        sc.cuda_free(p)


@pytest.mark.parametrize("mode", [1, 3, 4])
@pytest.mark.parametrize("N,C,H,W,F,K,st,pad", [(3, 17, 12, 13, 33, 3, 1, 1), (2, 32, 9, 9, 24, 2, 1, 0), (4, 24, 16, 16, 130, 5, 2, 2), (40, 32, 16, 16, 64, 3, 2, 1),
                                                (2, 8, 40, 40, 32, 7, 1, 3), (3, 31, 8, 8, 20, 1, 1, 0), (5, 40, 14, 14, 9, 3, 1, 1), (2, 32, 10, 9, 32, 4, 3, 2)])
def test_layers_of_up_to_32_channels(sc, mode, N, C, H, W, F, K, st, pad):
    """Two taps a k-step, an odd last one beside zeros; forward, both gradients and the transposed convolution, against float64."""
    import torch
    sc.set_precision(mode)
    rs = np.random.RandomState(N + C + H + F)
    OH, OW = (H + 2 * pad - K) // st + 1, (W + 2 * pad - K) // st + 1
    x, w, dy = (rs.standard_normal(s).astype(np.float32) for s in ((N, C, H, W), (F, C, K, K), (N, F, OH, OW)))
    xd, wd, gd = (sc.to_device_f32(t.ravel()) for t in (x, w, dy))
    y, dx, dw = (sc.cuda_malloc_f32(t.size) for t in (dy, x, w))
    sc.cuda_conv2d_fwd(xd, wd, y, N, C, H, W, F, K, K, pad, pad, st, st)
    sc.cuda_conv2d_bwd(wd, xd, gd, dx, dw, N, C, H, W, F, K, K, st, st, pad, pad)
    X, Wt = torch.from_numpy(x).double().requires_grad_(), torch.from_numpy(w).double().requires_grad_()
    Y = torch.nn.functional.conv2d(X, Wt, stride=st, padding=pad)
    Y.backward(torch.from_numpy(dy).double())
    assert rel_l2(sc.to_host_f32(y, dy.shape), Y.detach().numpy()) < TOL[mode]
    assert rel_l2(sc.to_host_f32(dx, x.shape), X.grad.numpy()) < TOL[mode]
    assert rel_l2(sc.to_host_f32(dw, w.shape), Wt.grad.numpy()) < (1e-3 if mode == 4 else TOL[mode])      # one fp16 product there
    for p in (xd, wd, gd, y, dx, dw):
        sc.cuda_free(p)


@pytest.mark.parametrize("mode", [3, 4])
def test_last_round_in_clusters(sc, mode):
    """148 tiles and a few more, with a long contraction: the last ones are shared by clusters, in a launch of their own."""
    sc.set_precision(mode)
    rs = np.random.RandomState(mode)
    N, C, H, F = 605, 256, 4, 250                              # 9680 x 250 x 2304: 76 x 2 tiles
    x, b = rs.standard_normal((N, C, H, H)).astype(np.float32), rs.standard_normal(F).astype(np.float32)
    w = (rs.standard_normal((F, C, 3, 3)) / np.sqrt(9 * C)).astype(np.float32)
    xd, wd, bd = (sc.to_device_f32(t.ravel()) for t in (x, w, b))
    y = sc.cuda_malloc_f32(N * F * H * H)
    sc.shadow_free(sc.conv2d_bias_act_fwd_s(xd, wd, bd, y, N, C, H, H, F, 3, 3, 1, 1, 1, 1, 1, 0))
    import torch
    dev = lambda t: torch.from_numpy(t).double().cuda()                          # noqa: E731
    ref = (torch.nn.functional.conv2d(dev(x), dev(w), padding=1) + dev(b).view(1, -1, 1, 1)).relu().cpu().numpy()
    assert rel_l2(sc.to_host_f32(y, ref.shape), ref) < TOL[mode]
    for p in (xd, wd, bd, y):
        sc.cuda_free(p)
