"""One training step of the MLP and of the VGG-style network against double precision, with the step's own decisions held fixed.

Another order of the same float32 sums moves a forward value by its last bits, and where that changes a ReLU's sign or a pool's index one
contribution to a gradient is there or not: a handful of those is 1e-3 of the VGG network's first-layer gradient, whatever the precision of
the sums.  Here the masks and indices that the step chose are read back, every gradient is computed in 64 bits with them, and what is left is
rounding (tests/test_gpu_batchnorm_step.py does the same for a network with batch normalisation)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _in_double(layers, params, X, Y, decided):
    """Loss and gradients with the given ReLU masks and pool indices; a convolution's ReLU behind its pool, which takes one value a window."""
    import torch
    leaves, h = [], torch.from_numpy(X).double()
    for L, P, d in zip(layers, params, decided):
        if P is not None:
            W, b = (torch.from_numpy(np.asarray(p, np.float64)).requires_grad_() for p in P)
            leaves += [W, b]
        if L["type"] == "conv":
            h = torch.nn.functional.conv2d(h, W, b.flatten(), padding=1)
        elif L["type"] == "maxpool":
            N, C, H, Wd = h.shape
            index, positive = (torch.from_numpy(a) for a in d)
            w = h.reshape(N, C, H // 2, 2, Wd // 2, 2).permute(0, 1, 2, 4, 3, 5).reshape(N, C, H // 2, Wd // 2, 4)
            h = w.gather(4, index.unsqueeze(4)).squeeze(4) * positive
        elif L["type"] == "flatten":
            h = h.flatten(1)
        else:
            h = h @ W + b
            if d is not None:
                h = h * torch.from_numpy(d)
    p = torch.softmax(h, 1).clamp(1e-7, 1 - 1e-7)            # the loss's own bounds (Seera.py:955-969)
    loss = -(torch.from_numpy(Y).double() * torch.log(p)).sum(1).mean()
    loss.backward()
    return float(loss.detach()), [t.grad.numpy() for t in leaves]


# Three times what was measured on these seeds.  Mode 3 rounds like float32: 5.0e-6.  Mode 4 forms weight gradients from one fp16 copy of each operand,
# whose roundings are 2e-4 of a term and partly cancel in the sum: 8.6e-5.  Mode 5 rounds each gradient on its way down as well: 2.9e-4.
FLOAT32, ONE_COPY, ONE_PASS = 1.5e-5, 2.6e-4, 9e-4
CASES = [("c2", 4096, None, ONE_PASS), ("c2", 1000, None, ONE_PASS), ("c2", 1000, (3, 3), FLOAT32),
         ("c3", 512, None, ONE_COPY), ("c3", 100, None, ONE_COPY), ("c3", 100, (3, 3), FLOAT32)]


@pytest.mark.parametrize("name,n,precision,bound", CASES)
def test_gradients_with_the_steps_own_decisions(name, n, precision, bound):
    from ml_framework_b200 import seera_cuda as sc, train, workloads as wl
    sc.init(0)
    work = wl.WORKLOADS[name]()
    precision = precision or train.policy_for(work)
    worst = 0.0
    for seed in (3, 11, 29)[:1 if n > 100 else 3]:
        tr = train.Trainer(work, seed=seed, precision=precision)
        X, Y = work.batch(n, seed)
        loss = tr.forward_backward(X, Y)
        got = [a for G in tr.host_grads() if G is not None for a in G]
        decided = []
        for L, layer in zip(work.layers, tr.model.model[1:]):
            if L["type"] == "maxpool":
                decided.append((layer.mask.to_host_i32().astype(np.int64), layer.outputs.to_numpy() > 0))
            else:
                decided.append(layer.outputs.to_numpy() > 0 if L["type"] == "dense" and L["act"] == "relu" else None)
        want_loss, want = _in_double(work.layers, work.params(seed), X, Y, decided)
        assert abs(loss.item() - want_loss) < 1e-5 * abs(want_loss)      # logits of tens, 3e-7 to 1e-6 off
        errors = [rel_l2(g, w) for g, w in zip(got, want)]
        print("\n[%s, %d samples, seed %d, precision %s] gradients against double precision %s" % (name, n, seed, precision, " ".join("%.1e" % e for e in errors)))
        worst = max(worst, *errors)
    assert worst < bound
    sc.set_precision(0)
