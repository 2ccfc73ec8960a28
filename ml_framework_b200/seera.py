"""Training front end on the B200 engine: Sequential, layers, Loss, SGD, Adam, autograd4nn, Tensor.

Mirrors the user-facing API of the reference (Seera.py:26-1086, Seera_Engine.py:22-26) - same class
names, constructor arguments, method names (`forward`, `zero_grad`, `fit`, `step`, `set_weights`,
`get_weights`, the attribute spelled `bais`) and error behaviour - so a training script written for
the reference's `device="cuda"` path runs here with the import line changed.  What differs is the
machinery underneath:

  * autograd works per LAYER, not per scalar op.  A layer's forward enqueues its contraction plus
    ONE fused bias+activation pass, and records a backward closure that enqueues ONE fused
    activation-gradient+bias-gradient pass and the dX / dW contractions.  The reference builds a node
    per elementary op with five placeholder buffers each (Seera_init.py:75-80) and walks them in
    Seera_Engine.backward_step (Seera_Engine.py:259-598).
  * all parameters live in one contiguous device arena, with matching arenas for gradients and
    optimizer state: the optimizer is a single kernel launch over the arena (Seera.py:1038-1063 issues
    ~30 launches per tensor) and a data-parallel run all-reduces the gradient arena in place.
  * weights are updated in place; device addresses of parameters are stable across steps.
  * nothing blocks: calls enqueue on the engine's stream, the loss value is read when asked for.

There is no CPU path here: `device` must be "cuda" and the compiled engine must be present.
"""
from __future__ import annotations

import math
import pickle
import threading
import weakref

import numpy as np

from . import seera_cuda as sc
from .cuTen import cuten

_ACT = {None: 0, "relu": 1, "sigmoid": 2, "tanh": 3}
_ACTIVATIONS = ("relu", "sigmoid", "softmax", "tanh")
f32 = np.float32


_numel = math.prod
_wrap = cuten._wrap
_malloc = sc.cuda_malloc_f32
_bare = object.__new__


def _new(shape):
    return _wrap(_malloc(_numel(shape)), shape)


# One submission for the launches of a phase (seera_batch_begin / _end): inside, the engine notes its launches down, and the end hands
# them over as one graph - a fraction of the host time per launch and no gaps between them on the device.  A model's first pass at a size
# runs launch by launch, which leaves no executable behind and lets the device start at once.  Only what is this module's own runs inside a
# batch: a caller's layer, loss, optimizer or gradient function may launch, wait or record events on the stream by itself.
_batch_begin, _batch_end = sc.batch_begin, sc.batch_end        # (_batch_begin None: every pass launch by launch)


class _Inside(threading.local):
    n = 0                            # batches that this thread has open: what runs inside one has been looked over


_inside = _Inside()


def _open_batch(model, kind, size):
    """True if a batch was opened, for a kind of pass that the model has made at this size before; the caller then owes a _close_batch()."""
    if _batch_begin is None:
        return False
    if (kind, size) not in model._passes:
        if len(model._passes) > 4096:
            model._passes.clear()
        model._passes.add((kind, size))
        return False
    _batch_begin(kind)
    _inside.n += 1
    return True


def _close_batch():
    _inside.n -= 1
    _batch_end()


_FORWARD, _BACKWARD, _STEP = 1, 2, 3     # kinds of pass


# ─────────────────────────────────────────────────────────────────────────────────────────────
# Tensor: a device value, its gradient, and the closure that propagates the gradient
# ─────────────────────────────────────────────────────────────────────────────────────────────
class Tensor:
    # What an instance starts from.  The eager path makes one of these per layer and call, so only what differs is stored on one.
    dtype = "float32"
    is_leaf = False
    grad = None                      # cuten, set by backward
    _parents = ()
    _backward = None                 # fn(grad: cuten) -> None, deposits into parents via _accumulate
    _softmax_logits = None           # for a softmax output: the Tensor of logits it came from
    _grad_slot = None                # for a parameter: its view into the model's gradient arena
    _takes_pooled = False            # its backward takes the gradient of a 2x2 max-pool of it in pooled form
    _copies = None                   # channels-last copies of the value, made by its producer for a convolution
    _rows = None                     # row-major copies of the value, made by its producer for a Dense layer
    _pass = None                     # (input shape, reference to the model) of the pass it came from

    def __init__(self, value, dtype="float32", is_leaf=False, device="cuda"):
        if isinstance(value, Tensor):
            value = value.value
        if not isinstance(value, cuten):
            value = cuten(np.ascontiguousarray(np.asarray(value, dtype=np.float32)))
        self.value = value
        if dtype != "float32":
            self.dtype = dtype
        if is_leaf:
            self.is_leaf = is_leaf

    @classmethod
    def _of(cls, value, parents, backward):
        """The output of an operation on the device."""
        t = _bare(cls)
        t.value = value
        t._parents = parents
        t._backward = backward
        return t

    # the reference reads gradients as `t.node.cp` (Seera_init.py:53-55)
    @property
    def node(self):
        return self

    @property
    def cp(self):
        return self.grad

    @cp.setter
    def cp(self, g):
        self.grad = g

    @property
    def shape(self):
        return self.value.shape

    def _grad_target(self):
        """Buffer a backward kernel should write this tensor's gradient contribution into: the arena
        slot when the gradient restarts from zero, otherwise a fresh buffer to be added."""
        if self.grad is None and self._grad_slot is not None:
            return self._grad_slot
        return _new(self.value.shape)

    def _accumulate(self, g):
        """Add a gradient contribution: a cuten of this tensor's shape, or a _PooledGrad (the gradient of a 2x2 max-pool
        of this tensor, still in pooled form) when it is the only contribution."""
        if self.grad is None:
            self.grad = g
        else:
            if isinstance(self.grad, _PooledGrad):
                self.grad = self.grad.materialize()
            if isinstance(g, _PooledGrad):
                g = g.materialize()
            out = _new(self.value.shape)
            sc.cuda_elemadd(self.grad.main_ptr, g.main_ptr, out.main_ptr, self.value.size)
            self.grad = out

    def to_numpy(self):
        return self.value.to_host_f32().copy()

    def item(self):
        a = self.value.to_host_f32()
        if a.size != 1:
            raise ValueError("Can only convert tensors with a single element to Python scalars")
        return a.item()

    def mean(self):
        if self.value.size == 1:
            return self
        raise NotImplementedError("Tensor.mean on a non-scalar: losses of this front end are already scalar")

    def detach(self):
        return Tensor(self.value, is_leaf=True)

    @classmethod
    def zeros(cls, shape, dtype="float32", device="cuda"):
        return cls(cuten.zeros(shape), is_leaf=True)

    @classmethod
    def ones(cls, shape, dtype="float32", device="cuda"):
        return cls(cuten.ones(shape), is_leaf=True)

    def __repr__(self):
        return f"Tensor(GPU)\n({self.value.to_host_f32()},\nshape={self.value.shape})"


tensor = Tensor


# Conv2D followed by a 2x2 / stride-2 MaxPool2D runs as one launch (pool in the convolution's epilogue) where the engine
# can do it; the convolution's own full-resolution output is then never materialised.  Set to False to keep every
# layer's output in memory.
FUSE_POOL = True
# A 2x2 unpooling that feeds a ConvTranspose2D leaves its output unmade until somebody reads it (see _Unpooled).
_LAZY_UNPOOL = True
# A Dense layer that feeds another Dense layer can have its GEMM epilogue write the 16-bit copies of its output that the next
# layer's GEMM reads (seera_matmul_bias_act_fwd_s, c_copies).  Off: at the sizes measured (4096 x 1024 outputs, one tile per
# CTA) the two-byte stores lengthen an epilogue that nothing overlaps by more than the next layer's vectorised conversion
# launch costs (MLP configuration: step 0.317 ms with it, 0.287 ms without).
import os as _os
DENSE_EPILOGUE_COPIES = _os.environ.get("SEERA_DENSE_EPILOGUE_COPIES", "0") != "0"


class _PooledGrad:
    """Gradient of a 2x2 / stride-2 max-pool output, kept in pooled form with the pool's argmax mask.  A consumer that
    can route it itself (Conv2D backward: one kernel forms dz from it) takes it as is; anything else materialises the
    full-resolution gradient with cuda_maxpool_bwd."""
    __slots__ = ("gp", "mask", "shape", "pooled")

    def __init__(self, gp, mask, shape, pooled=None):
        self.gp, self.mask, self.shape, self.pooled = gp, mask, tuple(shape), pooled

    def materialize(self):
        N, C, H, W = self.shape
        dx = _new(self.shape)
        sc.cuda_maxpool_bwd(self.gp.main_ptr, self.mask.main_ptr, dx.main_ptr, N, C, H, W, 2, 2, 0, 0, 2, 2)
        return dx


class _Formed(cuten):
    """A tensor whose values are formed from another's when its address is asked for.  One that is left unformed by a recording is formed
    anew each time it is asked for: every replay changes what it is formed from."""
    source = None
    stale = False                    # the values are those of an earlier replay, for all that is known here

    @classmethod
    def _of(cls, source, shape):
        t = cls._wrap(None, shape)
        t.source = source
        t.stale = sc.is_capturing()
        return t

    @property
    def main_ptr(self):
        if self._ptr is None:
            self._ptr = _malloc(self.size)
            if not self.stale:
                self._form()
        if self.stale:
            self.stale = not sc.is_capturing()           # inside the recording: from here on its replays form them
            self._form()
        return self._ptr

    @main_ptr.setter
    def main_ptr(self, value):
        self._ptr = value


class _Unpooled(_Formed):
    """The 2x2 nearest unpooling of `source`.  The transposed convolution that reads it can work from the source directly, and then it
    never is."""

    @classmethod
    def of(cls, low):
        N, C, H, W = low.shape
        return cls._of(low, (N, C, 2 * H, 2 * W))

    def _form(self):
        sc.cuda_unpooling_fwd(self.source.main_ptr, self._ptr, *self.source.shape, 2, 2)


class _Softmax(_Formed):
    """The row softmax of the logits `source`.  The cross-entropy, which has to form it anyway, writes it on its way (claim), and a training
    step then needs no pass for it."""

    @classmethod
    def of(cls, z):
        return cls._of(z, z.shape)

    def claim(self):
        """Address for a caller that writes the values itself."""
        if self._ptr is None:
            self._ptr = _malloc(self.size)
        if self.stale:
            self.stale = not sc.is_capturing()
        return self._ptr

    def _form(self):
        sc.cuda_softmax_fwd(self.source.main_ptr, self._ptr, *self.shape)


class _KeptCopies:
    """Owner of the channels-last copies a forward call kept for its backward call (0: none kept)."""
    __slots__ = ("h",)

    def __init__(self, h=0):
        self.h = h

    def release(self, free=sc.shadow_free):           # (held here: the module's names may be gone when the interpreter ends)
        if self.h:
            free(self.h)
            self.h = 0

    __del__ = release


class _KeptRows:
    """Owner of row-major operand copies a Dense forward call kept or handed on (0: none)."""
    __slots__ = ("h",)

    def __init__(self, h=0):
        self.h = h

    def release(self, free=sc.rows_free):
        if self.h:
            free(self.h)
            self.h = 0

    __del__ = release


_Function = type(lambda: None)


class autograd4nn:
    """Reverse pass from a scalar loss: `autograd4nn(loss)` (same call shape as Seera_Engine.py:24-26)."""

    def __init__(self, hook):
        self.hook = hook
        self.backward()

    def backward(self):
        order, own = self._order()
        opened = False
        if own and self.hook._pass is not None:
            size, model = self.hook._pass
            model = model()
            opened = model is not None and model._exchanges_nothing() and _open_batch(model, _BACKWARD, size)
        try:
            self._run(order)
        finally:
            if opened:
                _close_batch()

    def _order(self):
        """Every tensor that the gradient passes, parents first, and whether all of it is this module's own."""
        order, seen, own = [], set(), True
        stack = [self.hook]
        while stack:                                   # iterative DFS: no recursion limit on deep nets
            t = stack.pop()
            if t is None:                              # everything above its tensor has been placed
                order.append(stack.pop())
                continue
            if t in seen:
                continue
            seen.add(t)
            back = t._backward
            if back is not None and (back.__class__ is not _Function or back.__module__ != __name__):
                own = False
            stack.append(t)
            stack.append(None)
            for p in t._parents:
                if not p.is_leaf:                      # a leaf keeps its gradient and passes nothing on
                    stack.append(p)
        return order, own

    def _run(self, order):
        for t in order:
            if not t.is_leaf:
                t.grad = None
        self.hook.grad = cuten.ones_like(self.hook.value)
        for t in reversed(order):
            back, g = t._backward, t.grad
            if back is not None and g is not None:
                if g.__class__ is _PooledGrad and not t._takes_pooled:
                    t.grad = g = g.materialize()
                back(g)


# ─────────────────────────────────────────────────────────────────────────────────────────────
# Layers
# ─────────────────────────────────────────────────────────────────────────────────────────────
class Layer:
    # which layers read this one's output (set while a model is put together): a producer can then hand on more than its values
    # (weak references and no `self` in a gradient function: a model that is dropped returns its memory at once, and the next one finds it)
    _pool_consumer = None
    _feeds_conv = _feeds_dense = _feeds_convT = _feeds_copies = False
    _fused = None                    # a pool that the layer folded into its own launch: (pooled, mask, copies)
    _model = None

    def __init__(self):
        self.inputs = []
        self.outputs = []
        self.activations = {a: a for a in _ACTIVATIONS}

    def __call__(self, input_layer):
        if not isinstance(input_layer, Layer):
            raise TypeError("The input should be a Layer")
        self.inpobj = input_layer
        return self


class Input(Layer):
    def __init__(self, shape):
        super().__init__()
        self.shape = shape
        self.weights = 0
        self.bais = 0
        self.inputs = None

    def forward(self):
        self.outputs = self.inputs
        return self.outputs

    def __repr__(self):
        return f"Input Layer with shape {self.shape}"


def _initial(kind_scale, shape):
    kind, scale = kind_scale
    if kind == "normal":
        return (np.random.randn(*shape) * scale).astype(np.float32)
    if kind == "uniform":
        return np.random.uniform(-scale, scale, shape).astype(np.float32)
    return (np.zeros if kind == "zeros" else np.ones)(shape, dtype=np.float32)


def _initializers(fan_in, fan_out):
    return {
        "zeros": ("zeros", 0), "ones": ("ones", 1), "random_normal": ("normal", 1), "random_uniform": ("uniform", 0.05),
        "he_normal": ("normal", np.sqrt(2 / fan_in)), "he_uniform": ("uniform", np.sqrt(6 / fan_in)),
        "glorot_normal": ("normal", np.sqrt(2 / (fan_in + fan_out))), "glorot_uniform": ("uniform", np.sqrt(6 / (fan_in + fan_out))),
        "lecun_normal": ("normal", np.sqrt(1 / fan_in)), "lecun_uniform": ("uniform", np.sqrt(3 / fan_in)),
    }


def _pair(v):
    return (v, v) if isinstance(v, int) else tuple(v)


class _ParamLayer(Layer):
    """Shared parameter handling: host initial values until the model places them in its arena."""

    def _check(self, activation, initializer, table):
        if activation not in self.activations:
            raise ValueError('Activation must be "relu", "sigmoid", "softmax", or "tanh"')
        if initializer not in table:
            raise ValueError(f"Initializer must be one of {list(table.keys())}")

    def set_weights(self, W, B):
        if isinstance(W, Tensor):
            W, B = W.to_numpy(), B.to_numpy()
        elif not isinstance(W, np.ndarray):
            raise TypeError("Weights must be Tensor or numpy array")
        W = np.ascontiguousarray(W, np.float32)
        B = np.ascontiguousarray(B, np.float32)
        self._w_init, self._b_init = W, B
        if isinstance(self.weights, Tensor) and tuple(self.weights.value.shape) == W.shape:
            sc.upload_f32(self.weights.value.main_ptr, W)            # keeps the arena slot and its address
            sc.upload_f32(self.bais.value.main_ptr, B)
        else:
            self.weights = Tensor(W, is_leaf=True)
            self.bais = Tensor(B, is_leaf=True)

    def get_weights(self):
        return self.weights, self.bais

    def update_params(self, vW, vB):
        """w -= vW, b -= vB with device tensors (Seera.py:140-147), in place."""
        for t, v in ((self.weights, vW), (self.bais, vB)):
            neg = v * (-1)
            sc.cuda_elemadd(t.value.main_ptr, neg.main_ptr, t.value.main_ptr, t.value.size)

    # shared by Dense, Conv2D, ConvTranspose2D
    def _output(self, x, z, node_backward, takes_pooled=False, softmax=None):
        """The layer's output Tensor around `z`, which holds act(contraction + bias), or the logits of a softmax (`softmax`, where its values
        came with them)."""
        node = Tensor._of(z, (x, self.weights, self.bais), node_backward)
        if takes_pooled:
            node._takes_pooled = True
        if self.layeract != "softmax":
            return node
        y = softmax or _Softmax.of(z)

        def softmax_backward(g):
            dz = _new(y.shape)
            sc.cuda_softmax_vjp(y.main_ptr, g.main_ptr, dz._ptr, y.shape[0], y.shape[1])
            node._accumulate(dz)
        out = Tensor._of(y, (node,), softmax_backward)
        out._softmax_logits = node
        return out


def _grads_in_arena(owner, W, b):
    """Tells the model's hook that a layer's gradients sit in the arena: a bucket may go out."""
    model = owner and owner()
    if model is not None and model._on_grad_ready is not None and W.grad is W._grad_slot and b.grad is b._grad_slot:
        model._on_grad_ready(W)


def _deliver(owner, x, W, b, dx, dw, db):
    """Gradients of one backward call to the input and the parameters."""
    b._accumulate(db)
    W._accumulate(dw)
    _grads_in_arena(owner, W, b)
    if dx is not None:
        x._accumulate(dx)


_HEAD_COLUMNS = 16                   # the engine's head kernels hold whole rows of that many columns


class Dense(_ParamLayer):
    def __init__(self, in_units, out_units, activation=None, kernel_initializer="glorot_uniform",
                 bias_initializer="zeros", kernel_regularizer=None, bias_regularizer=None):
        super().__init__()
        table = _initializers(in_units, out_units)
        self._check(activation, kernel_initializer, table)
        self.layeract, self.in_units, self.out_units = activation, in_units, out_units
        self._w_init = _initial(table[kernel_initializer], (in_units, out_units))
        self._b_init = _initial(table[bias_initializer], (1, out_units))
        self.weights = Tensor(self._w_init, is_leaf=True)
        self.bais = Tensor(self._b_init, is_leaf=True)

    def __call__(self, input_layer):
        super().__call__(input_layer)
        input_layer._feeds_dense = True       # a Dense producer then also emits the row-major copies of its output this layer reads
        return self

    def forward(self):
        x = self.inputs = self.inpobj.outputs
        W, b = self.weights, self.bais
        xv, wv = x.value, W.value
        shape = xv.shape
        if len(shape) != 2 or shape[1] != self.in_units:
            raise ValueError(f"[cuTen]: matmul: inner dimensions must agree, got {xv.shape} @ {wv.shape}")
        M, K, N = shape[0], self.in_units, self.out_units
        z = _new((M, N))
        code = _ACT.get(self.layeract, 0)                    # a softmax follows the product as a pass of its own
        given = x._rows                                      # copies written by the Dense layer before
        want_out = DENSE_EPILOGUE_COPIES and self._feeds_dense and self.layeract != "softmax"
        ha = hw = ho = 0
        prob = None
        model = self._model and self._model()
        if model is not None and model._whole and self.layeract == "softmax" and N <= _HEAD_COLUMNS:
            prob = _Softmax.of(z)                            # a prediction's, with its logits if one launch makes both
            if not sc.matmul_softmax_fwd(xv.main_ptr, wv.main_ptr, b.value.main_ptr, z._ptr, prob.claim(), M, N, K):
                prob = None
        if prob is None:
            ha, hw, ho = sc.matmul_bias_act_fwd_s(xv.main_ptr, wv.main_ptr, b.value.main_ptr, z._ptr, M, N, K, code, given.h if given else 0, want_out)
        kept_a, kept_w = _KeptRows(ha) if ha else None, _KeptRows(hw) if hw else None
        need_dx, owner = not x.is_leaf, self._model

        def backward(g):
            # activation slope, bias gradient, dA and dB in one call; it reads the copies the forward call kept
            db, dw = b._grad_target(), W._grad_target()
            dx = _new(shape) if need_dx else None
            a = kept_a or given
            sc.matmul_act_bwd(xv._ptr, wv._ptr, z._ptr if code else 0, g.main_ptr, dx._ptr if need_dx else 0, dw._ptr, db._ptr, M, N, K, code,
                              a.h if a else 0, kept_w.h if kept_w else 0)
            for k in (kept_a, kept_w, given):
                if k:
                    k.release()
            _deliver(owner, x, W, b, dx, dw, db)
        self.outputs = out = self._output(x, z, backward, softmax=prob)
        if want_out:
            out._rows = _KeptRows(ho)
        return out

    def __repr__(self):
        return f"Dense({self.in_units}→{self.out_units}, act={self.layeract}, params={self.in_units * self.out_units + self.out_units})"


class Conv2D(_ParamLayer):
    def __init__(self, out_channels, in_channels, kernel_size, activation, stride=1, zero_padding=0,
                 kernel_initializer="he_normal", bias_initializer="zeros"):
        super().__init__()
        fan_in = in_channels * kernel_size[0] * kernel_size[1]
        table = _initializers(fan_in, out_channels * kernel_size[0] * kernel_size[1])
        self._check(activation, kernel_initializer, table)
        self.layeract, self.in_channels, self.out_channels = activation, in_channels, out_channels
        self.kernel_size, self.stride, self.zero_padding = tuple(kernel_size), _pair(stride), _pair(zero_padding)
        self._w_init = _initial(table[kernel_initializer], (out_channels, in_channels) + self.kernel_size)
        self._b_init = np.zeros((1, out_channels, 1, 1), np.float32)
        self.weights = Tensor(self._w_init, is_leaf=True)
        self.bais = Tensor(self._b_init, is_leaf=True)

    def __call__(self, input_layer):
        super().__call__(input_layer)
        input_layer._feeds_conv = True        # a pooling producer then also emits the channels-last copies this layer reads
        if self.out_channels not in (1, 2, 4):        # those few read their input in place
            input_layer._feeds_copies = True
        return self

    def forward(self):
        x = self.inputs = self.inpobj.outputs
        W, b = self.weights, self.bais
        xv, wv = x.value, W.value
        given = x._copies                                    # copies made by the producer of x
        if len(xv.shape) == 3:
            xv, given = xv.reshape((1,) + tuple(xv.shape)), None
        shape = xv.shape
        if len(shape) != 4:
            raise ValueError("[cuTen]: conv2d expects 4-D tensors (N,C,H,W) and (F,C,KH,KW)")
        if self.layeract == "softmax":
            raise ValueError("[Engine]: Softmax VJP requires at least 2D")
        N, C, H, Wd = shape
        F, (KH, KW), (sh, sw), (ph, pw) = self.out_channels, self.kernel_size, self.stride, self.zero_padding
        OH, OW = (H + 2 * ph - KH) // sh + 1, (Wd + 2 * pw - KW) // sw + 1
        code = _ACT[self.layeract]
        owner, pool = self._model, self._pool_consumer and self._pool_consumer()
        self._fused = None
        if FUSE_POOL and pool is not None and sc.conv2d_pool_fusable(N, C, H, Wd, F, KH, KW, sh, sw, ph, pw):
            # the pool is folded into this layer's epilogue: z stays a shape without memory
            z = _wrap(0, (N, F, OH, OW))
            z._owns_memory = False
            half = (N, F, OH // 2, OW // 2)
            pooled = _new(half)
            pmask = _wrap(sc.cuda_malloc_i32(pooled.size), half, "int32")
            args = (xv.main_ptr, wv.main_ptr, b.value.main_ptr, pooled._ptr, pmask._ptr, N, C, H, Wd, F, KH, KW, ph, pw, sh, sw, code,
                    given.h if given else 0, pool._feeds_conv)
            h, hw, hp = sc.conv2d_bias_act_pool_fwd_k(*args)
            self._fused = (pooled, pmask, _KeptCopies(hp) if hp else None)
            hy = 0
        else:
            z = _new((N, F, OH, OW))
            args = (xv.main_ptr, wv.main_ptr, b.value.main_ptr, z._ptr, N, C, H, Wd, F, KH, KW, ph, pw, sh, sw, code, given.h if given else 0)
            h, hw, hy = sc.conv2d_bias_act_fwd_k(*args, self._feeds_copies)
        kept, kept_w = _KeptCopies(h) if h else None, _KeptRows(hw) if hw else None
        need_dx = not x.is_leaf

        def backward(g):
            # pool routing, activation slope, bias gradient, dX and dW in one call
            db, dw = b._grad_target(), W._grad_target()
            dx = _new(shape) if need_dx else None
            if g.__class__ is _PooledGrad:
                gptr, gpptr, mptr, ypptr = 0, g.gp.main_ptr, g.mask._ptr, g.pooled.main_ptr if g.pooled is not None else 0
            else:
                gptr, gpptr, mptr, ypptr = g.main_ptr, 0, 0, 0
            k = kept or given
            args = (wv._ptr, xv._ptr, z._ptr, gptr, gpptr, mptr, ypptr, dx._ptr if need_dx else 0, dw._ptr, db._ptr,
                    N, C, H, Wd, F, KH, KW, sh, sw, ph, pw, code, k.h if k else 0)
            sc.conv2d_act_bwd_k(*args, kept_w.h if kept_w else 0)
            for k in (kept, kept_w, given):
                if k:
                    k.release()
            _deliver(owner, x, W, b, dx, dw, db)
        self.outputs = out = self._output(x, z, backward, takes_pooled=True)
        if hy:
            out._copies = _KeptCopies(hy)
        return out

    def __repr__(self):
        return f"Conv2D({self.in_channels}→{self.out_channels}, kernel={self.kernel_size}, act={self.layeract})"


class ConvTranspose2D(_ParamLayer):
    def __init__(self, out_channels, in_channels, kernel_size, activation, stride=1, zero_padding=0,
                 kernel_initializer="he_normal"):
        super().__init__()
        fan_in = in_channels * kernel_size[0] * kernel_size[1]
        table = _initializers(fan_in, out_channels * kernel_size[0] * kernel_size[1])
        for k in ("lecun_normal", "lecun_uniform"):
            table.pop(k)
        self._check(activation, kernel_initializer, table)
        self.layeract, self.in_channels, self.out_channels = activation, in_channels, out_channels
        self.kernel_size, self.stride, self.zero_padding = tuple(kernel_size), _pair(stride), _pair(zero_padding)
        self._w_init = _initial(table[kernel_initializer], (in_channels, out_channels) + self.kernel_size)
        self._b_init = np.zeros((1, out_channels, 1, 1), np.float32)
        self.weights = Tensor(self._w_init, is_leaf=True)
        self.bais = Tensor(self._b_init, is_leaf=True)

    def __call__(self, input_layer):
        super().__call__(input_layer)
        input_layer._feeds_convT = True       # an unpooling producer then leaves its output to be read at the low resolution
        if self.out_channels * self.kernel_size[0] * self.kernel_size[1] > 64:        # shorter patches read their input in place
            input_layer._feeds_copies = True
        return self

    def forward(self):
        x = self.inputs = self.inpobj.outputs
        W, b = self.weights, self.bais
        xv, wv = x.value, W.value
        shape = xv.shape
        if len(shape) != 4:
            raise ValueError("[cuTen]: conv2d_transpose expects 4-D tensors (N,Cin,H,W) and (Cin,Cout,KH,KW)")
        if self.layeract == "softmax":
            raise ValueError("[Engine]: Softmax VJP requires at least 2D")
        N, Cin, H, Wd = shape
        Cout, (KH, KW), (sh, sw), (ph, pw) = self.out_channels, self.kernel_size, self.stride, self.zero_padding
        Ho, Wo = (H - 1) * sh - 2 * ph + KH, (Wd - 1) * sw - 2 * pw + KW
        code = _ACT[self.layeract]
        z = _new((N, Cout, Ho, Wo))
        if (xv.__class__ is _Unpooled and xv._ptr is None and H % 2 == 0 and Wd % 2 == 0
                and sc.unpool2_convT_fusable(N, Cin, H // 2, Wd // 2, Cout, KH, KW, sh, sw, ph, pw)):
            return self._forward_unpooled(x, xv.source, z, code)
        need_dx, owner = not x.is_leaf, self._model
        given = x._copies
        h = sc.conv2DTranspose_bias_act_fwd_k(xv.main_ptr, wv.main_ptr, b.value.main_ptr, z._ptr, N, Cin, H, Wd, Cout, KH, KW, sh, sw, ph, pw,
                                              code, given.h if given else 0)
        kept = _KeptCopies(h) if h else None

        def backward(g):
            # activation slope, bias gradient and both products in one call
            db, dw = b._grad_target(), W._grad_target()
            dx = _new(shape) if need_dx else None
            k = kept or given
            sc.conv2DTranspose_act_bwd_k(wv._ptr, xv._ptr, z._ptr, g.main_ptr, dx._ptr if need_dx else 0, dw._ptr, db._ptr, N, Cin, H, Wd, Cout,
                                         KH, KW, sh, sw, ph, pw, code, k.h if k else 0)
            for k in (kept, given):
                if k:
                    k.release()
            _deliver(owner, x, W, b, dx, dw, db)
        self.outputs = self._output(x, z, backward)
        return self.outputs

    def _forward_unpooled(self, x, low, z, code):
        """The unpooling before this layer and the layer in one, from the low-resolution tensor and with its gradient as result."""
        W, b = self.weights, self.bais
        N, Cin, H, Wd = low.shape
        sc.unpool2_convT_bias_act_fwd(low.main_ptr, W.value.main_ptr, b.value.main_ptr, z._ptr, N, Cin, H, Wd, code)
        source = x._parents[0]                    # what was unpooled: its gradient goes to it directly
        need_dx, owner = not source.is_leaf, self._model

        def backward(g):
            db, dw = b._grad_target(), W._grad_target()
            dlow = _new(low.shape) if need_dx else None
            sc.unpool2_convT_act_bwd(W.value._ptr, low._ptr, z._ptr if code else 0, g.main_ptr, dlow._ptr if need_dx else 0, dw._ptr, db._ptr,
                                     N, Cin, H, Wd, code)
            _deliver(owner, source, W, b, dlow, dw, db)
        self.outputs = self._output(x, z, backward)
        return self.outputs

    def __repr__(self):
        return (f"ConvTranspose2D({self.in_channels}→{self.out_channels}, kernel={self.kernel_size}, "
                f"stride={self.stride}, act={self.layeract})")


class _BatchNorm(_ParamLayer):
    """Batch normalisation on the device (the reference computes it on the host even in its GPU path: Seera.py:511-623,
    Seera_init.py:870-921, Seera_Engine.py:381-415).  gamma / beta are the layer's `weights` / `bais` (as in the reference)
    and live in the model's parameter arena; the running statistics are device buffers, readable as NumPy arrays through
    `running_mean` / `running_var`.  In a data-parallel run each rank normalises with the statistics of its own shard, unless
    `sync` is set (also by `dp.attach_nccl(..., sync_batchnorm=True)`): then the statistics, and the sums of the backward
    formula, are those of all ranks' shards together, so that a sharded step equals the step on the joined batch."""

    def __init__(self, num, momentum=0.1, eps=1e-5, sync=False):
        super().__init__()
        self.momentum, self.eps, self.training, self.sync = momentum, eps, True, bool(sync)
        self._w_init = np.ones((num,), np.float32)
        self._b_init = np.zeros((num,), np.float32)
        self.weights = Tensor(self._w_init, is_leaf=True)
        self.bais = Tensor(self._b_init, is_leaf=True)
        self._rm = cuten(np.zeros(num, np.float32))
        self._rv = cuten(np.ones(num, np.float32))
        self._num = num

    gamma = property(lambda self: self.weights)
    beta = property(lambda self: self.bais)

    @property
    def running_mean(self):
        return self._rm.to_host_f32().copy()

    @running_mean.setter
    def running_mean(self, v):
        sc.upload_f32(self._rm.main_ptr, np.ascontiguousarray(v, np.float32).reshape(self._num))

    @property
    def running_var(self):
        return self._rv.to_host_f32().copy()

    @running_var.setter
    def running_var(self, v):
        sc.upload_f32(self._rv.main_ptr, np.ascontiguousarray(v, np.float32).reshape(self._num))

    def _shape_ok(self, shape):
        raise NotImplementedError

    def forward(self):
        x = self.inputs = self.inpobj.outputs
        xv = x.value
        shape = xv.shape
        self._shape_ok(shape)
        N, C = shape[0], shape[1]
        S = _numel(shape[2:])
        g, b = self.weights, self.bais
        y, mean, si = _new(shape), _new((C,)), _new((C,))
        fwd, bwd = (sc.batchnorm_fwd_sync, sc.batchnorm_bwd_sync) if self.sync else (sc.batchnorm_fwd, sc.batchnorm_bwd)
        fwd(xv.main_ptr, g.value.main_ptr, b.value.main_ptr, self._rm.main_ptr, self._rv.main_ptr, y._ptr, mean._ptr, si._ptr, N, C, S,
            float(self.momentum), float(self.eps), bool(self.training))
        need_dx, owner = not x.is_leaf, self._model

        def backward(dy):
            dg, db = g._grad_target(), b._grad_target()
            dx = _new(shape)
            bwd(dy.main_ptr, xv._ptr, mean._ptr, si._ptr, g.value._ptr, dx._ptr, dg._ptr, db._ptr, N, C, S)
            g._accumulate(dg)
            b._accumulate(db)
            _grads_in_arena(owner, g, b)
            if need_dx:
                x._accumulate(dx)
        self.outputs = out = Tensor._of(y, (x, g, b), backward)
        return out


class BatchNorm1d(_BatchNorm):
    def __init__(self, num_features, momentum=0.1, eps=1e-5, sync=False):
        super().__init__(num_features, momentum, eps, sync)
        self.num_features = num_features

    def _shape_ok(self, shape):
        if len(shape) != 2 or shape[1] != self.num_features:
            raise ValueError(f"BatchNorm1d({self.num_features}) expects (N, {self.num_features}), got {tuple(shape)}")

    def __repr__(self):
        return f"BatchNorm1d({self.num_features})"


class BatchNorm2d(_BatchNorm):
    def __init__(self, num_channels, momentum=0.1, eps=1e-5, sync=False):
        super().__init__(num_channels, momentum, eps, sync)
        self.num_channels = num_channels

    def _shape_ok(self, shape):
        if len(shape) != 4 or shape[1] != self.num_channels:
            raise ValueError(f"BatchNorm2d({self.num_channels}) expects (N, {self.num_channels}, H, W), got {tuple(shape)}")

    def __repr__(self):
        return f"BatchNorm2d({self.num_channels})"


class Concatenate(Layer):
    """Joins the outputs of two layers along axis 1 (Seera.py:486-505); one strided-copy launch forward, one backward."""

    def __call__(self, *input_layers):
        if len(input_layers) != 2:
            raise ValueError("Only 2 layers supported for concatenation.")
        for l in input_layers:
            if not isinstance(l, Layer):
                raise TypeError("All inputs must be Layer instances.")
        self.input_layers = input_layers
        return self

    def forward(self):
        a, b = self.inputs = [l.outputs for l in self.input_layers]
        av, bv = a.value, b.value
        y = av.concatenate2D(bv) if len(av.shape) >= 4 else av.concatenate1D(bv)

        def backward(g):
            da, db = cuten._concat_backward(g, av, bv)
            a._accumulate(da)
            b._accumulate(db)
        self.outputs = out = Tensor._of(y, (a, b), backward)
        return out

    def __repr__(self):
        return "Concatenate Layer"


class MaxPool2D(Layer):
    def __init__(self, pool_size=(2, 2), stride=1, padding=0):
        super().__init__()
        if not isinstance(pool_size, tuple):
            raise ValueError("kernelsize should be a tuple (height, width)")
        self.pool_size, self.stride, self.padding = pool_size, _pair(stride), _pair(padding)

    def __call__(self, input_layer):
        if not isinstance(input_layer, Layer):
            raise TypeError("Input must be a Layer instance.")
        self.inpobj = input_layer
        if (tuple(self.pool_size), self.stride, self.padding) == ((2, 2), (2, 2), (0, 0)):
            input_layer._pool_consumer = weakref.ref(self)     # a Conv2D producer may fold this pool into its own launch
        return self

    def forward(self):
        x = self.inputs = self.inpobj.outputs
        xv = x.value
        if len(xv.shape) != 4:
            raise ValueError("[cuTen]: maxpool2d expects 4-D tensor (N,C,H,W)")
        N, C, H, W = shape = xv.shape
        (KH, KW), (sh, sw), (ph, pw) = self.pool_size, self.stride, self.padding
        OH, OW = (H + 2 * ph - KH) // sh + 1, (W + 2 * pw - KW) // sw + 1
        if OH * OW > H * W:
            raise ValueError("[cuTen]: maxpool2d with more outputs than inputs is not supported")
        tiles_exactly = (KH, KW, sh, sw, ph, pw) == (2, 2, 2, 2, 0, 0) and H % 2 == 0 and W % 2 == 0
        fused = self.inpobj._fused
        if fused is not None:                     # the producing convolution already pooled its output
            y, mask, copies = fused
            self.inpobj._fused = None
        else:
            y = _new((N, C, OH, OW))
            mask = _wrap(sc.cuda_malloc_i32(y.size), y.shape, "int32")
            copies = None
            if tiles_exactly and self._feeds_conv:   # also leaves the channels-last copies of y for that convolution
                h = sc.maxpool2x2_fwd_s(xv.main_ptr, y._ptr, mask._ptr, N, C, H, W)
                copies = _KeptCopies(h) if h else None
            else:
                sc.cuda_maxpool_fwd(xv.main_ptr, y._ptr, mask._ptr, N, C, H, W, KH, KW, ph, pw, sh, sw)
        self.mask = mask

        def backward(g):
            if tiles_exactly and x._takes_pooled:
                x._accumulate(_PooledGrad(g, mask, shape, y))   # the producer routes it through the mask itself
                return
            dx = _new(shape)
            sc.cuda_maxpool_bwd(g.main_ptr, mask._ptr, dx._ptr, N, C, H, W, KH, KW, ph, pw, sh, sw)
            x._accumulate(dx)
        self.outputs = out = Tensor._of(y, (x,), backward)
        if copies is not None:
            out._copies = copies
        return out

    def __repr__(self):
        return f"MaxPool2D(pool={self.pool_size}, stride={self.stride})"


class Unpool2D_Nearest(Layer):
    def __init__(self, size=(2, 2)):
        super().__init__()
        self.size = size

    def __call__(self, input_layer):
        if not isinstance(input_layer, Layer):
            raise TypeError("Input must be a Layer instance.")
        self.inpobj = input_layer
        return self

    def forward(self):
        x = self.inputs = self.inpobj.outputs
        xv = x.value
        if len(xv.shape) != 4:
            raise ValueError("[cuTen]:unpool expects 4-D tensor (N,C,H,W)")
        sw, sh = self.size                       # the reference unpacks (sw, sh) (Seera_init.py:793)
        N, C, H, W = shape = xv.shape
        if self._feeds_convT and (sw, sh) == (2, 2) and _LAZY_UNPOOL:
            y = _Unpooled.of(xv)
        else:
            y = _new((N, C, H * sh, W * sw))
            sc.cuda_unpooling_fwd(xv.main_ptr, y._ptr, N, C, H, W, sh, sw)

        def backward(g):
            dx = _new(shape)
            sc.cuda_unpooling_bwd(g.main_ptr, dx._ptr, N, C, H, W, sh, sw)
            x._accumulate(dx)
        self.outputs = out = Tensor._of(y, (x,), backward)
        return out

    def __repr__(self):
        return f"Unpool2D_Nearest(size={self.size})"


class Flatten(Layer):
    def __call__(self, input_layer):
        if not isinstance(input_layer, Layer):
            raise TypeError("Input must be a Layer instance.")
        self.inpobj = input_layer
        return self

    def forward(self):
        x = self.inputs = self.inpobj.outputs
        shape = x.value.shape
        self.outputs = out = Tensor._of(x.value.flatten(), (x,), lambda g: x._accumulate(g.reshape(shape)))
        return out

    def __repr__(self):
        return "Flatten Layer"


_OWN_LAYERS = {c: c.forward for c in (Input, Dense, Conv2D, ConvTranspose2D, BatchNorm1d, BatchNorm2d, Concatenate, MaxPool2D, Unpool2D_Nearest,
                                       Flatten)}


# ─────────────────────────────────────────────────────────────────────────────────────────────
# Sequential
# ─────────────────────────────────────────────────────────────────────────────────────────────
def _train_step(model, optimizer, lossf, y):
    """One step on the model's current input: forward, loss, backward, update.  The loss."""
    loss = lossf(model.forward(), y)
    model.zero_grad()
    autograd4nn(loss)
    optimizer.step()
    return loss


def _own_step(optimizer, lossf):
    return optimizer.__class__ in (SGD, Adam) and getattr(lossf, "__func__", None) in _LOSSES


# Full batches left to run from which recording the step pays: recording costs the host an eager step, a replay half of one (small CNN
# at batch 64: 130 and 70 us a step, of which the device works 50).  500 samples by 64: 1160 -> 905 us, 2048: 4430 -> 2390 us.
_RECORD_FROM = 3


class _RecordedStep:
    """A training step recorded once, for `fit`: inputs and targets are copied into its own buffers, replays run on those."""

    @staticmethod
    def fits(model, optimizer, lossf):
        """Steps whose every part is this module's own: what a caller's layer, loss or optimizer does on the host would not be repeated."""
        return (not sc.is_capturing() and not sc.profile_enabled()
                and model._exchanges_nothing() and _own_step(optimizer, lossf) and optimizer.model is model
                and not optimizer.updates_by_bucket and model._own_passes())

    def __init__(self, model, optimizer, lossf, xshape, yshape, classes):
        self.model, self.optimizer = model, optimizer
        self.x, n = _new(xshape), yshape[0]
        self.y = cuten._wrap(sc.cuda_malloc_i32(n), (n,), "int32") if classes else _new(yshape)
        model.model[0].inputs = Tensor(self.x, is_leaf=True)
        optimizer._scalars_in_graph = True        # the update's scalars travel with the recorded launch
        sc.graph_begin()
        try:
            target = self.y
            if classes:
                target = _new((n, classes))
                sc.onehot_f32(self.y.main_ptr, target.main_ptr, n, classes)
            self.keep = Tensor(target, is_leaf=True)
            self.loss = _train_step(model, optimizer, lossf, self.keep)
        finally:
            optimizer._scalars_in_graph = False
            self.graph = sc.graph_end()

    def load(self, x, y, last_loss, kept):
        """Inputs and targets of the next replay; the loss of the step before goes to the address `kept`, which no replay overwrites."""
        sc.copy_three(self.x.main_ptr, x.main_ptr, self.x.size, self.y.main_ptr, y.main_ptr, self.y.size,
                      kept, last_loss.value.main_ptr if last_loss is not None else 0, 0 if last_loss is None else 1)

    def replay(self):
        sc.graph_set_scalars(self.graph, self.optimizer._scalars())
        sc.graph_launch(self.graph)
        return self.loss

    def release(self):
        if self.graph:
            sc.graph_destroy(self.graph)
            self.graph = None


class Sequential:
    _whole = False                   # in predict: a softmax that the last layer's launch can form is formed there

    def __init__(self, layers, device="cuda"):
        if not isinstance(layers, list):
            raise TypeError("Layers must be a list")
        if not isinstance(layers[0], Input):
            raise TypeError("First layer must be an Input layer")
        if device != "cuda":
            raise ValueError("this engine has no CPU path: Sequential(..., device=\"cuda\")")
        self.device = device
        self.model = [layers[0]] + [layer(layers[i]) for i, layer in enumerate(layers[1:])]
        self.world, self._allreduce, self._on_grad_ready = 1, None, None
        self._modal = [l for l in self.model if hasattr(l, "training")]       # layers that behave differently in evaluation
        self._passes = set()                          # kinds and sizes of passes made (see _open_batch)
        self._build_arena()
        self._ref = weakref.ref(self)
        for l in self.param_layers:
            l._model = self._ref

    # one contiguous block each for parameters and gradients; slots are 64-float aligned
    def _build_arena(self):
        self.param_layers = [l for l in self.model if isinstance(l, _ParamLayer)]
        offs, total = [], 0
        for l in self.param_layers:
            for init in (l._w_init, l._b_init):
                offs.append((total, init.shape, init.size))
                total += (init.size + 63) // 64 * 64
        self.n_arena = total
        host = np.zeros(max(total, 1), np.float32)
        for (o, _, n), init in zip(offs, [a for l in self.param_layers for a in (l._w_init, l._b_init)]):
            host[o:o + n] = init.ravel()
        self.params = cuten(host)
        self.grads = cuten._wrap(sc.cuda_zeros_f(max(total, 1)), (max(total, 1),))
        it = iter(offs)
        for l in self.param_layers:
            for name in ("weights", "bais"):
                o, shape, n = next(it)
                v = cuten._wrap(self.params.main_ptr + 4 * o, shape)
                v._owns_memory, v._base = False, self.params
                t = Tensor(v, is_leaf=True)
                t._arena_off, t._arena_n = o, n
                t._grad_slot = self._grad_view(t)
                setattr(l, name, t)
        self._grad_fresh = True

    def _grad_view(self, t):
        v = cuten._wrap(self.grads.main_ptr + 4 * t._arena_off, t.value.shape)
        v._owns_memory, v._base = False, self.grads
        return v

    def rehome_grads(self, ptr):
        """Use the caller's device block (at least n_arena floats, zeroed, kept alive by the caller) as the gradient arena
        from now on - e.g. memory registered with a communicator, so that collectives work on it in place."""
        g = cuten._wrap(int(ptr), (max(self.n_arena, 1),))
        g._owns_memory = False
        self.grads = g
        for t in self.parameters():
            t._grad_slot = self._grad_view(t)
            t.grad = None

    def parameters(self):
        return [t for l in self.param_layers for t in (l.weights, l.bais)]

    def forward(self, X=None):
        if X is not None:
            if isinstance(X, np.ndarray):
                X = Tensor(X, is_leaf=True)
            if not isinstance(X, Tensor):
                raise TypeError("Input must be a Tensor or numpy array.")
            self.model[0].inputs = X
        size = None
        if _inside.n:                                 # part of a training step's, whose first part ends with the forward
            _batch_begin(_STEP)
            _inside.n += 1
            opened = True
        else:
            opened = self._batchable() and _open_batch(self, _FORWARD, size := self.model[0].inputs.value.shape)
        try:
            out = None
            for layer in self.model:
                out = layer.forward()
        finally:
            if opened:
                _close_batch()
        if size is not None:
            out._pass = size, self._ref
        return out

    def _batchable(self):
        """Whether a pass over the current input may run as one batch: with gradients exchanged between ranks during backward, other
        streams take part in it."""
        return (self._allreduce is None and self._on_grad_ready is None and self.model[0].inputs.__class__ is Tensor and self._own_passes())

    def _exchanges_nothing(self):
        return self._allreduce is None and self._on_grad_ready is None

    def _own_passes(self):
        if self.__class__ is not Sequential and self.__class__.forward is not Sequential.forward:
            return False
        try:
            for l in self.model:
                if l.forward.__func__ is not _OWN_LAYERS.get(l.__class__):
                    return False
        except AttributeError:                        # a function in the place of the method
            return False
        return True

    def predict(self, X):
        """Forward in evaluation mode: BatchNorm layers normalise with their running statistics (Seera.py:690-700)."""
        self._set_mode(False)
        self._whole = True
        try:
            return self.forward(X)
        finally:
            self._whole = False
            self._set_mode(True)

    def _set_mode(self, training=True):
        for l in self._modal:
            l.training = training

    def zero_grad(self):
        """Parameter gradients restart from zero: the next backward writes them instead of adding."""
        for l in self.param_layers:
            l.weights.grad = l.bais.grad = None

    def get_params(self):
        for l in self.param_layers:
            print(l.get_weights())

    def summary(self):
        print("=" * 60 + "\nModel Summary\n" + "=" * 60)
        for i, l in enumerate(self.model):
            print(f"  Layer {i}: {l}")
        print("=" * 60)

    def gather_grads(self):
        """Copy every parameter gradient into its slot of the gradient arena (no-op for slots already there)."""
        for t in self.parameters():
            g = t.grad
            if g is t._grad_slot and g is not None:
                continue
            dst = self.grads.main_ptr + 4 * t._arena_off
            if g is None:
                sc.cuda_memset(dst, 0, 4 * t._arena_n)
            elif g.main_ptr != dst:
                sc.cuda_memcopy_devicetodevice(dst, g.main_ptr, t._arena_n)
                t.grad = self._grad_view(t)

    def fit(self, X_train, y, Optimizer, Loss, Epochs, batch_size=1, Loss_interval=20, num_classes=None):
        """Training loop with the reference's signature, shuffling and history (Seera.py:715-788).  The input side is a
        pipeline: each batch is gathered straight into one of two page-locked staging buffers and uploaded on the copy
        stream while the previous step runs, and the loss of a step is read back one step later, so the compute stream
        never waits for a transfer.  `y` may be the reference's one-hot / target array, or, with `num_classes`, a 1-D
        integer label array: 4 bytes per sample cross PCIe and the one-hot rows are formed on the device.
        After a first full batch the step is recorded, where the rest of the run pays for it (see _RecordedStep), and the other full
        batches are replays: of an eager step of a small network the host's work is more than half."""
        X_train = np.ascontiguousarray(X_train, np.float32)
        labels = num_classes is not None and np.ndim(y) == 1
        y = np.ascontiguousarray(y, np.int32 if labels else np.float32)
        n = X_train.shape[0]
        bs = int(batch_size)
        xrow, yrow = int(np.prod(X_train.shape[1:])), int(np.prod(y.shape[1:]))
        # two sets of staging / device buffers, sized for a full batch
        stage = []
        for _ in range(2):
            hx, hy = sc.host_alloc_pinned(bs * xrow * 4), sc.host_alloc_pinned(bs * yrow * 4)
            stage.append({"hx": hx, "hy": hy, "vx": sc.host_view(hx, bs * xrow * 4).view(np.float32),
                          "vy": sc.host_view(hy, bs * yrow * 4).view(np.int32 if labels else np.float32),
                          "dx": _new((bs,) + X_train.shape[1:]), "dy": _new((bs,) + y.shape[1:]) if not labels else None,
                          "dl": cuten._wrap(sc.cuda_malloc_i32(bs), (bs,), "int32") if labels else None})
        hl = sc.host_alloc_pinned(8)
        slots = sc.host_view(hl, 8).view(np.float32)
        kept = _new((2,))                       # the losses of two steps, where no replay overwrites them
        history = []

        def eager_step(st, m):
            xb = Tensor(cuten._wrap(st["dx"].main_ptr, (m,) + X_train.shape[1:]), is_leaf=True)
            xb.value._owns_memory = False
            if labels:
                yv = _new((m, int(num_classes)))
                sc.onehot_f32(st["dl"].main_ptr, yv.main_ptr, m, int(num_classes))
            else:
                yv = cuten._wrap(st["dy"].main_ptr, (m,) + y.shape[1:])
                yv._owns_memory = False
            self.model[0].inputs = xb
            opened = _own_step(Optimizer, Loss) and self._batchable() and _open_batch(self, _STEP, xb.value.shape)
            try:
                return _train_step(self, Optimizer, Loss, Tensor(yv, is_leaf=True))
            finally:
                if opened:
                    _close_batch()
        full_left = (n // bs) * Epochs          # full batches still to run
        recorded, recordable, ran_one = None, _RecordedStep.fits(self, Optimizer, Loss), False
        try:
            for epoch in range(Epochs):
                perm = np.random.permutation(n)
                starts = list(range(0, n, bs))

                def upload(k):                      # batch k -> staging set k % 2 -> its device buffers (copy stream)
                    st, idx = stage[k & 1], perm[starts[k]:starts[k] + bs]
                    m = len(idx)
                    np.take(X_train.reshape(n, xrow), idx, axis=0, out=st["vx"][:m * xrow].reshape(m, xrow))
                    np.take(y.reshape(n, yrow), idx, axis=0, out=st["vy"][:m * yrow].reshape(m, yrow))
                    sc.copy_upload(st["dx"].main_ptr, st["hx"], m * xrow * 4)
                    sc.copy_upload((st["dl"] if labels else st["dy"]).main_ptr, st["hy"], m * yrow * 4)
                    return m
                total, pending = 0.0, None          # pending: loss tensor of the previous step, not read back yet
                sc.copy_wait_compute()              # whatever still reads the staging sets comes first
                sizes = {0: upload(0)}
                for k in range(len(starts)):
                    st, m = stage[k & 1], sizes[k]
                    sc.compute_wait_copy()          # batch k has landed
                    if m == bs:
                        full_left -= 1
                        if recorded is None and recordable and ran_one and full_left + 1 >= _RECORD_FROM:
                            recorded = _RecordedStep(self, Optimizer, Loss, (m,) + X_train.shape[1:],
                                                     (m,) if labels else (m,) + y.shape[1:], int(num_classes) if labels else 0)
                        ran_one = True
                    at, source = 4 * ((k - 1) & 1), None if pending is None else pending.value.main_ptr
                    if m == bs and recorded is not None:
                        recorded.load(st["dx"], st["dl"] if labels else st["dy"], pending, kept.main_ptr + at)
                        source = kept.main_ptr + at
                    sc.copy_wait_compute()          # once step k - 1 has run, set (k + 1) % 2 is free and its loss final
                    if pending is not None:
                        sc.copy_download(hl + at, source, 4)
                    if m == bs and recorded is not None:
                        loss = recorded.replay()
                    else:
                        loss = eager_step(st, m)
                    if pending is not None:         # the device is already busy with step k
                        sc.copy_synchronize()
                        total += float(slots[(k - 1) & 1])
                    if k + 1 < len(starts):
                        sizes[k + 1] = upload(k + 1)
                    pending = loss
                sc.copy_wait_compute()
                sc.copy_download(hl + 4 * ((len(starts) - 1) & 1), pending.value.main_ptr, 4)
                sc.copy_synchronize()
                total += float(slots[(len(starts) - 1) & 1])
                history.append(total / len(starts))
                if epoch % Loss_interval == 0 or epoch == Epochs - 1:
                    print(f"Epoch {epoch + 1}/{Epochs} — Loss: {history[-1]:.6f}")
        finally:
            sc.stream_synchronize()
            sc.copy_synchronize()
            if recorded is not None:
                recorded.release()
            for st in stage:
                sc.host_free_pinned(st["hx"]); sc.host_free_pinned(st["hy"])
            sc.host_free_pinned(hl)
        return np.array(history)

    def _fit_unpipelined(self, X_train, y, Optimizer, Loss, Epochs, batch_size=1):
        """The same loop with a synchronous upload and loss read per step (the reference's structure); kept as the
        yardstick for fit()."""
        history = []
        n = X_train.shape[0]
        for epoch in range(Epochs):
            perm = np.random.permutation(n)
            Xs, ys = X_train[perm], y[perm]
            total, batches = 0.0, 0
            for s in range(0, n, batch_size):
                e = min(s + batch_size, n)
                ypred = self.forward(Tensor(Xs[s:e], is_leaf=True))
                loss = Loss(ypred, Tensor(ys[s:e], is_leaf=True))
                self.zero_grad()
                autograd4nn(loss)
                Optimizer.step()
                total += float(loss.value.to_host_f32().ravel()[0])
                batches += 1
            history.append(total / batches)
        return np.array(history)

    # checkpoint: layer configs + host copies of the weights (same record layout as Seera.py:790-860)
    def save(self, filepath, optimizer=None, rank=None):
        """Layer records as the reference writes them (Seera.py:790-860).  With `optimizer`, a last record of class
        "__optimizer__" carries its kind, hyper-parameters, step count and state arenas (Adam m / v, SGD velocity), so
        that training resumes exactly; the reference drops that state.  In a data-parallel run only rank 0 writes
        (`rank`, else the RANK environment variable): the ranks hold identical weights and optimizer state."""
        import os
        if int(os.environ.get("RANK", "0") if rank is None else rank) != 0:
            return
        data = []
        for l in self.model:
            info = {"class": l.__class__.__name__, "config": {}}
            if isinstance(l, Input):
                info["config"]["shape"] = l.shape
            elif isinstance(l, Dense):
                info["config"] = {"in_units": l.in_units, "out_units": l.out_units, "layeract": l.layeract}
            elif isinstance(l, (Conv2D, ConvTranspose2D)):
                info["config"] = {"out_channels": l.out_channels, "in_channels": l.in_channels, "kernel_size": l.kernel_size,
                                  "layeract": l.layeract, "stride": l.stride, "zero_padding": l.zero_padding}
            elif isinstance(l, MaxPool2D):
                info["config"] = {"pool_size": l.pool_size, "stride": l.stride, "padding": l.padding}
            elif isinstance(l, _BatchNorm):
                info["config"] = {"num_features" if isinstance(l, BatchNorm1d) else "num_channels": l._num, "momentum": l.momentum,
                                  "eps": l.eps, "running_mean": l.running_mean, "running_var": l.running_var}
            elif isinstance(l, Unpool2D_Nearest):
                info["config"] = {"size": l.size}
            if isinstance(l, _ParamLayer):
                info["weights"], info["bais"] = l.weights.to_numpy(), l.bais.to_numpy()
            data.append(info)
        if optimizer is not None:
            data.append({"class": "__optimizer__", "config": optimizer.state_dict()})
        with open(filepath, "wb") as f:
            pickle.dump(data, f)

    @classmethod
    def load(cls, filepath, with_optimizer=False):
        """Rebuilds the model; with_optimizer=True returns (model, optimizer) with the saved optimizer state restored
        (optimizer is None when the file holds none)."""
        with open(filepath, "rb") as f:
            data = pickle.load(f)
        layers, opt_state = [], None
        for info in data:
            c, k = info["config"], info["class"]
            if k == "__optimizer__":
                opt_state = c
                continue
            if k == "Input":
                l = Input(c["shape"])
            elif k == "Dense":
                l = Dense(c["in_units"], c["out_units"], activation=c["layeract"])
            elif k in ("Conv2D", "ConvTranspose2D"):
                l = (Conv2D if k == "Conv2D" else ConvTranspose2D)(c["out_channels"], c["in_channels"], c["kernel_size"],
                                                                 activation=c["layeract"], stride=c.get("stride", 1),
                                                                 zero_padding=c.get("zero_padding", 0))
            elif k == "MaxPool2D":
                l = MaxPool2D(pool_size=c["pool_size"], stride=c["stride"], padding=c["padding"])
            elif k in ("BatchNorm1d", "BatchNorm2d"):
                l = BatchNorm1d(c["num_features"], c["momentum"], c["eps"]) if k == "BatchNorm1d" else \
                    BatchNorm2d(c["num_channels"], c["momentum"], c["eps"])
                l.running_mean, l.running_var = c["running_mean"], c["running_var"]
            elif k in ("Unpool2D_Nearest", "UpSampling2D_Nearest"):
                l = Unpool2D_Nearest(size=c["size"])
            elif k == "Flatten":
                l = Flatten()
            elif k == "Concatenate":
                l = Concatenate()
            else:
                raise ValueError(f"Unknown layer type: {k}")
            if "weights" in info:
                l._w_init = np.ascontiguousarray(info["weights"], np.float32)
                l._b_init = np.ascontiguousarray(info["bais"], np.float32)
            layers.append(l)
        model = cls(layers)
        if not with_optimizer:
            return model
        return model, (_Optimizer.from_state(model, opt_state) if opt_state is not None else None)


# ─────────────────────────────────────────────────────────────────────────────────────────────
# Losses
# ─────────────────────────────────────────────────────────────────────────────────────────────
def _scale_gradients(g):
    """In the fp16 precision modes the backward pass scales its gradient copies by a power of two taken from the largest
    entry of the loss gradient (fp16's exponent range is 2^-14 .. 2^16; a converging run's gradients leave it downwards)."""
    if sc.get_precision() in (4, 5):
        sc.grad_scale_of_loss(g.main_ptr, g.size)           # (g is the loss's own: nobody has written it since)


class Loss:
    """Each loss is the mean over the batch THIS process holds.  In a data-parallel run the ranks' gradients are averaged
    by the optimizer (dp.attach sets the 1/world factor there), so no scale is applied here."""

    def categorical_cross_entropy(self, y_pred, y, epsilon=1e-7):
        """mean over the batch of -sum(y * log(clip(y_pred, eps, 1-eps)))  (Seera.py:955-969)."""
        if y_pred._softmax_logits is None:
            raise NotImplementedError("categorical_cross_entropy expects the output of a softmax layer")
        logits = y_pred._softmax_logits
        z, yv = logits.value, y.value
        N, C = z.shape
        if tuple(yv.shape) != (N, C):
            raise ValueError(f"[cuTen]: Shapes {tuple(yv.shape)} and {(N, C)} not broadcastable")
        rows, loss, dz = _new((N,)), _new((1,)), _new((N, C))
        p = y_pred.value
        sc.softmax_cce_fwd_bwd(z.main_ptr, yv.main_ptr, p.claim() if p.__class__ is _Softmax else p.main_ptr, rows._ptr, loss._ptr, dz._ptr,
                               N, C, float(epsilon), float(f32(1.0 / N)))
        # the gradient arrives as the all-ones seed of a scalar loss
        out = Tensor._of(loss, (logits,), lambda g: (_scale_gradients(dz), logits._accumulate(dz)))
        out._keep = (rows, yv)
        out._pass = y_pred._pass
        return out

    def _elementwise(self, kernel, y_pred, y, *extra):
        p, yv = y_pred.value, y.value
        if p.size != yv.size:
            raise ValueError(f"[cuTen]: Shapes {tuple(p.shape)} and {tuple(yv.shape)} not broadcastable")
        part, loss, dp = _new((sc.mse_partials(p.size),)), _new((1,)), _new(p.shape)
        kernel(p.main_ptr, yv.main_ptr, part.main_ptr, loss.main_ptr, dp.main_ptr, p.size,
               float(f32(1.0 / p.size)), *extra)
        out = Tensor._of(loss, (y_pred,), lambda g: (_scale_gradients(dp), y_pred._accumulate(dp)))
        out._keep = (part, yv)
        out._pass = y_pred._pass
        return out

    def mse(self, y_pred, y):
        """mean((y_pred - y)^2) over all elements (Seera.py:943-945)."""
        return self._elementwise(sc.mse_fwd_bwd, y_pred, y)

    def mae(self, y_pred, y):
        """mean(|y_pred - y|) over all elements (Seera.py:947-949)."""
        return self._elementwise(sc.mae_fwd_bwd, y_pred, y)

    def binary_cross_entropy(self, y_pred, y, epsilon=1e-15):
        """mean(-y log(p + eps) - (1 - y) log(1 - p + eps)) over all elements (Seera.py:951-953)."""
        return self._elementwise(sc.bce_fwd_bwd, y_pred, y, float(epsilon))


_LOSSES = (Loss.categorical_cross_entropy, Loss.mse, Loss.mae, Loss.binary_cross_entropy)


# ─────────────────────────────────────────────────────────────────────────────────────────────
# Optimizers: one fused launch over the whole parameter arena
# ─────────────────────────────────────────────────────────────────────────────────────────────
class _Optimizer:
    """The scalars of a step travel with the update's launch, and in a recorded step they are replaced in the graph before each replay
    (graph_set_scalars).  Where the update is enqueued apart from them - bucket by bucket during backward, or behind a sum over the
    ranks outside the recording - its kernel reads them from a small device buffer, which `advance()` refreshes."""

    def __init__(self, model):
        if not isinstance(model, Sequential):
            raise TypeError("Model should be Sequential")
        self.model = model
        self.use_gpu = True
        self._hyper = cuten(np.zeros(16, np.float32))
        self._hyper_host = np.zeros(16, np.float32)
        # data parallel: the bucket hooks apply the update range by range behind each bucket's sum (dp.update_in_buckets);
        # step() then only completes the sums
        self.updates_by_bucket = False
        self._advanced = False
        # a recording whose replays replace the scalars in the graph itself (Trainer.capture), instead of reading them from the
        # device buffer
        self._scalars_in_graph = False

    def _state(self):
        n = max(self.model.n_arena, 1)
        return cuten._wrap(sc.cuda_zeros_f(n), (n,))

    def _grads_ready(self):
        m = self.model
        m.gather_grads()
        if m._allreduce is not None:
            m._allreduce(m.grads)

    def _grad_scale(self):
        return 1.0 / self.model.world if self.model._allreduce is not None else 1.0

    def _upload(self, values):
        h = self._hyper_host                      # pageable memory: the copy has left it when upload_f32 returns
        h[:len(values)] = values
        sc.upload_f32(self._hyper._ptr, h)

    @staticmethod
    def from_state(model, state):
        if state["kind"] == "adam":
            o = Adam(model, lr=state["lr"], beta1=state["beta1"], beta2=state["beta2"], eps=state["eps"])
            o.t = state["t"]
            arenas = (("m", o.m), ("v", o.v))
        else:
            o = SGD(model, lr=state["lr"], momentum=state["momentum"])
            arenas = (("velocity", o.velocity),)
        for name, dst in arenas:
            a = np.ascontiguousarray(state[name], np.float32)
            if a.size != dst.size:
                raise ValueError(f"optimizer state '{name}' has {a.size} values, the model's arena {dst.size}")
            sc.upload_f32(dst.main_ptr, a)
        return o

    def begin_step(self):
        """Call before backward when the update runs bucket by bucket during it: the step's scalars must be on the device before
        the first bucket's update is enqueued.  A no-op otherwise and inside a capture (replays refresh the scalars themselves)."""
        if self.updates_by_bucket and not sc.is_capturing() and not self._advanced:
            self.advance()
            self._advanced = True

    def update_range(self, begin, end):
        """The update of arena slots [begin, end) alone (the same arithmetic as the whole-arena launch)."""
        if not sc.is_capturing() and not self._advanced:        # first range of a step whose caller did not call begin_step()
            self.advance()
            self._advanced = True
        if end > begin:
            self._enqueue(begin, end)

    def advance(self):
        """Puts the scalars of the next update on the device and counts it."""
        self._upload(self._scalars())

    def step(self):
        """One update; outside a capture this also advances the step count."""
        by_bucket = self.updates_by_bucket and self.model._allreduce is not None
        capturing = sc.is_capturing()
        scalars = None
        if by_bucket:
            if not capturing and not self._advanced:
                self.advance()
        elif not capturing or self._scalars_in_graph:
            scalars = self._scalars(count=not capturing)      # by value with the launch: nothing to upload
        self._advanced = False
        self._grads_ready()
        if not by_bucket:
            self._enqueue(scalars=scalars)


class SGD(_Optimizer):
    """vel = momentum*vel + lr*g ; w -= vel   (Seera.py:986-1008)."""

    def __init__(self, model, lr, momentum=0):
        super().__init__(model)
        self.lr, self.momentum = lr, momentum
        self.velocity = self._state()

    def _scalars(self, count=True):
        return [self.lr, self.momentum, self._grad_scale()]

    def state_dict(self):
        return {"kind": "sgd", "lr": self.lr, "momentum": self.momentum, "velocity": self.velocity.to_host_f32().copy()}

    def _enqueue(self, begin=0, end=None, scalars=None):
        m = self.model
        end = m.n_arena if end is None else end
        o = 4 * begin
        at = (m.params.main_ptr + o, m.grads.main_ptr + o, self.velocity.main_ptr + o, end - begin)
        if scalars is None:
            sc.cuda_sgd_step_dev(*at, self._hyper.main_ptr)
        else:
            sc.cuda_sgd_step(*at, *scalars)


class Adam(_Optimizer):
    """m, v exponential averages with bias correction, t starting at 1 (Seera.py:1014-1086)."""

    def __init__(self, model, lr=0.001, beta1=0.9, beta2=0.999, eps=1e-8):
        super().__init__(model)
        self.lr, self.beta1, self.beta2, self.eps, self.t = lr, beta1, beta2, eps, 1
        self.m, self.v = self._state(), self._state()

    def _scalars(self, count=True):
        """The update's scalars at the current step; `count` moves on to the next step."""
        b1, b2, t = self.beta1, self.beta2, self.t
        if count:
            self.t = t + 1
        return [self.lr, b1, 1 - b1, b2, 1 - b2, self.eps, 1 - b1 ** t, 1 - b2 ** t, self._grad_scale()]

    def state_dict(self):
        return {"kind": "adam", "lr": self.lr, "beta1": self.beta1, "beta2": self.beta2, "eps": self.eps, "t": self.t,
                "m": self.m.to_host_f32().copy(), "v": self.v.to_host_f32().copy()}

    def _enqueue(self, begin=0, end=None, scalars=None):
        md = self.model
        end = md.n_arena if end is None else end
        o = 4 * begin
        at = (md.params.main_ptr + o, md.grads.main_ptr + o, self.m.main_ptr + o, self.v.main_ptr + o, end - begin)
        if scalars is None:
            sc.cuda_adam_step_dev(*at, self._hyper.main_ptr)
        else:
            sc.cuda_adam_step(*at, *scalars)
