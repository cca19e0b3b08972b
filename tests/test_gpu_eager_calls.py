"""Eager calls that csrc/eager.cpp takes give what the Python implementations give, over the forms of
arguments it accepts; what it does not accept goes on in Python."""
import subprocess
import sys
import threading
from pathlib import Path

import pytest
import torch

from pfeife_b200 import ops
from pfeife_b200.ops import _lib

pytestmark = pytest.mark.gpu
DT = {"fp16": torch.float16, "bf16": torch.bfloat16}


@pytest.fixture(autouse=True)
def _module():
    assert _lib.eager() is not None


def _r(*shape, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(dtype)


def _f(*shape):
    return torch.randn(*shape, device="cuda")


def _strided(t):
    """The same values with another order in memory: rows twice as far apart."""
    return torch.stack([t, t + 1], dim=-2)[..., 0, :]


def _shifted(t):
    """The same values one place off a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    return buf[1:].copy_(t.reshape(-1)).view(t.shape)


def _cases(dt):
    cos, sin = ops.rope_tables(20, 32, device="cuda")
    ids = torch.randint(0, 50, (37,), device="cuda")
    ids[::5] = -100
    w, b, x = _r(48, 64, dtype=dt, scale=.2), _f(48), _r(3, 7, 64, dtype=dt)
    w2, b2, res = _r(64, 48, dtype=dt, scale=.2), _f(64), _r(3, 7, 48, dtype=dt)
    qkv, q = _r(2, 20, 3, 4, 32, dtype=dt), _r(2, 20, 4, 32, dtype=dt)
    kv = _r(2, 9, 2, 4, 32, dtype=dt)
    img, cw = _r(1, 16, 16, 64, dtype=dt), _r(128, 64, 3, 3, dtype=dt, scale=.1)
    lin = lambda act: lambda *a: ops.linear(*a, activation=act)
    norm = lambda x, g, b, r: ops.layer_norm(x, g, b, 1e-5, residual=r)
    out = {
        "linear": (lin(None), (x, w, b)), "linear_no_bias": (lin(None), (x, w)),
        "linear_half_bias": (lin(None), (x[0], w, b.to(dt))), "linear_strided": (lin(None), (_strided(x), w, b)),
        "linear_class_token": (lambda x, w, b: ops.linear(x[:, 0], w, b), (x, w, b)),
        "linear_transposed": (lambda x, w: ops.linear(x.transpose(0, 1), w), (x, w)),
        "linear_odd_width": (lin(None), (x, w[:45], b[:45])),
        "linear_odd_depth": (lin(None), (x[..., :60], w[:, :60].contiguous(), b)),
        "linear_wide_rows": (lin(None), (x[..., :40], w[:, :40], b)),
        "linear_residual": (lambda x, w, b, r: ops.linear(x, w, b, residual=r), (x, w, b, res)),
        "linear_strided_residual": (lambda x, w, r: ops.linear(x, w, None, "gelu", r), (x, w, _strided(res))),
        "mlp": (lambda *a: ops.mlp(*a), (x, w, b, w2, b2)),
        "mlp_no_bias": (lambda x, w, w2: ops.mlp(x, w, None, w2, None, "gelu_tanh"), (x, w, w2)),
        "mlp_one_bias": (lambda x, w, w2, b2, r: ops.mlp(x, w, None, w2, b2, "gelu", r), (x, w, w2, b2, x + 1)),
        "mlp_silu": (lambda *a: ops.mlp(*a, activation="silu"), (x, w, b, w2, b2)),
        "norm": (lambda x, g, b: ops.layer_norm(x, g, b), (x, _f(64), _f(64))),
        "norm_residual": (norm, (x, _f(64), _f(64), x + 1)),
        "norm_strided": (norm, (_strided(x), _f(64), _f(64), _strided(x + 1))),
        "norm_one_row": (lambda x, g, b: ops.layer_norm(x, g, b), (x[0, 0], _f(64), _f(64))),
        "norm_no_bias": (lambda x, g: ops.layer_norm(x, g, None), (x, _f(64))),
        "norm_half_gain": (lambda x, g, b: ops.layer_norm(x, g, b), (x, _f(64).to(dt), _f(64))),
        "rms": (lambda x, g: ops.rms_norm(x, g), (x, _f(64))),
        "rms_residual": (lambda x, g, r: ops.rms_norm(x, g, residual=r), (x, _f(64), x + 1)),
        "qkv": (ops.attention_qkv, (qkv,)), "qkv_causal": (lambda t: ops.attention_qkv(t, True, 0.3), (qkv,)),
        "qkv_strided": (ops.attention_qkv, (_strided(qkv),)),
        "qkv_shifted": (ops.attention_qkv, (_shifted(qkv),)),
        "qkv_transposed": (lambda t: ops.attention_qkv(t.transpose(0, 1)), (qkv,)),
        "attention": (lambda q, kv: ops.attention(q, kv[:, :, 0], kv[:, :, 1]), (q, kv)),
        "attention_causal": (lambda q, k: ops.attention(q, k, k + 1, causal=True), (q, q + 2)),
        "attention_odd_strides": (lambda q, k: ops.attention(q[..., :24], k[..., :24], k[..., 8:]), (q, q + 1)),
        "rope": (lambda t: ops.rope_qkv(t, cos, sin), (qkv,)),
        "rope_strided": (lambda t: ops.rope_qkv(t, cos, sin), (_strided(qkv),)),
        "swiglu": (ops.swiglu, (x,)), "geglu": (ops.geglu, (x,)), "swiglu_strided": (ops.swiglu, (_strided(x),)),
        "loss": (lambda x: ops.cross_entropy(x, ids), (_r(37, 50, dtype=dt),)),
        "loss_fp32": (lambda x: ops.cross_entropy(x, ids), (_f(37, 50),)),
        "loss_strided": (lambda x: ops.cross_entropy(x, ids, ignore_index=3), (_strided(_r(37, 50, dtype=dt)),)),
        "loss_3d": (lambda x: ops.cross_entropy(x, ids[:36].view(4, 9)), (_r(4, 9, 50, dtype=dt),)),
        "group_norm": (lambda x, g, b: ops.group_norm(x, g, b, 32, silu=True), (img, _f(64), _f(64))),
        "group_norm_strided": (lambda x, g, b: ops.group_norm(x.transpose(1, 2), g, b, 8), (img, _f(64), _f(64))),
        "norm_shifted": (norm, (_shifted(x), _shifted(_f(64)), _shifted(_f(64)), _shifted(x + 1))),
        "swiglu_shifted": (ops.swiglu, (_shifted(x),)),
        "loss_shifted": (lambda x: ops.cross_entropy(x, ids), (_shifted(_r(37, 50, dtype=dt)),)),
        "group_norm_shifted": (lambda x, g, b: ops.group_norm(x, g, b, 8), (_shifted(img), _shifted(_f(64)), _f(64))),
        "conv": (lambda x, w, b: ops.conv2d(x, w, b, 1, 1), (img, cw, _f(128))),
        "conv_no_bias": (lambda x, w: ops.conv2d(x, w, None, 1, 1), (img, cw)),
        "conv_5x5": (lambda x, w: ops.conv2d(x, w, None, 1, 2), (img, _r(128, 64, 5, 5, dtype=dt, scale=.1))),
        "conv_stride": (lambda x, w, b: ops.conv2d(x, w, b, 2, 1), (_r(2, 32, 32, 64, dtype=dt), cw, _f(128))),
        "conv_no_padding": (lambda x, w: ops.conv2d(x, w, None, 1, 0), (_r(1, 18, 18, 64, dtype=dt), cw)),
        "conv_1x1": (lambda x, w: ops.conv2d(x, w, None), (img, cw[:, :, :1, :1].contiguous())),
        "conv_weight_order": (lambda x, w: ops.conv2d(x, w.permute(0, 3, 1, 2), None, 1, 1),
                              (img, cw.permute(0, 2, 3, 1).contiguous())),
    }
    return out


PYTHON = {"linear_odd_width", "linear_odd_depth", "mlp_silu", "norm_half_gain", "rope_strided", "swiglu_strided",
          "qkv_shifted", "norm_shifted", "swiglu_shifted", "group_norm_shifted", "loss_3d", "conv_stride", "conv_no_padding", "conv_1x1"}


# of these, the ones that are native where nothing is recorded
UNRECORDED = {"linear_odd_width", "conv_stride", "conv_no_padding"}


def _launches():
    return _lib._eager.launches() if _lib._eager is not None else 0


def _outputs(fn, leaves, needs):
    """(Native launches of the forward and of the backward, outputs and gradients of the `needs`.)"""
    leaves = [t.detach().requires_grad_(i in needs) for i, t in enumerate(leaves)]
    before = _launches()
    out = fn(*leaves)
    forward = _launches()
    out = out if isinstance(out, tuple) else (out,)
    assert out[0].grad_fn is not None
    wrt = [t for t in leaves if t.requires_grad]
    g = torch.Generator(device="cuda").manual_seed(3)
    # gradients that arrive in another order of memory, and one output that has none
    grads = [torch.randn(o.shape, device="cuda", generator=g).to(o.dtype) for o in out]
    grads = [_strided(t) if t.dim() > 1 else t for t in grads]
    got = torch.autograd.grad(out, wrt, grads, allow_unused=True, retain_graph=len(out) > 1)
    if len(out) > 1:
        got += torch.autograd.grad(out[1:], wrt, grads[1:], allow_unused=True)
    return (forward - before, _launches() - forward), out + tuple(got)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("name", list(_cases(torch.bfloat16)) if torch.cuda.is_available() else [])
def test_native_calls_equal_pythons(name, dtype, monkeypatch):
    """The same kernels on the same data: equal bits, but for the sums by atomics (bias gradients of products),
    whose order differs: by a rounding of 32 bits, or of the 16 that a bias of those has."""
    torch.manual_seed(len(name))
    fn, leaves = _cases(DT[dtype])[name]
    every = set(range(len(leaves)))
    for needs in [every] + [every - {i} for i in every if len(every) > 1]:
        native, got = _outputs(fn, leaves, needs)
        assert all(n > 0 for n in native) if name not in PYTHON else native == (0, 0)
        before = _launches()
        with torch.no_grad():
            plain = fn(*leaves)
        if name not in PYTHON or name in UNRECORDED:
            assert _launches() > before
        with monkeypatch.context() as m:
            m.setattr(_lib, "_eager", None)
            want = _outputs(fn, leaves, needs)[1]
            with torch.no_grad():
                plain_want = fn(*leaves)
        for a, b in zip(plain if isinstance(plain, tuple) else (plain,),
                        plain_want if isinstance(plain_want, tuple) else (plain_want,)):
            assert torch.equal(a, b) and a.stride() == b.stride() and not a.requires_grad
        assert len(got) == len(want)
        for a, b in zip(got, want):
            assert (a is None) == (b is None)
            if a is not None:
                assert a.dtype == b.dtype and a.shape == b.shape
                if a.dim() == 1 and name.startswith(("linear", "mlp", "conv")):
                    torch.testing.assert_close(a, b, rtol=2.0 ** -7 if a.dtype != torch.float32 else 1e-5, atol=1e-5)
                else:
                    assert torch.equal(a, b)


def _reversed(t):
    """The same values with the dimensions the other way round in memory."""
    order = tuple(reversed(range(t.dim())))
    return t.permute(order).contiguous().permute(order)


def _spread(t):
    """The same values with a gap after each."""
    return torch.stack([t, t + 1], dim=-1)[..., 0]


def _wider(t):
    return t.float() if t.dtype in DT.values() else t


UNPACK = {"same": lambda t: t, "clone": lambda t: t.clone(), "reversed": _reversed,
          "shifted": lambda t: _shifted(t) if t.dim() > 0 else t,
          "rows_apart": lambda t: _strided(t) if t.dim() > 1 else t, "spread": _spread, "wider": _wider,
          "wider_images": lambda t: _wider(t) if t.dim() > 2 else t,
          "double": lambda t: t.double() if t.dtype == torch.float32 else t}


def _hooked(fn, leaves, how):
    """(outputs, None), or (None, what was raised) under hooks that unpack `how`."""
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, UNPACK[how]):
        try:
            return _outputs(fn, leaves, set(range(len(leaves))))[1], None
        except (AssertionError, RuntimeError) as e:
            return None, type(e)


def _agree(got, want):
    for a, b in zip(got, want):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.dtype == b.dtype and a.shape == b.shape
            # results of 8 bits, and probabilities of 8 bits where a formula in fp32 has more
            assert (a.double() - b.double()).norm() <= 2.0 ** -7 * b.double().norm()


@pytest.mark.parametrize("how", UNPACK)
@pytest.mark.parametrize("name", list(_cases(torch.bfloat16)) if torch.cuda.is_available() else [])
def test_what_the_formulas_in_python_unpack(name, how, monkeypatch):
    """Hooks on saved tensors that return the same values in another order or type: the gradients of a call
    without hooks.  Products refuse operands with gaps between a row's values, and a pre-activation and
    logits of another type."""
    torch.manual_seed(len(name))
    fn, leaves = _cases(torch.bfloat16)[name]
    monkeypatch.setattr(_lib, "_eager", None)
    want = _outputs(fn, leaves, set(range(len(leaves))))[1]
    got, error = _hooked(fn, leaves, how)
    if error is None:
        _agree(got, want)
    elif how == "shifted":              # what TMA reads has to lie on 16 bytes
        assert error is _lib.KernelError and name.startswith(("linear", "mlp", "conv", "attention"))
    else:
        assert name.startswith(("linear", "mlp", "loss", "conv_1x1")) and how not in ("same", "clone", "rows_apart")


@pytest.mark.parametrize("how", UNPACK)
@pytest.mark.parametrize("name", list(_cases(torch.bfloat16)) if torch.cuda.is_available() else [])
def test_what_native_backwards_unpack(name, how, monkeypatch):
    """The same of the nodes in C++, which raise what the formulas in Python raise."""
    torch.manual_seed(len(name))
    fn, leaves = _cases(torch.bfloat16)[name]
    want = _outputs(fn, leaves, set(range(len(leaves))))[1]
    got, error = _hooked(fn, leaves, how)
    with monkeypatch.context() as m:
        m.setattr(_lib, "_eager", None)
        assert error == _hooked(fn, leaves, how)[1]
    if error is None:
        _agree(got, want)


@pytest.mark.parametrize("python", [False, True])
@pytest.mark.parametrize("name", ["norm_residual", "rms", "norm_one_row", "swiglu", "geglu", "group_norm", "rope", "qkv",
                                  "attention"])
def test_gradients_off_their_vectors(name, python, monkeypatch):
    """A gradient that is a view into a buffer, off the 16 bytes that the kernels read it by."""
    fn, leaves = _cases(torch.bfloat16)[name]
    if python:
        monkeypatch.setattr(_lib, "_eager", None)
    leaves = [t.detach().requires_grad_() for t in leaves]
    out = fn(*leaves)
    out = out if isinstance(out, tuple) else (out,)
    dy = [torch.randn(o.shape, device="cuda").to(o.dtype) for o in out]
    got, want = (torch.autograd.grad(out, leaves, g, retain_graph=True) for g in ([_shifted(t) for t in dy], dy))
    _agree(got, want)


def test_rotary_tables_in_any_order():
    x, dy = _r(2, 20, 3, 4, 32).requires_grad_(), _r(2, 20, 3, 4, 32)
    tables = ops.rope_tables(20, 32, device="cuda")
    want = ops.rope_qkv(x, *tables)
    for order in (_reversed, _spread, _strided, _shifted):
        got = ops.rope_qkv(x, *map(order, tables))
        assert torch.equal(got, want)
        assert torch.equal(*(torch.autograd.grad(y, x, dy, retain_graph=True)[0] for y in (got, want)))


def test_results_may_be_changed_in_place_and_inputs_may_not():
    x, w = _r(8, 64).requires_grad_(), _r(64, 64).requires_grad_()
    y = ops.linear(x * 1, w)
    y.add_(1)                                      # not a view, not needed by the backward
    y.sum().backward()
    h = x * 1
    z = ops.layer_norm(h, _f(64), _f(64))
    h.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        z.sum().backward()
    y = ops.linear(x, w)
    y.sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        y.sum().backward()


def test_what_observes_ops_sees_them():
    from torch.utils._python_dispatch import TorchDispatchMode
    x, w = _r(8, 64), _r(64, 64)
    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Watch():
        ops.linear(x, w)
    assert any("pfeife" in s for s in seen)
    before = _lib._eager.launches()
    with torch.autocast("cuda", dtype=torch.float16):
        assert ops.linear(x, w).dtype == torch.float16
    ops.linear(torch.nn.Parameter(x).as_subclass(type("Sub", (torch.Tensor,), {})), w)
    assert _lib._eager.launches() == before
    assert isinstance(ops.linear(torch.nn.Parameter(x), w), torch.Tensor)
    assert _lib._eager.launches() > before


def test_refused_calls_raise_what_they_raised():
    x, w = _r(8, 64), _r(64, 64)
    with pytest.raises(AssertionError):
        ops.linear(x, _r(64, 32))
    with pytest.raises(_lib.KernelError):
        ops.linear(_shifted(x), w)
    y = ops.linear(x.requires_grad_(), w)
    with pytest.raises(_lib.KernelError):
        y.backward(_shifted(torch.ones_like(y)))


FIRST_CALL = """
import torch
from pfeife_b200 import ops
from pfeife_b200.ops import _lib
x, w = (torch.randn(64, 64, device="cuda").bfloat16() for _ in range(2))
seen = []
def call(x):
    ops.linear(x, w)
    seen.append(_lib._eager.launches())
with torch.inference_mode():
    call(x)
    call(x + 1)
call(x)
with torch.no_grad():
    call(x.requires_grad_())
y = ops.linear(x, w)
y.sum().backward()
assert seen == [1, 2, 3, 4] and _lib._eager.launches() > 5 and type(y.grad_fn).__name__ == "CppFunction", seen
"""


def test_the_first_call_may_be_in_inference_mode():
    """In a process of its own: what a call learns of tensors does not depend on the mode it is made in."""
    root = Path(__file__).resolve().parent.parent
    subprocess.run([sys.executable, "-c", FIRST_CALL], cwd=root, check=True, timeout=300)


def test_threads_and_streams():
    """Calls from several threads, each on a stream of its own."""
    x, w, b = _r(64, 256), _r(256, 256, scale=.1), _f(256)
    want, errors = ops.mlp(x, w, b, w, b), []

    def work():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
                for _ in range(50):
                    leaf = x.clone().requires_grad_()
                    y = ops.mlp(leaf, w, b, w, b)
                    y.sum().backward()
                    assert torch.equal(y, want) and leaf.grad is not None
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
