"""An eager call on plain tensors goes straight to its implementation; transforms, tracers, hooks and
higher derivatives still have to work as they do through the dispatcher.  On CPU the direct way is
switched on for CPU tensors."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from pfeife_b200 import ops
from pfeife_b200.ops import functional

DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


@pytest.fixture(params=DEVICES)
def device(request, monkeypatch):
    monkeypatch.setattr(functional, "_FIRST_DEVICE", -1 if request.param == "cpu" else 0)
    return request.param


class Watch(TorchDispatchMode):
    """Lets every op be seen, which keeps all calls on the dispatcher."""

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def _cases(device):
    """name -> (function of the leaves, leaves)"""
    dt = torch.float32 if device == "cpu" else torch.bfloat16
    g = torch.Generator().manual_seed(5)

    def r(*shape, scale=1.0, dtype=dt):
        return (torch.randn(*shape, generator=g) * scale).to(device=device, dtype=dtype)

    def v(n):
        return r(n, dtype=torch.float32)

    cos, sin = ops.rope_tables(16, 16, device=device)
    ids = torch.randint(0, 24, (2, 16), generator=g).to(device)
    return {
        "linear": (lambda x, w, b, res: ops.linear(x, w, b, "gelu", res),
                   [r(16, 64), r(32, 64, scale=0.2), v(32), r(16, 32)]),
        "mlp": (lambda x, w1, b1, w2, b2, res: ops.mlp(x, w1, b1, w2, b2, "gelu", res),
                [r(16, 64), r(96, 64, scale=0.2), v(96), r(64, 96, scale=0.2), v(64), r(16, 64)]),
        "layer_norm": (lambda x, w, b, res: ops.layer_norm(x, w, b, 1e-5, residual=res)[0],
                       [r(16, 64), v(64), v(64), r(16, 64)]),
        "rms_norm": (lambda x, w: ops.rms_norm(x, w), [r(16, 64), v(64)]),
        "gelu": (ops.gelu, [r(16, 64)]),
        "swiglu": (ops.swiglu, [r(16, 64)]),
        "cross_entropy": (lambda x: ops.cross_entropy(x, ids.view(-1)), [r(32, 24)]),
        "cross_entropy_rows": (lambda x: ops.cross_entropy(x, ids.view(-1), reduction="none"),
                               [r(32, 24)]),
        "mse": (lambda a: ops.mse_loss(a, a.detach() + 1), [r(16, 64)]),
        "embedding": (lambda t: ops.embedding(ids, t, dt), [r(24, 32)]),
        "rope": (lambda x: ops.rope(x, cos, sin), [r(2, 16, 2, 16)]),
        "rope_qkv": (lambda x: ops.rope_qkv(x, cos, sin), [r(2, 16, 3, 2, 16)]),
        "attention": (lambda q, k, v: ops.attention(q, k, v, causal=True),
                      [r(2, 16, 2, 16), r(2, 16, 2, 16), r(2, 16, 2, 16)]),
        "attention_qkv": (lambda qkv: ops.attention_qkv(qkv), [r(2, 16, 3, 2, 16)]),
        "conv2d": (lambda x, w, b: ops.conv2d(x, w, b, 1, 1),
                   [r(1, 8, 8, 16), r(24, 16, 3, 3, scale=0.2), v(24)]),
        "group_norm": (lambda x, w, b: ops.group_norm(x, w, b, 4, silu=True),
                       [r(2, 4, 4, 32), v(32), v(32)]),
        "upsample": (ops.upsample_nearest2x, [r(2, 4, 4, 32)]),
    }


NAMES = list(_cases("cpu"))
# two correct computations of one 16-bit result differ by a rounding; sums with atomics by less
TOL = {"cpu": 1e-5, "cuda": 2.0 ** -7}


def _near(a, b, device):
    a, b = a.double(), b.double()
    assert a.shape == b.shape and (a - b).norm() <= TOL[device] * b.norm() + 1e-6


@pytest.mark.parametrize("name", NAMES)
def test_gradients_of_several_vectors_at_once(name, device):
    fn, leaves = _cases(device)[name]
    leaves = [t.requires_grad_() for t in leaves]
    y = fn(*leaves)
    assert "Direct" in y.grad_fn.name() or name == "cross_entropy_rows"      # (a view of it)
    vs = torch.stack([torch.ones_like(y), torch.randn_like(y), torch.zeros_like(y)])
    batched = torch.autograd.grad(y, leaves, vs, is_grads_batched=True, retain_graph=True)
    for i in range(len(vs)):
        one = torch.autograd.grad(y, leaves, vs[i], retain_graph=True)
        for a, b in zip(batched, one):
            _near(a[i], b, device)


def test_lazily_negated_inputs(device, monkeypatch):
    """A view with the negative bit set holds the wrong sign in memory: no implementation gets one."""
    for op in (functional.act_fwd, functional.act_bwd):
        def plain(x, *args, plain=op.plain):
            assert not x.is_neg()
            return plain(x, *args)
        monkeypatch.setattr(op, "plain", plain)
    dtype = torch.float32 if device == "cpu" else torch.bfloat16
    x = torch.randn(8, 64).to(device=device, dtype=dtype)
    flip = torch._neg_view(x).requires_grad_()
    y, want = ops.gelu(flip), ops.gelu((-x).requires_grad_())
    _near(y, want, device)
    v = torch.randn_like(x)
    for out in (y, want):
        (g,) = torch.autograd.grad(out, out.grad_fn.next_functions[0][0].variable, torch._neg_view(v),
                                   retain_graph=True)
        (w,) = torch.autograd.grad(out, out.grad_fn.next_functions[0][0].variable, -v)
        _near(g, w, device)


def test_wrappers_that_outlive_their_transform(device):
    """A tensor kept from inside a transform has no memory of its own; the dispatcher unwraps it."""
    dtype = torch.float32 if device == "cpu" else torch.bfloat16
    x, kept = torch.randn(8, 64).to(device=device, dtype=dtype), []
    torch.func.grad(lambda t: (kept.append(t), t.sum())[1])(x)
    torch.func.functionalize(lambda t: (kept.append(t), t + 1)[1])(x)
    for t in kept:
        assert not functional._plain_call((t,))
    assert torch.equal(ops.gelu(kept[0]), ops.gelu(x))


@pytest.mark.parametrize("name", ["rope", "rope_qkv", "upsample", "linear", "mlp"])
def test_second_derivatives_where_the_backward_is_linear(name, device):
    """The gradients of rope, of upsampling and of a residual are linear in the result's gradient
    and are made of ops that can be differentiated again."""
    fn, leaves = _cases(device)[name]
    leaves = [t.requires_grad_() for t in leaves]
    x = leaves[-1]                       # the residual, or the only input
    out = []
    for watched in (False, True):
        v = torch.full_like(fn(*leaves), 0.5).requires_grad_()
        if watched:
            with Watch():
                (gx,) = torch.autograd.grad(fn(*leaves), x, v, create_graph=True)
                (gv,) = torch.autograd.grad(gx.square().sum(), v)
        else:
            (gx,) = torch.autograd.grad(fn(*leaves), x, v, create_graph=True)
            (gv,) = torch.autograd.grad(gx.square().sum(), v)
        out.append((gx.detach(), gv))
    for a, b in zip(*out):
        assert torch.equal(a, b) and b.any()


def test_second_derivatives_of_the_others_are_refused(device):
    fn, leaves = _cases(device)["linear"]
    leaves = [t.requires_grad_() for t in leaves]
    (gx,) = torch.autograd.grad(fn(*leaves).sum(), leaves[0], create_graph=True)
    with pytest.raises(RuntimeError):
        gx.sum().backward()


@pytest.mark.parametrize("name", ["linear", "layer_norm", "rope", "rope_qkv", "cross_entropy",
                                  "attention_qkv"])
def test_symbolic_traces_beside_real_tensors(name, device):
    """A proxy input next to tensors that exist (weights, tables): the call is recorded."""
    fn, leaves = _cases(device)[name]
    rest = leaves[1:]
    if name == "attention_qkv":
        fn = lambda qkv: ops.attention_qkv(qkv, scale=0.25)
    if name == "cross_entropy":
        ids = torch.arange(32, device=device) % 24
        fn = lambda x: functional._call(functional.ce_mean_fwd, x, ids, -100)
    gm = torch.fx.symbolic_trace(lambda x: fn(x, *rest))
    assert any("pfeife" in str(n.target) for n in gm.graph.nodes)
    with torch.no_grad():
        assert torch.equal(gm(leaves[0]), fn(*leaves))


@pytest.mark.parametrize("name", NAMES)
def test_recomputing_checkpoints(name, device):
    """Saved tensors come back through hooks that may themselves run recorded ops, once each."""
    from torch.utils.checkpoint import checkpoint
    fn, leaves = _cases(device)[name]
    leaves = [t.requires_grad_() for t in leaves]
    y = fn(*leaves)
    want = torch.autograd.grad(y, leaves, torch.ones_like(y))
    y = checkpoint(lambda *a: fn(a[0] * 1, *a[1:]), *leaves, use_reentrant=False)
    got = torch.autograd.grad(y, leaves, torch.ones_like(y))
    for a, b in zip(got, want):
        _near(a, b, device)


def test_unpacking_hooks_run_recorded(device):
    seen = []

    def unpack(t):
        leaf = torch.ones(2, device=t.device, requires_grad=True)
        with torch.enable_grad():
            seen.append((leaf * 2).requires_grad)
        return t

    fn, leaves = _cases(device)["linear"]
    leaves = [t.requires_grad_() for t in leaves]
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        y = fn(*leaves)
    torch.autograd.grad(y, leaves, torch.ones_like(y))
    assert seen and all(seen)


def test_calls_inside_another_op_are_not_recorded(device):
    """Below autograd (the implementation of a user's own op) a call keeps no graph, whatever its
    weights ask for."""
    w = torch.randn(32, 64).to(device=device, dtype=torch.float32 if device == "cpu" else torch.bfloat16)
    x, w = torch.ones_like(w), w.requires_grad_()
    with torch._C._AutoDispatchBelowAutograd():
        assert ops.linear(x, w).grad_fn is None
    assert ops.linear(x, w).grad_fn is not None
