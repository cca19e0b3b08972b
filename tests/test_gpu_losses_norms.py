"""Losses, norms and eager calls at the edges of their kernels' vector, slab and tile splits, against
64-bit PyTorch."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

# unit roundoff of the result types
U = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -24}


def close(got, want, rel):
    """2-norm of the difference, relative; `rel` is the rounding of the result's type plus the
    1e-5 of fp32 sums."""
    got, want = got.double(), want.double()
    assert torch.isfinite(got).all()
    assert (got - want).norm() <= (rel + 1e-5) * want.norm() + 1e-12


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,V", [(1, 1), (3, 7), (5, 1000), (17, 2049), (591, 33), (592, 4103),
                                    (2, 50257), (1200, 1003)])
def test_cross_entropy_edges(rows, V, dtype):
    from pfeife_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows + V)
    x = (torch.randn(rows, V, device="cuda", generator=g) * 3).to(dtype).requires_grad_()
    t = torch.randint(0, V, (rows,), device="cuda", generator=g)
    t[::3] = -100
    xr = x.detach().double().requires_grad_()
    for reduction in ("mean", "sum", "none"):
        loss = ops.cross_entropy(x, t, reduction=reduction)
        want = F.cross_entropy(xr, t, reduction="none")
        want = want if reduction == "none" else want.sum() / (
            max(1, int((t != -100).sum())) if reduction == "mean" else 1)
        w = torch.randn(loss.shape, device="cuda", generator=g) + 2
        (dx,) = torch.autograd.grad(loss, x, w)
        (dr,) = torch.autograd.grad(want, xr, w.double())
        close(loss, want, 0.0)
        # fp16: small probabilities over many rows are subnormal, half a step of 2^-24 each
        sub = 2.0 ** -25 * dr.numel() ** 0.5 if dtype == torch.float16 else 0.0
        assert (dx.double() - dr).norm() <= (U[dtype] + 1e-5) * dr.norm() + sub


@pytest.mark.parametrize("rows", [16384, 16385, 20000, 700001])
def test_cross_entropy_of_many_rows(rows):
    """Per-pixel losses: several CTAs sum the rows; the mean is that of the rows that count."""
    from pfeife_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, 5, device="cuda", generator=g).requires_grad_()
    t = torch.randint(0, 5, (rows,), device="cuda", generator=g)
    t[1::3] = -100
    xr = x.detach().double().requires_grad_()
    loss, want = ops.cross_entropy(x, t), F.cross_entropy(xr, t)
    close(loss, want, 0.0)
    close(torch.autograd.grad(loss, x)[0], torch.autograd.grad(want, xr)[0], 0.0)


def test_cross_entropy_masked_vocabulary_and_all_ignored():
    """Logits of -inf and of the type's lowest value have no probability; a batch without a row
    that counts has loss 0 and no gradient."""
    from pfeife_b200 import ops
    x = torch.randn(9, 3000, device="cuda").to(torch.bfloat16)
    x[:, :1024] = float("-inf")
    x[:, 2000:] = torch.finfo(torch.bfloat16).min
    t = torch.randint(1024, 2000, (9,), device="cuda")
    x.requires_grad_()
    loss = ops.cross_entropy(x, t)
    (dx,) = torch.autograd.grad(loss, x)
    xr = x.detach().double().requires_grad_()
    want = F.cross_entropy(xr, t)
    (dr,) = torch.autograd.grad(want, xr)
    close(loss, want, 0.0)
    close(dx, dr, U[torch.bfloat16])
    none = torch.full_like(t, -100)
    y = torch.randn(9, 3000, device="cuda").to(torch.bfloat16).requires_grad_()
    loss = ops.cross_entropy(y, none)
    (dy,) = torch.autograd.grad(loss, y)
    assert float(loss.detach()) == 0.0 and not dy.any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [9, 700])       # both sizes of CTA
@pytest.mark.parametrize("V", [2, 7, 10, 1000, 2048, 3001])
def test_cross_entropy_keeps_nan_and_skips_masked(V, rows, dtype):
    """A NaN logit outside the target's column makes the row's loss NaN, whatever part of the row a
    thread owns; -inf logits (a masked vocabulary) count as zero probability."""
    from pfeife_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(V + rows)
    x = torch.randn(rows, V, device="cuda", generator=g).to(dtype)
    t = torch.zeros(rows, dtype=torch.int64, device="cuda")
    masked = torch.rand(rows, V, device="cuda", generator=g) < 0.7
    masked[:, 0] = False
    x = x.masked_fill(masked, float("-inf"))
    want = F.cross_entropy(x.double(), t, reduction="none")
    got = ops.cross_entropy(x, t, reduction="none")
    # the targets' own rounding aside, fp32 sums: u of the loss and of the logits it is the difference of
    assert torch.allclose(got.double(), want, rtol=1e-5, atol=1e-5)
    r = torch.arange(rows, device="cuda")
    one = x.clone()
    one[r, 1 + r % (V - 1)] = float("nan")
    run = x.clone()                       # eight NaNs side by side: the whole of one 16-byte load
    for k in range(8):
        run[r, (1 + (8 * r + k) % (V - 1))] = float("nan")
    for bad in (one, run):
        assert torch.isnan(ops.cross_entropy(bad, t, reduction="none")).all()
        assert torch.isnan(ops.cross_entropy(bad, t))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("silu", [True, False])
@pytest.mark.parametrize("B,H,W,C,G", [(1, 1, 1, 32, 8), (2, 5, 7, 8, 2), (3, 16, 16, 32, 8),
                                       (1, 37, 37, 320, 32), (2, 9, 3, 2048, 32),
                                       (1, 4, 4, 2560, 32), (5, 64, 64, 96, 32)])
def test_group_norm_edges(B, H, W, C, G, silu, dtype):
    from pfeife_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(C + H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x = (rnd(B, H, W, C) * 2 + rnd(C)).to(dtype).requires_grad_()
    w, b = (1 + 0.2 * rnd(C)).requires_grad_(), (0.2 * rnd(C)).requires_grad_()
    dy = rnd(B, H, W, C).to(dtype)
    xr, wr, br = (t.detach().double().requires_grad_() for t in (x, w, b))
    want = F.group_norm(xr.permute(0, 3, 1, 2), G, wr, br, 1e-5).permute(0, 2, 3, 1)
    want = F.silu(want) if silu else want
    wants = torch.autograd.grad(want, (xr, wr, br), dy.double())
    for _ in range(2):               # the second time into recycled scratch
        y = ops.group_norm(x, w, b, G, 1e-5, silu)
        grads = torch.autograd.grad(y, (x, w, b), dy)
        close(y, want, U[dtype])
        for got, ref in zip(grads, wants):
            # groups of a few values lose digits in E[x^2] - E[x]^2 and in the differences of dx
            close(got, ref, (U[dtype] if got.dtype == dtype else 0.0) + (2e-4 if H * W < 64 else 0))


def _block(x, res, w, b, w1, b1, qkv):
    from pfeife_b200 import ops
    y, h = ops.layer_norm(x, w, b, 1e-5, residual=res)
    y = ops.mlp(y, w1, b1, w1.t().contiguous(), None, "gelu", residual=h)
    a = ops.attention_qkv(ops.linear(y, qkv).view(2, 16, 3, 4, 16), causal=True)
    return ops.cross_entropy(a.reshape(-1, 64).float() * 4, torch.arange(32, device=x.device))


def test_eager_calls_equal_dispatched_ones():
    """An eager call goes straight to its implementation and gives the bits that the same call gives
    through the dispatcher (under a dispatch mode, where every op must stay visible)."""
    from torch.utils._python_dispatch import TorchDispatchMode
    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    g = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    mk = [rnd(2, 16, 64).half(), rnd(2, 16, 64).half(), 1 + 0.1 * rnd(64), 0.1 * rnd(64),
          (0.1 * rnd(64, 64)).half(), 0.1 * rnd(64), (0.2 * rnd(192, 64)).half()]
    results = []
    for watch in (False, True):
        leaves = [t.clone().requires_grad_() for t in mk]
        if watch:
            with Watch():
                loss = _block(*leaves)
                loss.backward()
        else:
            loss = _block(*leaves)
            loss.backward()
        assert ("Direct" in loss.grad_fn.name()) is not watch
        results.append([loss.detach()] + [t.grad for t in leaves])
    assert any("pfeife::linear_fwd" in s or "pfeife.linear_fwd" in s for s in seen)
    assert any("attn_qkv_bwd" in s for s in seen)
    for i, (a, b) in enumerate(zip(*results)):
        if i == 6:      # b1: its column sums are added with atomics, in any order
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-6)
        else:           # dq comes from one key tile, the norm's sums in a fixed order
            assert torch.equal(a, b)


def test_eager_backward_launches_each_kernel_once():
    """The packed attention backward is one native call, whichever way the op was called."""
    from pfeife_b200 import ops
    from pfeife_b200.ops import _lib
    qkv = torch.randn(1, 64, 3, 2, 32, device="cuda").half().requires_grad_()
    o = ops.attention_qkv(qkv)
    before = _lib.launch_count()
    (dqkv,) = torch.autograd.grad(o, qkv, torch.ones_like(o))
    assert _lib.launch_count() == before + 1 and dqkv.is_contiguous()


def test_eager_calls_keep_autograd_rules():
    """Saved-tensor hooks see what the ops save, a second backward is refused, results may be changed
    in place, and no graph is kept without gradients."""
    from pfeife_b200 import ops
    x = torch.randn(8, 64, device="cuda").half().requires_grad_()
    w = torch.randn(32, 64, device="cuda").half().requires_grad_()
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(),
                                                  lambda t: t.cuda()):
        y = ops.linear(x, w, activation="gelu")
    assert torch.Size([8, 64]) in packed and torch.Size([32, 64]) in packed
    dx, dw = torch.autograd.grad(y, (x, w), torch.ones_like(y), retain_graph=True)
    z = ops.linear(x, w, activation="gelu")
    rx, rw = torch.autograd.grad(z, (x, w), torch.ones_like(z))
    assert torch.equal(dx, rx) and torch.equal(dw, rw)
    z = ops.linear(x, w)
    (gx,) = torch.autograd.grad(z, x, torch.ones_like(z), create_graph=True)
    with pytest.raises(RuntimeError):
        gx.sum().backward()
    with torch.no_grad():
        assert ops.linear(x, w).grad_fn is None
    assert ops.linear(x.detach(), w.detach()).grad_fn is None
    # results may be changed in place, with and without a graph
    x3 = x.detach().view(2, 4, 64).requires_grad_()
    y = ops.linear(x3, w)
    y += 1.0
    (gx,) = torch.autograd.grad(y.float().square().sum(), x3)
    z = ops.linear(x3, w) + 1.0
    (rx,) = torch.autograd.grad(z.float().square().sum(), x3)
    assert torch.equal(gx, rx)
    with torch.no_grad():
        y = ops.linear(x3, w)
    y.add_(ops.linear(x3, w))
    assert y.requires_grad


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,N", [(1, 8), (7, 24), (8, 192), (9, 256), (300, 264), (2371, 1408),
                                    (5, 2040), (4999, 2048), (33, 2056), (640, 520)])
def test_norm_backward_tiles(rows, N, rms):
    """Gradients of the residual norm at the edges of the row tiles and column shares; twice, the
    second time into recycled scratch, and into existing gradients."""
    from pfeife_b200 import ops
    from pfeife_b200.ops import kernels as kx
    g = torch.Generator(device="cuda").manual_seed(rows + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    dtype = torch.bfloat16
    x, res, gy, gh = ((rnd(rows, N) * 2).to(dtype) for _ in range(4))
    w, b = 1 + 0.1 * rnd(N), 0.1 * rnd(N)
    xr, wr, br = (t.double().requires_grad_() for t in ((x + res), w, b))
    if rms:
        want = xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-5) * wr
    else:
        want = F.layer_norm(xr, (N,), wr, br, 1e-5)
    wants = torch.autograd.grad(want, (xr, wr) if rms else (xr, wr, br), gy.double())
    for _ in range(2):
        leaves = [t.clone().requires_grad_() for t in (x, res, w, b)]
        if rms:
            y, h = ops.rms_norm(leaves[0], leaves[2], 1e-5, residual=leaves[1])
        else:
            y, h = ops.layer_norm(*[leaves[i] for i in (0, 2, 3)], 1e-5, residual=leaves[1])
        wrt = (leaves[0], leaves[2]) if rms else (leaves[0], leaves[2], leaves[3])
        grads = torch.autograd.grad((y, h), wrt, (gy, gh))
        close(y, want, U[dtype])
        # dx is rounded once, after the gradient of the sum was added to it
        close(grads[0], wants[0] + gh.double(), 1.5 * U[dtype])
        for got, ref in zip(grads[1:], wants[1:]):
            close(got, ref, 1e-5)
    _, _, mean, rstd = kx.norm_fwd(x + res, w, None if rms else b, 1e-5, rms)
    dw, db = torch.ones(N, device="cuda"), torch.ones(N, device="cuda")
    kx.norm_bwd(gy, x + res, w, mean, rstd, rms, dgamma=dw, dbeta=None if rms else db,
                accumulate=True, want_dbeta=False)
    close(dw, wants[1] + 1, 1e-5)
    if not rms:
        close(db, wants[2] + 1, 1e-5)


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,N", [(1, 4096), (2, 2056), (3, 3072), (591, 3080), (2500, 4096)])
def test_norm_backward_wide_rows(rows, N, rms):
    """Rows that one CTA holds two at a time: fewer batches than the ring has stages, an odd last
    row, threads without columns, several batches per CTA."""
    test_norm_backward_tiles(rows, N, rms)


@pytest.mark.parametrize("silu", [True, False])
@pytest.mark.parametrize("B,H,W,C,G", [(1, 5, 5, 3200, 32), (1, 5, 5, 3328, 32), (2, 64, 41, 320, 32)])
def test_group_norm_forms_of_the_backward(B, H, W, C, G, silu):
    """The largest CTA with a ring of pixels, the form without one, and more pixels per thread than a
    ring has places."""
    test_group_norm_edges(B, H, W, C, G, silu, torch.bfloat16)


def test_norm_backward_wide_rows_on_some_of_the_sms():
    """The caller's number of SMs bounds the CTAs, each of which writes one row of scratch."""
    from pfeife_b200.ops import _lib
    rows, N, sms = 1000, 3072, 16
    L = _lib.calls()
    h, dy = (torch.randn(rows, N, device="cuda").to(torch.bfloat16) for _ in range(2))
    w = torch.ones(N, device="cuda")
    mean, rstd = torch.zeros(rows, device="cuda"), torch.ones(rows, device="cuda")
    scratch = torch.full((L.pf_norm_bwd_ctas(rows, sms), 2, N), float("nan"), device="cuda")
    dx, dw, db = torch.empty_like(h), torch.empty_like(w), torch.empty_like(w)
    assert L.pf_norm_bwd(dy, h, w, mean, rstd, None, dx, dw, db, scratch, rows, N, 1, 0, _lib.PF_BF16, sms,
                         _lib.stream_of(h)) == 0
    assert scratch[:sms].isfinite().all() and scratch[sms:].isnan().all()
    want = (dy.double() * h.double()).sum(0)
    assert (dw - want).norm() <= 1e-5 * want.norm()


@pytest.mark.parametrize("silu", [True, False])
@pytest.mark.parametrize("C", [6144, 6152, 6400, 6408, 8192])
def test_group_norm_of_many_channels(C, silu):
    """Sums of more than 6144 channels take more than 48 KB of shared memory, and beyond 6400 a CTA has
    more than 800 threads."""
    test_group_norm_edges(1, 5, 5, C, 8, silu, torch.bfloat16)
