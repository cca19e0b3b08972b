"""UNet kernels (implicit-GEMM and im2col convolution, GroupNorm+SiLU, upsample) and the Llama / UNet model
families on the GPU against fp32 CPU references."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _close(a, b, tol):
    err = (a.float().cpu() - b.float().cpu()).abs().max().item()
    mag = b.float().abs().max().item()
    assert err <= tol * max(1.0, mag), f"err {err} vs magnitude {mag}"


@pytest.mark.parametrize("cin,cout,k,stride", [(16, 32, 3, 1), (32, 32, 3, 2), (24, 40, 1, 1),
                                               (4, 32, 3, 1), (32, 4, 3, 1)])
def test_conv2d_nhwc(cin, cout, k, stride):
    from pfeife_b200 import ops
    torch.manual_seed(0)
    x = torch.randn(2, 16, 16, cin)
    w = torch.randn(cout, cin, k, k) * 0.1
    b = torch.randn(cout)
    xr, wr, br = (t.clone().requires_grad_() for t in (x, w, b))
    yr = F.conv2d(xr.permute(0, 3, 1, 2), wr, br, stride=stride, padding=k // 2).permute(0, 2, 3, 1)
    yr.sum().backward()
    xg = x.cuda().to(torch.bfloat16).requires_grad_()
    wg = w.cuda().to(torch.bfloat16).requires_grad_()
    bg = b.cuda().requires_grad_()
    y = ops.conv2d(xg, wg, bg, stride, k // 2)
    y.float().sum().backward()
    _close(y, yr.detach(), 3e-2)
    _close(xg.grad, xr.grad, 3e-2)
    _close(wg.grad, wr.grad, 3e-2)
    _close(bg.grad, br.grad, 3e-2)


@pytest.mark.parametrize("cin,cout,hw,k,stride", [
    (64, 128, 16, 3, 1),      # implicit GEMM forward and dgrad, tiles of 8 output rows
    (128, 64, 32, 3, 1),      # tiles of 4 output rows; 2048 output pixels
    (64, 64, 32, 3, 2),       # stride 2: implicit forward (16 x 16 outputs), col2im dgrad
    (128, 192, 64, 3, 1),     # two output rows per tile, several k-blocks per tap
    (64, 72, 16, 3, 1),       # Cout not a multiple of 64: implicit forward, GEMM + col2im dgrad
])
def test_conv2d_implicit_gemm(cin, cout, hw, k, stride):
    """Shapes the implicit-GEMM path covers (C % 64 == 0, whole output rows per 128-pixel tile):
    values and all gradients against an fp32 reference, with a random upstream gradient so that
    a misplaced filter tap cannot cancel out."""
    from pfeife_b200 import ops
    from pfeife_b200.ops import kernels as kx
    torch.manual_seed(1)
    x = torch.randn(2, hw, hw, cin)
    w = torch.randn(cout, cin, k, k) * 0.05
    b = torch.randn(cout)
    assert kx.conv_gemm_supported(x, k, k, stride, k // 2)
    xr, wr, br = (t.clone().requires_grad_() for t in (x, w, b))
    yr = F.conv2d(xr.permute(0, 3, 1, 2), wr, br, stride=stride, padding=k // 2).permute(0, 2, 3, 1)
    gy = torch.randn(yr.shape)
    yr.backward(gy)
    xg = x.cuda().to(torch.bfloat16).requires_grad_()
    wg = w.cuda().to(torch.bfloat16).requires_grad_()
    bg = b.cuda().requires_grad_()
    y = ops.conv2d(xg, wg, bg, stride, k // 2)
    y.backward(gy.cuda().to(y.dtype))
    torch.cuda.synchronize()
    kx.check_status()
    _close(y, yr.detach(), 3e-2)
    _close(xg.grad, xr.grad, 3e-2)
    _close(wg.grad, wr.grad, 3e-2)
    _close(bg.grad, br.grad, 3e-2)


@pytest.mark.parametrize("silu", [False, True])
def test_group_norm_silu(silu):
    from pfeife_b200 import ops
    torch.manual_seed(0)
    x = torch.randn(2, 16, 16, 64)
    g, b = torch.randn(64) * 0.5 + 1, torch.randn(64) * 0.1
    xr, gr, br = (t.clone().requires_grad_() for t in (x, g, b))
    yr = F.group_norm(xr.permute(0, 3, 1, 2), 8, gr, br, 1e-5)
    yr = (F.silu(yr) if silu else yr).permute(0, 2, 3, 1)
    dy = torch.randn(2, 16, 16, 64)
    yr.backward(dy)
    xg = x.cuda().to(torch.bfloat16).requires_grad_()
    gg, bg = g.cuda().requires_grad_(), b.cuda().requires_grad_()
    y = ops.group_norm(xg, gg, bg, 8, 1e-5, silu)
    y.backward(dy.cuda().to(torch.bfloat16))
    _close(y, yr.detach(), 3e-2)
    _close(xg.grad, xr.grad, 5e-2)
    _close(gg.grad, gr.grad, 5e-2)
    _close(bg.grad, br.grad, 5e-2)


def test_upsample():
    from pfeife_b200 import ops
    x = torch.randn(2, 8, 8, 32, device="cuda").to(torch.bfloat16).requires_grad_()
    y = ops.upsample_nearest2x(x)
    y.float().pow(2).sum().backward()
    xr = x.detach().float().requires_grad_()
    yr = xr.repeat_interleave(2, 1).repeat_interleave(2, 2)
    yr.pow(2).sum().backward()
    _close(y, yr.detach(), 1e-2)
    _close(x.grad, xr.grad, 3e-2)


def _model_grads(model, loss_of, device, dtype):
    import copy
    m = copy.deepcopy(model).to(device)
    if dtype is not None:
        with torch.autocast("cuda", dtype=dtype):
            loss = loss_of(m)
    else:
        loss = loss_of(m)
    loss.backward()
    return float(loss.detach()), {n: p.grad.detach().float().cpu() for n, p in m.named_parameters()}


def test_llama_model_gpu_matches_cpu():
    from pfeife_b200.models.llama import Llama, causal_lm_loss, llama_config
    torch.manual_seed(0)
    model = Llama(llama_config("llama_tiny", hidden_size=128, num_heads=4, intermediate_size=256))
    ids = torch.randint(0, 256, (2, 32))
    lc, gc = _model_grads(model, lambda m: causal_lm_loss(m(ids).float(), ids), "cpu", None)
    lg, gg = _model_grads(model, lambda m: causal_lm_loss(m(ids.cuda()), ids.cuda()), "cuda",
                          torch.bfloat16)
    assert lg == pytest.approx(lc, rel=2e-2)
    for n in gc:
        _close(gg[n], gc[n], 8e-2)


def test_unet_model_gpu_matches_cpu():
    from pfeife_b200 import ops
    from pfeife_b200.models.unet import UNet, unet_config
    torch.manual_seed(0)
    model = UNet(unet_config("unet_tiny"))
    B = 2
    args = (torch.randn(B, 4, 16, 16), torch.randint(0, 1000, (B,)), torch.randn(B, 7, 32),
            torch.randn(B, 16), torch.randn(B, 6))
    noise = torch.randn(B, 4, 16, 16)
    lc, gc = _model_grads(model, lambda m: F.mse_loss(m(*args).float(), noise), "cpu", None)
    cargs = tuple(a.cuda() for a in args)
    lg, gg = _model_grads(
        model, lambda m: F.mse_loss(m(cargs[0].to(torch.bfloat16), *cargs[1:]).float(),
                                    noise.cuda()), "cuda", torch.bfloat16)
    assert lg == pytest.approx(lc, rel=3e-2)
    worst = max((gg[n] - gc[n]).abs().max().item() / max(1e-3, gc[n].abs().max().item())
                for n in gc)
    assert worst < 0.25


@pytest.mark.parametrize("w_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,H,Cin,Cout,K,stride", [
    (1, 8, 64, 64, 3, 1), (2, 16, 64, 72, 3, 2), (1, 16, 4, 320, 3, 1), (1, 16, 96, 4, 3, 1),
    (1, 9, 13, 21, 3, 1), (1, 16, 128, 65, 1, 1), (1, 12, 8, 8, 5, 1), (1, 11, 3, 9, 9, 1)])
def test_conv_weight_orders(B, H, Cin, Cout, K, stride, w_dtype):
    """Output and gradients with the packed weights (padding, flipped taps, gradient order) against
    64 bits; every product sums 16-bit values in fp32 and rounds once (twice through col2im)."""
    from pfeife_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(Cin * 31 + Cout)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x = rnd(B, H, H, Cin).to(torch.bfloat16).requires_grad_()
    # fp32 weights that bf16 holds exactly: the cast in front of the product changes nothing
    w = (0.1 * rnd(Cout, Cin, K, K)).to(torch.bfloat16).to(w_dtype).requires_grad_()
    b = rnd(Cout).requires_grad_()
    y = ops.conv2d(x, w, b, stride, K // 2)
    dy = rnd(*y.shape).to(torch.bfloat16)
    grads = torch.autograd.grad(y, (x, w, b), dy)
    xr, wr, br = (t.detach().double().requires_grad_() for t in (x, w, b))
    yr = torch.nn.functional.conv2d(xr.permute(0, 3, 1, 2).cpu(), wr.cpu(), br.cpu(),
                                    stride=stride, padding=K // 2).permute(0, 2, 3, 1)
    wants = torch.autograd.grad(yr, (xr, wr, br), dy.double().cpu())
    u = 2.0 ** -8
    for got, want in ((y, yr), (grads[0], wants[0]), (grads[1], wants[1]), (grads[2], wants[2])):
        want = want.to(got.device)
        assert (got.double() - want).norm() <= 1.5 * u * want.norm()
    assert grads[1].dtype == w_dtype


@pytest.mark.parametrize("w_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [1, 3])
@pytest.mark.parametrize("layout", ["transposed", "sliced", "channels_last", "expanded"])
def test_conv_weight_views(layout, K, w_dtype):
    """Weights that are views of something else: the same values as a contiguous copy gives."""
    from pfeife_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(K)
    rnd = lambda *s: (0.1 * torch.randn(*s, device="cuda", generator=g)).to(w_dtype)
    Cout, Cin = 64, 72
    w = {"transposed": lambda: rnd(Cin, Cout, K, K).transpose(0, 1),
         "sliced": lambda: rnd(Cout, Cin + 3, K, K)[:, 3:],
         "channels_last": lambda: rnd(Cout, Cin, K, K).to(memory_format=torch.channels_last),
         "expanded": lambda: rnd(Cout, 1, K, K).expand(Cout, Cin, K, K)}[layout]()
    x = torch.randn(2, 8, 8, Cin, device="cuda", generator=g).to(torch.bfloat16)
    out = []
    for weight in (w, w.clone(memory_format=torch.contiguous_format)):
        leaves = x.clone().requires_grad_(), weight.detach().requires_grad_()
        y = ops.conv2d(*leaves, None, 1, K // 2)
        out.append((y,) + torch.autograd.grad(y, leaves, torch.ones_like(y)))
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("Cout,Cin,taps", [
    (8, 8, 1), (1, 1, 1), (21, 13, 1), (9, 4104, 1), (64, 64, 4), (64, 520, 9), (17, 455, 9),
    (72, 9, 25), (16, 96, 49), (5, 3, 49), (33, 120, 63), (24, 65, 64), (7, 16, 65)])
def test_conv_weight_kernels_move_every_element(Cout, Cin, taps):
    """Packed, flipped and gradient orders at the edges of the tiles (64 taps, whole and ragged
    vectors, several shares of the channels), bit for bit."""
    from pfeife_b200.ops import kernels as kx
    cout8, cin8 = (Cout + 7) // 8 * 8, (Cin + 7) // 8 * 8
    w = torch.randn(Cout, Cin, taps, 1, device="cuda").to(torch.bfloat16)
    full = w.new_zeros(cout8, cin8, taps)
    full[:Cout, :Cin] = w[..., 0]
    shifted = torch.empty(w.numel() + 1, dtype=w.dtype, device="cuda")[1:].view(w.shape).copy_(w)
    for src in (w, shifted):                      # 16-byte aligned or not
        assert torch.equal(kx.conv_pack(src, cout8, cin8),
                           full.permute(0, 2, 1).reshape(cout8, -1))
        assert torch.equal(kx.conv_pack(src, cout8, cin8, flip=True),
                           full.flip(2).permute(1, 2, 0).reshape(cin8, -1))
    sums = torch.randn(cout8, taps * cin8, device="cuda")
    want = sums.view(cout8, taps, cin8)[:Cout, :, :Cin].permute(0, 2, 1).reshape(w.shape)
    for dtype in (torch.float32, torch.bfloat16, torch.float16):
        got = kx.conv_unpack(sums, w.shape, cin8, dtype)
        assert got.is_contiguous() and torch.equal(got, want.to(dtype))


@pytest.mark.parametrize("batch,hw,cin,cout,stride", [
    (1, 8, 64, 64, 1),        # one k-block per image row group, one tile, nothing to split
    (3, 8, 128, 72, 1),       # k-blocks of eight output rows, image after image
    (2, 32, 64, 320, 1),      # the reduction in several parts
    (2, 128, 64, 64, 1),      # a k-block is half an output row
    (2, 32, 64, 128, 2),      # stride 2: 16 x 16 outputs
])
def test_conv_wgrad_steps_through_pixels(batch, hw, cin, cout, stride):
    """Weight gradients over every way a k-block of 64 output pixels can lie in an image, also into a
    buffer that holds something else before.  Products are exact in
    fp32, so only the order of the sums differs: 2^-24 of the root of the number of terms."""
    from pfeife_b200.ops import kernels as kx
    torch.manual_seed(3)
    x = torch.randn(batch, hw, hw, cin, device="cuda").to(torch.bfloat16)
    ho = (hw - 1) // stride + 1
    dy = torch.randn(batch, ho, ho, cout, device="cuda").to(torch.bfloat16)
    assert kx.conv_wgrad_supported(x, cout, 3, 3, stride, 1)
    out = torch.full((cout, 9 * cin), 7.0, device="cuda")
    kx.conv_wgrad(dy.view(-1, cout), x, 3, 3, stride, 1, out=out)
    more = kx.conv_wgrad(dy.view(-1, cout), x, 3, 3, stride, 1, out=out.clone(), accumulate=True)
    ref = torch.nn.grad.conv2d_weight(x.double().permute(0, 3, 1, 2), (cout, cin, 3, 3),
                                      dy.double().permute(0, 3, 1, 2), stride=stride, padding=1)
    ref = ref.permute(0, 2, 3, 1).reshape(cout, 9 * cin)
    kx.check_status()
    assert ((out - ref).norm() / ref.norm()).item() < 1e-5
    assert ((more - 2 * ref).norm() / ref.norm()).item() < 2e-5


@pytest.mark.parametrize("cout,hw", [(4, 16), (8, 32), (56, 16), (3, 128), (60, 16), (64, 16)])
def test_conv_input_gradient_of_few_filters(cout, hw, monkeypatch):
    """Up to 64 filters: the gradient is padded to the width the implicit GEMM reads.  fp32 sums and one
    rounding: the error is that of the exact result rounded to 16 bits, give or take the roundings that
    fp32 sums of up to 576 terms turn (columns of 16 bits would add as much again)."""
    from pfeife_b200 import ops
    from pfeife_b200.ops import kernels as kx
    torch.manual_seed(6)
    x = torch.randn(2, hw, hw, 64, device="cuda").to(torch.bfloat16).requires_grad_()
    w = (torch.randn(cout, 64, 3, 3, device="cuda") * 0.1).to(torch.bfloat16)
    gy = torch.randn(2, hw, hw, cout, device="cuda").to(torch.bfloat16)
    y = ops.conv2d(x, w, None, 1, 1)
    calls, conv_gemm = [], kx.conv_gemm
    monkeypatch.setattr(kx, "conv_gemm", lambda *a, **k: calls.append(1) or conv_gemm(*a, **k))
    dx, = torch.autograd.grad(y, x, gy)
    assert calls
    ref = torch.nn.grad.conv2d_input((2, 64, hw, hw), w.double(), gy.double().permute(0, 3, 1, 2),
                                     padding=1).permute(0, 2, 3, 1)
    assert (dx - ref).norm() < 1.1 * (ref.to(torch.bfloat16) - ref).norm()


@pytest.mark.parametrize("KH,KW,pad,H,W,cout", [
    (1, 3, 0, 32, 36, 8), (3, 1, 1, 28, 28, 4), (1, 3, 0, 32, 36, 64), (3, 5, 1, 32, 34, 128),
    (1, 1, 1, 16, 32, 8), (5, 5, 1, 18, 34, 8), (3, 3, 1, 16, 32, 4)])
def test_conv_gradients_of_any_kernel_shape(KH, KW, pad, H, W, cout):
    """The implicit route of the input gradient has one padding for both axes: kernels that are not square
    go through the column buffer.  One rounding, of the columns too on that route: sqrt(2) 2^-9 at most
    on average."""
    from pfeife_b200 import ops
    torch.manual_seed(7)
    x = torch.randn(1, H, W, 64, device="cuda").to(torch.bfloat16).requires_grad_()
    w = (torch.randn(cout, 64, KH, KW, device="cuda") * 0.1).to(torch.bfloat16).requires_grad_()
    y = ops.conv2d(x, w, None, 1, pad)
    xd, wd = x.detach().double().permute(0, 3, 1, 2), w.detach().double()
    gy = torch.randn(y.shape, device="cuda").to(torch.bfloat16)
    gd = gy.double().permute(0, 3, 1, 2)
    dx, dw = torch.autograd.grad(y, (x, w), gy)
    ref = torch.nn.functional.conv2d(xd, wd, padding=pad).permute(0, 2, 3, 1)
    refx = torch.nn.grad.conv2d_input(xd.shape, wd, gd, padding=pad).permute(0, 2, 3, 1)
    refw = torch.nn.grad.conv2d_weight(xd, wd.shape, gd, padding=pad)
    for got, want in ((y, ref), (dx, refx), (dw, refw)):
        assert got.shape == want.shape
        assert ((got - want).norm() / want.norm()).item() < 1.5 * 2.0 ** -9


@pytest.mark.parametrize("batch,hw,cin,cout,stride", [(2, 32, 64, 320, 1), (2, 128, 320, 8, 1),
                                                      (4, 64, 320, 320, 2)])
def test_conv_weight_gradients_repeat(batch, hw, cin, cout, stride):
    """The same bits every time, written and accumulated, where the reduction is divided."""
    from pfeife_b200.ops import _lib, kernels as kx
    torch.manual_seed(4)
    x = torch.randn(batch, hw, hw, cin, device="cuda").to(torch.bfloat16)
    ho = (hw - 1) // stride + 1
    dy = torch.randn(batch * ho * ho, cout, device="cuda").to(torch.bfloat16)
    assert _lib.calls().pf_gemm_workspace(cout, 9 * cin, batch * ho * ho, 0, 2, 148, 0) > 0
    start = torch.randn(cout, 9 * cin, device="cuda")
    first = None
    for _ in range(20):
        got = (kx.conv_wgrad(dy, x, 3, 3, stride, 1),
               kx.conv_wgrad(dy, x, 3, 3, stride, 1, out=start.clone(), accumulate=True))
        first = first or got
        assert all(torch.equal(a, b) for a, b in zip(got, first))
    assert torch.equal(first[1], start + first[0])
    kx.check_status()
