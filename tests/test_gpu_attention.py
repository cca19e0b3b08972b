"""tcgen05 flash attention (forward and backward) against an fp32 PyTorch reference."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def ref_attn(q, k, v, causal, scale):
    qf, kf, vf = (t.float().permute(0, 2, 1, 3) for t in (q, k, v))
    s = qf @ kf.transpose(-1, -2) * scale
    if causal:
        sq, sk = s.shape[-2:]
        mask = torch.ones(sq, sk, dtype=torch.bool, device=s.device).tril(sk - sq)
        s = s.masked_fill(~mask, float("-inf"))
    p = torch.softmax(s, -1)
    return (p @ vf).permute(0, 2, 1, 3), torch.logsumexp(s, -1)


CASES = [  # B, H, Sq, Sk, D, causal
    (2, 3, 197, 197, 64, False),     # ViT-L
    (1, 2, 257, 257, 88, False),     # ViT-g/14 head dim
    (1, 2, 300, 300, 128, True),     # Llama-style causal
    (2, 2, 128, 77, 64, False),      # UNet cross attention
    (1, 1, 1024, 1024, 64, False),
    (1, 2, 64, 64, 32, True),
    # a few rows past a multiple of 128: leftover queries / keys run on CUDA cores
    (2, 2, 259, 259, 64, True),
    (1, 2, 130, 257, 96, False),
    (1, 2, 260, 384, 32, False),
    (1, 2, 256, 258, 64, False),
    (1, 2, 261, 261, 64, False),     # five leftover rows: a ragged tensor-core tile instead
    (1, 2, 258, 300, 64, True),      # causal with Sq != Sk: ragged key tiles in the backward
    (1, 4, 1024, 1024, 128, True),   # several query tiles per head, many key tiles each
    (3, 5, 384, 640, 64, False),     # more work items than one wave of a small grid
    (4, 3, 17, 17, 64, False),       # far fewer rows than one tile (reduced ViT of the tests)
    (2, 4, 16, 16, 32, True),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,Sq,Sk,D,causal", CASES)
def test_attention_fwd_bwd(dtype, B, H, Sq, Sk, D, causal):
    from pfeife_b200.ops import kernels as kx
    g = torch.Generator(device="cuda").manual_seed(0)
    mk = lambda S: torch.randn(B, S, H, D, device="cuda", generator=g).to(dtype)
    q, k, v = mk(Sq), mk(Sk), mk(Sk)
    do = mk(Sq)
    scale = 1.0 / math.sqrt(D)
    o, lse = kx.attn_fwd(q, k, v, causal, scale)
    dq, dk, dv = kx.attn_bwd(do, q, k, v, o, lse, causal, scale)
    torch.cuda.synchronize()
    kx.check_status()
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    o_ref, lse_ref = ref_attn(qr, kr, vr, causal, scale)
    o_ref.backward(do.float())
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert (o.float() - o_ref).abs().max() <= tol * 2
    assert (lse - lse_ref).abs().max() <= 2e-2
    for got, want, name in ((dq, qr.grad, "dq"), (dk, kr.grad, "dk"), (dv, vr.grad, "dv")):
        err = (got.float() - want).abs().max().item()
        mag = want.abs().max().item()
        assert err <= tol * 4 * max(1.0, mag), f"{name}: err {err} (max |ref| {mag})"


@pytest.mark.parametrize("D", [64, 128])
def test_attention_forward_when_the_row_maximum_keeps_growing(D):
    """Later key tiles carry much larger scores than earlier ones, so the maximum that scales
    the probabilities has to be raised (and the accumulated output rescaled) several times
    within one row; keys of the last tile are tiny again (no rescale there)."""
    from pfeife_b200.ops import kernels as kx
    B, H, Sq, Sk = 1, 2, 256, 768
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(B, Sq, H, D, device="cuda", generator=g).to(torch.bfloat16)
    k = torch.randn(B, Sk, H, D, device="cuda", generator=g)
    ramp = torch.tensor([0.1, 1.0, 4.0, 12.0, 30.0, 0.05], device="cuda").repeat_interleave(128)
    k = (k * ramp[None, :, None, None]).to(torch.bfloat16)
    v = torch.randn(B, Sk, H, D, device="cuda", generator=g).to(torch.bfloat16)
    scale = 1.0 / math.sqrt(D)
    o, lse = kx.attn_fwd(q, k, v, False, scale)
    torch.cuda.synchronize()
    kx.check_status()
    o_ref, lse_ref = ref_attn(q, k, v, False, scale)
    assert torch.isfinite(o.float()).all()
    assert (o.float() - o_ref).abs().max() <= 4e-2
    assert ((lse - lse_ref).abs() / lse_ref.abs().clamp_min(1.0)).max() <= 1e-2


def test_attention_on_fused_qkv_views():
    """q, k, v as strided slices of one [B, S, 3, H, D] projection, through autograd."""
    from pfeife_b200 import ops
    B, S, H, D = 2, 257, 4, 88
    qkv = (torch.randn(B, S, 3, H, D, device="cuda") * 0.5).to(torch.float16).requires_grad_()
    out = ops.attention(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2])
    out.float().sum().backward()
    ref_in = qkv.detach().float().requires_grad_()
    o_ref, _ = ref_attn(ref_in[:, :, 0], ref_in[:, :, 1], ref_in[:, :, 2], False, 1 / math.sqrt(D))
    o_ref.sum().backward()
    assert (out.float() - o_ref).abs().max() <= 1e-2
    assert (qkv.grad.float() - ref_in.grad).abs().max() <= 5e-2


def test_packed_qkv_attention_writes_fused_gradient():
    from pfeife_b200 import ops
    B, S, H, D = 2, 300, 2, 64
    qkv = (torch.randn(B, S, 3, H, D, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_()
    out = ops.attention_qkv(qkv, causal=True)
    out.float().sum().backward()
    ref_in = qkv.detach().float().requires_grad_()
    o_ref, _ = ref_attn(ref_in[:, :, 0], ref_in[:, :, 1], ref_in[:, :, 2], True, 1 / math.sqrt(D))
    o_ref.sum().backward()
    assert (out.float() - o_ref).abs().max() <= 2e-2
    assert (qkv.grad.float() - ref_in.grad).abs().max() <= 1e-1


BWD_EDGES = [  # B, H, Sq, Sk, D, causal: tile edges, remainders, every head-dim class, empty key tiles
    (1, 1, 1, 1, 8, False), (2, 3, 127, 128, 24, False), (1, 2, 129, 129, 32, False),
    (2, 2, 257, 257, 88, True), (1, 2, 144, 272, 40, False), (1, 2, 385, 100, 64, False),
    (1, 2, 100, 385, 64, True), (1, 2, 385, 100, 64, True), (1, 1, 300, 128, 72, True),
    (2, 5, 513, 640, 128, True), (1, 3, 640, 513, 128, False), (40, 10, 65, 65, 96, False),
    (7, 25, 130, 258, 128, False), (3, 67, 272, 272, 64, True),
    # whole rounds of query tile pairs, then single tiles whose keys are shared out (one, some, empty)
    (5, 31, 300, 300, 64, False), (1, 150, 40, 200, 32, False), (2, 75, 256, 128, 96, False),
    (1, 1, 1024, 1024, 128, True), (1, 3, 700, 1500, 64, True),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,Sq,Sk,D,causal", BWD_EDGES)
def test_attention_fwd_bwd_at_tile_edges(dtype, B, H, Sq, Sk, D, causal):
    """Outputs and gradients against 64 bits.  P, dS and the results are rounded to 16 bits, each
    with a relative error of up to u = 2^-8 / 2^-11 and of u / 2 on average; 2 u bounds the 2-norm
    of their sum."""
    from pfeife_b200.ops import kernels as kx
    g = torch.Generator(device="cuda").manual_seed(Sq * 7 + Sk)
    mk = lambda S: torch.randn(B, S, H, D, device="cuda", generator=g).to(dtype)
    q, k, v, do = mk(Sq), mk(Sk), mk(Sk), mk(Sq)
    scale = 1.0 / math.sqrt(D)
    o, lse = kx.attn_fwd(q, k, v, causal, scale)
    grads = kx.attn_bwd(do, q, k, v, o, lse, causal, scale)
    again = kx.attn_bwd(do, q, k, v, o, lse, causal, scale)   # buffers with earlier contents
    torch.cuda.synchronize()
    kx.check_status()
    qr, kr, vr = (t.double().requires_grad_() for t in (q, k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", qr, kr) * scale
    if causal:
        seen = torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").tril(Sk - Sq)
        s = s.masked_fill(~seen, -1e30)      # rows that see no key: zeroed below
        p = torch.softmax(s, -1) * seen
    else:
        p = torch.softmax(s, -1)
    o_ref = torch.einsum("bhqk,bkhd->bqhd", p, vr)
    o_ref.backward(do.double())
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    wants = (o_ref.detach(), qr.grad, kr.grad, vr.grad)
    for name, got, want in zip(("o", "dq", "dk", "dv"), (o,) + grads, wants):
        assert torch.isfinite(got.float()).all(), name
        # the floor is what rounding dS, of the size of the probabilities' products, leaves in
        # gradients that cancel (one key: dq and dk are zero)
        floor = u * D ** 0.5 * want.numel() ** 0.5 * 0.5 if Sk == 1 else 0.0
        assert (got.double() - want).norm() <= 2 * u * want.norm() + floor, name
    for a, b in zip(grads, again):
        assert (a.float() - b.float()).norm() <= u * a.float().norm()


@pytest.mark.parametrize("Sq,Sk,H", [(250, 1500, 600), (256, 1409, 666), (129, 1408, 600)])
def test_attention_forward_with_pairs_beyond_whole_rounds(Sq, Sk, H):
    """More than four rounds of pairs of query tiles on 148 SMs: the pairs left over are split and go to
    a launch of their own from 12 key tiles on, and stay whole below (the last case).  Heads on both
    sides of the line against 64 bits; u / 2 per rounding (probabilities, result) on average."""
    from pfeife_b200.ops import kernels as kx
    g = torch.Generator(device="cuda").manual_seed(Sk)
    q, k, v = (torch.randn(1, S, H, 32, device="cuda", generator=g).to(torch.bfloat16)
               for S in (Sq, Sk, Sk))
    o, lse = kx.attn_fwd(q, k, v, False, 32 ** -0.5)
    kx.check_status()
    pick = [0, 147, 591, 592, H - 1]
    s = torch.einsum("qhd,khd->hqk", q[0, :, pick].double(), k[0, :, pick].double()) * 32 ** -0.5
    want = torch.einsum("hqk,khd->qhd", s.softmax(-1), v[0, :, pick].double())
    assert ((o[0, :, pick] - want).norm() / want.norm()).item() < 2 * 2.0 ** -8
    assert (lse[0, pick] - s.logsumexp(-1)).abs().max().item() < 1e-4


WHOLE = [  # B, H, Sq, Sk, D, causal: enough heads that the backward takes each whole, with one and with two
    # tokens beyond full tiles, ragged tiles, key tiles that not every query tile sees
    (10, 14, 257, 257, 88, False), (8, 20, 129, 129, 32, False), (16, 19, 130, 130, 64, False),
    (24, 16, 258, 258, 48, False), (4, 37, 513, 513, 40, False), (10, 14, 257, 257, 128, False),
    (7, 20, 300, 300, 64, True), (7, 20, 130, 300, 96, True), (7, 20, 300, 130, 72, False),
    (7, 20, 256, 256, 8, False), (37, 8, 385, 257, 32, False),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,Sq,Sk,D,causal", WHOLE)
def test_attention_backward_of_whole_heads(dtype, B, H, Sq, Sk, D, causal):
    """The same bounds as at the tile edges; and dQ, whose sums one thread keeps, repeats bit for bit."""
    from pfeife_b200.ops import kernels as kx
    test_attention_fwd_bwd_at_tile_edges(dtype, B, H, Sq, Sk, D, causal)
    q, do = (torch.randn(B, Sq, H, D, device="cuda").to(dtype) for _ in range(2))
    k, v = (torch.randn(B, Sk, H, D, device="cuda").to(dtype) for _ in range(2))
    o, lse = kx.attn_fwd(q, k, v, causal, D ** -0.5)
    first, second = (kx.attn_bwd(do, q, k, v, o, lse, causal, D ** -0.5) for _ in range(2))
    assert all(torch.equal(a, b) for a, b in zip(first, second))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,Sq,Sk,D,causal", [
    (40, 10, 64, 64, 128, False), (2, 5, 33, 17, 88, False), (5, 40, 128, 32, 64, False), (7, 50, 17, 65, 32, True),
    (3, 7, 1, 40, 72, False), (2, 5, 65, 64, 48, False)])
def test_attention_backward_of_few_rows(dtype, B, H, Sq, Sk, D, causal):
    """One tile of either kind whose outputs leave without boxes, up to as many rows, and one row more."""
    test_attention_backward_of_whole_heads(dtype, B, H, Sq, Sk, D, causal)


@pytest.mark.parametrize("B,H,S,D", [(23, 20, 129, 32), (30, 15, 130, 64)])
def test_attention_backward_of_leftover_tokens_of_many_heads(B, H, S, D):
    """More heads than three to an SM of 148, which take the form of fewer registers."""
    test_attention_backward_of_whole_heads(torch.bfloat16, B, H, S, S, D, False)


@pytest.mark.parametrize("D,left,causal", [(32, 1, False), (64, 3, True), (88, 4, False), (128, 1, True)])
def test_attention_forward_of_leftover_rows(D, left, causal):
    """Rows beyond full tiles against 64 bits (u / 2 on average for rounding the result; the probabilities
    stay in fp32), fewer keys than lanes among them, and a NaN key, which reaches every row that sees it."""
    from pfeife_b200.ops import kernels as kx
    for Sk in (5, 128 + left, 700):
        q, k, v = (torch.randn(2, S, 3, D, device="cuda").to(torch.bfloat16) for S in (128 + left, Sk, Sk))
        o, lse = kx.attn_fwd(q, k, v, causal, D ** -0.5)
        qr, kr, vr = (t.double() for t in (q, k, v))
        want, lse_want = (t[..., -left:, :, :] if t.dim() == 4 else t[..., -left:]
                          for t in ref_attn64(qr, kr, vr, causal, D ** -0.5))
        assert (o[:, -left:].double() - want).norm() <= 2.0 ** -8 * want.norm()
        assert (lse[..., -left:] - lse_want).abs().max() < 1e-4
        k[:, 2] = float("nan")
        o, _ = kx.attn_fwd(q, k, v, causal, D ** -0.5)
        assert torch.isnan(o[:, -left:].float()).all()
    kx.check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Sq,Sk,H,D,causal", [
    (300, 300, 304, 64, False), (384, 130, 270, 40, False), (387, 387, 304, 32, False), (640, 257, 200, 64, False),
    (1000, 350, 160, 32, False), (1300, 800, 420, 64, False), (1024, 1024, 420, 48, True), (1153, 1153, 470, 32, True)])
def test_attention_forward_of_one_issuing_thread(Sq, Sk, H, D, causal, dtype):
    """Many heads of an odd number of query tiles, the last key tile ragged, or of long rows under a causal mask:
    one thread issues the products of both sides of a pair.  Every tile of the first, a middle and the last head against 64 bits."""
    from pfeife_b200.ops import kernels as kx
    q = torch.randn(1, Sq, H, D, device="cuda").to(dtype)
    k, v = (torch.randn(1, Sk, H, D, device="cuda").to(dtype) for _ in range(2))
    o, lse = kx.attn_fwd(q, k, v, causal, D ** -0.5)
    kx.check_status()
    for h in (0, H // 2, H - 1):
        want, lse_want = ref_attn64(*(t[:, :, h:h + 1].double() for t in (q, k, v)), causal, D ** -0.5)
        for r in range(0, Sq, 128):
            got = o[:, r:r + 128, h:h + 1].double()
            assert (got - want[:, r:r + 128]).norm() <= 2 * 2.0 ** -8 * want[:, r:r + 128].norm()
        assert (lse[:, h] - lse_want[:, 0]).abs().max() < 1e-4
    assert torch.isfinite(o).all()


@pytest.mark.parametrize("S,H,D,causal", [(1024, 160, 32, False), (1025, 152, 64, False), (1537, 110, 128, False),
                                          (2050, 58, 64, False), (257, 150, 88, True), (129, 1200, 32, False)])
def test_attention_forward_of_several_launches(S, H, D, causal):
    """Launches of a call that run beside one another: inputs overwritten before it and right after it, results
    used at once, eagerly and replayed, give the bits of calls that have the device to themselves; the
    last rows (of the last launch) and one head are within u of 64 bits."""
    from pfeife_b200.ops import kernels as kx
    sets = [[torch.randn(1, S, H, D, device="cuda").to(torch.bfloat16) for _ in range(3)] for _ in range(3)]
    want = []
    for q, k, v in sets:
        torch.cuda.synchronize()
        want.append(kx.attn_fwd(q, k, v, causal, D ** -0.5))
        torch.cuda.synchronize()
    q, k, v = (t.clone() for t in sets[0])
    outs = [[torch.zeros_like(t) for t in w] for w in want]

    def all_sets():
        for i, given in enumerate(sets):
            for t, g in zip((q, k, v), given):
                t.copy_(g)
            for t, r in zip(outs[i], kx.attn_fwd(q, k, v, causal, D ** -0.5)):
                t.copy_(r)

    def check():
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert all(torch.equal(a, b) for a, b in zip(o, w))
            for t in o:
                t.zero_()

    for _ in range(3):
        all_sets()
        check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        all_sets()
    for _ in range(3):
        graph.replay()
        check()
    for h in (0, H - 1):
        o64, lse64 = ref_attn64(*(t[:, :, h:h + 1].double() for t in sets[0]), causal, D ** -0.5)
        o, lse = want[0][0][:, :, h:h + 1].double(), want[0][1][:, h:h + 1]
        for rows in (slice(None), slice(-(S % 128 or 128), None)):
            assert (o[:, rows] - o64[:, rows]).norm() <= 2.0 ** -8 * o64[:, rows].norm()
        assert (lse - lse64).abs().max() < 1e-4
    kx.check_status()


def ref_attn64(q, k, v, causal, scale):
    s = torch.einsum("bqhd,bkhd->bhqk", q, k) * scale
    if causal:
        s = s.masked_fill(~torch.ones(s.shape[-2:], dtype=torch.bool, device="cuda").tril(
            k.shape[1] - q.shape[1]), float("-inf"))
    return torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1), v), s.logsumexp(-1)


@pytest.mark.parametrize("tokens,heads,dim", [(129, 50, 64), (129, 50, 128), (130, 50, 32), (257, 70, 88), (385, 70, 64),
                                               (129, 3, 64), (257, 3, 88)])
def test_infinities_in_the_last_token(tokens, heads, dim):
    """Leftover rows on CUDA cores: a token whose lane has none beside it is read there too, and must not count.
    An infinity in its value reaches its own column of every row, and nothing else.  The first sizes take the
    tokens out of the tiles in the backward as well, the last do not."""
    from pfeife_b200 import ops

    torch.manual_seed(tokens + dim)
    q, k, v, do = (torch.randn(2, tokens, heads, dim, device="cuda").bfloat16() for _ in range(4))
    inf_v, inf_do = v.clone(), do.clone()
    inf_v[:, -1, :, 5] = float("inf")
    inf_do[:, -1, :, 5] = float("-inf")

    def run(v, do):
        leaves = [t.detach().requires_grad_() for t in (q, k, v)]
        o = ops.attention(*leaves)
        return o.detach(), torch.autograd.grad(o, leaves, do)[2]

    (o, dv), (inf_o, _), (_, inf_dv) = run(v, do), run(inf_v, do), run(v, inf_do)
    other = [c for c in range(dim) if c != 5]
    for got, finite, inf in ((inf_o, o, float("inf")), (inf_dv, dv, float("-inf"))):
        assert (got[..., 5] == inf).all()
        assert torch.equal(got[..., other], finite[..., other])
