"""tcgen05 GEMM against an fp32 PyTorch reference: every operand-major combination, ragged
tile edges, every epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, a_mn, b_mn):
    A = a.float().t() if a_mn else a.float()
    B = b.float().t() if b_mn else b.float()
    return A @ B.t()


def _mk(M, N, K, a_mn, b_mn, dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn((K, M) if a_mn else (M, K), device="cuda", generator=g).to(dtype)
    b = torch.randn((K, N) if b_mn else (N, K), device="cuda", generator=g).to(dtype)
    return a, b


def _close(out, ref, K, dtype):
    tol = (2e-2 if dtype == torch.bfloat16 else 4e-3) * (K ** 0.5)
    err = (out.float() - ref).abs().max().item()
    assert err <= tol, f"max abs err {err} > {tol}"
    # relative bound: all that separates the two is the rounding of the output to 16 bits (and
    # of 16-bit intermediates some epilogues save), far below one percent of the result's norm
    rel = ((out.float() - ref).norm() / ref.norm().clamp_min(1e-20)).item()
    rtol = 1e-2 if dtype == torch.bfloat16 else 2e-3
    assert rel <= rtol, f"relative error {rel} > {rtol}"


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (300, 200, 136),
                                   (6168, 1408, 1408), (1000, 128, 72)])
@pytest.mark.parametrize("form", [4096, 2048])   # single-CTA tiles / CTA-pair tiles
def test_gemm_layouts(a_mn, b_mn, dtype, M, N, K, form):
    from pfeife_b200.ops import kernels as kx
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operands need a 16-byte aligned pitch")
    a, b = _mk(M, N, K, a_mn, b_mn, dtype)
    out = kx.gemm(a, b, a_mn=a_mn, b_mn=b_mn, tile_n=form)
    torch.cuda.synchronize()
    kx.check_status()
    _close(out, _ref(a, b, a_mn, b_mn), K, dtype)


# bit 10: direct-store epilogue, bit 11: CTA-pair form, bit 12: single-CTA form
@pytest.mark.parametrize("tile_n", [4096 + 128, 4096 + 256, 4096 + 1024 + 256, 2048, 2048 + 1024, 0])
def test_gemm_tile_variants_and_fp32_out(tile_n):
    from pfeife_b200.ops import kernels as kx
    a, b = _mk(520, 776, 320, False, False, torch.bfloat16)
    out = kx.gemm(a, b, out_dtype=torch.float32, tile_n=tile_n)
    torch.cuda.synchronize()
    _close(out, _ref(a, b, False, False), 320, torch.float32)


@pytest.mark.parametrize("tile_n", [4096, 4096 + 1024, 2048, 2048 + 1024])
@pytest.mark.parametrize("M,N,K", [(400, 384, 192), (6168, 1408, 320)])
def test_gemm_epilogues(tile_n, M, N, K):
    """Every fused epilogue through the TMA-store path and the direct-store path (bit 10), on
    single-CTA tiles (bit 12) and on CTA-pair tiles (bit 11)."""
    from pfeife_b200.ops import kernels as kx
    dtype = torch.bfloat16
    a, b = _mk(M, N, K, False, False, dtype)
    a = a * 0.1
    bias = torch.randn(N, device="cuda")
    res = torch.randn(M, N, device="cuda").to(dtype)
    ref = _ref(a, b, False, False) + bias
    # bias + residual
    out = kx.gemm(a, b, bias=bias, residual=res, tile_n=tile_n)
    _close(out, ref + res.float(), K, dtype)
    # bias + GELU with saved pre-activation
    aux = torch.empty(M, N, device="cuda", dtype=dtype)
    out = kx.gemm(a, b, bias=bias, aux=aux, epilogue=kx.EPI_GELU, tile_n=tile_n)
    _close(aux, ref, K, dtype)
    _close(out, torch.nn.functional.gelu(ref), K, dtype)
    # dGELU: out = acc * gelu'(aux)
    z = torch.randn(M, N, device="cuda").to(dtype)
    out = kx.gemm(a, b, aux=z, epilogue=kx.EPI_DGELU, tile_n=tile_n)
    zf = z.float().requires_grad_()
    torch.nn.functional.gelu(zf).sum().backward()
    _close(out, _ref(a, b, False, False) * zf.grad, K, dtype)
    # fp32 accumulate (gradient bucket), both operands MN-major as in wgrad
    at, bt = a.t().contiguous(), b.t().contiguous()
    bucket = torch.ones(M, N, device="cuda")
    kx.gemm(at, bt, a_mn=True, b_mn=True, out=bucket, accumulate=True, tile_n=tile_n)
    kx.gemm(at, bt, a_mn=True, b_mn=True, out=bucket, accumulate=True, tile_n=tile_n)
    torch.cuda.synchronize()
    kx.check_status()
    _close(bucket, 1.0 + 2.0 * _ref(a, b, False, False), K, torch.float32)


@pytest.mark.parametrize("M,N,K", [(512, 512, 4096), (1408, 1408, 6168), (304, 704, 2048)])
@pytest.mark.parametrize("form", [0, 4096])
def test_gemm_accumulate_with_split_reduction(M, N, K, form):
    """Few output tiles and a long reduction: the gradient-accumulating GEMM divides each tile's
    k-blocks among several work items that all add into the fp32 output."""
    from pfeife_b200.ops import kernels as kx
    a, b = _mk(M, N, K, True, True, torch.bfloat16, seed=3)
    a, b = a * 0.1, b * 0.1
    out = torch.full((M, N), 0.5, device="cuda")
    kx.gemm(a, b, a_mn=True, b_mn=True, out=out, accumulate=True, tile_n=form)
    kx.gemm(a, b, a_mn=True, b_mn=True, out=out, accumulate=True, tile_n=form)
    torch.cuda.synchronize()
    kx.check_status()
    _close(out, 0.5 + 2.0 * _ref(a, b, True, True), K, torch.float32)


def test_gemm_strided_views():
    """Operands that are column slices of a wider tensor (fused QKV) keep their pitch."""
    from pfeife_b200.ops import kernels as kx
    big = torch.randn(512, 3 * 256, device="cuda").to(torch.bfloat16)
    w = torch.randn(128, 256, device="cuda").to(torch.bfloat16)
    q = big[:, 256:512]
    out = torch.empty(512, 2 * 128, device="cuda", dtype=torch.bfloat16)
    kx.gemm(q, w, out=out[:, 128:])
    torch.cuda.synchronize()
    _close(out[:, 128:], q.float() @ w.float().t(), 256, torch.bfloat16)


@pytest.mark.parametrize("world,rank,ends", [(2, 0, None), (2, 1, None), (4, 2, None),
                                             (3, 1, (500, 1100, 1536)), (2, 1, (1536, 1536))])
def test_gemm_allgather_one_device(world, rank, ends):
    """The all-gather GEMM with every "peer" copy on this GPU: one launch copies the rows the
    other ranks own into the local weight while it computes, and the product must match
    x @ W^T.  Each copy is current only in the rows its rank owns (the rest is poisoned)."""
    from pfeife_b200.ops import kernels as kx
    from pfeife_b200.parallel.dp_fused import _table
    M, N, K = 700, 1536, 320
    ends = ends or tuple((r + 1) * (N // world) for r in range(world))
    starts = (0,) + tuple(ends[:-1])
    torch.manual_seed(world * 10 + rank)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.1).to(torch.bfloat16)
    copies = []
    for r in range(world):
        c = torch.full_like(w, float("nan"))
        c[starts[r]:ends[r]] = w[starts[r]:ends[r]]
        copies.append(c)
    w_full = copies[rank]
    ready = torch.zeros((N + 255) // 256 + 1, dtype=torch.int32, device="cuda")
    out = kx.gemm_allgather(x, w_full, _table([c.data_ptr() for c in copies]), world, rank, ends,
                            ready)
    torch.cuda.synchronize()
    kx.check_status()
    assert torch.equal(w_full, w)
    assert int(ready[-1]) == N - (ends[rank] - starts[rank])
    _close(out, x.float() @ w.float().t(), K, torch.bfloat16)


def test_gather_rows_one_device():
    """Stand-alone row gather: rows owned by the other ranks arrive from their copies."""
    from pfeife_b200.ops import kernels as kx
    from pfeife_b200.parallel.dp_fused import _table
    N, K, world, rank = 1000, 264, 4, 2
    ends = (100, 400, 650, 1000)
    starts = (0,) + ends[:-1]
    w = torch.randn(N, K, device="cuda").to(torch.float16)
    copies = []
    for r in range(world):
        c = torch.zeros_like(w)
        c[starts[r]:ends[r]] = w[starts[r]:ends[r]]
        copies.append(c)
    kx.gather_rows(copies[rank], _table([c.data_ptr() for c in copies]), world, rank, ends)
    torch.cuda.synchronize()
    assert torch.equal(copies[rank], w)


@pytest.mark.parametrize("M,N", [(4736, 512), (4737, 512), (129, 136), (136, 4096)])
@pytest.mark.parametrize("K", [72, 1088])
def test_gemm_around_one_round_of_small_tiles(M, N, K):
    """Sizes on both sides of the line up to which 128 x 128 tiles all run at once (148 SMs)."""
    from pfeife_b200.ops import kernels as kx
    a, b = _mk(M, N, K, False, False, torch.bfloat16)
    out = kx.gemm(a, b, out_dtype=torch.float32)
    ref = a.double() @ b.double().t()
    kx.check_status()
    # products of 16-bit values are exact in fp32; K fp32 additions in some order, whose roundings add
    # up like a random walk over sums that grow like one: sqrt(K) 2^-24 at most
    assert ((out - ref).norm() / ref.norm()).item() < K ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [(320, 72, 32768, True, True), (8, 2880, 4096, True, True),
                                             (128, 128, 512, False, False), (136, 72, 4160, False, True)])
def test_gemm_fp32_output_split_into_many_parts(M, N, K, a_mn, b_mn):
    """Few tiles under a long reduction, written and not accumulated, into an output that held something
    else before."""
    from pfeife_b200.ops import kernels as kx
    a, b = _mk(M, N, K, a_mn, b_mn, torch.bfloat16)
    out = torch.full((M, N), float("nan"), device="cuda")
    kx.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out)
    ref = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    kx.check_status()
    # products of 16-bit values are exact in fp32; K fp32 additions in some order, whose roundings add
    # up like a random walk over sums that grow like one: sqrt(K) 2^-24 at most
    assert ((out - ref).norm() / ref.norm()).item() < K ** 0.5 * 2.0 ** -24


def _pieces(z):
    """fp32 values as the sum of three bf16 columns of a GEMM operand."""
    a = torch.zeros(z.numel(), 64, device="cuda", dtype=torch.bfloat16)
    rest = z.clone()
    for j in range(3):
        a[:, j] = rest.to(torch.bfloat16)
        rest = rest - a[:, j].float()
    assert not rest.any()
    b = torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    b[:, :3] = 1
    return a, b


# (x, gelu(x)) as the bits of fp32: what the formula gives when each of its steps rounds once
GELU_BITS = [
    (0xc0f24df9, 0xaa1dfac3), (0xc0c3eae2, 0xb142a258), (0xc0a381d2, 0xb55dcbf1),
    (0xc0971fcc, 0xb6b8aed8), (0xc07f9b80, 0xb9082db1), (0xc090bfc8, 0xb7671e4c),
    (0xc0012341, 0xbd343b7f), (0xbfc13a61, 0xbdcabafc), (0xc0074344, 0xbd15967a),
    (0xbf3ff460, 0xbe2e0cb2), (0xbf06f443, 0xbe216d2f), (0xbf51ac69, 0xbe2d1785),
    (0x3e8c2846, 0x3e2a6456), (0x3e5d506f, 0x3e01977e), (0x3ed7f86c, 0x3e8f477c),
    (0x3f05ac43, 0x3ebaef04), (0x3f78d47c, 0x3f4fa452), (0x3f836242, 0x3f5ebca0),
    (0x4005bd43, 0x400349ec), (0x402e9d57, 0x402e0f12), (0x402f4958, 0x402ebf02)]


def test_gelu_epilogue_keeps_its_bits():
    """A last bit of GELU turns 16-bit roundings that every later layer carries on: the logits of a
    whole model change with it.  Values at which fused or folded steps give other bits."""
    from pfeife_b200.ops import kernels as kx
    bits = torch.tensor(GELU_BITS, dtype=torch.int64).to(torch.int32).cuda()
    z = bits[:, 0].contiguous().view(torch.float32)
    a, b = _pieces(z)
    out = torch.empty(z.numel(), 64, device="cuda")
    kx.gemm(a, b, out=out)
    assert torch.equal(out, z[:, None].expand_as(out))
    kx.gemm(a, b, out=out, epilogue=kx.EPI_GELU)
    kx.check_status()
    assert torch.equal(out.view(torch.int32), bits[:, 1:].expand_as(out))


def test_dgelu_epilogue_by_value():
    """GELU' over [-8, 8], where a norm shows nothing of the tail.  Against the same formula in 64 bits
    (Abramowitz and Stegun 7.1.26): its exponent, up to 46 in fp32, gives 46 ln 2 / 2^24 = 2e-6, every
    other step some 2^-23; between -2 and 8, where terms cancel, absolutely, with 1.5e-7 of the
    formula's own."""
    from pfeife_b200.ops import kernels as kx
    z = torch.linspace(-8, 8, 8192, device="cuda")
    a, b = _pieces(z)
    aux = kx.gemm(a, b, out_dtype=torch.float32)
    one = torch.zeros_like(a)
    one[:, 0] = 1
    got = kx.gemm(one, b, out_dtype=torch.float32, aux=aux, epilogue=kx.EPI_DGELU)[:, 0].double()
    kx.check_status()
    x = aux[:, 0].double()
    s = x.abs() * 0.5 ** 0.5
    t = 1 / (1 + 0.3275911 * s)
    poly = ((((1.061405429 * t - 1.453152027) * t + 1.421413741) * t - 0.284496736) * t
            + 0.254829592) * t
    e = torch.exp(-s * s)
    y = 0.5 * poly * e
    want = torch.where(x >= 0, 1 - y, y) + x * e * 0.3989422804014327
    tail = x < -2
    assert ((got - want) / want)[tail].abs().max().item() < 1e-5
    exact = 0.5 * torch.erfc(-x * 0.5 ** 0.5) + x * torch.exp(-x * x / 2) * 0.3989422804014327
    assert (got - exact)[~tail].abs().max().item() < 4e-7


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [(320, 72, 32768, True, True), (130, 260, 4104, False, False),
                                             (8, 2880, 16384, True, True), (592, 1408, 6168, True, True)])
def test_gemm_split_outputs_repeat(M, N, K, a_mn, b_mn):
    """An fp32 output has the same bits every time, however its reduction is divided; also into rows
    longer than the output's, whose rest stays as it is."""
    from pfeife_b200.ops import _lib, kernels as kx
    assert _lib.calls().pf_gemm_workspace(M, N, K, 0, 0, 148, 0) > 0
    a, b = _mk(M, N, K, a_mn, b_mn, torch.bfloat16)
    first = kx.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
    for _ in range(20):
        assert torch.equal(kx.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32), first)
    wide = torch.full((M, N + 8), 3.0, device="cuda")
    kx.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=wide[:, :N])
    assert torch.equal(wide[:, :N], first) and (wide[:, N:] == 3).all()
    kx.check_status()
