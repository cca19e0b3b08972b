"""How Python values reach the kernel library's entry points: through the module built for this Python and
through ctypes where there is none.  The entry points called here return before they touch a device."""
import ctypes

import pytest
import torch

from pfeife_b200 import ops
from pfeife_b200.csrc import build
from pfeife_b200.ops import _lib


@pytest.fixture(params=["module", "ctypes"])
def calls(request, monkeypatch):
    if not build.KERNEL_LIB.exists():
        pytest.skip("the kernel library is not built")
    library = ctypes.CDLL(str(build.KERNEL_LIB), mode=ctypes.RTLD_GLOBAL)
    if request.param == "ctypes":
        monkeypatch.setattr(_lib, "_CALLS_LIB", build.PKG / "missing.so")
    elif not build.CALLS_LIB.exists():
        pytest.skip("the module is not built: this Python has no headers")
    out = _lib.load_calls(library)
    assert isinstance(out, _lib._CtypesCalls) == (request.param == "ctypes")
    return out


def _gemm(calls, a, b, M=8, dtype=_lib.PF_BF16, lda=64, alpha=1.0):
    return calls.pf_gemm(a, b, None, M, 8, 64, lda, 64, 8, 0, 0, dtype, dtype, None, 0, None, 0, None, 0,
                         0, 0, alpha, None, 148, 0, None, 0, None)


def test_values_arrive(calls):
    assert calls.pf_norm_bwd_ctas(1, 148) == 1
    assert calls.pf_norm_bwd_ctas(1 << 40, 148) == calls.pf_norm_bwd_ctas(1 << 20, 148) > 148
    assert calls.pf_gemm_workspace(320, 72, 65536, False, 0, 148, 0) > 0
    assert calls.pf_gemm_workspace(320, 72, 65536, 1, 0, 148, 0) == 0
    t = torch.zeros(64, 64, dtype=torch.bfloat16)
    assert _gemm(calls, t, t, M=0) == 0
    assert _gemm(calls, t, t, dtype=7) == -1
    assert _gemm(calls, t, t, lda=63) == -2
    assert _gemm(calls, t[0, 1:], t) == -2                 # 2 bytes off, as a tensor and as a number
    assert _gemm(calls, t.data_ptr(), t.data_ptr() + 2) == -2
    assert calls.pf_rope_qkv(t, t, None, None, 0, 1, 1, 16, 0, _lib.PF_BF16, None) == 0
    # strides as a tuple: rows of queries that are no multiple of 16 bytes
    z = (64, 64, 64)
    args = [t, t, t, t, t, 1, 1, 8, 8, 64, (64, 60, 64), z, z, 0, 1.0, _lib.PF_BF16, None, None]
    assert calls.pf_attn_fwd(*args) == -2


VECTORS = {             # entry points that read and write 16 bytes at a time: arguments, and which of them are operands
    "pf_norm_fwd": (lambda t: [t, t, t, t, t, t, None, None, 1, 64, 0.0, 0, 2, None], range(6)),
    "pf_norm_bwd": (lambda t: [t, t, t, None, None, t, t, None, None, t, 1, 64, 0, 0, 2, 148, None], (0, 1, 2, 5, 6, 9)),
    "pf_glu_fwd": (lambda t: [t, t, 1, 64, 0, 2, 148, None], range(2)),
    "pf_glu_bwd": (lambda t: [t, t, t, 1, 64, 0, 2, 148, None], range(3)),
    "pf_elementwise": (lambda t: [t, t, t, 64, 20, 2, 148, None], range(3)),
    "pf_groupnorm_fwd": (lambda t: [t, None, None, t, None, None, None, 1, 1, 64, 8, 0.0, 0, 2, 148, None], (0, 3)),
    "pf_groupnorm_bwd": (lambda t: [t, t, None, None, None, None, t, None, None, None, None, 1, 1, 64, 8, 0, 2, 148,
                                    None], (0, 1, 6)),
    "pf_im2col": (lambda t: [t, t, 1, 1, 1, 64, 1, 1, 1, 1, 1, 0, 64, 2, 148, None], range(2)),
    "pf_col2im": (lambda t: [t, t, 1, 1, 1, 64, 1, 1, 1, 1, 1, 0, 64, 2, 148, None], range(2)),
    "pf_upsample2x": (lambda t: [t, t, 1, 1, 1, 64, 0, 2, 148, None], range(2)),
    "pf_conv_pack": (lambda t: [None, t, 8, 8, 1, 8, 8, 0, None], (1,)),
    "pf_nonfinite": (lambda t: [t, 64, None, 148, None], (0,)),
    "pf_adamw": (lambda t: [t, t, t, t, None, 64, None, None, 0.0, 0.0, 0.0, 0.0, 0.0, 1, None, 1.0, 1, 0, 0, 148, None],
                 range(4)),
}


@pytest.mark.skipif(torch.cuda.is_available(), reason="where there is no device, what is not refused is not launched")
@pytest.mark.parametrize("name", VECTORS)
def test_operands_off_their_vectors_are_refused(calls, name):
    arguments, operands = VECTORS[name]
    aligned = torch.zeros(256)
    assert aligned.data_ptr() % 16 == 0
    for i in operands:
        for off in (2, 4, 8, 14):
            args = arguments(aligned.data_ptr())
            args[i] += off
            assert getattr(calls, name)(*args) == -2


DEALT, WHOLE, LEFTOVER = "key tiles dealt", "whole heads", "leftover tokens beside them"


@pytest.mark.skipif(torch.cuda.is_available(), reason="the plan is asked for 148 SMs, as where there is no device")
@pytest.mark.parametrize("heads,queries,keys,dim,causal,route", [
    # whole heads while they cost no round, and while their sums are small
    (144, 250, 250, 64, 0, WHOLE), (150, 250, 250, 64, 0, DEALT), (8, 250, 250, 64, 0, DEALT), (57, 257, 257, 88, 0, DEALT),
    (144, 760, 760, 64, 0, WHOLE), (144, 890, 890, 64, 0, DEALT), (144, 1020, 300, 64, 0, WHOLE),
    (144, 1020, 512, 64, 0, DEALT), (144, 380, 380, 128, 0, WHOLE), (144, 510, 510, 128, 0, DEALT),
    (144, 1020, 1020, 32, 0, WHOLE), (144, 1100, 1100, 32, 0, DEALT),
    (144, 630, 630, 128, 1, WHOLE), (144, 760, 760, 128, 1, DEALT), (294, 1020, 1020, 128, 1, WHOLE),
    (144, 300, 256, 64, 1, DEALT),
    (144, 630, 200, 128, 0, WHOLE), (144, 760, 200, 128, 0, DEALT), (144, 500, 380, 88, 0, WHOLE), (144, 630, 380, 88, 0, WHOLE),
    (144, 630, 500, 88, 0, DEALT), (144, 380, 630, 88, 0, WHOLE), (144, 380, 630, 128, 0, DEALT), (144, 250, 630, 128, 0, WHOLE),
    (132, 898, 898, 32, 1, DEALT), (144, 898, 898, 32, 1, WHOLE), (144, 642, 642, 88, 1, DEALT), (294, 898, 898, 88, 1, DEALT),
    (294, 898, 898, 64, 1, WHOLE), (294, 642, 642, 88, 1, WHOLE),
    # leftover tokens where that saves what it costs
    (160, 257, 257, 64, 0, LEFTOVER), (96, 129, 129, 64, 0, LEFTOVER), (57, 129, 129, 64, 0, DEALT), (57, 257, 257, 64, 0, LEFTOVER),
    (384, 257, 257, 88, 0, LEFTOVER), (160, 257, 257, 88, 0, DEALT), (140, 257, 257, 128, 0, LEFTOVER),
    (304, 257, 257, 128, 0, DEALT), (144, 1025, 1025, 64, 0, DEALT),
    (96, 130, 130, 64, 0, WHOLE), (304, 130, 130, 64, 0, LEFTOVER), (160, 130, 130, 64, 0, DEALT), (384, 258, 258, 64, 0, LEFTOVER),
    (294, 258, 258, 64, 0, WHOLE), (96, 130, 130, 32, 0, LEFTOVER), (57, 258, 258, 32, 0, DEALT), (304, 386, 386, 32, 0, LEFTOVER),
    (384, 259, 259, 64, 0, DEALT), (384, 258, 258, 88, 0, DEALT)])
def test_the_plan_of_the_attention_backward(calls, heads, queries, keys, dim, causal, route):
    """Which way a call goes, by the scratch that it asks for: the lines were measured from both sides."""
    tiles, columns, left = (queries + 127) // 128, (dim + 31) // 32 * 32, queries % 128
    full = queries // 128
    sizes = {DEALT: heads * queries * dim, WHOLE: min(heads, 148) * tiles * 128 * columns,
              LEFTOVER: min(heads, 148) * full * 128 * columns + heads * left * 3 * full * 128}
    assert len(set(sizes.values())) == 3
    assert calls.pf_attn_bwd_scratch(1, heads, queries, keys, dim, causal) == (sizes[route] + 255) // 256


def test_what_does_not_fit_is_refused(calls):
    t = torch.zeros(64, 64, dtype=torch.bfloat16)
    with pytest.raises(TypeError):
        calls.pf_norm_bwd_ctas(1)
    with pytest.raises(TypeError):
        calls.pf_norm_bwd_ctas(1.5, 148)
    with pytest.raises((TypeError, AttributeError)):
        _gemm(calls, "tensor", t)
    with pytest.raises(TypeError):
        _gemm(calls, t, t, alpha="1")
    if not isinstance(calls, _lib._CtypesCalls):           # ctypes wraps numbers and takes any tuple
        with pytest.raises(OverflowError):
            calls.pf_norm_bwd_ctas(1, 1 << 31)
        with pytest.raises(OverflowError):
            calls.pf_norm_bwd_ctas(1 << 63, 148)
        with pytest.raises(ValueError):
            calls.pf_attn_fwd(t, t, t, t, t, 1, 1, 8, 8, 64, (1,) * 9, None, None, 0, 1.0, 2, None, None)


def test_a_tensor_on_the_cpu_is_refused():
    with pytest.raises(_lib.KernelError):
        _lib.stream_of(torch.zeros(1))


def test_the_module_is_optional(monkeypatch, tmp_path, capsys):
    """Without Python's headers everything else is built, and no module of another state stays."""
    left = tmp_path / "calls.so"
    left.write_bytes(b"")
    monkeypatch.setattr(build, "CALLS_LIB", left)
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    monkeypatch.setattr(build, "_stale", lambda *a: False)
    build.build()
    assert not left.exists() and "ctypes" in capsys.readouterr().out


@pytest.mark.parametrize("library", ["missing", "of_a_parent"])
def test_calls_on_the_cpu_load_nothing(library, monkeypatch, tmp_path):
    """Beside CUDA, whether the library is not built or the process was forked from one that holds CUDA."""
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    for name, value in (("_lib", None), ("_tried", False), ("_calls", None), ("_eager", None), ("_eager_tried", False)):
        monkeypatch.setattr(_lib, name, value)
    if library == "missing":
        monkeypatch.setattr(_lib, "_KERNEL_LIB", tmp_path / "missing.so")
    else:
        monkeypatch.setattr(_lib, "_KERNEL_LIB", tmp_path)

        def init():
            raise RuntimeError("Cannot re-initialize CUDA in forked subprocess")
        monkeypatch.setattr(torch.cuda, "init", init)
    x, w, g = torch.randn(2, 16, 32, requires_grad=True), torch.randn(32, 32), torch.ones(32)
    qkv, cos_sin = torch.randn(2, 8, 3, 2, 16), ops.rope_tables(8, 16)
    image = torch.randn(1, 4, 4, 32)
    for y in (ops.linear(x, w), ops.mlp(x, w, None, w, None), ops.layer_norm(x, g, g), ops.rms_norm(x, g),
              ops.swiglu(x), ops.geglu(x), ops.cross_entropy(x[0], torch.zeros(16, dtype=torch.int64)),
              ops.rope_qkv(qkv, *cos_sin), ops.attention_qkv(qkv), ops.attention(*qkv.unbind(2)),
              ops.group_norm(image, g, g, 4), ops.conv2d(image, torch.randn(8, 32, 3, 3), padding=1)):
        assert torch.isfinite(y).all()
        if y.requires_grad:
            y.sum().backward()
    assert not _lib._tried and not _lib._eager_tried


def test_eager_calls_without_their_sources(monkeypatch, tmp_path):
    (tmp_path / "eager.so").write_bytes(b"")
    monkeypatch.setattr(build, "eager_lib", lambda: tmp_path / "eager.so")
    monkeypatch.setattr(build, "EAGER_SRC", tmp_path / "eager.cpp")
    monkeypatch.setattr(_lib, "lib", lambda: object())
    monkeypatch.setattr(_lib, "_eager", None)
    monkeypatch.setattr(_lib, "_eager_tried", False)
    assert _lib.eager() is None and _lib.eager() is None
