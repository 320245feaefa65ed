"""The native half of the ops (csrc/host.cpp): it takes the ordinary call and declines everything else to the Python
function, so a call has the same outcome whichever of the two decides."""

from __future__ import annotations

import pytest
import torch

from cross_dsl_kernels_b200 import _native, ops, w4a16

NAMES = ("rmsnorm", "linear", "w4a16", "append", "attention", "swiglu")


class _Declines:
    """Stands in for the native module: every call goes on to the Python path."""

    def __getattr__(self, name):
        return lambda *args: None


def _both(monkeypatch, call):
    """The call's outcome (value, or exception type and text) on the native path and on the Python path."""
    out = []
    for native in (True, False):
        with monkeypatch.context() as m:
            if not native:
                m.setattr(_native, "host", lambda: _Declines())
            try:
                out.append(call())
            except Exception as e:
                out.append((type(e), str(e)))
    return out


def test_it_declines_what_is_not_on_a_gpu_and_odd_argument_lists():
    host = _native.host()
    x = torch.zeros(2, 8)
    assert host.rmsnorm(x, x, x[0], 1e-6, True, False) is None
    assert host.linear(x, x, None, "NK", 0, False) is None
    assert host.swiglu(x, False) is None
    for name in NAMES:
        assert getattr(host, name)() is None
        assert getattr(host, name)(*[None] * 20) is None


def test_it_is_built_for_one_torch_and_one_python_and_may_be_missing(monkeypatch):
    """Its name carries what it was compiled against; where it was not built, every call goes to the Python functions."""
    from cross_dsl_kernels_b200 import build
    ours = _native.host_path()
    assert ours.exists() and build.host_target() == ours and not build.needs_build()
    monkeypatch.setattr(torch, "__version__", "99.0+other")
    assert _native.host_path() != ours and build.needs_build()
    _native.host.cache_clear()
    try:
        with pytest.warns(RuntimeWarning, match="not built"):
            host = _native.host()
        assert all(getattr(host, name)(1, 2) is None for name in NAMES)
        with pytest.raises(ValueError, match="CUDA"):
            ops.swiglu(torch.zeros(2, 8))
    finally:
        _native.host.cache_clear()
    assert f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}" in build._host_command(ours)


def test_the_library_builds_without_a_torch_that_has_cuda(monkeypatch):
    import torch.utils.cpp_extension
    from cross_dsl_kernels_b200 import build
    monkeypatch.setattr(torch.utils.cpp_extension, "library_paths", lambda *a, **k: [])
    assert build.host_target() is None and not build.needs_build()


@pytest.mark.gpu
def test_ordinary_calls_give_the_same_bits(monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(0)

    def normal(*shape, dtype=torch.float32):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)

    x, r, w = normal(3, 520, dtype=torch.bfloat16), normal(3, 520, dtype=torch.bfloat16), normal(520, dtype=torch.bfloat16)
    xf, wk = normal(3, 256), normal(256, 72)
    xh = normal(2, 256, dtype=torch.float16)
    packed = torch.randint(0, 256, (48, 128), generator=g, device="cuda", dtype=torch.uint8)
    scales, out = (0.01 + 0.01 * torch.rand(48, 2, generator=g, device="cuda")).half(), torch.empty(2, 48, device="cuda", dtype=torch.float16)
    qkv = normal(3, 8 * 64, dtype=torch.float16).view(3, 8, 64)  # q, k and v are column slices of one matrix
    table, pos, seq = torch.tensor([[1, 0], [3, 2], [4, 5]], device="cuda"), torch.tensor([0, 17, 31], device="cuda"), torch.arange(3, device="cuda")
    cos, sin = normal(32, 32), normal(32, 32)
    kc, vc = torch.zeros(6, 16, 2, 64, device="cuda", dtype=torch.float16), torch.zeros(6, 16, 2, 64, device="cuda", dtype=torch.float16)

    def append():
        got = ops.rope_gqa_paged_kv_append(qkv[:, :4], qkv[:, 4:6], qkv[:, 6:], cos, sin, pos, table, seq, kc, vc, page_size=16,
                                           rope_dim=64, interleaved=False)
        return got, kc.clone(), vc.clone()

    calls = [lambda: ops.fused_residual_rmsnorm(x, r, w, 1e-5), lambda: ops.fused_residual_rmsnorm(x, r, w, 1e-5, return_residual=False)[:1],
             lambda: (ops.decode_linear(xf, wk, None),), lambda: (ops.decode_linear(xf, wk, wk[0].clone(), split_k=2),),
             lambda: (w4a16.w4a16_linear(xh, packed, scales),), lambda: (w4a16.w4a16_linear(xh, packed, scales, out=out).clone(),), append,
             lambda: (ops.paged_decode_attention(qkv[:, :4].contiguous(), kc, vc, pos, table, seq, page_size=16),),
             lambda: (ops.swiglu(x),), lambda: (ops.swiglu(x[:, 8:72]),)]
    for call in calls:
        native, python = _both(monkeypatch, call)
        assert len(native) == len(python) and all(torch.equal(a, b) for a, b in zip(native, python))
    assert w4a16.w4a16_linear(xh, packed, scales, out=out) is out
    assert ops.fused_residual_rmsnorm(x, r, w, 1e-5, return_residual=False)[1] is None
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):  # the current stream is what it launches on
        y = ops.decode_linear(xf, wk)
    side.synchronize()
    assert torch.equal(y, ops.decode_linear(xf, wk))


@pytest.mark.gpu
def test_refused_calls_are_refused_alike(monkeypatch):
    x = torch.ones(2, 8, device="cuda")
    h, p, s = x.half(), torch.zeros(4, 4, device="cuda", dtype=torch.uint8), torch.ones(4, 1, device="cuda").half()
    calls = [lambda: ops.fused_residual_rmsnorm(x, x, x[0].half(), 1e-6), lambda: ops.fused_residual_rmsnorm(x, x, x[0], 0.0),
             lambda: ops.fused_residual_rmsnorm(x, x, x[0], float("nan")), lambda: ops.fused_residual_rmsnorm(x.t(), x.t(), x[:, 0], 1e-6),
             lambda: ops.fused_residual_rmsnorm(x, x[:1], x[0], 1e-6), lambda: ops.fused_residual_rmsnorm(x.cpu(), x, x[0], 1e-6),
             lambda: ops.fused_residual_rmsnorm(x[:0], x[:0], x[0], 1e-6), lambda: ops.decode_linear(x, x, weight_layout="KK"),
             lambda: ops.decode_linear(x, x, weight_layout="NK", split_k=3), lambda: ops.decode_linear(x, x.t(), weight_layout="KN"),
             lambda: ops.decode_linear(x, x, x[0], weight_layout="NK"), lambda: ops.swiglu(x[:, :7]), lambda: ops.swiglu(x.t()),
             lambda: w4a16.w4a16_linear(h, p, s, group_size=48), lambda: w4a16.w4a16_linear(x, p, s),
             lambda: w4a16.w4a16_linear(h, p, s, out=h[:, :4]), lambda: w4a16.w4a16_linear(h.requires_grad_(), p, s)]
    for call in calls:
        native, python = _both(monkeypatch, call)
        assert native == python and native[0] is ValueError
