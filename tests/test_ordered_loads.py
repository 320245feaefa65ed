"""What a kernel reads of the preceding kernel's output must be read behind its wait for that kernel.

A load through the read-only path counts as invariant, and the compiler may move it in front of ``pdl_wait()``: a stale
operand, on no more than the compiler's choice.  So the sources of the kernels that wait are checked for such loads of
anything but the constant operands the dependent-launch contract names, and dependent steps are run on operands that the
preceding kernel has just written over other values."""

from __future__ import annotations

import re

import pytest
import torch

from conftest import ROOT

CSRC = ROOT / "cross_dsl_kernels_b200" / "csrc"
CONSTANTS = {"weight", "wv", "packed", "wp", "scales", "sp", "bias", "cos", "sin", "crow", "srow", "at"}  # at: of the scales
READ_ONLY = re.compile(r"\b(__ldg|ld_cached16|ld_stream16|ld_stream_f1|ld_stream_f4)\(\s*(?:reinterpret_cast<[^>]*>\()?(?:a\.)?(\w+)")


def _waiting_kernels():
    """(name, parameters, body) of each kernel that waits for the preceding one."""
    for path in sorted(CSRC.glob("*.cu")):
        for part in re.split(r"(?=__global__ )", path.read_text())[1:]:
            part = part[:part.index("\n}\n")]
            head = re.search(r"(\w+_kernel)\(", part)
            if head and "pdl_wait();" in part:
                params, body = part[head.end():].split("{", 1)
                yield head.group(1), params, body


def test_no_invariant_load_of_what_the_preceding_kernel_wrote():
    kernels = list(_waiting_kernels())
    assert {"rmsnorm_row_kernel", "w4a16_mma_kernel", "w4a16_rx_kernel", "rope_append_kernel", "swiglu_kernel", "gemv_mma_kernel",
            "paged_decode_attention_kernel", "paged_decode_attention_tc_kernel"} <= {name for name, _, _ in kernels}
    for name, params, body in kernels:
        assert "const T* __restrict__" not in re.sub(r"const T\* __restrict__ weight\b", "", params), name
        assert "const int64_t* __restrict__" not in params, name
        for load, operand in READ_ONLY.findall(body):
            assert operand in CONSTANTS, f"{name}: {load}({operand})"
    chunk = re.search(r"struct Chunk \{.*?\n\};", (CSRC / "rope_kv.cu").read_text(), re.S).group(0)
    row_at = re.search(r"struct RowAt \{.*?\n\};", (CSRC / "attention.cu").read_text(), re.S).group(0)
    assert not READ_ONLY.search(chunk) and not READ_ONLY.search(row_at)  # helpers that the kernels read through


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,k,n", [(1, 4096, 6144), (4, 1024, 4096), (8, 4096, 2048), (16, 2304, 4096)])
def test_dependent_steps_read_what_the_preceding_kernel_wrote(tokens, k, n):
    """norm -> projection -> append -> attention -> SwiGLU, captured with dependent launches, on new inputs for every round so that
    whatever a kernel finds too early is another round's data: the bits of the same ops launched one after the other."""
    from cross_dsl_kernels_b200.ops import fused_residual_rmsnorm, paged_decode_attention, rope_gqa_paged_kv_append, swiglu
    from cross_dsl_kernels_b200.timing import capture
    from cross_dsl_kernels_b200.w4a16 import w4a16_linear
    g = torch.Generator(device="cuda").manual_seed(tokens + k)
    dim, rounds, page, ctx = 128, 6, 16, 96
    heads = n // dim
    hkv = heads // 6 if heads % 6 == 0 else heads // 4
    hq = heads - 2 * hkv
    rows = [torch.randn(tokens, k, generator=g, device="cuda").half() for _ in range(rounds)]
    weight = torch.randn(k, generator=g, device="cuda").half()
    packed = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)
    scales = (0.001 + 0.002 * torch.rand(n, k // 128, generator=g, device="cuda")).half()
    cos, sin = torch.randn(ctx, dim // 2, generator=g, device="cuda"), torch.randn(ctx, dim // 2, generator=g, device="cuda")
    pos = torch.randint(0, ctx, (tokens,), generator=g, device="cuda")
    table = torch.randperm(tokens * ctx // page, generator=g, device="cuda").reshape(tokens, -1)
    seq = torch.arange(tokens, device="cuda")
    fresh = torch.randn(2, tokens * ctx // page, page, hkv, dim, generator=g, device="cuda").half()

    def step(dep, caches):
        outs = []
        for i in range(rounds):
            y, _ = fused_residual_rmsnorm(rows[i], rows[i - 1], weight, 1e-6, dependent_launch=dep)
            qkv = w4a16_linear(y, packed, scales, dependent_launch=dep)
            q, key, val = (t for t in qkv.view(tokens, heads, dim)[:, :hq + 2 * hkv].split((hq, hkv, hkv), dim=1))
            q = rope_gqa_paged_kv_append(q, key, val, cos, sin, pos, table, seq, *caches, page_size=page, rope_dim=dim,
                                         interleaved=False, dependent_launch=dep)
            for hint in (ctx, 0):  # both splits of the attention read
                outs.append(paged_decode_attention(q, *caches, pos, table, seq, page_size=page, context_hint=hint, dependent_launch=dep))
            outs.append(swiglu(qkv, dependent_launch=dep))
        return outs

    plain = [fresh[0].clone(), fresh[1].clone()]
    want = step(False, plain)
    caches = [fresh[0].clone(), fresh[1].clone()]
    outputs: list = []
    graph = capture([lambda: step(True, caches)], outputs=outputs)
    for _ in range(5):
        for t in outputs[0]:
            t.fill_(float("nan"))
        caches[0].copy_(fresh[0]), caches[1].copy_(fresh[1])
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outputs[0], want))
        assert all(torch.equal(a, b) for a, b in zip(caches, plain))
