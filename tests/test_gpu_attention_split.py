"""Attention over contexts of every mix: the even split over the CTAs, with and without scratch."""

from __future__ import annotations

import ctypes

import pytest
import torch

from conftest import rel_l2
from oracle import attention as oracle_attention

pytestmark = pytest.mark.gpu


def _paged(tokens, q_heads, kv_heads, dim, page, positions, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    per_seq = max(positions) // page + 1
    table = torch.randperm(tokens * per_seq, generator=g).reshape(tokens, per_seq)
    shape = (tokens * per_seq, page, kv_heads, dim)
    return (torch.randn(tokens, q_heads, dim, generator=g).to(dtype), torch.randn(shape, generator=g).to(dtype),
            torch.randn(shape, generator=g).to(dtype), torch.tensor(positions), table, torch.arange(tokens))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,dim,page,positions", [
    ((32, 8), 128, 16, [8191]),                                  # one long context over every CTA
    ((8, 1), 64, 16, [0, 3000, 63, 64, 1, 127, 128, 2047]),      # items inside one CTA, across two, across many
    ((4, 4), 256, 5, [700, 0, 0, 0, 15, 16, 31]),                # odd pages, whole tiles and single positions
    ((2, 2), 64, 16, [0] * 3),                                   # fewer tiles than CTAs
    ((4, 2), 64, 7, [i % 90 for i in range(300)]),               # more tokens than a block has threads
])
def test_attention_even_split(dtype, heads, dim, page, positions):
    """Contexts of every mix, dealt evenly to the CTAs: against the FP32 restatement, for each bound the caller may name
    (the grid follows it), with the same bits every time; and the split over heads and clusters that runs without scratch, which cuts
    the contexts elsewhere and so gives its own bits."""
    from cross_dsl_kernels_b200 import _native
    from cross_dsl_kernels_b200.ops import paged_decode_attention
    q, kc, vc, pos, table, seq = _paged(len(positions), *heads, dim, page, positions, dtype, seed=dim + len(positions))
    want = oracle_attention.paged_decode_attention(q, kc, vc, pos, table, seq, page_size=page)
    dev = [t.cuda() for t in (q, kc, vc, pos, table, seq)]
    rel = {torch.float32: 1e-5, torch.float16: 1e-3, torch.bfloat16: 5e-3}[dtype]  # of the existing attention tests
    for hint in (0, 1, 100, max(positions) + 1, 100000):
        got = paged_decode_attention(*dev, page_size=page, context_hint=hint)
        assert rel_l2(got.cpu(), want) <= rel
        assert torch.equal(got, paged_decode_attention(*dev, page_size=page, context_hint=hint)), "deterministic"
    bare = torch.empty_like(dev[0])
    status = _native.lib().xdk_paged_decode_attention(
        *(t.data_ptr() for t in dev), bare.data_ptr(), len(positions), *heads, dim, table.shape[1], page, 0, dim ** -0.5, 0,
        _native.dtype_code(dtype), 0, _native.stream_ptr(bare.device))
    _native.check(status, "attention without scratch")
    assert rel_l2(bare.cpu(), want) <= rel


def test_attention_not_a_number_and_empty_contexts_show():
    """A NaN in one row of K reaches exactly the heads that read it, split or not; a position of -1 (nothing to attend to)
    gives NaN, as 0 / 0 always did."""
    from cross_dsl_kernels_b200.ops import paged_decode_attention
    q, kc, vc, pos, table, seq = _paged(3, 8, 2, 128, 16, [4000, 5, 2000], torch.float16, seed=3)
    page, off = int(table[0, 2500 // 16]), 2500 % 16
    kc[page, off, 1] = float("nan")
    pos[1] = -1
    got = paged_decode_attention(*(t.cuda() for t in (q, kc, vc, pos, table, seq)), page_size=16).cpu()
    assert torch.isnan(got[0, 4:]).all() and torch.isfinite(got[0, :4]).all()
    assert torch.isnan(got[1]).all() and torch.isfinite(got[2]).all()


@pytest.mark.parametrize("heads,dim,tokens", [((8, 2), 64, 1), ((8, 2), 64, 4), ((8, 8), 128, 1), ((32, 8), 128, 2)])
def test_short_contexts_under_a_long_bound(heads, dim, tokens):
    """Few tiles on a grid sized for many: the CTAs without a share have no part in it, so a call takes about what the grid of
    splits takes (it took up to 2.7 times as long while they left empty partial results to add up)."""
    from cross_dsl_kernels_b200.ops import paged_decode_attention
    from cross_dsl_kernels_b200.timing import graph_median_us
    q, kc, vc, pos, table, seq = _paged(tokens, *heads, dim, 16, [8191] * tokens, torch.float16, seed=tokens)
    pos = torch.full((tokens,), 1000)
    want = oracle_attention.paged_decode_attention(q, kc, vc, pos, table, seq, page_size=16)
    dev = [t.cuda() for t in (q, kc, vc, pos, table, seq)]
    us = []
    for hint in (0, 8192, 1024):  # even, even, splits
        assert rel_l2(paged_decode_attention(*dev, page_size=16, context_hint=hint).cpu(), want) <= 1e-3
        us.append(graph_median_us([lambda: paged_decode_attention(*dev, page_size=16, context_hint=hint)] * 8)["median_us"])
    assert max(us[:2]) <= 1.5 * us[2], us


@pytest.mark.parametrize("page,pages", [(16, 64), (5, 100), (64, 20), (16, 200), (1, 1535), (1, 1537)])
def test_no_bound_is_that_of_the_page_table(page, pages):
    """A call without a context_hint is the call with what a row of the page table can hold: the same plan, the same bits."""
    from cross_dsl_kernels_b200 import _native
    from cross_dsl_kernels_b200.ops import paged_decode_attention
    tokens, heads, dim = 3, (6, 3), 64
    q, kc, vc, pos, table, seq = _paged(tokens, *heads, dim, page, [page * pages - 1, page * pages // 2, 0], torch.float32, seed=pages)
    dev = [t.cuda() for t in (q, kc, vc, pos, table, seq)]
    want = paged_decode_attention(*dev, page_size=page, context_hint=page * pages)
    for hint in (0, -1, -2 ** 63):
        assert torch.equal(paged_decode_attention(*dev, page_size=page, context_hint=hint), want)
    out = torch.empty_like(dev[0])  # a C caller sizes its scratch for no bound, and passes none
    size = _native.lib().xdk_paged_decode_attention_scratch_bytes(tokens, *heads, dim, 0, _native.XDK_F32)
    scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
    dst = _native.PeerOutStruct()
    dst.ptr[0], dst.world, dst.ld, dst.col0 = out.data_ptr(), 1, heads[0] * dim, 0
    status = _native.lib().xdk_paged_decode_attention_ws(
        *(t.data_ptr() for t in dev), ctypes.byref(dst), tokens, *heads, dim, pages, page, 0, dim ** -0.5, 0, _native.XDK_F32, scratch.data_ptr(), size,
        0, _native.stream_ptr(out.device))
    _native.check(status, "attention")
    assert torch.equal(out, want)
