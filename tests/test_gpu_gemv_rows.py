"""Projections of more than 16 rows at the edges of their plan: ragged blocks of rows, column groups, stages and K tails."""

from __future__ import annotations

import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["KN", "NK"])
@pytest.mark.parametrize("m,k,n", [(17, 4, 4), (32, 36, 60), (33, 260, 68), (48, 1028, 64), (49, 4100, 132), (64, 2048, 1000),
                                   (65, 516, 72), (130, 64, 200)])
def test_projection_of_more_rows_than_sixteen(layout, m, k, n):
    """Integer-valued operands: every order of the sums is exact.  Ragged rows, columns and last stages, every split."""
    from cross_dsl_kernels_b200.ops import decode_linear
    g = torch.Generator().manual_seed(m + k + n)
    x, w = torch.randint(-3, 4, (m, k), generator=g).float(), torch.randint(-3, 4, (k, n), generator=g).float()
    b = torch.randint(-9, 10, (n,), generator=g).float()
    want = (x.double() @ w.double() + b.double()).float()
    weight = (w if layout == "KN" else w.t().contiguous()).cuda()
    for split in (0, 1, 2, 4, 8):
        assert torch.equal(decode_linear(x.cuda(), weight, b.cuda(), weight_layout=layout, split_k=split).cpu(), want)
    xr = torch.randn(m, k, generator=g)
    wr = torch.randn(k, n, generator=g) / k ** 0.5
    got = decode_linear(xr.cuda(), (wr if layout == "KN" else wr.t().contiguous()).cuda(), weight_layout=layout).cpu()
    assert rel_l2(got, xr.double() @ wr.double()) <= 1e-6  # FP32 FMAs: about sqrt(K) 2^-24 for a sum of K terms


@pytest.mark.parametrize("layout", ["KN", "NK"])
def test_operands_that_do_not_split(layout):
    """An infinity, a value that rounds up to one, and a NaN: as FP32 products of the plain operands give them."""
    from cross_dsl_kernels_b200.ops import decode_linear
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(20, 128, generator=g), torch.randn(128, 32, generator=g).abs()
    x[3, 7], x[4, 8], x[5, 9], x[6, 10] = float("inf"), float("-inf"), float("nan"), torch.finfo(torch.float32).max
    want = x @ w
    got = decode_linear(x.cuda(), (w if layout == "KN" else w.t().contiguous()).cuda(), weight_layout=layout).cpu()
    assert torch.isnan(got[5]).all() and torch.equal(torch.isinf(got[3:7]), torch.isinf(want[3:7]))
    assert torch.equal(got[3], want[3]) and torch.equal(got[4], want[4])
    rest = [r for r in range(20) if r not in (3, 4, 5, 6)]
    assert rel_l2(got[rest], want[rest]) <= 1e-6
