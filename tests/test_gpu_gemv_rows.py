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


@pytest.mark.parametrize("layout,k,n,split", [("KN", 4096, 1024, True), ("KN", 14336, 4100, True), ("NK", 4096, 2372, True),
                                              ("NK", 8192, 4096, True), ("KN", 4096, 768, True), ("KN", 4096, 764, False), ("KN", 4092, 1024, False), ("KN", 64, 512, False),
                                              ("NK", 4096, 2368, False), ("NK", 2048, 4096, False), ("NK", 4, 8, False)])
def test_the_split_is_no_less_accurate_than_fp32_fmas(layout, k, n, split):
    """More than 16 rows: split-TF32 products where their error against 64 bits is no larger than that of the FP32 FMAs, the bits of
    those elsewhere, and always from the version-1 entry point."""
    from cross_dsl_kernels_b200 import _native
    from cross_dsl_kernels_b200.ops import decode_linear
    g = torch.Generator(device="cuda").manual_seed(k + n)
    ours, fmas = 0.0, 0.0
    for _ in range(4):
        x, w = torch.randn(24, k, generator=g, device="cuda"), torch.randn(k, n, generator=g, device="cuda") / k ** 0.5
        want, weight = x.double() @ w.double(), w if layout == "KN" else w.t().contiguous()
        got, strict = (decode_linear(x, weight, weight_layout=layout, strict_fp32=s) for s in (False, True))
        assert torch.equal(got, strict) != split
        ours, fmas = ours + rel_l2(got, want), fmas + rel_l2(strict, want)
        first = torch.empty_like(got)
        _native.check(_native.lib().xdk_gemv_f32(x.data_ptr(), weight.data_ptr(), None, first.data_ptr(), 24, k, n, int(layout == "NK"), 0,
                                                 None, 0, _native.stream_ptr(x.device)), "version 1")
        assert torch.equal(first, strict)
    assert ours <= fmas * 1.01  # means of four draws of 24 N outputs: they scatter by less than 1 %


@pytest.mark.parametrize("layout,k,n", [("KN", 4096, 768), ("KN", 4100, 1028), ("KN", 8192, 1200), ("KN", 4096, 512), ("NK", 4096, 2400)])
def test_the_bits_of_a_row_do_not_depend_on_the_rows_beside_it(layout, k, n):
    """More than 16 rows, up to several launches of them: the same bits for a row in every batch, and the right ones."""
    from cross_dsl_kernels_b200.ops import decode_linear
    g = torch.Generator(device="cuda").manual_seed(n)
    x, w = torch.randn(1300, k, generator=g, device="cuda"), torch.randn(k, n, generator=g, device="cuda") / k ** 0.5
    weight, bias = w if layout == "KN" else w.t().contiguous(), torch.randn(n, generator=g, device="cuda")
    whole = decode_linear(x, weight, bias, weight_layout=layout)
    assert rel_l2(whole, x.double() @ w.double() + bias.double()) <= 2e-7 * (k / 4096) ** 0.5  # 1.6e-7 of the product, and the bias's sum
    for m in (17, 32, 33, 64, 100, 288, 289, 592, 593, 1185):
        assert torch.equal(decode_linear(x[:m], weight, bias, weight_layout=layout), whole[:m])
        assert torch.equal(decode_linear(x[1300 - m:], weight, bias, weight_layout=layout), whole[1300 - m:])


@pytest.mark.parametrize("layout,n", [("KN", 772), ("KN", 1000), ("KN", 4100), ("KN", 20000), ("NK", 2380), ("NK", 20000)])
def test_outputs_that_are_not_finite_at_full_size(layout, n):
    """Rows of x and columns of W with infinities and NaNs, at every width of a pass: those outputs as FP32 FMAs give them, and for
    the price of a second pass (they used to take one thread each, up to fifty times as long)."""
    from cross_dsl_kernels_b200.ops import decode_linear
    m, k = 70, 4096
    g = torch.Generator(device="cuda").manual_seed(n)
    x, w = torch.randn(m, k, generator=g, device="cuda"), torch.randn(k, n, generator=g, device="cuda") / k ** 0.5
    bias = torch.randn(n, generator=g, device="cuda")
    clean = decode_linear(x, w if layout == "KN" else w.t().contiguous(), bias, weight_layout=layout)
    x[3, 5], x[17, k - 1], x[m - 1, 0] = float("inf"), float("nan"), float("-inf")
    x[20] *= 1e30  # times a column of 1e30: a true overflow
    w[7, 2], w[9, n - 1] = float("nan"), float("inf")
    w[:, 11] = 1e30
    weight = w if layout == "KN" else w.t().contiguous()

    def times(a, b):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        decode_linear(a, b, bias, weight_layout=layout)
        start.record()
        for _ in range(5):
            decode_linear(a, b, bias, weight_layout=layout)
        end.record()
        end.synchronize()
        return start.elapsed_time(end)

    got, strict = (decode_linear(x, weight, bias, weight_layout=layout, strict_fp32=s) for s in (False, True))
    odd = torch.zeros(m, n, dtype=torch.bool, device="cuda")
    odd[[3, 17, m - 1]] = True
    odd[:, [2, n - 1]] = True
    overflow = torch.zeros_like(odd)
    overflow[20, 11] = True  # an infinity or a NaN, by the order of the sum
    assert not torch.isfinite(strict[odd | overflow]).any() and not torch.isfinite(got[overflow]).any()
    assert torch.isfinite(strict[~(odd | overflow)]).all()
    assert torch.equal(got[odd].nan_to_num(nan=7.0, posinf=8.0, neginf=9.0), strict[odd].nan_to_num(nan=7.0, posinf=8.0, neginf=9.0))
    same = ~odd
    same[20], same[:, 11] = False, False
    assert torch.equal(got[same], clean[same])  # finite outputs keep their bits
    large = ~odd & ~overflow & ~same
    assert rel_l2(got[large], strict[large]) <= 1e-6
    assert times(torch.full_like(x, float("nan")), weight) <= 6 * times(torch.randn_like(x), torch.randn_like(weight))
