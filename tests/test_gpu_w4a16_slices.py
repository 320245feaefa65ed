"""The W4A16 kernel that keeps x in registers, at the shapes where its split of K and N changes, and the two shapes of the
direct-load kernel."""

from __future__ import annotations

import pytest
import torch

from cross_dsl_kernels_b200 import quantization as qz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n,group", [
    (128, 8, 32),         # half a slice, half a column group
    (384, 40, 64),        # a last slice of 128 k
    (1280, 9008, 128),    # five slices: three column sets per CTA, several passes each
    (3968, 2376, 128),    # the widest single CTA (15.5 slices)
    (4352, 4096, 256),    # 17 slices: the first shape that a cluster shares, an uneven second rank
    (11008, 1000, 128),   # 43 slices over three ranks
    (14336, 528, 64),     # few column groups: more ranks than K alone asks for
    (16384, 30000, 128),  # many passes per cluster
    (3072, 4800, 128),    # few rows: three CTAs per SM save the direct-load kernel a pass; three chunks in batches of two
    (2048, 28680, 64),    # and several passes of it, a ragged last one
    (32768, 24, 128),     # the longest K of the path
    (32896, 24, 128),     # and the first one past it
])
@pytest.mark.parametrize("m", [1, 8, 9, 16])
def test_w4a16_slices_ranks_and_sets(m, k, n, group):
    """Codes, scales and x are small integers and powers of two: every sum is exact, whatever the order, so each of the
    plans has to give the bits of a 64-bit product."""
    from cross_dsl_kernels_b200.w4a16 import w4a16_linear
    g = torch.Generator().manual_seed(k + n + m)
    q = torch.randint(-1, 2, (n, k), generator=g, dtype=torch.int8)
    packed = qz.pack_int4(q)
    scales = torch.full((n, -(-k // group)), 0.5).half() * (1 + torch.randint(0, 2, (n, -(-k // group)), generator=g)).half()
    x = (torch.randint(0, 16, (m, k), generator=g) == 0).half() * torch.randint(-1, 2, (m, k), generator=g).half()
    bias = torch.randint(-4, 5, (n,), generator=g).half()
    w = q.double() * scales.double().repeat_interleave(group, dim=1)[:, :k]
    want = (x.double() @ w.t() + bias.double()).half()  # sums stay below 2^10 in halves: exact in FP16
    for dependent in (False, True):
        got = w4a16_linear(x.cuda(), packed.cuda(), scales.cuda(), bias.cuda(), group_size=group, dependent_launch=dependent)
        assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("m,k", [(3, 384), (8, 1152), (9, 128), (16, 5504)])
def test_w4a16_large_scales_on_a_last_half_slice(m, k):
    """K % 256 = 128 leaves half of the last slice past K, where the copy fills the codes with zeros; a zero code stands for
    -8, and with a scale of 8192 or more -8 * scale is an infinity in FP16.  The quantizer gives such scales."""
    from cross_dsl_kernels_b200.w4a16 import w4a16_linear
    w = torch.zeros(24, k)
    w[:, ::37] = 60000.0
    packed, scales = qz.quantize_int4(w.half(), group_size=128)
    assert scales.max() >= 8192
    x = torch.zeros(m, k).half()
    x[:, ::37] = 2.0 ** -12
    got = w4a16_linear(x.cuda(), packed.cuda(), scales.cuda(), group_size=128).cpu()
    codes = qz.unpack_int4(packed, k).double()
    want = x.double() @ (codes * scales.double().repeat_interleave(128, dim=1)[:, :k]).half().double().t()
    assert torch.equal(got, want.half())


@pytest.mark.parametrize("k,n", [
    (128, 1000), (384, 2048), (896, 4696),  # short K of many rows: the stream kernel
    (7168, 2368),   # one column group per SM: the direct-load kernel up to M = 8
    (10240, 4096), (10240, 18904), (12288, 9432),  # the tcgen05 kernel from M = 9, and for whole strips below
    (14336, 14208),  # the kernel with x in registers
    (14336, 37888), (20480, 28672),  # more columns than its clusters take in one wave
])
def test_w4a16_on_both_sides_of_the_dispatch(k, n):
    """As above, on the GPU: the sums of small integers are exact in FP32, whichever kernel has the shape."""
    from cross_dsl_kernels_b200.w4a16 import w4a16_linear
    g = torch.Generator(device="cuda").manual_seed(k + n)
    low, high = (torch.randint(7, 10, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8) for _ in range(2))
    packed = low + 16 * high  # codes of -1, 0 and 1
    scales = torch.full((n, k // 128), 0.5, device="cuda").half()
    codes = torch.stack((packed & 15, packed >> 4), dim=2).flatten(1).float() - 8
    for m in (3, 8, 9, 16):
        x = (torch.randint(0, 16, (m, k), generator=g, device="cuda") == 0).half() * torch.randint(-1, 2, (m, k), generator=g, device="cuda").half()
        want = (x.float() @ codes.t() * 0.5).half()
        for dependent in (False, True):
            assert torch.equal(w4a16_linear(x, packed, scales, group_size=128, dependent_launch=dependent), want)
