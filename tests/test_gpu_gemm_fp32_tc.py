"""The fp32 product in bfloat16 terms against 64 bits, beside the CUDA-core product."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from inferx_b200.kernels import ops
    return ops


def _off(a, ref):
    return float((a.double() - ref).norm() / ref.norm())


# edges of the 128 x 128 tile and of the 64-entry step, odd widths (scalar stores), one step,
# two steps, runs of k of unequal length
@pytest.mark.parametrize("M,N,K", [(17, 8, 8), (127, 129, 64), (128, 128, 72), (129, 255, 128),
                                   (40, 1024, 2048), (600, 2048, 5632), (333, 1000, 1032),
                                   (65, 3, 4096)])
@pytest.mark.parametrize("splits", [None, 1, 3])
def test_against_64_bits(M, N, K, splits):
    ops = _ops()
    if splits == 3 and -(-K // 64) < 3:
        pytest.skip("fewer steps than runs")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    # magnitudes over six decades, so that terms of every size meet
    x = torch.randn(M, K, generator=g, device="cuda") * 10 ** (
        6 * torch.rand(M, K, generator=g, device="cuda") - 3)
    w = torch.randn(N, K, generator=g, device="cuda")
    ref = x.double() @ w.double().T
    for act in (None, "relu_squared"):
        want = ref if act is None else ref.clamp(min=0) ** 2
        got = ops.gemm_fp32_tc(x, w, act, splits=splits)
        plain = ops.gemm_generic(x, w.unsqueeze(0), None, None, dual=False, activation=act)
        # an error of this product is 2^-23 or so of a step's sum, a chain's grows with K; at
        # K of one step they are the same few 2^-24
        assert _off(got, want) <= max(1.05 * _off(plain, want), 2.0 ** -22)
    ops.check_async_errors()


def test_infinities_nan_and_sums_that_overflow():
    ops = _ops()
    x = torch.randn(130, 256, device="cuda")
    w = torch.randn(140, 256, device="cuda")
    x[3, 5], x[7, 9], w[11, 200], w[139, 0] = math.inf, math.nan, -math.inf, 3.4e38
    x[129, 0] = 0.5
    x[50] = 0.0
    x[50, 1] = 3.4e38                       # its first term rounds up to infinity
    ref = ops.gemm_generic(x, w.unsqueeze(0), None, None, dual=False)
    for splits in (1, 2):
        got = ops.gemm_fp32_tc(x, w, splits=splits)
        assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.isinf(), ref.isinf())
        inf = ref.isinf()
        assert torch.equal(got[inf], ref[inf])
        fine = ref.isfinite()
        torch.testing.assert_close(got[fine], ref[fine], rtol=1e-5, atol=1e-4)
    ops.check_async_errors()


def test_which_products_take_it():
    ops = _ops()
    w = torch.randn(24, 64, device="cuda")
    before = ops.LAUNCHES[0]
    x = torch.randn(33, 64, device="cuda")
    assert ops._splits_fp32(x, w) and not ops._splits_fp32(x[:16], w)
    assert not ops._splits_fp32(torch.randn(33, 60, device="cuda"), w[:, :60].contiguous())
    off = torch.randn(33 * 64 + 4, device="cuda")[4:].view(33, 64)      # a 16-byte mark
    assert not ops._splits_fp32(off, w)
    torch.testing.assert_close(ops.linear(off, w), off @ w.T, rtol=1e-4, atol=1e-4)
    assert ops.LAUNCHES[0] == before + 1


@pytest.mark.parametrize("scale_x,scale_w", [(1e-36, 1.0), (1e-38, 1.0), (1e-38, 1e6),
                                             (1e-20, 1e-20), (1e-30, 1e-10), (1e-33, 1e-3)])
@pytest.mark.parametrize("splits", [1, 4])
def test_operands_too_small_for_three_terms(scale_x, scale_w, splits):
    """Below 2^-110 the third term is a subnormal, below 2^-126 the second too: such sums are made
    from the operands themselves."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(40, 1024, generator=g, device="cuda") * scale_x
    w = torch.randn(130, 1024, generator=g, device="cuda") * scale_w
    x[7] = 0.0
    ref = x.double() @ w.double().T
    off = [_off(y, ref) for y in (ops.gemm_fp32_tc(x, w, splits=splits), ops.gemm_generic(
        x, w.unsqueeze(0), None, None, dual=False))]
    # a result that is itself subnormal carries 2^-150 of rounding in any order of sums
    floor = 2.0 ** -150 * ref.numel() ** 0.5 / float(ref.norm())
    assert off[0] <= max(off[1], 2.0 ** -22, 4 * floor), off


def test_sums_that_overflow_in_another_order():
    """What cancels in ascending k may pass infinity where products of 64 k are added together."""
    ops = _ops()
    x = torch.ones(20, 512, device="cuda")
    w = torch.zeros(24, 512, device="cuda")
    w[:, 0:512:4], w[:, 1:512:4] = 3e38, -3e38
    w[3, 2] = 1.0
    ref = ops.gemm_generic(x, w.unsqueeze(0), None, None, dual=False)
    for splits in (1, 2):
        got = ops.gemm_fp32_tc(x, w, splits=splits)
        assert got.isfinite().all() == ref.isfinite().all()
    ops.check_async_errors()


def test_short_inner_sizes_stay_on_the_cuda_cores():
    ops = _ops()
    for rows, k in ((33, 64), (64, 128), (130, 96)):
        x, w = torch.randn(rows, k, device="cuda"), torch.randn(48, k, device="cuda")
        plain = ops.gemm_generic(x, w.unsqueeze(0), None, None, dual=False)
        assert torch.equal(ops.linear(x, w), plain)
