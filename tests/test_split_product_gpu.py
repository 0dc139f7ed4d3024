"""The float32 product on the tensor cores (operands as sums of three bfloat16 values) at the edges of its tiles."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu

SHAPES = [0, 11, 12, 14, 21, 22, 24, 31]
# What is left out of a product is below 2^-26 of it; 64 columns' sum is cut off at most four times at 2^-23 of itself and
# then added with a rounding of 2^-24 (K / 64 of them), one more for a bias or an addition into C.  The sums are random
# walks, so 2-norms of errors add as squares: below 4e-7 of the result's for the K here.
BOUND = 4e-7


def off(y, want):
    return float((y.double().cpu() - want).norm() / want.norm())


@pytest.mark.parametrize("m", [17, 128, 129, 300])
@pytest.mark.parametrize("n,k", [(1, 8), (64, 64), (65, 72), (130, 200), (63, 576), (128, 1000)])
def test_against_64_bits(m, n, k):
    o = ops()
    g = torch.Generator().manual_seed(m + 10 * n + 100 * k)
    a, w = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g) / math.sqrt(k)
    bias = torch.randn(n, generator=g)
    want = a.double() @ w.double().T
    ad, wd, bd = a.to(DEV), w.to(DEV), bias.to(DEV)
    assert o.gemm_split_f32_takes(ad, wd)
    room = torch.empty(m * n + 1, device=DEV)
    for shape in SHAPES:
        for at in (0, 1):  # (a destination that is not 16-byte aligned)
            out = room[at:at + m * n].view(m, n).fill_(float("nan"))
            o.gemm_split_f32(ad, wd, bd, out, o.STORE_F32, shape)
            assert off(out, want + bias) < BOUND, (shape, at)
            again = torch.empty(m, n, device=DEV)
            o.gemm_split_f32(ad, wd, bd, again, o.STORE, shape)
            assert torch.equal(out, again)
            o.gemm_split_f32(ad, wd, None, out, o.ADD_F32, shape)
            assert off(out, 2 * want + bias) < BOUND, (shape, at)
    o.check_status(DEV)


@pytest.mark.parametrize("m", [17, 129, 300])
@pytest.mark.parametrize("inter,k", [(1, 8), (64, 72), (65, 200), (130, 576)])
def test_gated(m, inter, k):
    """silu(gate) * up in the epilogue, against 64 bits; an infinity among the sums of either."""
    o = ops()
    g = torch.Generator().manual_seed(m + 10 * inter + 100 * k)
    a, w = torch.randn(m, k, generator=g), torch.randn(2 * inter, k, generator=g) / math.sqrt(k)
    bias = torch.randn(2 * inter, generator=g)
    z = a.double() @ w.double().T + bias
    want = torch.nn.functional.silu(z[:, :inter]) * z[:, inter:]
    room = torch.empty(m * inter + 1, device=DEV)
    for shape in SHAPES:
        for at in (0, 1):
            out = room[at:at + m * inter].view(m, inter).fill_(float("nan"))
            o.gemm_split_f32(a.to(DEV), w.to(DEV), bias.to(DEV), out, o.GEMM_GATED, shape)
            assert off(out, want) < 2 * BOUND, (shape, at)  # (two sums, and expf's few units)
    a[3, 0] = math.inf
    z = a.double() @ w.double().T + bias
    want = torch.nn.functional.silu(z[:, :inter]) * z[:, inter:]
    o.gemm_split_f32(a.to(DEV), w.to(DEV), bias.to(DEV), out, o.GEMM_GATED)
    want[3][torch.isneginf(z[3, :inter])] = math.nan  # (g / (1 + exp(-g)) of minus infinity, as the kernel for rows has it)
    assert torch.equal(torch.isnan(out.cpu()), torch.isnan(want)) and torch.equal(torch.isinf(out.cpu()), torch.isinf(want))
    o.check_status(DEV)


@pytest.mark.parametrize("k", [576, 1536, 4096])
def test_no_further_from_64_bits_than_chains_of_multiply_adds(k):
    o = ops()
    g = torch.Generator().manual_seed(k)
    for draw in (torch.randn, torch.rand):  # (sums that cancel, and sums that only grow)
        a, w = draw(200, k, generator=g).to(DEV), draw(96, k, generator=g).to(DEV)
        want = (a.double() @ w.double().T).cpu()
        split, chain = torch.empty(200, 96, device=DEV), torch.empty(200, 96, device=DEV)
        o.gemm_split_f32(a, w, None, split, o.STORE)
        o.gemm_simt(a, w, None, chain, o.STORE)
        assert off(split, want) <= off(chain, want)


@pytest.mark.parametrize("shape", SHAPES)
def test_values_that_are_no_numbers_and_tiny_ones(shape):
    o = ops()
    g = torch.Generator().manual_seed(5)
    a, w = torch.randn(40, 136, generator=g), torch.randn(70, 136, generator=g)
    a[3, 5], a[7, 9], a[8, 135], w[2, 1], w[66, 130] = math.inf, math.nan, -math.inf, -math.inf, math.nan
    a[11], a[12] = a[11] * 1e-38, 0.0
    w[5, ::2] = 0.0
    want = a.double() @ w.double().T
    out = torch.empty(40, 70, device=DEV)
    o.gemm_split_f32(a.to(DEV), w.to(DEV), None, out, o.STORE, shape)
    out = out.cpu()
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    assert torch.equal(torch.isinf(out), torch.isinf(want)) and torch.equal(out[torch.isinf(out)] > 0, want[torch.isinf(want)] > 0)
    rows = torch.isfinite(want)
    rows[11] = False
    assert off(out[rows], want[rows]) < BOUND
    tiny = torch.isfinite(want[11])
    # (parts below 2^-133 are lost: 136 products of at most 2^-133 x 4)
    assert float((out[11].double() - want[11])[tiny].abs().max()) < 136 * 4 * 2.0 ** -133


def test_rows_off_the_32_byte_boundary_are_left_to_the_cuda_cores():
    o = ops()
    a, w = torch.zeros(32, 24, device=DEV), torch.zeros(8, 24, device=DEV)
    assert o.gemm_split_f32_takes(a, w) and not o.gemm_split_f32_takes(a[:16], w)
    assert not o.gemm_split_f32_takes(torch.zeros(32, 20, device=DEV), torch.zeros(8, 20, device=DEV))
    assert not o.gemm_split_f32_takes(torch.zeros(32 * 24 + 4, device=DEV)[4:].view(32, 24), w)
    with pytest.raises(o.KernelError):
        o.gemm_split_f32(torch.zeros(32 * 24 + 4, device=DEV)[4:].view(32, 24), w, None, torch.zeros(32, 8, device=DEV), o.STORE)
