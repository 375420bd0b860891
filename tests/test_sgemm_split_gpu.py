"""The float32 product on the tensor cores: every number of token columns, edges of its tiles, chunks, groups and slices, row
strides and base addresses that do not take 16-byte loads, and numbers that are not finite."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def product(a, w, out=None):
    from tokasaurus_b200.kernels import ops

    out = torch.empty(a.shape[0], w.shape[0], device=DEV) if out is None else out
    ops.sgemm_tn(a, w, out)
    return out


# N, K: one tile and slice; a tile's and a chunk's remainders; several slices of unequal length; many tiles (one slice)
@pytest.mark.parametrize("N,K", [(128, 128), (131, 190), (257, 576), (2048, 1100), (20000, 256)])
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 129, 700])
def test_split_product(M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    out = product(a, w)
    want = a.double() @ w.double().T
    # what is left out of a term is below 2^-24 of it, a sum of 128 terms truncated to 24 bits 16 times, then at most
    # K / 128 + 16 roundings of the running sum: 64 units in the last place of the sum of magnitudes covers all of it
    bound = 64 * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T)
    assert ((out.double() - want).abs() <= bound).all()
    assert (out.double() - want).norm() <= 4e-7 * want.norm()  # an FMA chain's own error is about 2^-25 sqrt(K)
    for row in {0, M // 2, M - 1}:  # a row's result does not depend on the other rows of the batch
        assert torch.equal(product(a[row:row + 1].contiguous(), w)[0], out[row])


def test_split_product_strides():
    g = torch.Generator().manual_seed(3)
    a0, w0 = torch.randn(40, 519, generator=g).to(DEV), torch.randn(200, 777, generator=g).to(DEV)
    for off, K in ((0, 512), (1, 512), (4, 515)):  # (strides 519 and 777: no 16-byte loads)
        a, w = a0[:, off:off + K], w0[:, off:off + K]
        out = torch.full((40, 300), 7.0, device=DEV)
        product(a, w, out[:, 50:250])
        assert torch.equal(out[:, 50:250], product(a.contiguous(), w.contiguous()))
        assert (out[:, :50] == 7).all() and (out[:, 250:] == 7).all()


@pytest.mark.parametrize("M", [3, 300])
def test_split_product_not_finite(M):
    """Infinities, NaN and sums beyond the largest number come out as the FMA chain has them, and only where they belong."""
    g = torch.Generator().manual_seed(5)
    a, w = torch.randn(M, 320, generator=g).to(DEV), torch.randn(256, 320, generator=g).to(DEV)
    a[1, 7], w[5, 9], w[6, 3] = math.inf, -math.inf, math.nan
    a[2] *= 2e38
    out = product(a, w)
    want = a.double() @ w.double().T
    fits = want.float()
    assert torch.equal(torch.isnan(out), torch.isnan(fits))
    assert torch.equal(out.isinf(), fits.isinf()) and torch.equal(out[out.isinf()], fits[fits.isinf()])
    fine = fits.isfinite() & (torch.arange(M, device=DEV)[:, None] != 2)
    assert ((out.double() - want)[fine].abs() <= 64 * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T)[fine]).all()
