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


# slices that a second kernel adds (one row and four rows a block) and blocks that do all of K
@pytest.mark.parametrize("M,N", [(3, 256), (300, 256), (3, 20000), (20, 20000), (50, 20000), (301, 20000)])
def test_split_product_not_finite(M, N):
    """Infinities, NaN and sums beyond the largest number come out as the FMA chain has them, and only where they belong."""
    g = torch.Generator().manual_seed(5)
    a, w = torch.randn(M, 320, generator=g).to(DEV), torch.randn(N, 320, generator=g).to(DEV)
    clean = product(a, w)
    a[1, 7], w[5, 9], w[N - 1, 3] = math.inf, -math.inf, math.nan
    a[2] *= 2e38
    out = product(a, w)
    want = a.double() @ w.double().T
    fits = want.float()
    assert torch.equal(torch.isnan(out), torch.isnan(fits))
    assert torch.equal(out.isinf(), fits.isinf()) and torch.equal(out[out.isinf()], fits[fits.isinf()])
    same = torch.ones(M, N, dtype=torch.bool, device=DEV)
    same[1:3], same[:, 5], same[:, N - 1] = False, False, False
    assert torch.equal(out[same], clean[same])
    for n in (0, 6, N - 2):  # the chain itself, on the host: a product and a sum of two float32 are rounded once in float64
        acc = torch.zeros((), dtype=torch.float32)
        for x, y in zip(a[2].cpu().double(), w[n].cpu().double()):
            acc = (x * y + acc.double()).float()
        torch.testing.assert_close(out[2, n].cpu(), acc, rtol=2.0 ** -22, atol=0, equal_nan=True)


@pytest.mark.parametrize("M,N,K", [(4, 2048, 8192), (500, 2048, 8192), (500, 16384, 1024)])
def test_split_product_not_finite_takes_no_age(M, N, K):
    """Rows of NaN (a step graph's padding may be) cost next to nothing: they took 45 to 300 times a clean product here.  A row with
    an infinity is summed again, by whole warps: within the time of some tens of products."""
    def time(bad, value):
        a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
        a[:bad, 5] = value
        out = torch.empty(M, N, device=DEV)
        product(a, w, out)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ev[0].record()
        for _ in range(5):
            product(a, w, out)
        ev[1].record()
        torch.cuda.synchronize()
        assert not out[:bad].isfinite().any() and out[bad:].isfinite().all()
        return ev[0].elapsed_time(ev[1])

    clean = time(0, 0.0)
    assert time(M, math.nan) < 4 * clean and time(1, math.inf) < 60 * clean


@pytest.mark.parametrize("M,N,K", [(4, 256, 512), (300, 20000, 128)])  # slices, and all of K in a block
def test_split_product_knows_the_step_s_status(M, N, K, monkeypatch):
    """A wait that runs out is reported to the status word of the step that the thread is in, as by every kernel that waits."""
    from tokasaurus_b200.kernels import ops

    seen, real = [], ops._fn

    def spy(lib, name):
        f = real(lib, name)
        return (lambda *a: seen.append(a[-2].value) or f(*a)) if name == "tkb_sgemm_tn_f32" else f

    monkeypatch.setattr(ops, "_fn", spy)
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.linear(a, w)
    with ops.reporting_to(status):
        out = ops.linear(a, w)
        with ops.reporting_to(None):
            ops.linear(a, w)
        ops.linear(a, w)
    ops.linear(a, w)
    assert seen == [None, status.data_ptr(), None, status.data_ptr(), None]
    assert int(status) == 0 and torch.equal(out, ops.linear(a, w))


@pytest.mark.parametrize("M,N", [(3, 256), (130, 20000)])
@pytest.mark.parametrize("small,large", [(1e-36, 1.0), (1e-40, 1e8), (1e-44, 1e14), (1e-30, 1e-6), (1e30, 1e4), (1e33, 1e-20), (1e-12, 1e12)])
def test_split_product_far_from_one(M, N, small, large):
    """All bits of numbers of every size: close to the smallest normal number, below it (where few bits are), and so large that they
    do not fit the cut form."""
    g = torch.Generator().manual_seed(9)
    a = (torch.randn(M, 300, generator=g, dtype=torch.float64) * small).float().to(DEV)
    w = (torch.randn(N, 300, generator=g, dtype=torch.float64) * large).float().to(DEV)
    for x, y in ((a, w), (w[:200].contiguous(), torch.cat([a, a[:1].expand(200, -1)]).contiguous())):  # small tokens, then small weights
        out = product(x, y)
        want = x.double() @ y.double().T
        # as for numbers around one, and half a unit of the smallest number for a result that is one
        bound = 64 * 2.0 ** -24 * (x.abs().double() @ y.abs().double().T) + 2.0 ** -149
        assert ((out.double() - want).abs() <= bound).all()


# rows that take 16-byte loads go to the kernel that brings the weights by TMA, others to the one that loads them itself; tokens are cut
# ahead from 65 rows on; few and many blocks a slice, K slices in one block and in several
@pytest.mark.parametrize("M", [3, 16, 31, 64, 65, 128, 300, 513])
@pytest.mark.parametrize("N,K", [(129, 132), (3072, 1028), (2048, 2052), (300, 4100)])
def test_both_split_kernels_give_the_same_bits(M, N, K):
    g = torch.Generator().manual_seed(M + N)
    a0, w0 = torch.randn(M, K + 1, generator=g).to(DEV), torch.randn(N, K + 1, generator=g).to(DEV)
    a, w = a0[:, 1:], w0[:, 1:]  # (rows start where no 16-byte load may)
    want = product(a, w)
    out = torch.full((M, N + 5), 7.0, device=DEV)
    product(a.contiguous(), w.contiguous(), out[:, :N])
    assert torch.equal(out[:, :N], want) and (out[:, N:] == 7).all()


def test_pieces_cut_ahead_are_bounded():
    """Large calls go in blocks of rows, so that the pieces cut ahead take 256 MB at most; the bits are those of smaller calls, and
    operands without 16-byte loads, whose kernel cuts itself, ask for none."""
    from tokasaurus_b200.kernels import ops

    lib = ops._libs.get("sgemm.cu")
    sizes = lambda a, w: (ops._ptr(a), ops._ptr(w), a.shape[0], w.shape[0], a.shape[1], a.stride(0), w.stride(0))  # noqa: E731
    w = torch.empty(20000, 8192, device=DEV)  # enough column tiles for whole sums in a block
    assert 0 < 4 * ops._sgemm_scratch(lib)(*sizes(torch.empty(8192, 8192, device=DEV), w)) <= 256 << 20
    odd = torch.empty(8192, 8193, device=DEV)[:, :8192]
    assert ops._sgemm_scratch(lib)(*sizes(odd, w)) == 0
    g = torch.Generator().manual_seed(9)
    K = 16384
    for M, N in ((2900, 1100), (2700, 2100)):  # two blocks of rows; sums in slices and whole
        a, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
        out = torch.full((M + 1, N), 7.0, device=DEV)
        ops.sgemm_tn(a, w, out[:M])
        assert (out[M] == 7).all()
        assert torch.equal(out[:M], torch.cat([product(x, w) for x in a.split(700)]))
        want = a.double() @ w.double().T
        assert (out[:M].double() - want).norm() <= 4e-7 * want.norm()
