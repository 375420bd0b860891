"""The FP32-pipe attention: blocks of several tokens and a block for every token give the same bits (segments' edges, windows
that start inside a segment, groups of heads that do and do not divide a block, tokens of several requests in one block), against
a float64 statement, with values behind a token's own key that are not numbers."""

import math

import pytest
import torch

from test_kernels_gpu import i32, make_paged, plain_attention, tol

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd,nh,nkv,window", [(64, 8, 2, None), (64, 8, 2, 100), (128, 6, 2, 129), (16, 40, 1, None),
                                               (80, 3, 3, 257), (256, 10, 2, None)])
def test_both_kernels_agree(dtype, hd, nh, nkv, window):
    from tokasaurus_b200.kernels import ops

    lens = [128, 5, 390, 1, 257]
    ps = 16
    kc, vc, indptr, pages, K, V = make_paged(dtype, len(lens), lens, nkv, hd, ps, 80, seed=hd)
    new = [128, 2, 140, 1, 1]  # the last tokens of every request are the step's
    token_seq = i32([s for s, n in enumerate(new) for _ in range(n)])
    positions = i32([lens[s] - n + i for s, n in enumerate(new) for i in range(n)])
    T = token_seq.numel()
    q = torch.randn(T, (nh + 2 * nkv) * hd, generator=torch.Generator().manual_seed(1)).to(dtype).to(DEV)
    scale = 1 / math.sqrt(hd)

    def run(rows, vcache=vc):
        n = T if rows is None else rows.numel()
        out = torch.full((n, nh * hd), 9.0, dtype=dtype, device=DEV)
        ops.attn_paged(q, q.shape[1], out, kc, vcache, token_seq, positions, indptr, pages, rows, n, nh, nkv, hd, ps, scale, window)
        return out

    out = run(None)  # 272 rows of 5 requests: blocks of several tokens
    picked = i32([0, 127, 128, 130, 200, 269, 270, 271])
    for t in picked.tolist():  # one row at a time: a block for every token
        assert torch.equal(run(i32([t]))[0], out[t])
        want = plain_attention(q[t, : nh * hd].view(nh, hd).cpu(), K[token_seq[t]], V[token_seq[t]], int(positions[t]), scale, window)
        torch.testing.assert_close(out[t].view(nh, hd).cpu().double(), want, **tol(dtype), check_dtype=False)
    # what stands behind a token's own key is not looked at: the last token's value of the third request is no number
    bad = vc.clone()
    page, slot = int(pages[int(indptr[2]) + (lens[2] - 1) // ps]), (lens[2] - 1) % ps
    bad[page, :, slot] = math.nan
    got = run(None, bad)
    last = 128 + 2 + 140 - 1
    keep = torch.arange(T, device=DEV) != last
    assert torch.equal(got[keep], out[keep]) and got[last].isnan().all()


@pytest.mark.parametrize("hd,nh,nkv,window", [(64, 8, 2, None), (128, 6, 6, 200), (256, 10, 2, None)])
@pytest.mark.parametrize("decoding,portion", [(5, 40), (1, 9), (70, 1100), (3, 2)])
def test_requests_that_decode_beside_portions(hd, nh, nkv, window, decoding, portion):
    """Steps of both: single tokens ahead of, between and behind portions, padding tokens at the end, more rows than a block scans at a
    time, rows in another order; every row has the bits that it has alone."""
    from tokasaurus_b200.kernels import ops

    new = [portion] + [1] * decoding + [portion // 2 + 1, 1, 3]
    lens = [n + 37 * (i % 11) * (n == 1) for i, n in enumerate(new)]
    ps = 16
    kc, vc, indptr, pages, K, V = make_paged(torch.float32, len(lens), lens, nkv, hd, ps, sum(-(-n // ps) for n in lens) + 2, seed=hd)
    seq = [s for s, n in enumerate(new) for _ in range(n)]
    pos = [lens[s] - n + i for s, n in enumerate(new) for i in range(n)]
    token_seq, positions = i32(seq + [-1] * 5), i32(pos + [0] * 5)
    T = len(seq)
    q = torch.randn(T + 5, (nh + 2 * nkv) * hd, generator=torch.Generator().manual_seed(1)).to(DEV)

    def run(rows, n):
        out = torch.full((n, nh * hd), 9.0, device=DEV)
        ops.attn_paged(q, q.shape[1], out, kc, vc, token_seq, positions, indptr, pages, rows, n, nh, nkv, hd, ps, 0.1, window)
        return out

    out = run(None, T + 5)
    g = torch.Generator().manual_seed(2)
    order = torch.randperm(T, generator=g).to(torch.int32)  # neighbours of other requests nearly everywhere
    assert torch.equal(run(order.to(DEV), T), out[order.long().to(DEV)])
    for t in [0, portion - 1, portion, portion + decoding - 1, T - 1, T - 4] + torch.randint(T, (6,), generator=g).tolist():
        assert torch.equal(run(i32([t]), 1)[0], out[t])
        want = plain_attention(q[t, : nh * hd].view(nh, hd).cpu(), K[seq[t]], V[seq[t]], pos[t], 0.1, window)
        torch.testing.assert_close(out[t].view(nh, hd).cpu().double(), want, **tol(torch.float32), check_dtype=False)


def test_requests_that_decode_do_not_wait_for_one_another():
    """One kv head a head: 24 requests' contexts in one block were walked one after the other."""
    from tokasaurus_b200.kernels import ops

    nh, hd, ps, n, ctx, portion = 16, 128, 16, 24, 1500, 200
    lens = [ctx] * n + [portion]
    kc, vc, indptr, pages, _, _ = make_paged(torch.float32, n + 1, lens, nh, hd, ps, sum(-(-x // ps) for x in lens), seed=1)

    def time(seqs, news):
        seq = [s for s, k in zip(seqs, news) for _ in range(k)]
        pos = [lens[s] - k + i for s, k in zip(seqs, news) for i in range(k)]
        T = len(seq)
        q, out = torch.randn(T, nh * hd, device=DEV), torch.empty(T, nh * hd, device=DEV)
        args = (q, nh * hd, out, kc, vc, i32(seq), i32(pos), indptr, pages, None, T, nh, nh, hd, ps, 0.1, None)
        ops.attn_paged(*args)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ev[0].record()
        for _ in range(10):
            ops.attn_paged(*args)
        ev[1].record()
        torch.cuda.synchronize()
        return ev[0].elapsed_time(ev[1])

    apart = time(range(n), [1] * n) + time([n], [portion])
    assert time(range(n + 1), [1] * n + [portion]) < 2 * apart  # (was 12 times)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd,nh,nkv", [(64, 8, 2), (256, 10, 2), (16, 40, 1)])
@pytest.mark.parametrize("new,pad", [([1, 1], 2), ([1, 9, 1], 5), ([40], 24), ([200, 1, 2], 53)])
def test_rows_of_padding_tokens_are_zero(dtype, hd, nh, nkv, new, pad):
    """A step graph's padding tokens: memory that nobody wrote (here NaN) does not go into the products behind."""
    from tokasaurus_b200.kernels import ops

    kc, vc, indptr, pages, _, _ = make_paged(dtype, len(new), new, nkv, hd, 16, 40, seed=1)
    seq = [s for s, n in enumerate(new) for _ in range(n)]
    token_seq, positions = i32(seq + [-1] * pad), i32([i for n in new for i in range(n)] + [0] * pad)
    T = len(seq)
    q = torch.randn(T + pad, nh * hd, generator=torch.Generator().manual_seed(1)).to(dtype).to(DEV)
    out = torch.full((T + pad, nh * hd), math.nan, dtype=dtype, device=DEV)
    ops.attn_paged(q, q.shape[1], out, kc, vc, token_seq, positions, indptr, pages, None, T + pad, nh, nkv, hd, 16, 0.1, None)
    assert (out[T:] == 0).all() and out[:T].isfinite().all()


@pytest.mark.parametrize("hd,nh,nkv", [(64, 8, 2), (256, 10, 2)])
@pytest.mark.parametrize("rows", [1, 40])
def test_scores_that_are_all_minus_infinity(hd, nh, nkv, rows):
    """A softmax over nothing but minus infinities is 0 / 0, as it is in float64; one score that is a number takes all the weight,
    and keys on pages that were given back count for nothing."""
    from tokasaurus_b200.kernels import ops

    L, ps = 300, 16
    kc, vc, indptr, pages, K, V = make_paged(torch.float32, 1, [L], nkv, hd, ps, 30, seed=2)
    kc[:, :, :, 3] = 1e30
    q = torch.randn(rows, nh * hd, generator=torch.Generator().manual_seed(1)).to(DEV)
    q.view(rows, nh, hd)[:, 0, 3] = -1e30  # head 0: every score is minus infinity
    q.view(rows, nh, hd)[:, 1:, 3] = 0
    token_seq, positions = i32([0] * rows), i32(range(L - rows, L))

    def run(ids):
        out = torch.full((rows, nh * hd), 9.0, device=DEV)
        ops.attn_paged(q, nh * hd, out, kc, vc, token_seq, positions, indptr, ids, None, rows, nh, nkv, hd, ps, 1.0, None)
        return out.view(rows, nh, hd)

    out = run(pages)
    assert out[:, 0].isnan().all() and out[:, 1:].isfinite().all()
    assert (run(torch.full_like(pages, -1)) == 0).all()  # no key at all
    target = 133
    kc[int(pages[target // ps]), 0, target % ps, 3] = 0
    torch.testing.assert_close(run(pages)[:, 0].cpu(), V[0][target, 0].expand(rows, hd), rtol=1e-6, atol=0)
