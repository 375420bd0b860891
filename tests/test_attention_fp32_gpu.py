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
