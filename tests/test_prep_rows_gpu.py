"""Preparing many tokens for sink attention (four a block, 128 columns a warp at a time) against the same tokens in calls of
fewer, which take a block each."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
DT = {"bfloat16": torch.bfloat16, "float32": torch.float32}


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("tokens,heads,kv,dim,vdim,bias,norm,rot,vk,own,write", [
    (592, 32, 8, 64, 64, True, 1, 64, False, True, True),
    (593, 3, 1, 64, 128, False, 2, 42, False, True, True),
    (607, 5, 5, 128, 64, True, 0, 128, False, True, True),
    (1001, 16, 4, 128, 128, True, 2, 6, True, True, True),
    (600, 6, 3, 64, 64, False, 1, 0, False, False, True),
    (599, 9, 3, 64, 64, True, 2, 32, False, True, False),
    (2049, 40, 8, 128, 64, True, 2, 128, False, True, True),
    (1603, 16, 4, 128, 128, False, 2, 128, False, True, True),
    (1490, 32, 8, 64, 64, True, 2, 64, False, True, True),
    (739, 16, 4, 64, 64, True, 2, 64, False, True, True),
    (743, 16, 4, 64, 64, True, 2, 64, False, True, True),
    (1537, 6, 2, 128, 64, False, 1, 64, False, True, True),
    (1601, 24, 8, 64, 64, False, 1, 42, True, True, True),
])
def test_prep_of_many_tokens_is_that_of_few(dtype, tokens, heads, kv, dim, vdim, bias, norm, rot, vk, own, write):
    from tokasaurus_b200.kernels import ops

    g = torch.Generator().manual_seed(tokens + heads)
    page, wide = 16, 4  # (columns behind the projections)
    width = (heads + (kv if own else 0)) * dim + (0 if vk or not own else kv * vdim)
    qkv = torch.randn(tokens, width + wide, generator=g).to(DEV)
    b = torch.randn(width, generator=g).to(DEV) if bias else None
    w = (torch.rand(2, dim, generator=g) + 0.5).to(DEV) if norm == 2 else None
    freq = (torch.rand(rot // 2, generator=g, dtype=torch.float64) + 1e-3).to(DEV) if rot else None
    first = tokens // 3  # two requests; some tokens belong to none
    seq = torch.tensor([0] * first + [1] * (tokens - first), dtype=torch.int32)
    pos = torch.cat([torch.arange(first), 9 + torch.arange(tokens - first)]).int()
    seq[5], seq[-1], seq[first] = -1, -1, -1
    pages = [-(-first // page), -(-(9 + tokens - first) // page)]
    order = torch.randperm(sum(pages), generator=g).int().to(DEV)
    indptr = torch.tensor([0, pages[0], sum(pages)], dtype=torch.int32, device=DEV)
    seq, pos = seq.to(DEV), pos.to(DEV)
    got = []
    for step in (tokens, 500):  # (500 tokens: a block each)
        q = torch.full((tokens, heads * dim), 7.0, dtype=DT[dtype], device=DEV)
        cache = torch.full((sum(pages), kv, page, dim + vdim), 7.0, dtype=DT[dtype], device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        for a in range(0, tokens, step):
            z = slice(a, a + step)
            ops.sink_attn_prep(qkv[z], b, norm > 0, 1e-6, q[z], cache, pos[z], seq[z], indptr, order, heads, kv, dim, vdim, page, write,
                               status, norm_w=w, rot_freq=freq, rot_dims=rot, rot_pairs=True, values_are_keys=vk, own_kv=own)
        assert int(status.item()) == 0
        got.append((q.double(), cache.double()))
    for x, y in zip(*got):  # every number goes through the same additions
        assert torch.equal(x, y)
