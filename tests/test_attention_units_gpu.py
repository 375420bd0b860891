"""Prompt portions on tcgen05 whose heads are shared out among units of a block: every number of key tiles for every number of units
that take them in turn, odd groups of heads, windows, and scores that are not finite."""

import math

import pytest
import torch

from test_kernels_gpu import DEV, i32, make_paged, run_mma_attention

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tokasaurus_b200.kernels import ops

    return ops


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("nh,nkv,ps,window", [(3, 1, 16, None), (4, 2, 5, None), (5, 1, 8, 100)])
@pytest.mark.parametrize("single", [False, True])
def test_numbers_of_key_tiles(ops, hd, nh, nkv, ps, window, single):
    """Portions that end 1 to 12 tiles of 64 keys behind their requests' beginnings: fewer tiles than units, as many, more, and
    rounds of the ring of tiles."""
    lens_kv = [2, 63, 65, 128, 129, 193, 257, 320, 383, 450, 513, 641, 767]
    lens_q = [2, 63, 3, 128, 100, 2, 65, 64, 5, 130, 2, 2, 66]
    got, want = run_mma_attention(ops, lens_q, lens_kv, nh, nkv, hd, ps, window, seed=hd + nh, tc=True, single_heads=single)
    assert not torch.isnan(got).any()
    torch.testing.assert_close(got, want, rtol=1.6e-2, atol=1.2e-2)  # the bound of the other tests of these kernels
    again, _ = run_mma_attention(ops, lens_q, lens_kv, nh, nkv, hd, ps, window, seed=hd + nh, tc=True, single_heads=single)
    assert torch.equal(got, again)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("value", [math.nan, math.inf])
def test_scores_that_are_not_finite(ops, hd, single, value):
    """A row of q that holds a NaN or an infinity is NaN, and nothing of it reaches other rows or heads."""
    import numpy as np
    from types import SimpleNamespace

    from tokasaurus_b200.parts.attention import plan_attention

    nh, nkv, ps, L, n = 3, 1, 16, 400, 150
    kc, vc, indptr, pages, _, _ = make_paged(torch.bfloat16, 1, [L], nkv, hd, ps, 30, seed=2)
    plan = plan_attention(SimpleNamespace(seq_q_len=np.asarray([n], dtype=np.int32), seq_kv_len=np.asarray([L], dtype=np.int32)), None,
                          query_tile=128)
    c = i32(plan["counts"])

    def run(qkv):
        out, status = torch.zeros(n, nh * hd, dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        ops.attn_prefill_tc(qkv.to(DEV), out, kc, vc, i32([0]), i32([n]), i32([L]), indptr, pages, i32(plan["tiles"]), c[2:3],
                            int(plan["counts"][2]), nh, nkv, hd, ps, hd ** -0.5, None, status, single_heads=single)
        assert int(status) == 0
        return out.view(n, nh, hd)

    qkv = torch.randn(n, (nh + 2 * nkv) * hd, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    want = run(qkv)
    qkv[77, hd + 3] = value
    got = run(qkv)
    assert got[77, 1].isnan().all()
    keep = torch.ones(n, nh, dtype=torch.bool)
    keep[77, 1] = False
    assert torch.equal(got[keep.to(DEV)], want[keep.to(DEV)])


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("L,n", [(150, 150), (400, 150), (20, 20)])
def test_scores_of_minus_infinity(ops, hd, single, L, n):
    """A score of minus infinity is a weight of zero: beside finite scores the row is what it is without that key, a row that sees
    no other score is 0 / 0, and the values of keys behind a row's own position do not reach it, however large they are."""
    import numpy as np
    from types import SimpleNamespace

    from tokasaurus_b200.parts.attention import plan_attention

    nh, nkv, ps = 3, 1, 1
    kc, vc, indptr, pages, k, v = make_paged(torch.bfloat16, 1, [L], nkv, hd, ps, L + 3, seed=4)
    table = pages[:L].long()
    kc[table, 0, 0, 5] = kc[table, 0, 0, 5].abs() + 0.5  # component 5 of every key is positive
    plan = plan_attention(SimpleNamespace(seq_q_len=np.asarray([n], dtype=np.int32), seq_kv_len=np.asarray([L], dtype=np.int32)), None,
                          query_tile=128)
    c = i32(plan["counts"])

    def run(qkv, kc, vc):
        out, status = torch.zeros(n, nh * hd, dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        ops.attn_prefill_tc(qkv.to(DEV), out, kc, vc, i32([0]), i32([n]), i32([L]), indptr, pages, i32(plan["tiles"]), c[2:3],
                            int(plan["counts"][2]), nh, nkv, hd, ps, hd ** -0.5, None, status, single_heads=single)
        assert int(status) == 0
        return out.view(n, nh, hd)

    qkv = torch.randn(n, (nh + 2 * nkv) * hd, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    qkv[:, 5: nh * hd: hd] = qkv[:, 5: nh * hd: hd].abs() + 0.5
    want = run(qkv, kc, vc)
    # every score of these rows is minus infinity
    rows = [0, 7, n - 1]
    bad = qkv.clone()
    bad[rows, hd + 5] = -math.inf
    got = run(bad, kc, vc)
    assert got[rows, 1].isnan().all()
    keep = torch.ones(n, nh, dtype=torch.bool)
    keep[rows, 1] = False
    assert torch.equal(got[keep.to(DEV)], want[keep.to(DEV)])
    # one key of minus infinity: rows that see it and others are as without it (float64 sums; the bound of the other tests)
    key = max(0, L - n) + 3
    gone = kc.clone()
    gone[table[key], 0, 0, 5] = -math.inf
    got = run(qkv, gone, vc)
    q = qkv[:, : nh * hd].view(n, nh, hd).double().to(DEV)
    s = torch.einsum("nhd,kd->nhk", q, kc[table, 0, 0].double()) * hd ** -0.5
    pos = torch.arange(L - n, L, device=DEV)
    hidden = (torch.arange(L, device=DEV)[None] > pos[:, None]) | (torch.arange(L, device=DEV)[None] == key)
    ref = torch.softmax(s.masked_fill(hidden[:, None], -math.inf), dim=2) @ vc[table, 0, 0].double()
    torch.testing.assert_close(got.double(), ref, rtol=1.6e-2, atol=1.2e-2)
    # the last token's value, which only its own row sees
    large = vc.clone()
    large[table[L - 1], 0, 0] = 3.0e38
    assert torch.equal(run(qkv, kc, large)[: n - 1], want[: n - 1])


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("nh,nkv,ps,window,single", [(3, 1, 16, None, False), (4, 2, 5, None, True), (5, 1, 8, 1350, False), (1, 1, 16, None, False)])
def test_lone_heads_with_many_key_tiles(ops, hd, nh, nkv, ps, window, single):
    """Around the number of key tiles from which a lone head's go to two units (heads of 128), odd and even numbers of them."""
    lens_kv = [1344, 1345, 1408, 1409, 1530, 2047]
    lens_q = [2, 130, 3, 2, 70, 5]
    got, want = run_mma_attention(ops, lens_q, lens_kv, nh, nkv, hd, ps, window, seed=hd + nh, tc=True, single_heads=single)
    torch.testing.assert_close(got, want, rtol=1.6e-2, atol=1.2e-2)  # the bound of the other tests of these kernels
