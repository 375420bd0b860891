"""Work items of the split-key attention in the order in which their blocks start: the same items give the same bits
whatever the order, and the planner's order names each item once, the longest first."""

import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from tokasaurus_b200.parts.attention import plan_attention
from tokasaurus_b200.parts.rope import RotaryEncoding

DEV = "cuda:0"


def plan_of(lens_kv, window, blocks_per_item, slots):
    host = SimpleNamespace(seq_q_len=np.ones(len(lens_kv), dtype=np.int32), seq_kv_len=np.asarray(lens_kv, dtype=np.int32))
    return plan_attention(host, window, blocks_per_item=blocks_per_item, slots=slots)


@pytest.mark.parametrize("lens_kv,window,slots", [([900, 70, 1, 3000, 64, 129], None, 64), ([500] * 9, None, 8), ([500, 40, 700], 300, 16),
                                                  (list(range(1, 4000, 61)), None, 592)])
def test_order_of_the_items(lens_kv, window, slots):
    plan = plan_of(lens_kv, window, 8, slots)
    n = int(plan["counts"][0])
    assert int(plan["counts"][8]) == int(8 * n > slots)
    if not plan["counts"][8]:
        return
    items, order = plan["items"][: 3 * n].reshape(-1, 3), plan["item_order"][: 4 * n].reshape(-1, 4)
    assert sorted(order[:, 3].tolist()) == list(range(n))
    assert (items[order[:, 3]] == order[:, :3]).all()
    span = np.minimum(np.asarray(lens_kv), window or 1 << 30)[order[:, 0]]
    keys = np.minimum(order[:, 2], span - order[:, 1])
    assert (keys > 0).all() and (np.diff(keys) <= 0).all()


def test_unequal_requests_end_sooner_cut_at_the_nearest_share():
    """32 requests of 512 to 4,096 keys over 37 slots: cut at the share below, most stay whole and the longest one is what
    a slot ends with beside another; requests of one length are cut as before."""
    lens = [512 + 3584 * ((i * 29) % 64) // 63 for i in range(32)]
    slots = 296
    plan = plan_of(lens, None, 8, slots)
    items = plan["item_order"].reshape(-1, 4)
    assert int(plan["counts"][0]) == len(items) and items[:, 2].max() < 0.8 * max(lens)
    assert slots // 8 < len(items) <= slots // 8 + 32


@pytest.mark.parametrize("slots,ordered", [(64, True), (4096, False)])
def test_order_of_the_wanted_rows(slots, ordered):
    """The wanted rows' items of more than a wave have an order of their own, also padded to a graph's sizes."""
    from tokasaurus_b200.kernels import ops
    from tokasaurus_b200.parts.attention import AttentionPlanning

    lens_q, lens_kv = [5, 1, 300, 7, 64], [700, 40, 3000, 7, 1200]
    ends = np.cumsum(lens_q) - 1
    positions = np.concatenate([np.arange(n - q, n) for q, n in zip(lens_q, lens_kv)])
    host = SimpleNamespace(seq_q_len=np.asarray(lens_q, dtype=np.int32), seq_kv_len=np.asarray(lens_kv, dtype=np.int32),
                           logit_rows=ends.astype(np.int32), token_ids=positions, positions=positions,
                           token_seq=np.repeat(np.arange(5), lens_q), table_indptr=[np.arange(6)])
    plan = plan_attention(host, None, blocks_per_item=8, slots=slots)
    n, word = int(plan["counts"][3]), int(plan["counts"][10])
    assert word == n | (0 if ordered else ops.ITEMS_LISTED) and ordered == (8 * n > slots)
    grown = AttentionPlanning.pad_plan(None, plan, dict(items=50, dec=9, tiles=20, row_items=n + 7, rows=6))
    assert grown["row_item_order"].shape[0] == 4 * (n + 7)
    if ordered:
        items, order = plan["row_items"][: 3 * n].reshape(-1, 3), grown["row_item_order"][: 4 * n].reshape(-1, 4)
        assert sorted(order[:, 3].tolist()) == list(range(n)) and (items[order[:, 3]] == order[:, :3]).all()
        keys = np.minimum(order[:, 2], np.asarray(lens_kv)[order[:, 0]] - order[:, 1])
        assert (keys > 0).all() and (np.diff(keys) <= 0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("hd,nh,nkv,ps", [(64, 32, 8, 16), (128, 24, 8, 16), (48, 6, 3, 4), (80, 34, 2, 16), (256, 4, 1, 16)])
@pytest.mark.parametrize("tma", [True, False])
@pytest.mark.parametrize("fused", [True, False])
def test_order_gives_the_same_bits(hd, nh, nkv, ps, tma, fused):
    from test_kernels_gpu import i32, make_paged

    from tokasaurus_b200.kernels import ops

    lens_kv = [1030, 1, 65, 700, 256, 64, 333]
    B = len(lens_kv)
    kc, vc, indptr, pages, _, _ = make_paged(torch.bfloat16, B, lens_kv, nkv, hd, ps, sum(-(-n // ps) for n in lens_kv) + 3, seed=hd)
    blocks = nkv * ((nh // nkv + 15) // 16)
    plan = plan_of(lens_kv, None, blocks, 8 * blocks)
    assert plan["counts"][8] == 1
    n_items = int(plan["counts"][0])
    g = torch.Generator().manual_seed(hd)
    qkv = torch.randn(B, (nh + 2 * nkv) * hd, generator=g).to(torch.bfloat16).to(DEV)
    c, status = i32(plan["counts"]), torch.zeros(1, dtype=torch.int32, device=DEV)
    rot = hd if hd % 4 == 0 else 0
    inv = RotaryEncoding(rot, 10000.0).inv_freq().to(DEV)

    def run(order):
        k, v, out = kc.clone(), vc.clone(), torch.full((B, nh * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
        args = (qkv, k, v, i32(list(range(B))), i32(lens_kv), indptr, pages, i32(plan["items"]), c[0:1], n_items + 5 * (order is None),
                i32(plan["dec_seqs"]), i32(plan["dec_item_start"]), c[1:2], B, out, nh, nkv, hd, ps, 1 / math.sqrt(hd), None)
        pad = torch.zeros(15, dtype=torch.int32, device=DEV)
        args = args[:7] + (torch.cat([args[7], pad]),) + args[8:]
        entry = torch.cat([i32(plan["item_entry"]), pad])
        if fused:
            ops.attn_decode_rope_mma(*args, inv, rot, True, status, item_entry=entry, tma=tma, item_order=order)
        else:
            ops.attn_decode_mma(*args, item_entry=entry, tma=tma, status=status, item_order=order)
        return out, k, v

    want, got = run(None), run(i32(plan["item_order"]))
    assert int(status) == 0 and not want[0].isnan().any()
    for a, b in zip(want, got):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.gpu
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("hd,nh,nkv", [(64, 32, 8), (128, 24, 8), (80, 34, 2)])
def test_a_grid_larger_than_the_items_serves_both_orders(hd, nh, nkv, fused):
    """The launch of a step graph: more places than items, and a word on the device that says whether this step is ordered."""
    from test_kernels_gpu import i32, make_paged

    from tokasaurus_b200.kernels import ops

    ps, lens_kv = 16, [1030, 1, 65, 700, 256, 64, 333]
    B, blocks = len(lens_kv), nkv * ((nh // nkv + 15) // 16)
    kc, vc, indptr, pages, _, _ = make_paged(torch.bfloat16, B, lens_kv, nkv, hd, ps, sum(-(-n // ps) for n in lens_kv) + 3, seed=hd)
    plan = plan_of(lens_kv, None, blocks, 8 * blocks)
    n_items = int(plan["counts"][0])
    cap = n_items + 9
    grown = lambda x, n: i32(np.concatenate([x[:n], np.zeros(n // n_items * cap - n, dtype=np.int32)]))  # noqa: E731
    items, entry = grown(plan["items"], 3 * n_items), grown(plan["item_entry"], n_items)
    qkv = torch.randn(B, (nh + 2 * nkv) * hd, generator=torch.Generator().manual_seed(hd)).to(torch.bfloat16).to(DEV)
    c, status = i32(plan["counts"]), torch.zeros(1, dtype=torch.int32, device=DEV)
    rot = hd if hd % 4 == 0 else 0
    inv = RotaryEncoding(rot, 10000.0).inv_freq().to(DEV)

    def run(order, n):
        k, v, out = kc.clone(), vc.clone(), torch.full((B, nh * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
        args = (qkv, k, v, i32(list(range(B))), i32(lens_kv), indptr, pages, items, i32([n]), cap, i32(plan["dec_seqs"]),
                i32(plan["dec_item_start"]), c[1:2], B, out, nh, nkv, hd, ps, 1 / math.sqrt(hd), None)
        if fused:
            ops.attn_decode_rope_mma(*args, inv, rot, True, status, item_entry=entry, item_order=order)
        else:
            ops.attn_decode_mma(*args, item_entry=entry, status=status, item_order=order)
        return out.view(torch.int16), k.view(torch.int16), v.view(torch.int16)

    want = run(None, n_items)
    assert int(status) == 0 and not want[0].view(torch.bfloat16).isnan().any()
    order = grown(plan["item_order"], 4 * n_items)
    for got in (run(order, n_items), run(torch.zeros_like(order), n_items | ops.ITEMS_LISTED), run(None, n_items | ops.ITEMS_LISTED)):
        assert all(torch.equal(a, b) for a, b in zip(want, got))
