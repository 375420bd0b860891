"""Routed experts whose row tiles are fetched and stored in part: token counts around whole pieces of eight and around a tile,
every token choosing the same experts (a tile as full as it gets), weights on the input, padding tokens that choose nothing."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


class Step:
    def __init__(self, token_seq):
        self.n_tokens, self.token_seq = token_seq.numel(), token_seq
        self.status = torch.zeros(1, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("expert,weigh_input", [("silu_gated", False), ("silu_gated", True), ("gelu", False)])
@pytest.mark.parametrize("T", [6, 8, 9, 16, 63, 64, 120, 121, 128, 129, 300])
def test_routed_experts_of_any_number_of_tokens(T, expert, weigh_input):
    from tokasaurus_b200.engine.runtime import Runtime
    from tokasaurus_b200.parts import RoutedExperts

    W, I, E, top = 256, 128, 6, 2
    names = (lambda e: (f"g{e}", f"u{e}", f"d{e}")) if expert == "silu_gated" else (lambda e: (f"u{e}", f"d{e}"))
    part = RoutedExperts(W, I, E, top, "r", None, names, expert=expert, weigh_input=weigh_input, out_dtype=torch.float32)
    g = torch.Generator().manual_seed(T)
    w = {"r": torch.randn(E, W, generator=g)}
    for e in range(E):
        for n in names(e):
            w[n] = torch.randn(*((W, I) if n[0] == "d" else (I, W)), generator=g).mul((I if n[0] == "d" else W) ** -0.5).bfloat16()
    h = torch.randn(T, W, generator=g).bfloat16()
    if T % 3 == 0:  # every token like the first: two experts take them all
        h = (h[:1].float() + 0.01 * h.float()).bfloat16()
    part.bind({n: t.to(DEV) for n, t in w.items()}, Runtime.make(DEV, "bfloat16"))
    seq = torch.arange(T, dtype=torch.int32)
    seq[T // 2] = -1  # a padding token
    out = part.forward(Step(seq.to(DEV)), h.to(DEV)).double().cpu()
    x = h.double()
    vals, idx = torch.topk(x @ w["r"].double().T, top)
    share = torch.softmax(vals, -1)
    want = torch.zeros(T, W, dtype=torch.float64)
    for e in range(E):
        s = (share * (idx == e)).sum(-1, keepdim=True)
        z = x * s if weigh_input else x
        up = z @ w[f"u{e}"].double().T
        a = torch.nn.functional.silu(z @ w[f"g{e}"].double().T) * up if expert == "silu_gated" else torch.nn.functional.gelu(up)
        y = a @ w[f"d{e}"].double().T
        want += torch.where(s > 0, y if weigh_input else y * s, torch.zeros(()).double())
    live = seq >= 0
    # the inner values and each expert's output are rounded to bfloat16: 2^-9 of each, twice
    assert (out - want)[live].norm() <= 2.0 ** -7 * want[live].norm()
    assert ((out - want)[live].abs() <= 2.0 ** -5 * want[live].abs().amax(-1, keepdim=True)).all()


@pytest.mark.parametrize("T", [6, 9, 16, 40])
def test_a_table_that_names_an_expert_twice(T):
    """Experts chosen by token id: a table may name one expert several times, so a tile holds more rows than there are tokens."""
    from tokasaurus_b200.engine.runtime import Runtime
    from tokasaurus_b200.parts import RoutedExperts

    W, I, E, top, V = 256, 128, 5, 3, 50
    names = lambda e: (f"g{e}", f"u{e}", f"d{e}")  # noqa: E731
    part = RoutedExperts(W, I, E, top, None, None, names, out_dtype=torch.float32, table_name="t", vocab=V)
    g = torch.Generator().manual_seed(T)
    table = torch.randint(0, E, (V, top), generator=g, dtype=torch.int32)
    table[: V // 2] = 3  # half of all tokens: one expert, three times
    w = {"t": table}
    for e in range(E):
        for n in names(e):
            w[n] = torch.randn(*((W, I) if n[0] == "d" else (I, W)), generator=g).mul((I if n[0] == "d" else W) ** -0.5).bfloat16()
    h = torch.randn(T, W, generator=g).bfloat16()
    ids = torch.arange(T, dtype=torch.int32) % V
    part.bind({n: t.to(DEV) for n, t in w.items()}, Runtime.make(DEV, "bfloat16"))
    step = Step(torch.arange(T, dtype=torch.int32, device=DEV))
    step.token_ids, step.seq_slot, step.last_token = ids.to(DEV), torch.zeros(T, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    out = part.forward(step, h.to(DEV)).double().cpu()
    x, want = h.double(), torch.zeros(T, W, dtype=torch.float64)
    for e in range(E):
        share = (table[ids.long()] == e).sum(-1, keepdim=True) / top
        y = (torch.nn.functional.silu(x @ w[f"g{e}"].double().T) * (x @ w[f"u{e}"].double().T)) @ w[f"d{e}"].double().T
        want += share * y
    assert (out - want).norm() <= 2.0 ** -7 * want.norm()


@pytest.mark.parametrize("rows,tile_rows", [(1, 8), (8, 8), (9, 16), (120, 120), (128, 128)])
def test_clamped_units_on_short_tiles(rows, tile_rows):
    """The grouped product with the clamped unit in its epilogue: two groups, tiles of which only the first rows are anybody's; what is
    behind them is neither read nor written."""
    from tokasaurus_b200.kernels import ops

    K, N, limit, alpha = 256, 192, 1.5, 1.702
    g = torch.Generator().manual_seed(rows)
    a = torch.full((256, K), float("nan")).bfloat16()
    for t in range(2):
        a[128 * t:128 * t + tile_rows] = torch.randn(tile_rows, K, generator=g).bfloat16()
    gate, up = (torch.randn(2, N, K, generator=g).mul(K ** -0.5).bfloat16() for _ in range(2))
    w = torch.stack([ops.interleave_gate_up(gate[e].to(DEV), up[e].to(DEV)) for e in range(2)]).contiguous()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = ops.gemm_tcgen05_grouped(a.to(DEV), w, torch.tensor([1, 0], dtype=torch.int32, device=DEV), status, gated=True,
                                   clamp=(limit, alpha), tile_rows=tile_rows).double().cpu()
    assert int(status) == 0
    for t, e in ((0, 1), (1, 0)):
        x = a[128 * t:128 * t + rows].double()
        gv = (x @ gate[e].double().T).clamp(max=limit)
        uv = (x @ up[e].double().T).clamp(-limit, limit)
        want = gv * torch.sigmoid(alpha * gv) * (uv + 1)
        assert (out[128 * t:128 * t + rows] - want).abs().max() <= 2.0 ** -7 * want.abs().max()
