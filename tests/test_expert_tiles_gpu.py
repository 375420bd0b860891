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
