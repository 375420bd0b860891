"""Passes over rows in 16-byte pieces against float64, at the edges of their rules: parts of a warp's and a block's sizes, parts and
strides that take single values, gates before and behind the norm, weights used round and round; SiLU columns that end inside a
thread's four pieces."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("groups,part", [(3, 4), (16, 128), (2, 132), (1, 512), (1, 516), (2, 2048), (1, 4096), (1, 8192), (1, 8196),
                                         (2, 130), (1, 7)])
@pytest.mark.parametrize("gate_first,silu,odd", [(True, False, 0), (False, True, 0), (False, False, 0), (False, True, 1)])
def test_gated_group_norm(dtype, groups, part, gate_first, silu, odd):
    from tokasaurus_b200.kernels import ops

    g = torch.Generator().manual_seed(part + groups)
    rows, H = 5, groups * part
    both = torch.randn(rows, 2 * H + odd, generator=g).to(DEV)
    y, gate = both[:, :H], both[:, H + odd:]  # (odd: the gates start between 16-byte pieces, or the rows do)
    w = torch.rand(part if part % 4 == 0 else H, generator=g).to(DEV) + 0.5
    out = torch.full((rows + 1, H), 7.0, dtype=dtype, device=DEV)
    kw = {} if gate_first else dict(silu_gate=silu)
    ops.gated_group_norm(y, gate, w, out[:rows], groups, 1e-5, gate_first=gate_first, **kw)
    v, gg = y.double().view(rows, groups, part), gate.double().view(rows, groups, part)
    if gate_first:
        v = v * gg * torch.sigmoid(gg)
    n = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double().repeat(H // w.numel()).view(groups, part)
    if not gate_first:
        n = n * torch.sigmoid(gg) * (gg if silu else 1)
    n = n.view(rows, H)
    # float32: a few roundings of each value and of the statistics; bfloat16: one rounding of the result
    bound = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -19) * n.abs() + 1e-12
    assert ((out[:rows].double() - n).abs() <= bound).all() and (out[rows] == 7).all()


@pytest.mark.parametrize("cols,stride", [(4, 8), (1030, 1040), (1028, 1032), (6144, 8192), (4100, 4101), (8192, 8192)])
def test_silu_cols(cols, stride):
    from tokasaurus_b200.kernels import ops

    x = torch.randn(3, stride, generator=torch.Generator().manual_seed(cols)).to(DEV) * 4
    want = x.double()
    want[:, :cols] = want[:, :cols] * torch.sigmoid(want[:, :cols])
    ops.silu_cols(x, cols, ops.decay_recurrence_defines(128, 128, 32))
    assert ((x.double() - want).abs() <= 2.0 ** -20 * want.abs() + 1e-30).all()
