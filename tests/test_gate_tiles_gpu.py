"""Decays of gated linear attention for many tokens: the tiled kernel gives the bits of the kernel for few tokens."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("T,C,rank,off", [(650, 2000, 64, 8), (641, 2047, 17, 3), (704, 1920, 100, 4), (2500, 130, 33, 0)])
def test_tiles_give_the_same_bits(T, C, rank, off):
    from tokasaurus_b200.kernels import ops

    g = torch.Generator().manual_seed(T)
    width = off + C + rank + 5
    proj = torch.randn(T, width, generator=g).to(DEV)
    a2t, bias = torch.randn(rank, C, generator=g).to(DEV) * 0.3, torch.randn(C, generator=g).to(DEV)
    defines = ops.decay_recurrence_defines(64, 64)

    def gates(rows):
        p, f = rows.clone(), torch.full((rows.shape[0], C), float("nan"), device=DEV)
        ops.gla_gates(p, off + C, rank, a2t, bias, 16.0, f, off, C, 0.3, defines)
        return p, f

    p, f = gates(proj)
    want = torch.sigmoid(proj[:, off + C:off + C + rank].double() @ a2t.double() + bias.double()) ** (1 / 16.0)
    # a sum of `rank` terms of about 0.3 rounds to 1e-6, which the root divides by 16, and every function to 2 units in the last place
    torch.testing.assert_close(f.double(), want, rtol=2e-6, atol=0)
    for r0 in range(0, T, 40):  # 40 tokens: fewer tiles than SMs
        pp, ff = gates(proj[r0:r0 + 40].contiguous())
        assert torch.equal(ff, f[r0:r0 + 40]) and torch.equal(pp, p[r0:r0 + 40])
