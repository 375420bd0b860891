"""Decays of gated linear attention for many tokens: the tiled kernel gives the bits of the kernel for few tokens."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


# the last column tile with 80, 127, 5 and all 128 columns, one with two (64 and fewer: the second half of every thread has none)
@pytest.mark.parametrize("T,C,rank,off", [(1100, 2000, 64, 8), (1089, 2047, 17, 3), (2561, 1925, 100, 4), (1153, 1920, 33, 0), (8321, 130, 33, 0)])
def test_tiles_give_the_same_bits(T, C, rank, off):
    from tokasaurus_b200.kernels import ops

    tiles, sms = -(-T // 64) * -(-C // 128), torch.cuda.get_device_properties(0).multi_processor_count
    assert 4 * tiles >= 7 * sms if rank <= 64 else tiles >= 4 * sms  # the tiled kernel's calls
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
    for r0 in range(0, T, 320):  # too few tiles
        pp, ff = gates(proj[r0:r0 + 320].contiguous())
        assert torch.equal(ff, f[r0:r0 + 320]) and torch.equal(pp, p[r0:r0 + 320])
