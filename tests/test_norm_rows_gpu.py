"""The norm of many rows: a warp (two beyond 2,048 numbers) a row, at the edges of its range and of its blocks."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("rows,H", [(592, 1024), (593, 1028), (595, 2044), (597, 2048), (599, 2052), (601, 3000), (1030, 4096), (594, 4092),
                                    (887, 1024), (889, 1028), (891, 1536), (1479, 2048), (1483, 2044), (1776, 2048), (1777, 1540)])
@pytest.mark.parametrize("form", ["none", "bfloat16", "slice"])
def test_add_rmsnorm_of_many_rows(rows, H, form):
    from tokasaurus_b200.kernels import ops

    g = torch.Generator().manual_seed(rows + H)
    x = (torch.randn(rows, H, generator=g) * 3).to(DEV)
    d = torch.randn(rows, H, generator=g).to(DEV)
    delta = dict(none=None, bfloat16=d.bfloat16(), slice=d)[form]
    w = (torch.rand(H, generator=g) + 0.5).to(DEV)
    guard = torch.full((rows + 1, H), 7.0, device=DEV)
    guard[:rows] = x
    out = torch.full((rows + 1, H), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.add_rmsnorm(guard[:rows], delta, w, 1e-5, out[:rows])
    y = x if delta is None else x + delta.float()
    assert torch.equal(guard[:rows], y) and (guard[rows] == 7).all() and (out[rows] == 7).all()
    want = y.double() * torch.rsqrt(y.double().pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    # one rounding to 8 bits, and float32 statistics behind it
    torch.testing.assert_close(out[:rows].double(), want, rtol=2.0 ** -8, atol=1e-30)
