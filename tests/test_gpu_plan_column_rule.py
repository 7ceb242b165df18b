"""Blocks of real columns on row plans on both sides of the grouping rule: groups and
windows below and above two blocks per SM, a last group of one column alone or in a
group, of two and three, with padded leading dimensions and accumulation.  Grouped,
alone or one by one, the columns are those of single products bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def field_chain(ek, L, N):
    bond = ek.spin((1.0, "xx"), (1.0, "yy"), (0.8, "zz"))
    h = np.random.default_rng(4).uniform(-1, 1, L)
    return ek.operator([bond] * (L - 1) + [v * ek.spin("z") for v in h],
                       [[i, i + 1] for i in range(1, L)] + [[i] for i in range(1, L + 1)],
                       ek.ProjectedBasis(L=L, N=N))


@pytest.mark.parametrize("L,N", [(12, 6), (16, 8), (18, 9), (20, 10)])
@pytest.mark.parametrize("dt", ["float64", "float32"])
def test_block_equals_columns(ek, L, N, dt):
    import torch
    H = field_chain(ek, L, N)
    D, dt = H.size(1), getattr(torch, dt)
    for nv in (8, 9, 10, 11, 16, 17, 33):
        g = torch.Generator(device="cuda").manual_seed(nv)
        x = torch.randn((nv, D + 3), dtype=dt, device="cuda", generator=g)[:, :D].t()
        y = torch.randn((nv, D + 7), dtype=dt, device="cuda", generator=g)[:, :D].t()
        torch.cuda.synchronize()
        cols = [c for c in range(nv) if c < 2 or c >= nv - 4]
        xc = {c: x[:, c].clone() for c in cols}
        torch.cuda.synchronize()
        one = {c: H * xc[c] for c in cols}
        out = H * x
        assert all(torch.equal(out[:, c], one[c]) for c in cols)
        acc = torch.empty((nv, D + 7), dtype=dt, device="cuda")[:, :D].t()
        acc.copy_(y)
        torch.cuda.synchronize()
        ek.mul_(acc, H, x)
        torch.cuda.synchronize()
        assert all(torch.equal(acc[:, c], y[:, c] + one[c]) for c in cols)
