"""Eigenvalue steps between the steps of a block Lanczos: T's blocks are brought into
their final form in place, once each, so a run checked often ends with the values of
one checked at the end only; operators whose space closes early among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sector(ek, L, N, k):
    return ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.6, "zz")), 2,
                                 ek.TranslationalBasis(L=L, N=N, k=k))


@pytest.mark.parametrize("every", [1, 2, 5, 9])
@pytest.mark.parametrize("block", [8, 16, 24])
def test_checked_often_or_once(ek, every, block):
    ops = [sector(ek, 14, 7, k) for k in (0, 3)] + [sector(ek, 15, 6, 2)]
    m = 9
    once, _ = ek.block_lanczos(ops, block=block, m=m, nev=3, tol=0.0)
    # a tolerance no run meets: every check happens, none stops
    often, info = ek.block_lanczos(ops, block=block, m=m, nev=3, tol=1e-300, check_every=every)
    assert info["steps"] == m
    assert np.array_equal(once, often, equal_nan=True)


def test_closed_space_among_running_ones(ek):
    H, G = sector(ek, 14, 7, 1), sector(ek, 14, 7, 2)
    w, V = np.linalg.eigh(H.todense())
    rng = np.random.default_rng(2)
    x = V[:, :20] @ (rng.standard_normal((20, 8)) + 1j * rng.standard_normal((20, 8)))
    y = rng.standard_normal((G.size(1), 8)) + 1j * rng.standard_normal((G.size(1), 8))
    once, a = ek.block_lanczos([H, G], [x, y], block=8, m=12, nev=2)
    often, b = ek.block_lanczos([H, G], [x, y], block=8, m=12, nev=2, tol=1e-300, check_every=3)
    assert a["breakdowns"] == b["breakdowns"] == 1
    assert np.array_equal(once, often, equal_nan=True)
