"""Gram-Schmidt twice with the second sweep delayed by one step: a run over the
whole space must return every eigenvalue, which it does only while all Krylov
vectors stay orthogonal to rounding.

Column counts pass the kernels' edges (groups of four columns; 32, 64 and 128
columns, where the warps stop splitting rows; the 128-column coefficient chunk),
with fewer rows than a warp up to some rows per block, real and complex, alone
and in an uneven batch.  A backward stable Lanczos gives the eigenvalues of T to
a modest multiple of eps |H|: 1e-12 relative to the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fields(ek, L, N, seed=1):
    h = np.random.default_rng(seed).uniform(-2, 2, L)
    bond = ek.spin((1.0, "xx"), (1.0, "yy"), (1.0, "zz"))
    return ek.operator([bond] * (L - 1) + [v * ek.spin("z") for v in h],
                       [[i, i + 1] for i in range(1, L)] + [[i] for i in range(1, L + 1)],
                       ek.ProjectedBasis(L=L, N=N))


def momentum(ek, L, N, k):
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2,
                              ek.TranslationalBasis(L=L, N=N, k=k))
    return H + ek.trans_inv_operator(ek.spin((0.31, "xx"), (0.31, "yy"), (0.17, "zz")), [1, 3],
                                     H.B)


@pytest.mark.parametrize("make", [
    lambda ek: fields(ek, 5, 1),        # 5 rows
    lambda ek: fields(ek, 9, 2),        # 36
    lambda ek: fields(ek, 12, 2),       # 66
    lambda ek: fields(ek, 9, 4),        # 126
    lambda ek: fields(ek, 10, 5),       # 252
    lambda ek: momentum(ek, 9, 4, 2),   # 14 rows, complex
    lambda ek: momentum(ek, 13, 5, 3),  # 99
    lambda ek: momentum(ek, 15, 5, 2),  # 200
])
def test_whole_space_gives_every_eigenvalue(ek, make):
    H = make(ek)
    D = H.size(1)
    v0 = np.random.default_rng(D).standard_normal(D)
    ev, info, a, b = ek.lanczos_e0(H, v0, m=D, nev=D, return_coeffs=True)
    assert info["steps"] == D
    ref = np.linalg.eigvalsh(H.todense())
    assert np.allclose(ev, ref, rtol=0, atol=1e-12 * np.abs(ref).max())


def test_whole_space_in_an_uneven_batch(ek):
    ops = [fields(ek, L, N, seed=L) for L, N in ((5, 1), (10, 5), (9, 2), (7, 3))]
    ev, _ = ek.batch_lanczos_e0(ops, m=252, nev=5)
    for op, e in zip(ops, ev):
        ref = np.linalg.eigvalsh(op.todense())
        assert np.allclose(e, ref[:5], rtol=0, atol=1e-12 * np.abs(ref).max())
