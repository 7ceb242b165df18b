"""The device tridiagonal eigenvalues behind the batched Lanczos: the values a
run returns are the lowest ones of the recurrence it returns.

Sizes: orders at the edges of the kernel's eight-row groups (1, 7, 8, 9) and of
its 1,024-row shared-memory stage (1,023 .. 1,030), and one to nine eigenvalues
(one to eight thread groups, and a second pass).  Tolerance: a Sturm count is
exact for a matrix whose entries moved by a few eps (4 eps |T|), the interval
ends at eps |T|, and numpy's own solver adds a small multiple of the same:
32 eps |T| with |T| <= max|a| + 2 max|b|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(ek, L, seed):
    h = np.random.default_rng(seed).uniform(-3, 3, L)
    bond = ek.spin((1.0, "xx"), (1.0, "yy"), (1.0, "zz"))
    return ek.operator([bond] * (L - 1) + [v * ek.spin("z") for v in h],
                       [[i, i + 1] for i in range(1, L)] + [[i] for i in range(1, L + 1)],
                       ek.ProjectedBasis(L=L, N=L // 2))


def lowest(a, b, nev):
    b = b[: len(a) - 1]
    return np.linalg.eigvalsh(np.diag(a) + np.diag(b, 1) + np.diag(b, -1))[:nev]


@pytest.mark.parametrize("steps", [1, 7, 8, 9, 70, 1023, 1024, 1025, 1030])
@pytest.mark.parametrize("nev", [1, 3, 9])
def test_values_of_the_returned_recurrence(ek, steps, nev):
    if steps > 100 and nev == 3:
        pytest.skip("the long recurrences once with one and once with two passes")
    H = chain(ek, 14 if steps > 100 else 10, 3)
    v0 = np.random.default_rng(steps).standard_normal(H.size(1))
    ev, info, a, b = ek.lanczos_e0(H, v0, m=steps, nev=nev, return_coeffs=True)
    n = min(nev, info["steps"])
    assert info["steps"] == steps
    tol = 32 * np.finfo(float).eps * (np.abs(a).max() + 2 * np.abs(b).max())
    assert np.all(np.abs(ev[:n] - lowest(a, b, n)) <= tol)
    assert np.all(np.isnan(ev[n:]))


@pytest.mark.parametrize("nev", [1, 2, 5])
def test_uneven_batch_stops_where_each_operator_converges(ek, nev):
    """The check on the device: every operator's values are within the stop
    tolerance of its dense spectrum, whichever step it stopped at."""
    ops = [chain(ek, L, 10 + L) for L in (6, 8, 9, 11, 7)]
    ev, info = ek.batch_lanczos_e0(ops, m=150, nev=nev, tol=1e-13, check_every=4)
    assert info["steps"] < 150
    for op, e in zip(ops, ev):
        ref = np.linalg.eigvalsh(op.todense())[:nev]
        assert np.allclose(e, ref, rtol=0, atol=1e-10 * abs(ref[0]))
