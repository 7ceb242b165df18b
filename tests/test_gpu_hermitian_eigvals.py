"""Squared Schmidt values from the shared-memory tridiagonalisation: every order
a chain can cut (1 to 1,024, and 2,048, which real matrices no longer fit),
square and flat Schmidt matrices, real and complex, product states (rank one),
states of very small and large norm.  A backward stable solver is within a
modest multiple of n eps of the largest value; squares below n eps of it are
returned as zero: 8 n eps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(ek, v, L, nA, scale=1.0):
    s = ek.ent_spec(v * scale, list(range(1, nA + 1)), ek.TensorBasis(L=L)) / scale
    ref = np.linalg.svd(v.reshape(2 ** nA, -1), compute_uv=False)
    n = len(ref)
    assert len(s) == n and np.all(np.diff(s) <= 0)
    assert np.abs(s ** 2 - ref ** 2).max() <= 8 * n * np.finfo(float).eps * ref[0] ** 2


@pytest.mark.parametrize("L,nA", [(1, 0), (2, 1), (4, 2), (6, 3), (9, 4), (11, 5), (12, 6), (13, 7),
                                  (16, 8), (18, 9), (20, 10), (21, 10), (22, 11)])
@pytest.mark.parametrize("cx", [False, True])
def test_random_states(ek, L, nA, cx):
    rng = np.random.default_rng(L)
    v = rng.standard_normal(2 ** L) + (1j * rng.standard_normal(2 ** L) if cx else 0)
    check(ek, v / np.linalg.norm(v), L, nA)


@pytest.mark.parametrize("scale", [1.0, 1e-120, 1e120])
def test_rank_one_and_scales(ek, scale):
    rng = np.random.default_rng(1)
    a, b = rng.standard_normal(64), rng.standard_normal(64) + 1j * rng.standard_normal(64)
    v = np.kron(a, b)
    v /= np.linalg.norm(v)
    check(ek, v, 12, 6, scale)
    w = np.zeros(2 ** 10)
    w[5] = 1.0
    check(ek, w, 10, 5, scale)
