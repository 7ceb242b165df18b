"""Gram matrices with columns of tiny entries (1e-150 to 1e-170) beside entries of size
one, as nearly decoupled rows of a Schmidt matrix give: the squares of such a column
leave the range of doubles, the rest of the spectrum must not notice.  8 n eps of the
largest value, as for every other state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nA", [3, 6, 8])
@pytest.mark.parametrize("tiny", [1e-150, 1e-158, 1e-160, 1e-161, 1e-162, 1e-170])
@pytest.mark.parametrize("cx", [False, True])
def test_tiny_rows(ek, nA, tiny, cx):
    L, n = 2 * nA, 2 ** nA
    rng = np.random.default_rng(nA)
    M = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cx else 0)
    for r in (0, 1, n // 2):
        M[r] *= tiny
    M /= np.linalg.norm(M)
    s = ek.ent_spec(np.ascontiguousarray(M).ravel(), list(range(1, nA + 1)), ek.TensorBasis(L=L))
    ref = np.linalg.svd(M, compute_uv=False)
    assert np.abs(s ** 2 - ref ** 2).max() <= 8 * n * np.finfo(float).eps * ref[0] ** 2
