"""Where the strings stop: dense terms of three and four sites hold 36 to 256 strings
against 8 or 16 entries a column, and run on the row kernel; fields keep the strings.
Both sides of the rule against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = 9


def dense(k, n, cx):
    rng = np.random.default_rng(10 * k + n)
    mats = []
    for _ in range(n):
        a = rng.standard_normal((2 ** k, 2 ** k))
        if cx:
            a = a + 1j * rng.standard_normal((2 ** k, 2 ** k))
        mats.append((a + a.conj().T) / 2)
    return mats, [list(range(i + 1, i + k + 1)) for i in range(n)]


def fields(k, n, cx):
    rng = np.random.default_rng(n)
    x, y = np.array([[0, 1], [1, 0]]), np.array([[0, -1j], [1j, 0]])
    mats = [h * x + (0.3 * y if cx else 0) for h in rng.uniform(0.5, 1, n)]
    return mats, [[i + 1] for i in range(n)]


@pytest.mark.parametrize("make,k,n,strings", [
    (fields, 1, 1, True), (fields, 1, 9, True),
    (dense, 2, 8, False), (dense, 3, 1, False), (dense, 3, 7, False),
    (dense, 4, 1, False), (dense, 4, 2, False), (dense, 4, 6, False),
])
@pytest.mark.parametrize("cx", [False, True])
def test_dense_terms_run_on_the_row_kernel(ek, O, make, k, n, strings, cx):
    mats, inds = make(k, n, cx)
    H = ek.operator(mats, inds, ek.TensorBasis(L=L))
    ref = O.operator(mats, inds, O.tensor(L))
    if strings:
        H.configure_("fast")
    else:
        with pytest.raises(ek.EDKError, match="fast kernel does not apply"):
            H.configure_("fast")
    rng = np.random.default_rng(0)
    x = rng.standard_normal(2 ** L) + 1j * rng.standard_normal(2 ** L)
    y, r = H * x, ref.mul(x)
    assert np.linalg.norm(y - r) <= 1e-14 * np.linalg.norm(r)


def test_complex_fields_of_a_large_space_keep_the_strings(ek):
    mats, inds = fields(1, 17, True)
    ek.operator(mats, inds, ek.TensorBasis(L=17)).configure_("fast")
