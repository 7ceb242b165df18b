"""The Pauli-string form has the matrix elements of the row kernel: an element that
is zero does not read the vector (infinities and NaN stay in the rows that have an
element with them), and matrices whose entries the strings would round away run on
the row kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = 12


def operators():
    P, X = np.diag([1.0, 0.0]), np.array([[0.0, 1.0], [1.0, 0.0]])
    xx, yy = np.kron(X, X), np.fliplr(np.diag([-1.0, 1.0, 1.0, -1.0]))
    fields = [(np.linspace(0.4, 0.9, L)[i] * X, [i + 1]) for i in range(L)]
    bonds = [[i, i + 1] for i in range(1, L)]
    hop = np.zeros((4, 4))
    hop[1, 2] = hop[2, 1] = 0.7
    return {
        "projected flips": [(np.kron(P, np.kron(X, P)), [i, i + 1, i + 2]) for i in range(1, L - 1)],
        "bonds of many strengths": [((0.3 + 0.1 * i) * hop, b) for i, b in enumerate(bonds)] + fields,
        "pair creation": [(xx + 0.3 * yy, b) for b in bonds],
        "three couplings on one flip": [(np.kron(P, 0.1 * X), [1, 5]), (np.kron(P, 0.3 * X), [2, 5]),
                                        (np.kron(P, 0.7 * X), [3, 5])],
        "wide entries": [(np.array([[0, 0, 0, 1e10], [0, 0, 1e-10, 0], [0, 1e-10, 0, 0],
                                    [1e10, 0, 0, 0]]), b) for b in bonds[::3]],
    }


def dense(terms):
    H = np.zeros((2 ** L, 2 ** L))
    idx = np.arange(2 ** L)
    for m, sites in terms:
        k = len(sites)
        c = sum(((idx >> (L - s)) & 1) << (k - 1 - q) for q, s in enumerate(sites))
        for x in range(2 ** k):
            flip = sum(((x >> (k - 1 - q)) & 1) << (L - s) for q, s in enumerate(sites))
            H[idx ^ flip, idx] += m[c ^ x, c]
    return H


def build(ek, terms):
    return ek.operator([m for m, _ in terms], [s for _, s in terms], ek.TensorBasis(L=L))


@pytest.mark.parametrize("kind", list(operators()))
def test_each_entry_to_rounding(ek, kind):
    """y_i against its own row's sum of magnitudes: a row of n products of entries
    right to 8 eps."""
    terms = operators()[kind]
    H, Hd = build(ek, terms), dense(terms)
    x = np.random.default_rng(0).standard_normal(2 ** L)
    scale = np.abs(Hd) @ np.abs(x)
    for dt, eps in ((np.float64, 2.3e-16), (np.complex128, 2.3e-16), (np.float32, 1.2e-7)):
        xt = x.astype(dt)
        y = H * xt
        ref = Hd @ xt.astype(np.complex128 if dt == np.complex128 else np.float64)
        assert np.all(np.abs(y - ref) <= 32 * eps * scale)


@pytest.mark.parametrize("kind", list(operators()))
@pytest.mark.parametrize("dt", [np.float64, np.complex128, np.float32, np.complex64])
def test_non_finite_entries_stay_in_their_rows(ek, kind, dt):
    terms = operators()[kind]
    H, Hd = build(ek, terms), dense(terms)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(2 ** L).astype(dt)
    at = rng.choice(2 ** L, 5, replace=False)
    x[at] = np.array([np.inf, -np.inf, np.nan, np.inf, np.nan], dtype=dt)
    with np.errstate(all="ignore"):
        y = H * x
    touched = (Hd[:, at] != 0).any(axis=1)
    touched[at] = True  # (the diagonal is always multiplied)
    assert np.isfinite(y[~touched]).all()
