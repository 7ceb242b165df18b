"""Products on symmetry-group sectors: rows shared by sixteen or four lanes (few
rows) or held by one (many rows or columns), one-site rotations compared at the
zero-run tops (up to 27 sites, 28 to 32), generators that are no such rotation,
and the bond partition over the lanes at odd chain lengths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECTORS = [  # L, basis keywords
    (5, dict(N=2, k=2)),
    (8, dict(N=4, k=0, p=1, z=-1)),
    (9, dict(N=4, k=0, p=-1)),
    (12, dict(N=6, p=-1, z=1)),          # no rotation among the generators
    (12, dict(N=6, k=1, a=2)),           # two-site cell
    (14, dict(k=7, z=1)),                # no charge
    (27, dict(N=3, k=4)),                # last length with the shift in spare bits
    (28, dict(N=3, k=14, p=1)),
    (32, dict(N=3, k=5)),
]


@pytest.mark.parametrize("L,kw", SECTORS)
def test_group_product_matches_oracle(ek, O, L, kw):
    B, Bo = ek.basis(L=L, **kw), O.basis(L=L, **kw)
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2, B)
    Ho = O.trans_inv_operator(O.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2, Bo)
    D = B.size(1)
    rng = np.random.default_rng(L)
    x = rng.standard_normal(D) + 1j * rng.standard_normal(D)
    y = H * x
    ref = Ho.mul(x)
    # products of at most 2 L entries: 1e-13 is some 30 roundings of the row sum
    assert np.linalg.norm(y - ref) <= 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("lanes", [4, 1])
def test_shared_and_single_lane_rows_agree(ek, lanes):
    """The same sector as one column (sixteen lanes a row) and inside a block
    wide enough for four lanes or one per row."""
    B = ek.basis(L=18, N=9, k=0, p=1, z=1)
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (1.0, "zz")), 2, B)
    D = B.size(1)
    fit = 2 * 148 * 2048
    ncol = (fit // (16 * D) if lanes == 4 else fit // (4 * D)) + 1
    X = np.asfortranarray(np.random.default_rng(0).standard_normal((D, ncol)))
    Y = H * X
    for c in (0, ncol // 2, ncol - 1):
        y = H * np.ascontiguousarray(X[:, c])
        assert np.linalg.norm(Y[:, c] - y) <= 1e-14 * np.linalg.norm(y)


@pytest.mark.parametrize("L,N,k,p", [(7, 3, 2, None), (20, 10, 3, None), (27, 3, 5, None),
                                     (28, 3, 9, None), (32, 3, 7, None), (12, 6, 6, -1),
                                     (28, 3, 0, 1), (31, 3, 0, -1)])
def test_shift_of_the_first_minimum(ek, O, L, N, k, p):
    """index() positions and coefficients, periodic states among them."""
    if p is None:
        B, Bo = ek.TranslationalBasis(L=L, N=N, k=k), O.translational(L, k=k, N=N)
    else:
        B = ek.TranslationParityBasis(L=L, N=N, k=k, p=p)
        Bo = O.transparity(L, k=k, p=p, N=N)
    rng = np.random.default_rng(L)
    ones = L - N
    sites = [rng.choice(L, ones, replace=False) for _ in range(400)]
    states = np.array([sum(1 << int(v) for v in q) for q in sites], dtype=np.uint64)
    pos, coeff = B.index_states(states)
    for s, q, c in zip(states, pos, coeff):
        cr, qr = Bo.index([(int(s) >> (L - 1 - i)) & 1 for i in range(L)])
        assert q == (qr if cr != 0 else 0)
        assert cr == 0 or c == cr
