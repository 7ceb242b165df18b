"""Hashed momentum sectors large enough for canonicalisation at the zero-run tops (512
rows per SM): shift counted in spare bits (up to 27 sites) and apart (28 to 32).
index() against the oracle, with random states, one bit away from periodic ones and
the periodic ones themselves; products on the hash, as a block and on the
materialised matrix against the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SECTORS = [(24, 12, 12), (25, 10, 3), (28, 8, 5), (32, 7, 3)]


@pytest.fixture(params=SECTORS, ids=lambda p: f"L{p[0]}N{p[1]}k{p[2]}")
def sector(request, ek, O):
    L, N, k = request.param
    B, Bo = ek.TranslationalBasis(L=L, N=N, k=k), O.translational(L, k=k, N=N)
    assert B.size(1) >= 512 * 148 and B.get_search() == "hash"
    return L, N, B, Bo


def states(L, N):
    rng = np.random.default_rng(L)
    out = [sum(1 << int(v) for v in rng.choice(L, N, replace=False)) for _ in range(300)]
    mask = (1 << L) - 1
    for c in range(1, L):  # period c
        if L % c or N * c % L:
            continue
        for _ in range(8):
            cell = sum(1 << int(v) for v in rng.choice(c, N * c // L, replace=False))
            s = sum(cell << (c * i) for i in range(L // c))
            out.append(s)
            i, j = (int(v) for v in rng.choice(L, 2, replace=False))
            if ((s >> i) ^ (s >> j)) & 1:
                out.append(s ^ (1 << i) ^ (1 << j))
    run = (1 << N) - 1  # one run, at every shift
    out += [((run << i) | (run >> (L - i))) & mask for i in range(L)]
    return np.array(out, dtype=np.uint64)


def test_index(sector):
    L, N, B, Bo = sector
    st = states(L, N)
    pos, coeff = B.index_states(st)
    for s, q, c in zip(st, pos, coeff):
        cr, qr = Bo.index([(int(s) >> (L - 1 - i)) & 1 for i in range(L)])
        assert q == (qr if cr != 0 else 0)
        assert cr == 0 or c == cr


@pytest.mark.parametrize("two", [False, True])
def test_products(ek, O, sector, two):
    L, N, B, Bo = sector
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2, B)
    Ho = O.trans_inv_operator(O.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2, Bo)
    if two:
        H = H + ek.trans_inv_operator(ek.spin((0.3, "zzz"), (0.2, "xzx"), (0.2, "yzy")), 3, B)
        Ho = O.trans_inv_operator(O.spin((0.3, "zzz"), (0.2, "xzx"), (0.2, "yzy")), 3, Bo)
    D = B.size(1)
    rng = np.random.default_rng(N)
    x = rng.standard_normal(D) + 1j * rng.standard_normal(D)
    ref = Ho.mul(x)
    if two:
        ref = ref + O.trans_inv_operator(O.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2, Bo).mul(x)
    # rows of at most 2 L products: 1e-13 is some 30 roundings of the row sum
    assert np.linalg.norm(H * x - ref) <= 1e-13 * np.linalg.norm(ref)
    X = np.asfortranarray(np.stack([x, 1j * x, x, x, x], axis=1))
    assert np.linalg.norm((H * X)[:, 1] - 1j * ref) <= 1e-13 * np.linalg.norm(ref)
    H.sparse_()
    assert np.linalg.norm(H * x - ref) <= 1e-13 * np.linalg.norm(ref)
