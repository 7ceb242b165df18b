"""Block Lanczos steps enqueued eight at a time: step counts around the host's
looks, with and without a tolerance, and sectors whose Krylov space closes
between two looks, against the dense spectra (1e-9 as the single-vector runs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sector(ek, L, N, k):
    return ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.6, "zz")), 2,
                                 ek.TranslationalBasis(L=L, N=N, k=k))


def levels(H, nev):
    w = np.linalg.eigvalsh(H.todense())
    d = [w[0]]
    for x in w[1:]:
        if x - d[-1] > 1e-9:
            d.append(x)
    return np.array(d[:nev])


@pytest.mark.parametrize("steps,tol,every", [(7, 0.0, 10), (8, 0.0, 10), (9, 0.0, 3), (17, 0.0, 0),
                                             (25, 1e-11, 5), (25, 1e-11, 8), (25, 1e-11, 30)])
def test_step_counts_and_checks(ek, steps, tol, every):
    ops = [sector(ek, 14, 7, k) for k in (0, 3)] + [sector(ek, 15, 6, 2)]
    ev, info = ek.block_lanczos(ops, block=8, m=steps, nev=2, tol=tol, check_every=every)
    assert info["steps"] <= steps and info["matvecs"] == info["steps"] * 8 * 3
    assert (tol > 0 and every < steps) or info["steps"] == steps
    if steps >= 17:
        for H, e in zip(ops, ev):
            ref = levels(H, 2)
            assert np.allclose(e, ref, rtol=0, atol=1e-9 * abs(ref[0]))


@pytest.mark.parametrize("steps", [5, 11, 12])
def test_closed_krylov_space(ek, steps):
    """A start block inside an invariant subspace of 20 eigenvectors: the third
    block of eight would have rank four, so the space ends with two blocks, and
    the levels are the Ritz values of span{x, H x}; a random block goes on."""
    H, G = sector(ek, 14, 7, 1), sector(ek, 14, 7, 2)
    Hd = H.todense()
    w, V = np.linalg.eigh(Hd)
    rng = np.random.default_rng(2)
    x = V[:, :20] @ (rng.standard_normal((20, 8)) + 1j * rng.standard_normal((20, 8)))
    y = rng.standard_normal((G.size(1), 8)) + 1j * rng.standard_normal((G.size(1), 8))
    Q, _ = np.linalg.qr(np.hstack([x, Hd @ x]))
    ref = np.linalg.eigvalsh(Q.conj().T @ Hd @ Q)[:2]
    ev, info = ek.block_lanczos([H, G], [x, y], block=8, m=steps, nev=2)
    assert info["breakdowns"] == 1 and info["steps"] == steps
    assert np.allclose(ev[0], ref, rtol=0, atol=1e-9 * abs(w[0]))
    one, only = ek.block_lanczos([H], [x], block=8, m=steps, nev=2)
    assert only["breakdowns"] == 1 and only["steps"] == 2
    assert np.allclose(one[0], ref, rtol=0, atol=1e-9 * abs(w[0]))
