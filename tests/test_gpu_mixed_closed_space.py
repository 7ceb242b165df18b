"""Mixed precision in Krylov spaces that close before the step limit: sectors with
fewer levels than steps.  The last vector is then the rounding of the FP32
storage, which the second sweep takes in whole; the run has to end there.

Batches: every value returned is a level of the sector and the lowest is E0, within
1e-9 of the largest level (the FP64 refinement leaves rounding only).
Propagation: the whole space is exact for every time, so nothing restarts; the
states carry FP32 rounding of the vectors and of T, 6e-8 (1 + |H| t) a vector."""
import numpy as np
import pytest
from scipy.linalg import expm

pytestmark = pytest.mark.gpu


def sectors(ek, L):
    bond = ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz"))
    return [ek.trans_inv_operator(bond, 2, ek.TranslationalBasis(L=L, N=L // 2, k=k))
            for k in range(L)]


def check(ops, ev, nev):
    for H, e in zip(ops, ev):
        ref = np.linalg.eigvalsh(H.todense())
        tol = 1e-9 * max(1.0, np.abs(ref).max())
        got = e[np.isfinite(e)]
        assert len(got) >= min(nev, np.count_nonzero(np.diff(ref) > 1e-8) + 1)
        assert abs(got[0] - ref[0]) < tol
        assert np.abs(got[:, None] - ref[None, :]).min(axis=1).max() < tol


@pytest.mark.parametrize("nev", [1, 4])
@pytest.mark.parametrize("L", [6, 7, 8, 9])
def test_batches_of_short_chains(ek, L, nev):
    ops = sectors(ek, L)
    for seed in range(8):
        ev, _ = ek.batch_lanczos_e0(ops, m=200, nev=nev, tol=1e-12, precision="mixed", seed=seed)
        check(ops, ev, nev)


def test_short_chain_in_an_uneven_batch(ek):
    ops = sectors(ek, 7) + sectors(ek, 12)[:4]
    ev, _ = ek.batch_lanczos_e0(ops, m=200, nev=2, tol=1e-12, precision="mixed")
    check(ops, ev, 2)


def test_scaled_operators(ek):
    bond = 1e4 * ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz"))
    ops = [ek.trans_inv_operator(bond, 2, ek.TranslationalBasis(L=7, N=3, k=k)) for k in range(7)]
    for seed in range(8):
        ev, _ = ek.batch_lanczos_e0(ops, m=200, precision="mixed", seed=seed)
        check(ops, ev, 1)


@pytest.mark.parametrize("L,k", [(8, 0), (8, 3), (10, 1)])
def test_propagation_in_a_closed_space_needs_no_restart(ek, L, k):
    H = sectors(ek, L)[k]
    D = H.size(1)
    rng = np.random.default_rng(L + k)
    psi = rng.standard_normal(D) + 1j * rng.standard_normal(D)
    psi /= np.linalg.norm(psi)
    ts = np.array([0.5, 7.0, 30.0])
    out, d = ek.timeevolve(H, psi, ts, return_diagnostics=True, tol=1e-10, precision="mixed")
    assert d["restarts"] == 0 and d["matvecs"] <= D
    Hd = H.todense()
    norm = np.abs(np.linalg.eigvalsh(Hd)).max()
    for q, t in enumerate(ts):
        assert np.linalg.norm(out[:, q] - expm(-1j * t * Hd) @ psi) < 6e-8 * (1 + norm * t) * D
