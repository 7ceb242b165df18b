"""Krylov states combined several at a time: counts around the eight states of a
pass, through host and device results, across restarts and extensions, on every
kind of product the basis can be built with (row plan, tile, Pauli strings,
symmetry group, materialised) and with normalised output.  The controller's own
tolerance (1e-12 per interval) bounds the states: 1e-10 over the run."""
import numpy as np
import pytest
from scipy.linalg import expm

pytestmark = pytest.mark.gpu


def bond(S):
    return S((1.0, "xx"), (1.0, "yy"), (0.7, "zz"))


def problem(ek, kind):
    if kind == "ising":
        L = 8
        return ek.operator([ek.spin("zz")] * (L - 1) + [0.7 * ek.spin("x")] * L,
                           [[i, i + 1] for i in range(1, L)] + [[i] for i in range(1, L + 1)],
                           ek.TensorBasis(L=L))
    if kind == "group":
        B = ek.basis(L=12, N=6, k=0, p=1, z=-1)
    elif kind == "wide":
        B = ek.TranslationalBasis(L=34, N=3, k=5)
    else:
        B = ek.TranslationalBasis(L=12, N=6, k=3)
        if kind == "rank":
            B.set_search("rank")
    H = ek.trans_inv_operator(bond(ek.spin), 2, B)
    if kind == "sparse":
        H.sparse_()
    return H


@pytest.mark.parametrize("kind", ["hash", "rank", "sparse", "ising", "group", "wide"])
@pytest.mark.parametrize("nt", [1, 7, 8, 9, 20])
def test_states_match_the_dense_exponential(ek, kind, nt):
    import torch
    H = problem(ek, kind)
    Hd = H.todense()
    rng = np.random.default_rng(nt)
    psi = rng.standard_normal(H.size(1)) + 1j * rng.standard_normal(H.size(1))
    psi /= np.linalg.norm(psi)
    ts = np.sort(rng.uniform(0, 4, nt))
    kw = dict(tol=1e-12, m_init=8, m_max=16, extend_step=3)
    host, d = ek.timeevolve(H, psi, ts, return_diagnostics=True, **kw)
    dev = ek.timeevolve(H, torch.from_numpy(psi).cuda(), ts, **kw)
    assert np.array_equal(dev.cpu().numpy(), host)
    assert d.total_times_served == nt
    for q, t in enumerate(ts):
        assert np.linalg.norm(host[:, q] - expm(-1j * t * Hd) @ psi) < 1e-10
    unit = ek.timeevolve(H, 3.0 * psi, ts, normalize_output=True, **kw)
    assert np.allclose(unit, host, atol=1e-9)
