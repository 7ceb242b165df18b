"""The batched engine's step limit (edk.h): refused past it, before anything is built,
with a message that says so; the context stays usable.  Krylov bases of the propagator
have no such limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_step_limit(ek):
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2,
                              ek.TranslationalBasis(L=8, N=4, k=0))
    with pytest.raises(ek.EDKError, match="at most 12791 steps"):
        ek.batch_lanczos_e0([H], m=12792)
    assert ek.batch_lanczos_e0([H], m=12791)[1]["steps"] <= H.size(1)


def test_krylov_basis_past_it(ek):
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2,
                              ek.ProjectedBasis(L=16, N=8))
    D = H.size(1)  # 12,870
    psi = np.random.default_rng(0).standard_normal(D) + 0j
    psi /= np.linalg.norm(psi)
    ref = ek.timeevolve(H, psi, 0.7, tol=1e-11)
    out = ek.timeevolve(H, psi, 0.7, tol=1e-11, m_max=13000)
    assert np.linalg.norm(out - ref) < 1e-9
