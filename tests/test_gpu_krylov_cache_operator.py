"""A resumable Krylov cache follows its operator: materialising, clearing, another
search or another kernel between two calls changes how the product runs, never the
states, and no call reads tables that are gone.  Bases small enough to restart and
extend after every change; the states against the dense exponential, 1e-9 as in
test_gpu_krylov_cache.py."""
import numpy as np
import pytest
from scipy.linalg import expm

pytestmark = pytest.mark.gpu


def walk(ek, H, changes, m_init=5, m_max=9):
    Hd = H.todense()
    D = H.size(1)
    rng = np.random.default_rng(D)
    psi = rng.standard_normal(D) + 1j * rng.standard_normal(D)
    psi /= np.linalg.norm(psi)
    cache = ek.KrylovEvolutionCache(H, psi, tol=1e-12, m_init=m_init, m_max=m_max, extend_step=2)
    t = 0.0
    for change in changes:
        change()
        for dt in (0.02, 0.6):  # from the present basis, then past it
            t += dt
            got = cache.timeevolve_(t)
            assert np.linalg.norm(got - expm(-1j * t * Hd) @ psi) < 1e-9, t
    assert cache.diagnostics.restarts >= 1
    return cache


def momentum(ek, L=12, k=1):
    return ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), [1, 2],
                                 ek.TranslationalBasis(L=L, N=L // 2, k=k))


def test_matrix_made_and_cleared(ek):
    import torch
    H = momentum(ek)
    keep = []

    def clear():  # something else takes the memory the matrix had
        H.clear_sparse_cache_()
        keep.append([torch.full((1 << k,), float("nan"), device="cuda") for k in range(8, 22)])

    H.sparse_()
    walk(ek, H, [lambda: None, clear, H.sparse_, clear, lambda: (H.sparse_(), clear(), H.sparse_())])


def test_search_and_kernel_changed(ek):
    H = momentum(ek)
    walk(ek, H, [lambda: H.B.set_search("rank"), lambda: H.B.set_search("sorted"),
                 lambda: H.configure_("generic"), lambda: H.configure_("fast", 4),
                 lambda: (H.B.set_search("rank"), H.configure_("fast", 1)), H.autotune_])


def test_symmetry_group_rows_and_matrix(ek):
    """Without the matrix the product runs outside the batched kernels."""
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2,
                              ek.basis(L=12, N=6, p=-1, z=1))
    walk(ek, H, [lambda: None, H.sparse_, H.clear_sparse_cache_, H.sparse_])


def test_pauli_strings_and_matrix(ek):
    L = 7
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (0.4, "xz"), (0.4, "zx")), 2, ek.TensorBasis(L=L))
    walk(ek, H, [lambda: None, H.sparse_, H.clear_sparse_cache_])
