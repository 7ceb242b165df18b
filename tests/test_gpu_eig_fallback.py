"""A grid barrier of the tridiagonalisation that gives up (here after one poll) costs
the shared-memory route, not the call: the library's solver takes the same matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", ["0", "1"])
@pytest.mark.parametrize("cx", [False, True])
def test_spectrum_when_the_barrier_gives_up(ek, monkeypatch, polls, cx):
    L, nA = 16, 8
    rng = np.random.default_rng(3)
    v = rng.standard_normal(2 ** L) + (1j * rng.standard_normal(2 ** L) if cx else 0)
    v /= np.linalg.norm(v)
    B = ek.TensorBasis(L=L)
    monkeypatch.setenv("EDK_EIG_POLLS", polls)
    s = ek.ent_spec(v, list(range(1, nA + 1)), B)
    monkeypatch.delenv("EDK_EIG_POLLS")
    ref = np.linalg.svd(v.reshape(2 ** nA, -1), compute_uv=False)
    tol = 8 * len(ref) * np.finfo(float).eps * ref[0] ** 2
    assert np.abs(s ** 2 - ref ** 2).max() <= tol
    again = ek.ent_spec(v, list(range(1, nA + 1)), B)  # and the route is there as before
    assert np.abs(again ** 2 - ref ** 2).max() <= tol
