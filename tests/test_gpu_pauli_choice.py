"""Kernel choice of operators that have a Pauli-string form: "fast" selects the
strings, "generic" the row kernel, and the autotuner times both and names what it
installs.  The two sum a row in different orders, so the last bits of a product
tell which one ran."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ising(ek, L):
    rng = np.random.default_rng(L)
    h, g = rng.uniform(0.3, 1, L), rng.uniform(-1, 1, L)
    mats = [a * ek.spin("x") for a in h] + [a * ek.spin("z") for a in g] + [ek.spin("zz")] * (L - 1)
    inds = [[i] for i in range(1, L + 1)] * 2 + [[i, i + 1] for i in range(1, L)]
    return mats, inds


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
def test_generic_is_the_row_kernel(ek, monkeypatch, dt):
    L = 13
    B = ek.TensorBasis(L=L)
    mats, inds = ising(ek, L)
    H = ek.operator(mats, inds, B)
    monkeypatch.setenv("EDK_DISABLE_FAST", "1")
    rows = ek.operator(mats, inds, B)
    monkeypatch.delenv("EDK_DISABLE_FAST")
    x = np.random.default_rng(0).standard_normal(2 ** L).astype(dt)
    strings, ref = H * x, rows * x
    assert not np.array_equal(strings, ref)  # (different orders of summation)
    H.configure_("generic")
    assert np.array_equal(H * x, ref)
    H.configure_("fast")
    assert np.array_equal(H * x, strings)
    rows.configure_("generic")
    assert np.array_equal(rows * x, ref)


def test_autotune_times_both(ek):
    L = 14
    H = ek.operator(*ising(ek, L), ek.TensorBasis(L=L))
    x = np.random.default_rng(0).standard_normal(2 ** L)
    H.configure_("generic")
    rows = H * x
    H.configure_("fast")
    strings = H * x
    r = H.autotune_()
    assert {k for k, *_ in r["candidates"]} == {"fast", "generic"}
    assert np.array_equal(H * x, strings if r["kernel"] == "fast" else rows)


def test_solvers_follow_the_choice(ek):
    L = 10
    H = ek.operator(*ising(ek, L), ek.TensorBasis(L=L))
    e = [ek.lanczos_e0(H, m=120, tol=1e-13)[0][0]]
    H.configure_("generic")
    e.append(ek.lanczos_e0(H, m=120, tol=1e-13)[0][0])
    ref = np.linalg.eigvalsh(H.todense())[0]
    assert np.abs(np.array(e) - ref).max() < 1e-11
