"""Torch inputs that have to be copied first (gaps between the entries, real vectors
of a complex operator): the copy runs on torch's stream, the library on its own, so
the call has to wait for it.  A delay in front of the copy, and NaN in the memory it
will take, make a call that does not wait show."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def late():
    """Busy torch's stream for some milliseconds, the copy's memory full of NaN."""
    import torch

    def go(n, dtype):
        torch.cuda.synchronize()
        trash = torch.full((n,), float("nan"), dtype=dtype, device="cuda")
        torch.cuda.synchronize()
        del trash
        torch.cuda._sleep(40_000_000)
    return go


def momentum(ek, k, L=14):
    return ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2,
                                 ek.TranslationalBasis(L=L, N=L // 2, k=k))


def vector(D, cx=False, seed=0):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(D) + (1j * rng.standard_normal(D) if cx else 0)


@pytest.mark.parametrize("gap", [2, 3])
def test_strided_vector(ek, late, gap):
    import torch
    H = momentum(ek, 0)
    D = H.size(1)
    x = vector(D)
    wide = torch.zeros(D * gap, dtype=torch.float64, device="cuda")
    wide[::gap] = torch.from_numpy(x).cuda()
    late(D, torch.float64)
    y = H * wide[::gap]
    assert np.array_equal(y.cpu().numpy(), H * x)


def test_real_vector_of_a_complex_operator(ek, late):
    import torch
    H = momentum(ek, 3)
    x = vector(H.size(1))
    xd = torch.from_numpy(x).cuda()
    late(len(x), torch.complex128)
    y = H * xd
    assert np.array_equal(y.cpu().numpy(), H * x.astype(complex))


@pytest.mark.parametrize("kind", ["vector", "target", "both", "real"])
def test_mul_into_a_target(ek, late, kind):
    import torch
    H = momentum(ek, 3 if kind == "real" else 0)
    D = H.size(1)
    cx = kind == "real"
    x, t = vector(D), vector(D, cx, 1)
    ref = t + H * (x.astype(complex) if cx else x)

    def put(a, strided):
        a = torch.from_numpy(a).cuda()
        if not strided:
            return a
        wide = torch.zeros(2 * D, dtype=a.dtype, device="cuda")
        wide[::2] = a
        return wide[::2]

    xd, td = put(x, kind in ("vector", "both")), put(t, kind in ("target", "both"))
    late(D, torch.complex128 if cx else torch.float64)
    out = ek.mul_(td, H, xd)
    assert out is td
    assert np.allclose(td.cpu().numpy(), ref, rtol=0, atol=1e-13 * np.abs(ref).max())
    with pytest.raises(TypeError, match="target dtype"):
        ek.mul_(torch.zeros(D, dtype=torch.float32, device="cuda"), H, xd)


def test_mul_into_a_numpy_target_with_gaps(ek):
    H = momentum(ek, 0)
    D = H.size(1)
    x, wide = vector(D), np.zeros(2 * D)
    ek.mul_(wide[::2], H, x)
    assert np.array_equal(wide[::2], H * x) and not wide[1::2].any()


def test_evolution_and_entropy(ek, late):
    import torch
    H = momentum(ek, 0)
    D = H.size(1)
    psi = vector(D)
    psi /= np.linalg.norm(psi)
    ref = ek.timeevolve(H, psi.astype(complex), 0.4)
    xd = torch.from_numpy(psi).cuda()
    late(D, torch.complex128)
    assert np.allclose(ek.timeevolve(H, xd, 0.4).cpu().numpy(), ref, rtol=0, atol=1e-13)
    late(D, torch.complex128)
    cache = ek.KrylovEvolutionCache(H, xd)
    assert np.allclose(cache.timeevolve_(0.4).cpu().numpy(), ref, rtol=0, atol=1e-13)
    wide = torch.zeros(2 * D, dtype=torch.float64, device="cuda")
    wide[::2] = xd
    s = ek.ent_S(psi, [1, 2, 3], H.B)
    late(D, torch.float64)
    assert abs(ek.ent_S(wide[::2], [1, 2, 3], H.B) - s) < 1e-12
