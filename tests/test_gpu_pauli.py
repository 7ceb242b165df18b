"""Operators on the full space that are no flip-flop chains: the Pauli-string
kernel against the oracle and against the general row kernel.

Sizes: spaces smaller than one tile (1 .. 8 sites), one to a few tiles of 512
rows, and 2^19 rows (tiles of 2,048 with flips inside and across tiles); real
and complex, single and double precision, several columns, strided blocks and
accumulation.  Tolerance: a row sums at most 80 products, 1e-14 (1e-6 in single
precision) of the product's norm is several times their rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def model(S, L, kind):
    rng = np.random.default_rng(L)
    sites = [[i] for i in range(1, L + 1)]
    bonds = [[i, i + 1] for i in range(1, L)]
    mats, inds = [h * S("x") for h in rng.uniform(0.5, 1, L)], list(sites)
    if kind != "field":
        mats += [-S("zz")] * (L - 1) + [h * S("z") for h in rng.uniform(-1, 1, L)]
        inds += bonds + sites
    if kind == "real":  # pair creation, bonds of no order, three sites
        mats += [S("xx") + 0.3 * S("yy")] * (L - 1) + [0.2 * S("xzx")] * max(0, L - 2)
        inds += [b[::-1] for b in bonds] + [[i + 2, i, i + 1] for i in range(1, L - 1)]
    if kind == "complex":  # y fields and Dzyaloshinskii-Moriya bonds
        mats += [0.4 * S("y")] * L + [0.7 * (S("xy") - S("yx"))] * (L - 1)
        inds += sites + bonds
    return mats, inds


def pair(ek, O, L, kind):
    H = ek.operator(*model(ek.spin, L, kind), ek.TensorBasis(L=L))
    Ho = O.operator(*model(O.spin, L, kind), O.tensor(L))
    return H, Ho


@pytest.mark.parametrize("kind", ["field", "ising", "real", "complex"])
@pytest.mark.parametrize("L", [1, 2, 3, 8, 9, 11])
def test_product_matches_oracle(ek, O, L, kind):
    H, Ho = pair(ek, O, L, kind)
    rng = np.random.default_rng(7)
    x = rng.standard_normal(2 ** L) + 1j * rng.standard_normal(2 ** L)
    ref = Ho.mul(x)
    for dt, tol in ((np.complex128, 1e-14), (np.complex64, 1e-6)):
        y = H * x.astype(dt)
        assert y.dtype == dt and np.linalg.norm(y - ref) <= tol * np.linalg.norm(ref)
    if kind != "complex":
        ref = Ho.mul(x.real).real
        for dt, tol in ((np.float64, 1e-14), (np.float32, 1e-6)):
            y = H * x.real.astype(dt)
            assert y.dtype == dt and np.linalg.norm(y - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("kind,L", [("ising", 10), ("complex", 12), ("real", 19)])
def test_blocks_strides_and_accumulation_match_the_row_kernel(ek, monkeypatch, kind, L):
    import torch
    mats, inds = model(ek.spin, L, kind)
    B = ek.TensorBasis(L=L)
    H = ek.operator(mats, inds, B)
    monkeypatch.setenv("EDK_DISABLE_FAST", "1")
    G = ek.operator(mats, inds, B)  # the general row kernel
    D, nv = 2 ** L, 3
    dt = torch.complex128 if kind == "complex" else torch.float64
    g = torch.Generator(device="cuda").manual_seed(L)
    x = torch.randn((nv, D + 5), dtype=dt, device="cuda", generator=g)[:, :D].t()
    y0 = torch.randn((nv, D + 3), dtype=dt, device="cuda", generator=g)
    torch.cuda.synchronize()
    out = []
    for op in (H, G):
        y = y0.clone()[:, :D].t()
        torch.cuda.synchronize()
        ek.mul_(y, op, x)
        out.append(y)
    assert torch.linalg.vector_norm(out[0] - out[1]) <= 1e-14 * torch.linalg.vector_norm(out[1])


def test_ground_state_runs_on_the_strings(ek, O):
    H, Ho = pair(ek, O, 9, "ising")
    ev, info = ek.lanczos_e0(H, m=120, tol=1e-13)
    assert abs(ev[0] - np.linalg.eigvalsh(Ho.dense())[0]) <= 1e-11
