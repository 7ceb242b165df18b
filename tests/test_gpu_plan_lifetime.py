"""Row plans built together live as long as any operator of their batch: operators
go in any order, while products of others still run, and the memory is used again
only after the last."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(ek, L, seed):
    bond = ek.spin((1.0, "xx"), (1.0, "yy"), (0.8, "zz"))
    h = np.random.default_rng(seed).uniform(-1, 1, L)
    return ek.operator([bond] * (L - 1) + [v * ek.spin("z") for v in h],
                       [[i, i + 1] for i in range(1, L)] + [[i] for i in range(1, L + 1)],
                       ek.ProjectedBasis(L=L, N=L // 2))


def test_operators_of_a_batch_go_in_any_order(ek):
    Ls = [10, 12, 14, 16, 12, 10]
    for order in ([0, 1, 2, 3, 4, 5], [5, 3, 1, 0, 2, 4], [3, 2, 1, 5, 4, 0]):
        ops = [chain(ek, L, q) for q, L in enumerate(Ls)]
        xs = [np.random.default_rng(q).standard_normal(op.size(1)) for q, op in enumerate(ops)]
        ref = [op * x for op, x in zip([chain(ek, L, q) for q, L in enumerate(Ls)], xs)]
        ek.batch_lanczos_e0(ops, m=20)  # builds all plans at once
        for gone in order:
            ops[gone] = None
            chain(ek, 14, 50 + gone) * np.ones(3432)  # another plan from the same pool
            for q, op in enumerate(ops):
                if op is not None:
                    assert np.array_equal(op * xs[q], ref[q])


def test_last_operator_goes_while_its_product_runs(ek):
    import ctypes as C
    import torch
    E = ek._lib
    L = 20
    H = chain(ek, L, 0)
    D = H.size(1)
    x = torch.from_numpy(np.random.default_rng(1).standard_normal(D)).cuda()
    ref = (H * x).clone()
    y = torch.zeros(D, dtype=torch.float64, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
    E.check(E.load().edk_apply_async(H._h, E.F64, x.data_ptr(), y.data_ptr(), 1, D, D, 0,
                                     C.c_void_p(side.cuda_stream)))
    del H
    keep = [chain(ek, L, q) for q in range(1, 4)]
    for op in keep:
        op * x  # plans where the first one was
    torch.cuda.synchronize()
    assert torch.equal(y, ref)


def test_memory_of_a_batch_comes_back_with_its_operators(ek):
    """Six plans of some 166 MB built together: five operators go, their memory comes
    back (what the pool keeps for the next plans is 512 MB at most)."""
    import torch
    L = 26
    B = ek.ProjectedBasis(L=L, N=L // 2)
    bond = ek.spin((1.0, "xx"), (1.0, "yy"), (0.8, "zz"))
    ops = [ek.operator([(1 + 0.1 * q) * bond] * (L - 1), [[i, i + 1] for i in range(1, L)], B)
           for q in range(6)]
    ev, _ = ek.batch_lanczos_e0(ops, m=2)
    plan = 16 * B.size(1)
    before = torch.cuda.mem_get_info()[0]
    del ops[1:]
    torch.cuda.synchronize()
    back = torch.cuda.mem_get_info()[0] - before
    assert back >= 5 * plan - (512 << 20) - (64 << 20)
    # (alone the rows split differently over the blocks: other orders of summation)
    assert abs(ek.batch_lanczos_e0(ops, m=2)[0][0, 0] - ev[0, 0]) < 1e-12
