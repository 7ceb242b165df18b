"""Threads that share operators: every solver takes the operators' locks before its
first allocation on their stream, so no allocation lands in another thread's graph
capture.  Each call's result is that of the same call alone (1e-13: the norm of a
ground state is summed by atomics, in any order)."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def momentum(ek, L, k):
    return ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2,
                                 ek.TranslationalBasis(L=L, N=L // 2, k=k))


def run(jobs):
    alone = [f() for f in jobs]
    with ThreadPoolExecutor(len(jobs)) as pool:
        for _ in range(3):
            for a, b in zip(alone, [f.result() for f in [pool.submit(j) for j in jobs]]):
                for x, y in zip(a, b):
                    assert np.allclose(x, y, rtol=0, atol=1e-13 * np.abs(x).max(), equal_nan=True)


def test_ground_states_of_one_operator(ek):
    H = momentum(ek, 14, 0)
    v = np.random.default_rng(0).standard_normal((H.size(1), 4))

    def job(c, precision):
        def f():
            e, psi, _ = ek.ground_state(H, np.ascontiguousarray(v[:, c]), m=80, tol=1e-12,
                                        precision=precision)
            return np.atleast_1d(e), psi
        return f

    run([job(c, "fp64" if c % 2 else "mixed") for c in range(4)])


def test_batches_that_share_operators(ek):
    ops = [momentum(ek, 12, k) for k in range(6)]

    def job(sub):
        return lambda: (ek.batch_lanczos_e0(sub, m=60, nev=2, tol=1e-12)[0],)

    run([job(ops), job(ops[::-1]), job(ops[2:]), job([ops[3], ops[0]])])
