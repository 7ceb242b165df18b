"""alpha and beta of edk_lanczos_e0 hold max_steps entries: nothing is written past
them when the FP64 refinement of a mixed run takes more steps."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_nothing_past_max_steps(ek, group, precision):
    from edkit_b200 import _lib as E
    from edkit_b200.algorithms import _opts
    kw = dict(L=12, N=6, k=0)
    B = ek.basis(p=1, **kw) if group else ek.TranslationalBasis(**kw)
    H = ek.trans_inv_operator(ek.spin((1.0, "xx"), (1.0, "yy"), (0.7, "zz")), 2, B)
    m, guard = 5, 100
    v0 = np.random.default_rng(0).standard_normal(H.size(1))
    a, b, ev = np.full(m + guard, 7.25), np.full(m + guard, 7.25), np.zeros(1)
    d = E.LanczosDiag()
    o = _opts(m, 1, 1e-13, 5, precision, 20, True, False)
    E.check(E.load().edk_lanczos_e0(H._h, C.byref(o), E.ptr(v0), E.F64, E.HOST, E.ptr(ev),
                                    E.ptr(a), E.ptr(b), C.byref(d)))
    if not group:  # (there the last restart of several may end after a step)
        assert (d.steps > m) == (precision == "mixed")
    n = min(m, d.steps)
    assert np.all(a[n:] == 7.25) and np.all(b[n:] == 7.25)
    assert np.all(a[:n] != 7.25) and np.all(b[:n] != 7.25)
