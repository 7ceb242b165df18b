"""The library handles behind entanglement spectra and block Lanczos are shared:
several threads on their own bases at once, and bases that come and go."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_and_lifetimes(ek):
    def spectrum(L, seed):
        b = ek.TranslationalBasis(L=L, N=L // 2, k=0)
        v = np.random.default_rng(seed).standard_normal(b.size(1))
        v /= np.linalg.norm(v)
        return ek.ent_spec(v, list(range(1, L // 2 + 1)), b), ek.schmidt(
            v, list(range(1, L // 2 + 1)), b)

    got, failed = {}, []

    def work(t):
        try:
            for r in range(4):  # every basis is dropped before the next
                got[t, r] = spectrum(8 + 2 * (t % 3), 10 * t + r)
        except Exception as e:  # reported by the main thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for s, M in got.values():
        ref = np.linalg.svd(M, compute_uv=False)
        # squares of values below n eps of the largest are zero: 1e-7 of it
        assert np.allclose(s, ref, rtol=0, atol=1e-7 * ref[0])
