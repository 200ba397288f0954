"""Eigenphases of the device (cluster Householder reduction and bisection)
against numpy's eigenvalues of the same K."""
import numpy as np
import pytest

from scatt_b200 import solver as S
from scatt_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("l_cont", [0, 1, 3, 8, 12, 15, 20])      # orders 1, 4, 16, 81, 169, 256, 441
def test_eigenphases_match_numpy(l_cont):
    inp = synth.h2_like(Nr=201, dr=0.05, l_cont=l_cont)
    for r in S.ScanSolver(inp).solve([0.3, 0.9], opts=S.default_opts(allow_closed_channels=1, keep_window=0)):
        for K, phases in ((r.K_kme, r.eig_kme), (r.K_aa, r.eig_aa)):
            # the lower triangle is read; eigenvalues are backward stable: O(n eps |K|)
            lam = np.linalg.eigvalsh(K, UPLO="L")
            bound = 1e-14 * max(4, K.shape[0]) * max(np.max(np.abs(lam)), 1e-300)
            assert np.all(np.abs(np.sort(phases) - np.sort(np.arctan(lam))) <= bound + 1e-15)


def test_two_threads_with_different_orders():
    """Eigenphases of orders 169 and 4 computed at once, each as alone."""
    import threading

    opts = S.default_opts(allow_closed_channels=1, keep_window=0)
    inps = [synth.h2_like(Nr=201, dr=0.05, l_cont=l) for l in (12, 1)]
    want = [S.ScanSolver(i).solve([0.3, 0.9], opts=opts) for i in inps]
    got = [[], []]

    def work(k):
        sol = S.ScanSolver(inps[k])
        for _ in range(3 if k == 0 else 12):
            got[k].append(sol.solve([0.3, 0.9], opts=opts))

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert len(got[k]) == (3 if k == 0 else 12)
        for res in got[k]:
            for a, b in zip(res, want[k]):
                assert np.array_equal(a.eig_kme, b.eig_kme) and np.array_equal(a.eig_aa, b.eig_aa)
