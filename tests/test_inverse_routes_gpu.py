"""Which inverse the solver takes for S(n) and R(n): the general one where R is
one 64 x 64 tile (N_t <= 64), the symmetric sweep above; the gradients the
general one throughout."""
import numpy as np
import pytest

from scatt_b200 import _lib, synth
from scatt_b200 import adjoint as ADJ
from scatt_b200 import solver as S

pytestmark = pytest.mark.gpu

FIELDS = ("K_kme", "A", "B", "D", "d_raw", "partial_sigma")
OPTS = dict(allow_closed_channels=1)


def _solve(sol, Es, scheme, **kw):
    _lib.set_inverse_blocking(scheme)
    try:
        return sol.solve(Es, opts=S.default_opts(**OPTS, **kw))
    finally:
        _lib.set_inverse_blocking(0)


def _same(a, b):
    return all(np.array_equal(getattr(x, f), getattr(y, f)) for x, y in zip(a, b) for f in FIELDS)


@pytest.mark.parametrize("l_cont,n_orb,graphs", [(0, 1, 0), (3, 1, 0), (3, 3, 0), (3, 3, 1)])     # N_t 2, 32, 64
def test_one_tile_orders_take_the_general_inverse(l_cont, n_orb, graphs):
    sol = S.ScanSolver(synth.h2o_like(Nr=201, dr=0.05, l_cont=l_cont, lmax_orb=6, n_orb=n_orb))
    Es = [0.4, 0.6, 0.9]
    assert _same(_solve(sol, Es, 0, use_graphs=graphs), _solve(sol, Es, 2, use_graphs=graphs))


@pytest.mark.parametrize("l_cont,n_orb", [(3, 3), (4, 3), (6, 3), (7, 1)])     # N_t 64, 100, 196, 128 (S: 16 .. 64)
def test_the_gradients_forward_is_the_general_solve(l_cont, n_orb):
    sol = S.ScanSolver(synth.h2o_like(Nr=161, dr=1.4 / 160, l_cont=l_cont, lmax_orb=40, n_orb=n_orb))
    Es = [0.7, 0.9, 1.1]
    adj = ADJ.ScanAdjoint(sol, Es, segment=32, opts=S.default_opts(**OPTS))
    assert _same(adj.results, _solve(sol, Es, 2))
    # the default solve (sweep above one tile) differs by rounding only: the cross-solver bound of the dipoles
    for a, b in zip(adj.results, _solve(sol, Es, 0)):
        for f in FIELDS:
            x, y = getattr(a, f), getattr(b, f)
            assert np.max(np.abs(x - y)) <= 1e-10 * np.max(np.abs(y)), f


def test_device_memory_of_a_slot():
    """A slot of the scan at l_cont 20, N_t 1046 (a group of its own): 158 MB,
    none of it for the rescue's products, which the slots share."""
    import torch

    sol = S.ScanSolver(synth.h2o_like(Nr=131, dr=1.4 / 130, l_cont=20, lmax_orb=40, n_orb=5))
    opts = S.default_opts(allow_closed_channels=1, keep_window=0)
    used = []
    for slots in (16, 48):
        before = torch.cuda.mem_get_info()[0]
        scan = sol.scan(slots=slots, groups=slots, opts=opts)
        used.append(before - torch.cuda.mem_get_info()[0])
        scan.close()
    assert (used[1] - used[0]) / 32 <= 160e6


def test_orders_above_8192_are_refused():
    """N_t 8273 (64 orbitals at l_cont 22): an order that neither inverse takes."""
    sol = S.ScanSolver(synth.h2o_like(Nr=131, dr=1.4 / 130, l_cont=22, lmax_orb=2, n_orb=64))
    with pytest.raises(_lib.ScattError) as e:
        sol.solve([0.9], opts=S.default_opts(**OPTS, keep_window=0))
    assert e.value.code == 3                        # SCATT_ERR_SIZE
