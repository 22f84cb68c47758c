"""Reptation moves of several bead growths over real orbitals: a move draws 1 to
mdelta growths, and the determinant kernels of a later growth pass over the
reptiles whose move has none."""
import importlib
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(q, tmp_path, nu, nd, nrep, mdelta, moves, mode=1, timers=False):
    tables = importlib.import_module("2degas_b200.tables")
    d = tables.make_run(os.path.join(tmp_path, "d"), "c", nu, nd, 3.0, nconf=nrep, seed=7,
                        backflow=(0.2, 3.0, 1.8))
    s = q.System.read(d, "c")
    x = s.read_configs(d, ".0", 0, nrep)
    walk = np.cumsum(np.random.default_rng(3).normal(0.0, 0.02, (nrep, 12, x.shape[1])), axis=1)
    with q.Handle(s, capacity=nrep, seed=9) as h:
        h.set_move_inversion(mode)
        # every move forced
        h.rmc_init(nrep, (x[:, None, :] + walk).reshape(nrep * 12, -1), 12, 1, mdelta, 0.002, -0.4,
                   10 ** 9, 0)
        h.block_reset()
        if timers:
            h.phase_timers(True)
        h.rmc(moves)
        cycles = h.phase_timers(False)["cross"] if timers else 0
        return (h.block_get()[0],) + h.rmc_get_path(nrep - 1, 12), cycles


@pytest.mark.parametrize("nu,nd", [(13, 13), (21, 17), (37, 33), (45, 21), (121, 0)])
def test_moves_of_many_growths_equal_the_complex_route(q, tmp_path, nu, nd):
    (r, _), (c, _) = (_run(q, tmp_path, nu, nd, 6, 6, 3, mode) for mode in (1, 0))
    for u, v in zip(r, c):
        assert np.abs(u - v).max() <= 1e-9 * np.abs(v).max()


def test_no_determinant_work_for_growths_that_a_move_has_not(q, tmp_path):
    """16 moves of 64 reptiles with mdelta = 8 have 4.5 growths each (to 0.07): the
    Laplacian kernel's cycles are those of 4.5 growths, not of 8."""
    one = _run(q, tmp_path, 13, 13, 64, 1, 16, timers=True)[1]
    many = _run(q, tmp_path, 13, 13, 64, 8, 16, timers=True)[1]
    assert 3.0 * one < many < 6.0 * one
