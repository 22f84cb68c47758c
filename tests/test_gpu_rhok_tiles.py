"""rho_k of the pair kernels over k lists that span several tiles of the
lattice tables: vectors far out on the axes and diagonals appended to a deck's
list. A list of |n| <= 17 keeps the sums of every tile at once, one of |n| <=
33 fits two walker groups only with the tiles in turn, and at |n| = 57 the sums
of all tiles exceed any CTA. Every launch choice that such a deck's groups fit
steps the walkers as the oracle does: positions to 1e-11 and properties to 1e-9
of the largest value as elsewhere, rho_k to 1e-10 (57 multiplications per table
entry, phases to 57 * 2 pi and positions to 1e-12 give a few 1e-11)."""
import importlib
import math
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEED = 0xA11CE


def _deck(q, tmp_path, far, nu, nd, **kw):
    tables = importlib.import_module("2degas_b200.tables")
    d = tables.make_run(os.path.join(tmp_path, "d"), "c", nu, nd, 3.0, nconf=4, seed=5,
                        backflow=(0.2, 3.0, 1.8), **kw)
    unit = 2.0 * math.pi / math.sqrt((nu + nd) * math.pi)
    with open(os.path.join(d, "c.k"), "a") as f:
        for a, b in ((far, 0), (0, far), (far, far), (far - 9, -far), (8, 7), (7, -8), (8, far)):
            f.write(f" {a * unit!r} {b * unit!r}\n")
    s = q.System.read(d, "c")
    return s, s.read_configs(d, ".0", 0, 4)


@pytest.mark.parametrize("far", [17, 33, 57])
@pytest.mark.parametrize("nu,nd", [(13, 13), (5, 0), (9, 5)])
def test_long_lists_match_the_oracle(q, oracle_cls, tmp_path, far, nu, nd):
    s, x = _deck(q, tmp_path, far, nu, nd)
    o = oracle_cls(s)
    pop = o.population_init(x)
    o.vmc_philox(pop, 2, 0.02, 0, SEED, 0)
    for groups, mode, lanes in ((0, 1, 0), (1, 0, 4), (2, 1, 8), (2, 0, 0)):
        with q.Handle(s, capacity=4, seed=SEED) as h:
            h.set_launch(groups, 0)
            h.set_move_inversion(mode)
            h.set_pair_lanes(lanes)
            h.population_set(x)
            h.vmc(2, 0.02, 0)
            got = h.population_get()
        p, ref = got["p"], pop["p"]
        assert np.abs(got["x"] - pop["x"]).max() < 1e-11 * np.abs(pop["x"]).max()
        assert np.abs(p[:, :14] - ref[:, :14]).max() < 1e-9 * np.abs(ref[:, :14]).max()
        k = slice(s.s.n_scalar_props, s.nprops)
        assert np.abs(p[:, k] - ref[:, k]).max() < 1e-10 * np.abs(ref[:, k]).max()


def test_long_lists_can_be_tuned(q, tmp_path):
    s, x = _deck(q, tmp_path, 33, 13, 13, u3=True)
    with q.Handle(s, capacity=4, seed=SEED) as h:
        h.population_set(x)
        assert h.autotune()[2] > 0.0
        h.vmc(1, 0.02, 0)
