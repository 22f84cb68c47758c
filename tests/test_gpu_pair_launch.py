"""The pair kernels' launch where the caller leaves it to the size: walker groups
per CTA on both sides of each line of the rule, in walkers per SM, and the same
walkers bit for bit as with the choices made."""
import importlib
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(q, tmp_path, nu, nd, u3):
    tables = importlib.import_module("2degas_b200.tables")
    return q.System.read(tables.make_run(os.path.join(tmp_path, "d"), "c", nu, nd, 3.0, u3=u3,
                                         backflow=(0.2, 3.0, 1.8)), "c")


def _walkers(s, nw):
    half = s.s.el[0] / 2
    return np.random.default_rng(7).uniform(-half, half, (nw, 2 * s.N))


# up, down, u3, walkers per SM and groups below and from the line on
LINES = [(13, 13, False, 7, 1, 2), (13, 13, True, 6, 1, 2), (15, 15, False, 5, 1, 2),
         (16, 16, False, 4, 1, 2), (16, 16, True, 3, 1, 2), (25, 0, True, 6, 1, 2)]


@pytest.mark.parametrize("nu,nd,u3,line,below,above", LINES)
def test_groups_of_small_systems(q, tmp_path, nu, nd, u3, line, below, above):
    import torch

    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    s = _system(q, tmp_path, nu, nd, u3)
    for nw, groups in ((1, 1), (line * nsm - 1, below), (line * nsm, above)):
        with q.Handle(s, capacity=nw, seed=1) as h:
            h.population_set(_walkers(s, nw))
            h.set_autotune_scope(0)
            assert h.autotune()[0] == groups, nw


@pytest.mark.parametrize("nu,nd,u3,nw", [(16, 16, True, 450), (61, 61, True, 300),
                                         (61, 61, True, 150), (81, 81, False, 200)])
def test_the_rule_leaves_every_bit(q, tmp_path, nu, nd, u3, nw):
    s = _system(q, tmp_path, nu, nd, u3)
    got = []
    for groups, stage in ((0, 0), (1, 0), (1, 1), (2, 1)):
        with q.Handle(s, capacity=nw, seed=1) as h:
            h.set_launch(groups, stage)
            h.population_set(_walkers(s, nw))
            h.vmc(2, 0.02, 0)
            got.append(h.population_get())
    for g in got[1:]:
        for k in ("x", "g", "p"):
            assert np.array_equal(g[k], got[0][k]), k
