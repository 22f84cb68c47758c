"""Choices of a handle changed between two calls of a batch whose parameters are
the same: the second call runs with them, as the same calls made handle by
handle do, bit for bit (a replay of the first call's graph would keep the old
lanes, route or precision)."""
import importlib
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DELTA = 0.1


@pytest.fixture(scope="module")
def systems(q, tmp_path_factory):
    tables = importlib.import_module("2degas_b200.tables")
    d0 = tmp_path_factory.mktemp("batch")
    out = []
    for k, (nu, nd) in enumerate(((13, 13), (21, 21))):
        d = tables.make_run(os.path.join(d0, f"p{k}"), "c", nu, nd, 3.0, twist=True,
                            backflow=(0.2, 3.0, 1.8))
        out.append(q.System.read(d, "c"))
    return out


def _twist(s, h, i, j):
    s.set_twist(i, j)
    h.update_twist()


CHANGES = {
    "lanes": lambda s, h: h.set_pair_lanes(16),
    "groups": lambda s, h: h.set_launch(1, 1),
    "complex": lambda s, h: h.set_move_inversion(0),
    "batched inversion": lambda s, h: h.set_move_inversion(2),
    "layout": lambda s, h: h.set_inversion(1),
    "mixed": lambda s, h: h.set_precision("mixed"),
    "twist": lambda s, h: _twist(s, h, 1, 2),
    "timers": lambda s, h: h.phase_timers(True),
}


def _handles(q, systems, before):
    hs = []
    for k, s in enumerate(systems):
        s.set_twist(0, 0)
        h = q.Handle(s, capacity=24, seed=50 + k)
        L = s.s.el[0]
        h.population_set(np.random.default_rng(k).uniform(-L / 2, L / 2, (24, 2 * s.N)))
        for b in before:
            CHANGES[b](s, h)
        h.vmc(4, DELTA, 10 ** 9)
        h.block_reset()
        hs.append(h)
    return hs


@pytest.mark.parametrize("before,change", [((), c) for c in CHANGES] +
                         [(("complex",), "batched inversion")])
def test_a_change_between_two_calls_is_taken(q, systems, before, change):
    states = []
    for batched in (False, True):
        hs = _handles(q, systems, before)
        b = q.Batch(hs) if batched else None

        def call():
            if b:
                b.vmc(2, [DELTA, DELTA])
            else:
                for h in hs:
                    h.vmc(2, DELTA, 10 ** 9)

        call()
        for s, h in zip(systems, hs):
            CHANGES[change](s, h)
        call()
        if change == "twist":  # and Gamma again
            for s, h in zip(systems, hs):
                _twist(s, h, 0, 0)
            call()
        states.append([h.population_get() for h in hs])
        if change == "timers":
            assert all(h.phase_timers(False)["pairs"] > 0 for h in hs)
            call()  # the buffer is gone: the graph must not write to it
        if b:
            b.close()
        for h in hs:
            h.close()
    for u, v in zip(*states):
        for k in ("x", "g", "p"):
            assert np.array_equal(u[k], v[k]), k
