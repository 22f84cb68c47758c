"""A handle on a nearly full device: where everything but the real-orbital room of
the move scratch fits, the handle is made without that room, and its moves
are those of the complex kernels (to 1e-9 of the largest value, as the routes
agree elsewhere)."""
import importlib
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_create_falls_back_to_the_smaller_scratch(q, tmp_path):
    import torch

    tables = importlib.import_module("2degas_b200.tables")
    # 37 + 37: of the 2190 MB that a handle of this capacity takes the move scratch
    # is 1950, 780 of them the real orbitals' room; 120 MB too few hold the
    # scratch alone, but not beside the other 240
    cap = 16384
    d = tables.make_run(os.path.join(tmp_path, "d"), "c", 37, 37, 3.0, nconf=4,
                        backflow=(0.2, 3.0, 1.8))
    s = q.System.read(d, "c")
    x = s.read_configs(d, ".0", 0, 4)

    def chain(capacity, mode):
        with q.Handle(s, capacity=capacity, seed=3) as h:
            h.set_move_inversion(mode)
            h.population_set(x)
            h.vmc(2, 0.02, 0)
            return h.population_get()

    want = chain(4, 0)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    ballast = torch.empty(free - s.footprint(cap) + 120 * MB, dtype=torch.uint8, device="cuda")
    try:
        got = chain(cap, 1)
    finally:
        del ballast
        torch.cuda.empty_cache()
    for k in ("x", "g", "p"):
        assert np.abs(got[k] - want[k]).max() < 1e-9 * np.abs(want[k]).max(), k
