"""A handle on a nearly full device: where everything but the real-orbital room of
the move scratch fits, the handle is made without that room, and its moves
are those of the complex kernels (to 1e-9 of the largest value, as the routes
agree elsewhere). Host memory is page-locked for the staging of host-buffer
evaluations when a handle makes one, in the size that it needs."""
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


def _resident_shared():
    with open("/proc/self/status") as f:
        return sum(int(line.split()[1]) for line in f if line.startswith("RssShmem")) << 10


def test_handles_page_lock_no_staging_that_they_do_not_use(q, n26):
    q.Handle(n26, capacity=4096, seed=1).close()
    before = _resident_shared()
    hs = [q.Handle(n26, capacity=4096, seed=1) for _ in range(16)]
    grown = _resident_shared() - before
    for h in hs:
        h.close()
    assert grown < 16 * MB  # 16 x 4096 status words are 256 KB


def test_staging_grows_with_the_calls(q, n26, n26_configs):
    """Calls of every size, with those beyond the staging between them, return what
    one configuration at a time does."""
    x = np.tile(n26_configs, (64, 1))
    with q.Handle(n26, capacity=len(x), seed=1) as h:
        one = [h.compute_properties(x[k:k + 1]) for k in range(64)]
        for n in (2, 64, 3, 640, 4096, 65):
            for got, j in zip(h.compute_properties(x[:n]), range(4)):
                want = np.concatenate([o[j] for o in one])[np.arange(n) % 64]
                assert np.array_equal(got, want)
