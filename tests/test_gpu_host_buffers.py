"""Evaluations of host buffers that the caller has pinned: copied directly, without
the library's staging memory; pageable, pinned and absent buffers in any mixture
give the same results."""
import ctypes
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NW = 640


def _resident_shared():
    with open("/proc/self/status") as f:
        return sum(int(line.split()[1]) for line in f if line.startswith("RssShmem")) << 10


def _buffers(s, x, pinned):
    import torch

    out = []
    for k, pin in zip((2 * s.N, 2 * s.N, s.ntypes, s.nprops, 1), pinned):
        t = torch.zeros(len(x), k, dtype=torch.float64)
        out.append(t.pin_memory() if pin else t)
    out[0].copy_(torch.from_numpy(x))
    return out


def _call(h, buf, absent=None):
    p = [ctypes.cast(None if k == absent else b.data_ptr(), ctypes.POINTER(ctypes.c_double))
         for k, b in enumerate(buf)]
    h._chk(h.lib.qmc2d_compute_properties(h.h, len(buf[0]), *p))


@pytest.mark.parametrize("absent", [None, 1, 3])
def test_any_mixture_of_buffers(q, n26, n26_configs, absent):
    x = np.tile(n26_configs, (2, 1))
    with q.Handle(n26, capacity=len(x), seed=1) as h:
        want = h.compute_properties(x)
        for pinned in itertools.product((False, True), repeat=5):
            buf = _buffers(n26, x, pinned)
            _call(h, buf, absent)
            for k in range(1, 5):
                if k != absent:
                    assert np.array_equal(buf[k].numpy().ravel(), want[k - 1].ravel()), (pinned, k)


def test_pinned_buffers_take_no_staging_memory(q, n26, n26_configs):
    x = np.tile(n26_configs, (NW // len(n26_configs) + 1, 1))[:NW]
    buf = _buffers(n26, x, (True,) * 5)
    hs = [q.Handle(n26, capacity=NW, seed=1) for _ in range(8)]
    _call(hs[0], buf)
    before = _resident_shared()
    for h in hs[1:]:
        _call(h, buf)
    grown = _resident_shared() - before
    for h in hs:
        h.close()
    assert grown < 2 << 20  # seven stagings of 2 NW x 8 (4 N + 2 + n_props + 1) bytes are 14 MB or more
