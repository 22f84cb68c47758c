"""The real-orbital route of moves (Gamma-point determinants of an odd number of
plane waves as cosines and sines) against the complex kernels on the same
start: one VMC step with every move forced, on spins at the edges of the
kernels' tiles and register rows (one to 161 orbitals, equal and unequal
spins, with and without backflow displacement, mixed precision). Both routes
compute the same FP64 formulas in another order, so the step agrees as moves
agree with the oracle elsewhere in the suite (positions 1e-11, the rest 1e-9
of the largest value). A twist takes the complex kernels and Gamma, set
again, the real ones."""
import importlib
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHELLS = [(1, 1), (3, 1), (5, 5), (9, 0), (15, 13), (17, 17), (31, 25), (31, 33), (33, 0),
          (39, 41), (47, 49), (63, 0), (65, 63), (83, 0), (85, 45), (103, 0), (105, 0), (113, 0),
          (115, 33), (127, 0), (129, 31), (151, 0), (161, 0)]


def _deck(q, tmp_path, nu, nd, **kw):
    tables = importlib.import_module("2degas_b200.tables")
    n = 130 if nd == 0 and nu <= 29 else 6  # small populations of one small spin stay complex
    kw = dict(dict(rs=3.0, backflow=(0.2, 3.0, 1.8), nconf=n, seed=11), **kw)
    d = tables.make_run(os.path.join(tmp_path, "d"), "c", nu, nd, **kw)
    s = q.System.read(d, "c")
    return s, s.read_configs(d, ".0", 0, kw["nconf"])


def _step(q, s, x, mode, precision="fp64"):
    with q.Handle(s, capacity=len(x), seed=77) as h:
        h.set_precision(precision)
        h.set_move_inversion(mode)
        h.population_set(x)
        h.block_reset()
        h.vmc(1, 0.05 * 26 / s.N, 0)  # mage = age: every move is forced
        return h.population_get(), h.block_get()


def _same(a, b, tol):
    # a pair beyond the tables' cut has no drift and an infinite 1 / |g|: the
    # same entries have to be infinite
    fin = np.isfinite(b)
    if not np.array_equal(a[~fin], b[~fin]):
        return False
    a, b = a[fin], b[fin]
    return np.abs(a - b).max() <= tol * max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("nu,nd", SHELLS)
@pytest.mark.parametrize("bf", [0.2, 0.0])
def test_step_equals_the_complex_route(q, tmp_path, nu, nd, bf):
    s, x = _deck(q, tmp_path, nu, nd, backflow=(bf, 3.0, 1.8), u3=nu == 17)
    (r, rb), (c, cb) = _step(q, s, x, 1), _step(q, s, x, 0)
    assert _same(r["x"], c["x"], 1e-11)
    for k in ("g", "h", "p"):
        assert _same(r[k], c[k], 1e-9), k
    assert _same(rb[0], cb[0], 1e-9) and rb[1] == cb[1]


def test_mixed_precision_step(q, tmp_path):
    s, x = _deck(q, tmp_path, 21, 13)
    (r, _), (c, _) = _step(q, s, x, 1, "mixed"), _step(q, s, x, 0, "mixed")
    for k in ("g", "h", "p"):
        assert _same(r[k], c[k], 1e-9), k


@pytest.mark.parametrize("nu,nd", [(45, 45), (45, 47), (49, 31), (93, 69), (95, 67)])
def test_columns_of_one_type_per_cta(q, tmp_path, nu, nd):
    """Both sides of the sizes at which a Laplacian CTA takes one type's
    columns, and at which they no longer fit and are streamed."""
    s, x = _deck(q, tmp_path, nu, nd, backflow=(0.2, 3.0, 1.8))
    (r, _), (c, _) = _step(q, s, x, 1), _step(q, s, x, 0)
    assert _same(r["x"], c["x"], 1e-11)
    for k in ("g", "h", "p"):
        assert _same(r[k], c[k], 1e-9), k


@pytest.mark.parametrize("nu,nd", [(13, 13), (25, 0), (37, 33), (61, 61)])
def test_evaluation_equals_the_fused_kernel(q, tmp_path, nu, nd):
    """Evaluations on the handle's stream (through the move's kernels where the
    configurations are enough) and on a caller's (always the fused kernel)."""
    import torch

    n = 320 if nu < 30 else 5
    s, x = _deck(q, tmp_path, nu, nd, nconf=n)
    st = torch.cuda.Stream()
    with q.Handle(s, capacity=n, seed=1) as h:
        a = h.compute_properties(x)
        with torch.cuda.stream(st):
            xd = torch.from_numpy(x).cuda()
            o = [torch.zeros(n, k, dtype=torch.float64, device="cuda")
                 for k in (2 * s.N, s.ntypes, s.nprops, 1)]
        h.compute_properties_dev(n, xd.data_ptr(), *(t.data_ptr() for t in o),
                                 stream=st.cuda_stream)
        h.compute_properties_dev_status(n, st.cuda_stream)
    for u, v in zip(a, o):
        assert _same(u.reshape(n, -1), v.cpu().numpy(), 1e-9)


def test_reptation_equals_the_complex_route(q, tmp_path):
    s, x = _deck(q, tmp_path, 37, 29, u3=True)
    rng = np.random.default_rng(3)
    walk = np.cumsum(rng.normal(0.0, 0.02, size=(6, 12, x.shape[1])), axis=1)
    paths = (x[:, None, :] + walk).reshape(72, -1)
    out = []
    for mode in (1, 0):
        with q.Handle(s, capacity=6, seed=9) as h:
            h.set_move_inversion(mode)
            h.rmc_init(6, paths, 12, 1, 2, 0.002, -0.4, 10 ** 9, 0)  # every move forced
            h.block_reset()
            h.rmc(2)
            out.append((h.block_get()[0],) + h.rmc_get_path(5, 12))
    for u, v in zip(*out):
        assert _same(u, v, 1e-9)


def test_a_twist_and_gamma_again(q, tmp_path):
    s, x = _deck(q, tmp_path, 13, 13, twist=True)
    ref = {}
    for mode in (1, 0):
        with q.Handle(s, capacity=len(x), seed=5) as h:
            h.set_move_inversion(mode)
            out = []
            for tw in ((0, 0), (1, 2), (0, 0)):
                s.set_twist(*tw)
                h.update_twist()
                h.population_set(x)
                h.vmc(1, 0.05, 0)
                out.append(h.population_get()["p"])
            ref[mode] = out
    s.set_twist(0, 0)
    for a, b in zip(ref[1], ref[0]):
        assert _same(a, b, 1e-9)
    assert not _same(ref[1][1], ref[1][0], 1e-3)
