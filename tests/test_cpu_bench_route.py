"""What bench.py says of the orbital kernels it timed: the route from the move
inversion mode and layout that moves ran with, and the launches of a scope."""
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("scopes,mode,layout,real", [
    (5, None, 0, True), (5, 1, 0, True), (5, 2, 0, False), (0, 0, 0, False), (0, 1, 1, False),
    (5, 2, 1, False), (5, 1, 1, False)])
def test_the_route(bench, scopes, mode, layout, real):
    assert bench.takes_real(scopes, mode, layout) == real


@pytest.mark.parametrize("ns,backflow,n", [
    ([29, 29], 1, 2), ([29, 29], 0, 1), ([33, 29], 1, 3), ([45, 45], 1, 2), ([115, 31], 1, 4),
    ([161], 1, 3), ([113], 0, 1)])
def test_the_kernels_of_a_scope(bench, ns, backflow, n):
    assert len(bench.orbital_kernels(ns, True, backflow)) == n
    assert bench.orbital_kernels(ns, False, backflow) == ["orb_inv_kernel"]
