"""Configurations with a coordinate that is not a finite number: an evaluation
returns non-finite values wherever the complex kernels do, properties, rho_k of
every wave vector, drift and Laplacian, and leaves the other configurations
alone."""
import importlib
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NW = 600  # enough for the real-orbital kernels


def _evaluate(q, s, x, layout, fused=False):
    """fused: on a stream of the caller's, where the complex kernels evaluate with
    the default layout."""
    import torch

    stream = torch.cuda.Stream().cuda_stream if fused else None
    with q.Handle(s, capacity=len(x), seed=1) as h:
        h.set_inversion(layout)
        xd = torch.from_numpy(x).cuda()
        out = [torch.zeros(len(x), k, dtype=torch.float64, device="cuda")
               for k in (2 * s.N, s.ntypes, s.nprops, 1)]
        torch.cuda.synchronize()
        h.compute_properties_dev(len(x), xd.data_ptr(), *(o.data_ptr() for o in out),
                                 stream=stream)
        with pytest.raises(RuntimeError) as err:
            h.compute_properties_dev_status(len(x), stream=stream)
    return [o.cpu().numpy() for o in out[:3]], str(err.value)


def _case(q, tmp_path, nu, nd, value, axis, backflow):
    tables = importlib.import_module("2degas_b200.tables")
    d = tables.make_run(os.path.join(tmp_path, "d"), "c", nu, nd, 3.0, nconf=NW, seed=11,
                        backflow=(backflow, 3.0, 1.8))
    s = q.System.read(d, "c")
    x = s.read_configs(d, ".0", 0, NW).reshape(NW, -1)
    x[5::9, 2 * (s.N // 2) + axis] = value
    return s, x


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("nu,nd,axis,backflow", [(1, 0, 0, 0.2), (1, 1, 1, 0.2), (13, 13, 0, 0.2),
                                                 (13, 13, 1, 0.0), (29, 0, 1, 0.2),
                                                 (37, 21, 0, 0.2)])
def test_values_are_not_finite_where_the_complex_kernels_have_none(q, tmp_path, nu, nd, axis,
                                                                   backflow, value):
    s, x = _case(q, tmp_path, nu, nd, value, axis, backflow)
    real, cplx = (_evaluate(q, s, x, layout)[0] for layout in (0, 1))
    for u, v in zip(real, cplx):
        assert np.array_equal(np.isfinite(u), np.isfinite(v))


@pytest.mark.parametrize("nu,nd,axis,backflow", [(29, 0, 0, 0.2), (31, 13, 1, 0.0), (33, 13, 0, 0.0),
                                                 (37, 21, 0, 0.2), (57, 57, 1, 0.2), (115, 0, 0, 0.2),
                                                 (33, 129, 0, 0.0)])
def test_the_error_is_that_of_the_complex_kernels(q, tmp_path, nu, nd, axis, backflow):
    s, x = _case(q, tmp_path, nu, nd, np.nan, axis, backflow)
    assert _evaluate(q, s, x, 0)[1] == _evaluate(q, s, x, 0, fused=True)[1]
