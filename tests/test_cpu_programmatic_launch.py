"""Kernels launched while their predecessor drains (launch_pdl) must not read its
results through the read-only path (__ldg, ld.global.nc), which asks for data
that is constant for the kernel's whole life and whose loads no barrier holds
back: in the real-orbital sources it is for the wave vectors alone, and every
such kernel waits for its predecessors (pdl_wait) before anything else that it
reads from device memory."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2degas_b200",
                    "csrc")


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", ["real.cu", "real_det.cuh"])
def test_read_only_loads_are_of_the_wave_vectors(name):
    args = re.findall(r"__ldg\(([^)]*)", _text(name))
    assert all(re.match(r"(a\.)?gvec\b", a) for a in args), args


@pytest.mark.parametrize("name", ["real.cu", "kernels.cu", "rmc.cu"])
def test_every_programmatic_kernel_waits(name):
    text = _text(name)
    launched = set(re.findall(r"launch_pdl\(\s*(?:q2d::)?(\w+)", text)) - {"void", "k"}
    if "launch_pdl(k," in text:  # a kernel chosen by its template's arguments
        launched.add("real_inv_cta_kernel")
    assert launched
    for k in launched:
        body = re.split(r"__global__[^;{]*\b" + k + r"\(", text)[1].split("__global__")[0]
        assert "pdl_wait();" in body, k
