"""Offsets of the move scratch (move_scratch, real_layout) formed in a kernel stay
in registers: every thread of the move's kernels would otherwise write and read
them in local memory."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2degas_b200",
                    "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

KERNEL = """
#include "walker_eval.cuh"
__global__ void probe(const q2d::DevSys *s, double *x) {
  const q2d::MoveScratch l = q2d::move_scratch(*s);
  x[l.stride * blockIdx.x + l.rhok + threadIdx.x] = 1.0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_scratch_offsets_take_no_local_memory(tmp_path):
    src = tmp_path / "probe.cu"
    src.write_text(KERNEL)
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                        "-Xptxas", "-v", "-I", CSRC, "-c", str(src), "-o", str(tmp_path / "p.o")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert re.findall(r"(\d+) bytes stack frame", r.stderr) == ["0"]


def test_the_complex_kernels_take_the_offsets_from_the_host():
    """At 80 and 166 registers a thread they have none to form them with."""
    with open(os.path.join(CSRC, "kernels.cu")) as f:
        text = f.read()
    for k in ("orb_inv_kernel", "move_kernel"):
        head, body = re.split(r"__global__[^;{]*\b" + k + r"\(", text)[1].split("{", 1)
        assert "MoveScratch L" in head and "move_scratch(" not in body.split("__global__")[0]
