"""A refused dependent launch (``launch_pdl`` of ops/csrc/common.cuh) returns its error and leaves none for the next call."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "create_llm_by_cupy_b200" / "ops" / "csrc"

pytestmark = pytest.mark.gpu            # without a driver every call reports its absence

PROGRAM = r"""
#include "common.cuh"

__global__ void kernel(int* p) { if (p) *p = 1; }

int main() {
  // more threads than a block can have: refused on the host
  const cudaError_t e = b200::launch_pdl(kernel, dim3(1), dim3(4096), 0, nullptr, 0, static_cast<int*>(nullptr));
  const cudaError_t left = cudaGetLastError();
  printf("%d %d\n", int(e), int(left));
  return e != cudaSuccess && left == cudaSuccess ? 0 : 1;
}
"""


def test_refused_launch_leaves_no_error(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src, exe = tmp_path / "launch.cu", tmp_path / "launch"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
