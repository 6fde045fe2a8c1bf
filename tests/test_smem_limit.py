"""The shared-memory limit of a kernel is set on every device that launches it (no GPU: the runtime's two calls are replaced)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "oasr_b200" / "csrc"
PROGRAM = r"""
#include "smem_limit.cuh"
#include <cstdio>
static int device = 0, calls[70], failures = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
  if (failures > 0) { --failures; return cudaErrorInvalidValue; }
  calls[device] += bytes == 4096;
  return cudaSuccess;
}
void kernel(int) {}
int main() {
  static ob::SmemLimit limit;
  const int order[] = {0, 0, 3, 0, 3, 63, 63, 66, 66};
  for (int d : order) { device = d; if (limit.raise(kernel, 4096) != cudaSuccess) return 1; }
  device = 5; failures = 1;
  if (limit.raise(kernel, 4096) != cudaErrorInvalidValue || limit.raise(kernel, 4096) != cudaSuccess) return 2;
  std::printf("%d %d %d %d %d\n", calls[0], calls[3], calls[63], calls[66], calls[5]);
}
"""


def test_every_device_gets_the_limit_once_and_a_failure_is_tried_again(tmp_path):
    nvcc = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")
    (tmp_path / "t.cc").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", str(nvcc.parent.parent / "include"), "-o", "t", "t.cc"], cwd=tmp_path, check=True)
    assert subprocess.run(["./t"], cwd=tmp_path, check=True, capture_output=True, text=True).stdout.split() == ["1", "1", "1", "2", "1"]


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_no_launcher_keeps_one_flag_for_all_devices(name):
    assert not re.search(r"\bstatic\s+(std::atomic<)?bool>?\s+\w+\s*[={;]", (CSRC / name).read_text())
