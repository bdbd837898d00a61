"""Row energies read their source in 16-byte groups: a source that does not lie on them is refused on
the host, before any CUDA call (no GPU needed; the launcher is compiled into a small program)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "openclipp_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

MAIN = """
#include <cstdio>
#include "internal.h"
#include "row_energy.h"
namespace ocipb { unsigned long long g_launches; }
int main() {
  using namespace ocipb;
  alignas(16) static char b[4096];
  const RowEnergyJob good{b, 256, 512, b, 256, 512, 8, 2, 1, 3, 1};
  RowEnergyJob bad[5] = {good, good, good, good, good};
  bad[0].src += 4;
  bad[1].src_pitch += 8;
  bad[2].src_plane += 4;
  bad[3].dst += 2;
  bad[4].dst_pitch += 1;
  for (const RowEnergyJob& j : bad)
    if (launch_row_energies(F32, 3, j, nullptr, 1, 8, 2, 0) != cudaErrorInvalidValue) return 1;
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no CUDA compiler")
def test_misaligned_planes_are_refused(tmp_path):
    main, exe = tmp_path / "main.cu", tmp_path / "check"
    main.write_text(MAIN)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), "-o", str(exe), str(main),
                    os.path.join(CSRC, "row_energy.cu")], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
