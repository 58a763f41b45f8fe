"""Rows of the device integrals' Boys-function table: every argument below the
table's end reads a row of it, negative ones (a negative exponent) row 0.  Runs
the kernels' own functions on the host."""
import os
import subprocess

import pytest

from chem_gb300 import build

SRC = r"""
#include <cstdio>
#include <limits>
#include "eri3c_gpu.cuh"
using namespace gbjk;
int main() {
  const double lowest = std::numeric_limits<double>::lowest();
  const double inf = std::numeric_limits<double>::infinity();
  for (double T : {0.0, -0.0, 1e-300, -1e-300, 0.03, 1.0 / 32, -1.0 / 32, 32.96875, 32.97, 33.0,
                   -33.0, -1000.0, -1e9, lowest, -inf})
    std::printf("%a %d %d\n", T, eri_boys_row(eri_boys_arg(T)), kEriBoysRows);
  const double nan = std::numeric_limits<double>::quiet_NaN();
  std::printf("nan %d\n", eri_boys_arg(nan) != eri_boys_arg(nan) &&
                              eri_boys_arg(-nan) != eri_boys_arg(-nan));
}
"""


def test_rows(tmp_path):
    if not os.path.exists(build.NVCC):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "rows.cu", tmp_path / "rows"
    src.write_text(SRC)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-I" + build.CSRC, str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = [line.split() for line in out if line and not line.startswith("nan")]
    assert len(rows) == 15
    for t, row, n in rows:
        T = float.fromhex(t) if "inf" not in t else float(t)
        want = int(16 * T + 0.5) if T > 0 else 0
        assert 0 <= int(row) < int(n) and int(row) == want, t
    assert "nan 1" in out
