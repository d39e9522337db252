"""The row limit that keeps the x sweeps' 32-bit element indexes in range (host arithmetic, no device)."""

import os
import shutil
import subprocess

import pytest

from conftest import PKG

SRC = r"""
#include "sc_sweep_sizes.h"
#include <cstdio>
int main() {
  for (long long len = 2; len <= 1024; ++len) {
    const long long rows = sc::sweep_rows(len);
    // whole pairs; a last warp of up to 64 rows past the end; all 1024^2 rows of the largest plan at once
    if (rows % 2 || (rows + 64) * len > 2147483647LL || (len <= 514 && rows < 1024LL * 1024)) {
      std::printf("%lld: %lld rows\n", len, rows);
      return 1;
    }
  }
  return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs a host compiler")
def test_rows_of_one_launch_are_indexed_in_32_bits(tmp_path):
    (tmp_path / "rows.cpp").write_text(SRC)
    exe = tmp_path / "rows"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(tmp_path / "rows.cpp"), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == ""
