"""The kernels' scalar helpers (csrc/scalar.cuh), compiled for the host."""
import os
import subprocess

import pytest

from nonequilibriumgreensfunction_gb300 import _build

from conftest import REPO

CSRC = os.path.join(REPO, "nonequilibriumgreensfunction_gb300", "csrc")


def _run(tmp_path, body):
    src, exe = str(tmp_path / "t.cu"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write('#include <cstdio>\n#include "negf_internal.cuh"\nusing namespace negf;\nint main() {\n%s\n}\n'
                % body)
    subprocess.run([_build._nvcc(), *_build.NVCC_FLAGS, "-O1", "-I", CSRC, src, "-o", exe], check=True)
    return subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()


# A decimation step's largest change is NaN when any of a thread's elements is, the first, one in the
# middle or the last, and whatever follows it.
def test_largest_change_keeps_a_nan(tmp_path):
    got = _run(tmp_path, """
  const double nan = std::nan(""), inf = INFINITY;
  const double runs[][4] = {{nan, 1, 2, 3}, {1, nan, 2, 3}, {1, 2, 3, nan}, {inf, -nan, 1, 0}, {nan, inf, 0, 0},
                            {1, 3, 2, 0}, {0, 0, 0, 0}, {1, inf, 2, 3}};
  for (auto& r : runs) {
    double m = 0.0;
    for (double v : r) m = max_or_nan(m, v);
    std::printf("%llx ", bits_of(m));
  }""")
    nan, one = "7ff8000000000000", "4008000000000000"
    assert got == [nan] * 5 + [one, "0", "7ff0000000000000"]
