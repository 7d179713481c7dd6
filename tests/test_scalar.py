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


# FP64 <-> FP32 by integers against the conversions: the ends of FP32's normal range (exponents 896 to
# 898 and 1149 to 1151 of a double), carries into the next exponent and into infinity, ties to even both
# ways, subnormals, zeros, infinities, NaN, and random bits.
def test_conversions_round_as_the_conversions(tmp_path):
    got = _run(tmp_path, """
  long bad = 0, n = 0;
  auto one = [&](double x) {
    const float a = narrow(x), b = (float)x;
    bad += (a != a || b != b) ? !(a != a && b != b) : bits_of(a) != bits_of(b);
    const double w = widen(b), v = (double)b;
    bad += (w != w || v != v) ? !(w != w && v != v) : bits_of(w) != bits_of(v);
    ++n;
  };
  const unsigned long long low[] = {0, 1, 0x0FFFFFFF, 0x10000000, 0x10000001, 0x1FFFFFFF, 0x20000000, 0x30000000,
                                    0xFFFFFFFFFFFFFULL, 0xFFFFFEFFFFFFFULL, 0xFFFFFF0000000ULL, 0xFFFFFE0000000ULL,
                                    0xFFFFFF0000001ULL, 0xFFFFFEFFFFFFFULL};
  for (unsigned long long e = 0; e < 2048; ++e)
    for (unsigned long long m : low)
      for (int s = 0; s < 2; ++s) one(from_bits(((unsigned long long)s << 63) | (e << 52) | m));
  unsigned long long z = 1;
  for (int i = 0; i < 2000000; ++i) {
    z = z * 6364136223846793005ULL + 1442695040888963407ULL;
    const unsigned long long r = z ^ (z >> 29);
    one(from_bits(r));
    one(from_bits((r & 0x800FFFFFFFFFFFFFULL) | ((870 + (r >> 52) % 310) << 52)));   // around FP32's range
  }
  std::printf("%ld %ld", bad, n);""")
    assert got[0] == "0" and int(got[1]) > 4000000


# small_rcp against long double: parts of one size and far apart, exponents over the whole range and at
# the ends of the scaled one.  Bound: a part's error is at most 4 units of 2^-53 (the rounding of
# |a|^2, 1.5; of its product with the quotient's remainder, below 0.1; of the quotient, 1; of the
# reciprocal's own rounding in the correction, below 0.5) where the scaling is taken and 6 where crcp's
# six roundings are; a part that is no normal number may be off by two subnormal steps.
def test_reciprocal_of_a_small_block(tmp_path):
    got = _run(tmp_path, """
  long bad = 0, n = 0;
  unsigned long long z = 7;
  auto next = [&]() { z = z * 6364136223846793005ULL + 1442695040888963407ULL; return z ^ (z >> 29); };
  auto value = [&](int e) { return from_bits((next() & 0x800FFFFFFFFFFFFFULL) | ((unsigned long long)e << 52)); };
  auto one = [&](double2 a) {
    const double2 q = small_rcp(a);
    const int ex = (int)(bits_of(fmax(fabs(a.x), fabs(a.y))) >> 52);
    const long double s = std::ldexp(1.0L, -(ex - 1023)), x = a.x * s, y = a.y * s, d = x * x + y * y;
    const long double want[2] = {x / d * s, -y / d * s};
    const double have[2] = {q.x, q.y};
    const long double unit = std::ldexp(1.0L, -53) * (ex < 64 || ex > 1982 ? 6 : 4);
    for (int i = 0; i < 2; ++i)
      bad += !(std::fabs(have[i] - want[i]) <= unit * std::fabs(want[i]) + (std::fabs(want[i]) < std::ldexp(1.0L, -1021) ?
                                                                           std::ldexp(1.0L, -1073) : 0));
    ++n;
  };
  for (int i = 0; i < 300000; ++i) one({value(1023), value(1018 + (int)(next() % 10))});
  for (int e = 1; e < 2046; ++e)
    for (int f : {e, e - 1, e - 30, e - 60, e - 200, 1})
      if (f > 0) { one({value(e), value(f)}); one({value(f), value(e)}); one({value(e), 0.0}); one({0.0, value(e)}); }
  const double inf = INFINITY, nan = std::nan("");
  for (double2 a : {double2{0, 0}, double2{inf, 1}, double2{1, -inf}, double2{nan, 1}, double2{1, nan}, double2{0x1p-1074, 0}}) {
    const double2 p = small_rcp(a), q = crcp(a);
    bad += !((p.x == q.x || (p.x != p.x && q.x != q.x)) && (p.y == q.y || (p.y != p.y && q.y != q.y)));
  }
  std::printf("%ld %ld", bad, n);""")
    assert got[0] == "0" and int(got[1]) > 300000
