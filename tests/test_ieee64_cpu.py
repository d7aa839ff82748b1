"""fvm_ieee64.h on the host: products, quotients and square roots in integer
arithmetic equal the machine's own operations bit for bit, on random operands
of all magnitudes, on exact and nearly exact results (short and all-ones
significands), at the borders of the exponent window, on zeros, subnormals,
infinities and NaN, and with the float seeds off by their worst error
(rcp.approx: 1 ulp, rsqrt.approx: 2^-22.9; 2^-22 is given here)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fvm2d_gb300",
                    "csrc")
SOURCE = r"""
#include <cstdio>
#include <random>
#include "fvm_ieee64.h"
using namespace fvm;
static std::mt19937_64 rng(12345);
static double from(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
static double operand(int kind) {
  uint64_t u = rng(), k = rng(), e = (u >> 52) & 0x7ff;
  switch (kind) {
    case 0: break;                                                     // anything
    case 1: e = 1003 + k % 40; break;                                  // near one
    case 2: u &= ~((1ull << (k % 53)) - 1); e = 1023 + (k >> 8) % 3; break;   // short
    case 3: u |= (1ull << (k % 53)) - 1; e = 1023; break;              // long runs of ones
    case 4: e = k % 2 ? 766 + (k >> 8) % 5 : 1277 + (k >> 8) % 5; break;      // window's borders
    case 5: e = 723 + k % 600; break;
    default: {
      const uint64_t s[] = {0, 1ull << 63, 1, 0x7ff0000000000000ull, 0xfff0000000000000ull,
                            0x7ff8000000000000ull, 0x000fffffffffffffull, 0x0010000000000000ull,
                            0x7fefffffffffffffull, 0x3ff0000000000000ull, 0xbff0000000000000ull};
      return from(s[k % 11]);
    }
  }
  return from((u & 0x800fffffffffffffull) | (e << 52));
}
static long bad = 0;
static void same(const char *op, double a, double b, double x, double y) {
  if (memcmp(&x, &y, 8) && !(x != x && y != y) && bad++ < 5)
    printf("%s %a %a: %a, machine %a\n", op, a, b, x, y);
}
int main() {
  for (long i = 0; i < 3000000; i++) {
    const double a = operand((int)(rng() % 7)), b = operand((int)(rng() % 7)), c = a < 0 ? -a : a;
    same("mul", a, b, mul64(a, b), a * b);
    same("div", a, b, div64(a, b), a / b);
    same("div", a, a, div64(a, a), a / a);
    same("sqrt", a, a, sqrt64(a), sqrt(a));
    same("sqrt", c, c, sqrt64(c), sqrt(c));
    same("sqrt", c * c, c, sqrt64(c * c), sqrt(c * c));
    if (neg64(a) != (a < 0) || pos64(a) != (a > 0)) bad++;
  }
  printf("%ld differ\n", bad);
  return bad != 0;
}
"""


@pytest.mark.parametrize("off", ["0.0f", "0x1p-22f", "-0x1p-22f"])
def test_integer_arithmetic_equals_ieee(tmp_path, off):
    cxx = os.environ.get("CXX", "g++")
    if not shutil.which(cxx):
        pytest.skip("no C++ compiler")
    src = tmp_path / "t.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "t"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-DFVM_I64_OFF={off}",
                    f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
