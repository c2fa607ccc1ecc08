"""The twiddles of lines of any length (csrc/lines.cuh cis_ratio) are cos and sin rounded
once to float: compiled for the host from the header's own text, over every length up
to 320 and a sweep to 16384 (Bluestein's chirp has denominators of twice the length).
A sum cut at 1e-10 can miss the nearest float where the value lies within 1e-10 of the
middle of two: in at most 1e-10 / 3e-8 of the cases, taken tenfold."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import PKG_NAME, ROOT

PROGRAM = r"""
#include <cmath>
#include <cstdio>
struct float2 { float x, y; };
static float2 make_float2(float x, float y) { return {x, y}; }
static int __float2int_rn(float x) { return int(rintf(x)); }
#define PTY_DEVI static
%s
int main() {
  long n = 0, off = 0;
  double worst = 0.0;
  for (int den = 1; den <= 16384; den += den < 640 ? 1 : 61)
    for (int i = 0; i < den; ++i) {
      const float2 w = cis_ratio(i, den);
      long double a = -2.0L * 3.14159265358979323846264338L * i / den;
      long double c = cosl(a), s = sinl(a);
      if (4 * i %% den == 0) c = roundl(c), s = roundl(s);  // whole quarter turns are exact
      off += (w.x != float(c)) + (w.y != float(s));
      worst = std::fmax(worst, std::fmax(fabsl(w.x - c), fabsl(w.y - s)));
      n += 2;
    }
  printf("%%ld %%ld %%.9g\n", n, off, worst);
}
"""


def test_rounded_once(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("needs a host C++ compiler")
    text = open(os.path.join(ROOT, PKG_NAME, "csrc", "lines.cuh")).read()
    body = re.search(r"(PTY_DEVI float2 cis_ratio\(.*?\n}\n)", text, re.S).group(1)
    helper = re.search(r"(PTY_DEVI double2 cis_ratio64\(.*?\n}\n)", text, re.S)
    (tmp_path / "t.cpp").write_text(PROGRAM % ((helper.group(1) if helper else "") + body))
    exe = str(tmp_path / "t")
    subprocess.run([cxx, "-O2", "-std=c++17", str(tmp_path / "t.cpp"), "-lm", "-o", exe], check=True)
    n, off, worst = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert int(n) > 4_000_000
    assert int(off) <= 10 * 1e-10 / 3e-8 * int(n)
    assert float(worst) <= 2.0 ** -25 + 1e-9
