"""The launch helper (csrc/launch_retry.cuh, host code) against a fake runtime that keeps
a sticky last error until it is read: a failed first attempt followed by a good second
one is a success, one attempt that works is not repeated, and no failure leaves an
error behind for the next call."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG_NAME, ROOT

PROGRAM = r"""
#include <cassert>
#include "launch_retry.cuh"

struct Runtime {
  int fail_launches, fail_set_ups, last = 0, launches = 0, set_ups = 0, forced = 0;
  bool run() {
    return pty::launch_retry(
        [&](bool again) {
          ++set_ups;
          forced += again;
          if (fail_set_ups-- > 0) return last = 3, false;
          return true;
        },
        [&] {
          ++launches;
          return fail_launches-- > 0 ? last = 7 : 0;
        },
        [&] {
          const int e = last;
          last = 0;
          return e;
        });
  }
};

int main() {
  Runtime good{0, 0};
  assert(good.run() && good.launches == 1 && good.forced == 0 && good.last == 0);
  Runtime lost{1, 0};  // attributes gone: set up again, then queued
  assert(lost.run() && lost.launches == 2 && lost.set_ups == 2 && lost.forced == 1 && lost.last == 0);
  Runtime dead{2, 0};
  assert(!dead.run() && dead.launches == 2 && dead.last == 0);
  Runtime refused{0, 1};
  assert(!refused.run() && refused.launches == 0 && refused.last == 0);
  Runtime earlier{0, 0};  // an error left by someone else fails the first attempt only
  earlier.last = 5;
  assert(earlier.run() && earlier.last == 0);
  return 0;
}
"""


def test_launch_retry(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("needs a host C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, PKG_NAME, "csrc"), str(src), "-o",
                    str(exe)], check=True)
    subprocess.run([str(exe)], check=True)
