"""Kernel attributes are kept per function and device (parmoon_b200/csrc/func_attr.h):
a handle on a second GPU of the process gets its own.  The bookkeeping compiled for
the host with the runtime call replaced by a recorder, and no other place in the
sources that sets an attribute (once per process, on whatever device was current)."""
import glob
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "parmoon_b200", "csrc")

MAIN = r"""
#include "func_attr.h"
#include <cstdio>
int main() {
  pmg::FuncAttrs a;
  int f, g, calls = 0, rc = 0;
  auto set = [&] { calls++; return rc; };
  auto at = [&](const void *fn, int attr, int device, int value) { a.once(fn, attr, device, value, set); return calls; };
  std::printf("%d ", at(&f, 8, 0, 100));   // first use: 1
  std::printf("%d ", at(&f, 8, 0, 100));   // known: 1
  std::printf("%d ", at(&f, 8, 1, 100));   // another device: 2
  std::printf("%d ", at(&g, 8, 1, 100));   // another function: 3
  std::printf("%d ", at(&g, 9, 1, 100));   // another attribute: 4
  std::printf("%d ", at(&f, 8, 0, 200));   // another value: 5
  std::printf("%d ", at(&f, 8, 1, 100));   // the first device's value is its own: 5
  rc = 7;
  std::printf("%d ", a.once(&f, 8, 2, 100, set));  // a failure is returned: 7
  rc = 0;
  std::printf("%d ", a.once(&f, 8, 2, 100, set));  // and tried again: 0
  std::printf("%d\n", calls);
}
"""


def test_per_function_and_device(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, str(tmp_path / "main.cpp"), "-o", exe])
    assert subprocess.check_output([exe], text=True).split() == "1 1 2 3 4 5 5 7 0 7".split()


def test_one_place_sets_attributes():
    calls = [(os.path.basename(f), line.strip()) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")))
             for line in open(f) if "cudaFuncSetAttribute" in line]
    assert len(calls) == 1 and calls[0][0] == "pmg_api.cu", calls
