"""What the library keeps about a GPU is kept per GPU: csrc/per_device.cuh, compiled and run on the host,
and the sources without function-local counts or attributes of whichever device came first."""

import glob
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matfree_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.cuh"

struct Table { int device = -1, counts[36] = {}; };

int main() {
  mfg::PerDevice<Table> t;
  int made = 0;
  auto make = [&](int dev, bool works) {
    return [&made, dev, works](Table &x) { ++made; x.device = dev; return works; };
  };
  // a failure is not kept
  if (t.get(1, make(1, false)) || made != 1) return 1;
  const Table *a = t.get(0, make(0, true)), *b = t.get(1, make(1, true));
  if (!a || !b || a == b || a->device != 0 || b->device != 1 || made != 3) return 2;
  if (t.get(0, make(7, true)) != a || t.get(1, make(7, false)) != b || made != 3) return 3;
  if (t.get(-1, make(0, true)) || t.get(64, make(0, true)) || made != 3) return 4;
  // one value for all threads, complete when it is seen
  for (int round = 0; round < 50; ++round) {
    mfg::PerDevice<Table> s;
    std::atomic<int> calls{0}, wrong{0};
    std::vector<std::thread> ts;
    for (int i = 0; i < 8; ++i)
      ts.emplace_back([&, i] {
        for (int dev = 0; dev < 4; ++dev) {
          const Table *x = s.get(dev, [&](Table &y) {
            ++calls;
            for (int &c : y.counts) c = dev + 5;
            y.device = dev;
            return true;
          });
          if (!x || x->device != dev) ++wrong;
          else
            for (int c : x->counts) wrong += c != dev + 5;
        }
      });
    for (auto &th : ts) th.join();
    if (calls != 4 || wrong) return 5;
  }
  std::puts("ok");
}
"""


def test_one_value_per_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "ok\n"


@pytest.mark.parametrize("name", ["arnoldi_cluster.cu", "gs_cluster.cu", "dense_tcgen05.cu", "operators.cu",
                                  "tridiag_quadrature.cu"])
def test_no_count_of_the_first_device_is_kept(name):
    with open(os.path.join(CSRC, name)) as f:
        src = f.read()
    # function-local statics: the per-device tables, constants, and what is one for a process
    found = re.findall(r"^ +static (?!thread_local)([\w:]+(?:<[^>]*>)?) \w+[^;(]*;", src, re.M)
    assert set(found) <= {"PerDevice<CSlots>", "PerDevice<SplitKSlots>", "PerDevice<int>", "std::once_flag",
                          "PFN_cuTensorMapEncodeTiled_v12000", "const"}, found
    assert not re.search(r"static const (CSlots|SplitKSlots|GSlots<[^>]*>) \w+;", src)
