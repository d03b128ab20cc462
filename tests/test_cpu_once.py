"""pie_once.h: a kernel's attributes are set once per device, and nobody goes on without them (compiled and run on the host)."""
import shutil
import subprocess

import pytest

from proxy_inference_engine_b200._lib import CSRC

SOURCE = r"""
#include <atomic>
#include <thread>
extern "C" { typedef int cudaError_t; }
enum { cudaSuccess = 0 };
static thread_local int device = 0;
static int cudaGetDevice(int* d) { *d = device; return 0; }
#include "pie_once.h"

int main() {
  std::atomic<unsigned long long> served{0};
  // a second thread that comes while the first is still setting must set for itself
  std::atomic<int> sets{0};
  std::thread other;
  pie::once_per_device(served, [&] {
    ++sets;
    other = std::thread([&] { pie::once_per_device(served, [&] { ++sets; return 0; }); });
    other.join();
    return 0;
  });
  if (sets != 2) return 1;
  // afterwards nobody does, and another device does
  pie::once_per_device(served, [&] { ++sets; return 0; });
  if (sets != 2) return 2;
  device = 1;
  if (pie::once_per_device(served, [&] { ++sets; return 5; }) != 5 || sets != 3) return 3;   // a failure is reported
  pie::once_per_device(served, [&] { ++sets; return 0; });                                   // and tried again
  pie::once_per_device(served, [&] { ++sets; return 0; });
  return sets == 4 ? 0 : 4;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_attributes_are_set_before_anyone_goes_on(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text("")   # the stand-ins above
    (tmp_path / "once.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-pthread", "-I", str(tmp_path), "-I", CSRC, "once.cpp", "-o", "once"], cwd=tmp_path)
    assert subprocess.call([str(tmp_path / "once")]) == 0
