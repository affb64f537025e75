"""Kernel attributes belong to a device: the helper that sets them runs once for each current device, runs again after a
failure, and every kernel that needs one gets it through the helper.  (The helper is compiled against a cudaGetDevice
of the test's own: no GPU.)"""
import re
import subprocess

from xped_gb300.build import CSRC, CUDA_HOME

MAIN = r"""
#include <cstdio>
#include <stdexcept>
#include "per_device.hpp"
static int device = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
int main() {
  static xgb::PerDevice attr;
  int runs = 0;
  for (int d : {0, 1, 0, 2, 1, 0}) {
    device = d;
    attr.once([&] { ++runs; });
  }
  static xgb::PerDevice failing;
  int tries = 0;
  for (int i = 0; i < 3; ++i) {
    try {
      failing.once([&] { if (++tries == 1) throw std::runtime_error("once"); });
    } catch (const std::exception&) {
    }
  }
  std::printf("%d %d\n", runs, tries);
}
"""


def test_once_for_each_device(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(CSRC), "-I", str(CUDA_HOME / "include"),
                    str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split() == ["3", "2"]


def test_attributes_are_set_through_it():
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        for m in re.finditer(r"cudaFuncSetAttribute\(", text):
            opened = text.rfind(".once(", 0, m.start())
            assert opened >= 0 and "\n  });" not in text[opened:m.start()], (path.name, text[m.start():m.start() + 80])
