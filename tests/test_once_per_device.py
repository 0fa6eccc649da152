"""The once-per-device set-up of csrc/fl_once.h (CPU only): no caller returns before the set-up of its
device has ended, whichever thread runs it, and each device is set up once."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fluidity_b200" / "csrc"

PROGRAM = r"""
#include "fl_once.h"
#include <atomic>
#include <chrono>
#include <thread>
#include <vector>

int main() {
  static fl::OncePerDevice once;
  std::atomic<int> waiting{0}, runs[3] = {}, ready[3] = {}, early{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 12; ++t)
    threads.emplace_back([&, t] {
      const int device = t % 3;
      ++waiting;
      while (waiting < 12) std::this_thread::yield();
      once.run(device, [&] {
        ++runs[device];
        std::this_thread::sleep_for(std::chrono::milliseconds(50));
        ready[device] = 1;
      });
      if (!ready[device]) ++early;
    });
  for (auto& t : threads) t.join();
  if (early != 0) return 1;
  for (auto& r : runs)
    if (r != 1) return 2;
  int outside = 0;  // devices without a flag are set up every time
  for (int k = 0; k < 2; ++k) {
    once.run(-1, [&] { ++outside; });
    once.run(fl::OncePerDevice::kDevices, [&] { ++outside; });
  }
  return outside == 4 ? 0 : 3;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_no_caller_returns_before_its_device_is_set_up(tmp_path):
    src, exe = tmp_path / "once.cc", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)])
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


def test_every_kernel_attribute_is_set_through_it():
    """A kernel's attributes are set for the current device only: every place that sets one does so
    through OncePerDevice or, the cluster query, per device until its answer is stored."""
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        for at in (i for i in range(len(text)) if text.startswith("cudaFuncSetAttribute(", i)):
            before = text[:at]
            scope = before[max(before.rfind("once_on_device("), before.rfind("known[dev] == 0")):]
            assert scope.startswith(("once_on_device(", "known[dev]")) and "\n}\n" not in scope, (path.name, text[at:at + 80])
