"""What a process settles once a device: a kernel's shared memory is allowed on each device that launches it, never with one flag
for the process (no second GPU is needed: the devices and the driver's answers are made up)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "burn_transformers_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.cuh"

#define SAY(what) if (!(what)) { std::printf("%s\n", #what); return 1; }

int main() {
  bt::SharedMemoryAllowance kernel;
  std::vector<std::pair<int, size_t>> calls;
  auto on = [&](int dev, size_t bytes, bool works = true) {
    return kernel.allow(dev, bytes, [&](size_t n) { calls.push_back({dev, n}); return works; });
  };
  SAY(on(0, 55296) && on(0, 55296) && on(0, 100) && calls.size() == 1);      // once on the first device
  SAY(on(1, 55296) && calls.size() == 2 && calls[1].first == 1);             // again on the second
  SAY(on(0, 60000) && calls.size() == 3 && calls[2].second == 60000);        // more than before
  SAY(on(0, 55296) && calls.size() == 3);
  SAY(!on(2, 300000, false) && on(2, 300000) && calls.size() == 5);          // a refusal is not remembered as a success
  SAY(on(64, 8) && on(64, 8) && on(-1, 8) && calls.size() == 8);             // devices beyond those that are tracked
  bt::SharedMemoryAllowance shared;      // a smaller call that comes later must not take back what a larger one was allowed
  size_t now = 0;
  std::vector<std::thread> threads;
  for (int i = 1; i <= 16; ++i)
    threads.emplace_back([&, i] { for (size_t k = 0; k < 1000; ++k) shared.allow(3, i * 1000 + k, [&](size_t n) { now = n; return true; }); });
  for (auto& t : threads) t.join();
  SAY(now == 16999);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_shared_memory_is_allowed_device_by_device(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(CSRC), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    ran = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert ran.returncode == 0, ran.stdout


def test_no_kernel_keeps_one_flag_for_the_process():
    """A kernel's attribute is set in every call, or behind an allowance or an array that is kept per device."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        if "cudaFuncSetAttribute" not in text and "allow_shared_memory" not in text:
            continue
        found = re.findall(r"static (?:bool|size_t|int|long long) \w+(?:\[\w+\])?(?: =[^;]*)?;", text)
        assert not found, f"{path.name}: {found}"
