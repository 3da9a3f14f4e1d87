"""Launch attributes are set once on each device of a process, not once in the
process: the kernels' set-up over several devices and threads, on the host, and
no launcher that keeps it behind a flag of the process."""
import os
import re
import subprocess

from pdesolver_gb300 import build

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "eg_device_once.h"

std::atomic<int> calls[70];

void launch(int dev) {  // as a launcher does
  static EgDeviceOnce once;
  once(dev, [dev] { ++calls[dev]; });
}

int main() {
  std::vector<std::thread> t;
  for (int k = 0; k < 8; ++k)
    t.emplace_back([] {
      for (int dev = 0; dev < 64; ++dev) launch(dev);
    });
  for (auto& x : t) x.join();
  for (int dev = 0; dev < 64; ++dev)
    if (calls[dev] != 1) return 1;
  launch(64);  // beyond the flags: at every call
  launch(64);
  return calls[64] == 2 ? 0 : 2;
}
"""


def test_once_on_each_device(tmp_path):
    src = tmp_path / "once.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "once")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", build.CSRC, str(src), "-o", exe], check=True)
    assert subprocess.run([exe], timeout=60).returncode == 0


def test_no_launch_attribute_behind_a_flag_of_the_process():
    for name in sorted(os.listdir(build.CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(build.CSRC, name)) as f:
            text = f.read()
        for body in re.findall(r"static (?:const )?\w+ \w+ = \[\] \{(.*?)\n  \}\(\);", text, re.S):
            assert "cudaFuncSetAttribute" not in body, name
