"""Kernel attributes and addresses of __device__ variables belong to a device:
the host code that sets them does so once a device, not once a process."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "libemmi_mgfd_gb300", "csrc")

_PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "emmi_device_once.h"
// a kernel's attribute on each of four devices, one more past the flags
static std::atomic<int> calls[5];
static emmi::DeviceOnce once;
static bool launch(int dev) {
  const int d = dev < emmi::kOnceDevices ? dev : 4;
  emmi::device_once(once, dev, [d] { calls[d]++; });
  return calls[d] > 0;  // the opt-in is there: the launch is taken
}
int main() {
  std::atomic<int> refused{0};
  std::vector<std::thread> t;
  for (int i = 0; i < 8; i++)
    t.emplace_back([&] {
      for (int r = 0; r < 100; r++)
        for (int d : {0, 1, 2, 3, 100}) refused += !launch(d);
    });
  for (auto& v : t) v.join();
  std::printf("%d %d %d %d %d\n", refused.load(), calls[0].load(), calls[1].load(), calls[2].load(),
              calls[3].load());
  return 0;
}
"""


def test_every_device_is_set_up_once(tmp_path):
    src = tmp_path / "once.cpp"
    src.write_text(_PROGRAM)
    exe = str(tmp_path / "once")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, str(src), "-o", exe],
                   check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=60).stdout
    assert out.split() == ["0", "1", "1", "1", "1"]


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_nothing_of_a_device_is_set_under_a_flag_of_the_process(name):
    text = open(os.path.join(CSRC, name)).read()
    for body in re.findall(r"std::call_once\(.*?\}\s*\)\s*;", text, re.S):
        assert not re.search(r"cudaFuncSetAttribute|cudaGetSymbolAddress|init_\w+_kernels", body), body
