"""Set-up that belongs to a device (a kernel's shared-memory limit) is done on
each device, not once per process (csrc/per_device.h), on the CPU."""
import ctypes as C
import re
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "blocksp_b200" / "csrc"

HARNESS = r"""
#include <thread>
#include <vector>
#include "per_device.h"
// how often each of n devices was set up by calls from several threads
extern "C" void run(int n, int threads, int calls, int* setups) {
  static bsp::PerDevice flags[8];
  static int used = 0;
  bsp::PerDevice& f = flags[used++];
  std::vector<std::atomic<int>> c(n);
  auto call = [&](int d) {
    if (!f.has(d)) { c[d]++; f.set(d); }
  };
  std::vector<std::thread> t;
  for (int k = 0; k < threads; ++k)
    t.emplace_back([&, k] { for (int i = 0; i < calls; ++i) call((i + k) % n); });
  for (auto& x : t) x.join();
  for (int d = 0; d < n; ++d) setups[d] = c[d];
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("per_device")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-shared", "-fPIC", "-I", str(CSRC), "-o", str(d / "h.so"),
                    str(d / "h.cpp")], check=True)
    return C.CDLL(str(d / "h.so"))


@pytest.mark.parametrize("threads", [1, 4])
def test_every_device_is_set_up(lib, threads):
    n = (C.c_int * 8)()
    lib.run(8, threads, 800, n)
    assert all(1 <= v <= threads for v in n)


def test_devices_past_the_mask_are_never_skipped(lib):
    n = (C.c_int * 70)()
    lib.run(70, 1, 700, n)
    assert list(n[:64]) == [1] * 64 and list(n[64:]) == [10] * 6


def test_no_limit_is_set_once_per_process():
    """Every cudaFuncSetAttribute either runs at each launch or behind a
    per-device flag: no static of a plain type guards one."""
    for f in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]:
        text = f.read_text()
        for m in re.finditer(r"cudaFuncSetAttribute", text):
            assert not re.search(r"static\s+(bool|int)\s+\w+\s*=", text[max(0, m.start() - 400):m.start()]), f.name
