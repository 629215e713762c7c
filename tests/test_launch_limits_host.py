"""Kernels with more than the default shared memory are set up on every device they run on: the
launchers' table of limits against a fake CUDA runtime with several devices and failing calls."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monc_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROBE = r"""
#include "launch_limits.h"
#include <cstdio>
#include <map>
#include <thread>
#include <vector>

// the fake runtime: the calling thread's device, and per device and kernel the shared memory allowed
static thread_local int cur = 0;
static std::mutex mu;
static std::map<std::pair<int, const void*>, int> smem_of;
static int attribute_calls = 0, fail_attributes = 0;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = cur; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> l(mu);
  ++attribute_calls;
  if (fail_attributes > 0) { --fail_attributes; return cudaErrorInvalidValue; }
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_of[{cur, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
  *n = cur == 1 ? 0 : 2;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int dev) { *v = 100 + dev; return cudaSuccess; }
}
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  using namespace mgpu;
  int k1, k2;
  static LaunchTable t;
  auto get = [&] { return launch_limits(t, {&k1, &k2}, 256, 100000); };
  for (int round = 0; round < 2; ++round)
    for (int dev = 0; dev < 3; ++dev) {
      cur = dev;
      const LaunchLimits l = get();
      CHECK(l.nsm == 100 + dev);
      CHECK(l.occ == (dev == 1 ? 1 : 2));  // never 0
      CHECK((smem_of[{dev, &k1}] == 100000 && smem_of[{dev, &k2}] == 100000));
    }
  CHECK(attribute_calls == 3 * 4);  // once a device
  // a kernel that could not be set up is tried again
  cur = 3;
  fail_attributes = 1;
  get();
  CHECK(!smem_of.count({3, &k1}));
  get();
  CHECK((smem_of[{3, &k1}] == 100000));
  // devices beyond the table are set up on every call
  cur = LAUNCH_DEVICES;
  CHECK(get().nsm == 100 + LAUNCH_DEVICES);
  CHECK((smem_of[{LAUNCH_DEVICES, &k2}] == 100000));
  // threads on several devices at the same time
  static LaunchTable t2;
  smem_of.clear();
  std::vector<std::thread> ts;
  std::vector<int> bad(8, 0);
  for (int q = 0; q < 8; ++q)
    ts.emplace_back([&, q] {
      cur = q % 4;
      for (int n = 0; n < 1000; ++n) bad[q] += launch_limits(t2, {&k1}, 256, 5).nsm != 100 + cur;
    });
  for (auto& th : ts) th.join();
  for (int b : bad) CHECK(b == 0);
  for (int dev = 0; dev < 4; ++dev) CHECK((smem_of[{dev, &k1}] == 5));
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")), reason="no CUDA headers")
def test_limits_are_set_up_on_every_device(tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", os.path.join(CUDA, "include"), str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_every_launcher_of_the_dynamics_uses_the_table():
    """No launcher raises a limit, or keeps an occupancy, once a process."""
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read()
        assert not re.search(r"static int \w*occ|static int \w*nsm", text), f
        if f not in ("launch_limits.h", "fft.cu"):  # fft.cu keeps a flag a device
            assert "cudaFuncSetAttribute" not in text, f
