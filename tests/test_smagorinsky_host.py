"""The subgrid model of a run with fewer than two q fields, on the CPU: the device function compiled for
the host, with q-field accessors that count their reads.  Such a model has no liquid field to
read, and the kernels leave the accessors unset."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monc_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROBE = r"""
#include <cuda_runtime.h>
#undef __device__
#undef __forceinline__
#define __device__
#define __forceinline__ inline
#include <cmath>
#include <cstdio>
using std::acos; using std::copysign; using std::cos; using std::exp; using std::fabs; using std::log; using std::pow;
using std::signbit; using std::sqrt;
template <class T> T __ldg(const T* p) { return *p; }
inline double __drcp_rn(double x) { return 1.0 / x; }
inline float __frcp_rn(float x) { return 1.0f / x; }
#include "dycore_device.host.h"
using namespace mgpu;
static int reads = 0;
struct Profile { double operator()(int, int k) const { return 1.0 + 0.01 * k; } };
struct Field { double operator()(int k, int, int) const { return 0.1 * k; } };
// one accessor type serves theta and the q fields, as in the kernels
struct Counted { int q; double operator()(int k, int, int) const { reads += q; return 0.1 * k; } };
int main() {
  for (int nq = 0; nq <= 2; ++nq)
    for (int passive_q = 0; passive_q <= 1; ++passive_q) {
      Scalars s{};
      s.nx = s.ny = s.nz = 8;
      s.subb = 40.0; s.subc = 16.0; s.suba = 1.4; s.ric = 0.25; s.ricinv = 4.0; s.eps = 0.01; s.repsh = 50.0;
      s.passive_q = passive_q; s.nq = nq; s.iql = nq > 1;
      reads = 0;
      double vis = 0.0, diff = 0.0;
      const Counted th{0}, q{1};
      smagorinsky_from_strain<double, Profile, Field, Counted>(s, Profile{}, 1e-4, Field{}, th, &q, &q, 3, 0, 0, vis, diff);
      if ((reads > 0) != (nq == 2 && !passive_q)) {
        std::printf("nq %d passive_q %d: %d reads of the q fields\n", nq, passive_q, reads);
        return 1;
      }
    }
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")), reason="no CUDA headers")
@pytest.mark.parametrize("contracted", [False, True], ids=["separate", "contracted"])
def test_fewer_than_two_q_fields_are_not_read(tmp_path, contracted):
    text = open(os.path.join(CSRC, "dycore_device.cuh")).read()
    for t in ("64", "32"):  # the host has no PTX
        c = "d" if t == "64" else "f"
        text = text.replace(f'asm("div.rn.f{t} %0, %1, %2;" : "={c}"(q) : "{c}"(x), "{c}"(r));', "q = x / r;")
    assert "asm(" not in text
    (tmp_path / "dycore_device.host.h").write_text(text.replace('"mgpu_internal.h"', f'"{CSRC}/mgpu_internal.h"'))
    (tmp_path / "probe.cpp").write_text(PROBE)
    exe = tmp_path / "probe"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", *(["-DMGPU_CONTRACTED"] if contracted else []), "-I", str(tmp_path),
                    "-I", os.path.join(CUDA, "include"), str(tmp_path / "probe.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
