"""The TVD kernels' reciprocal (csrc/reciprocal.cuh) against the correctly rounded 1.0 / x over its
range: at most one unit in the last place, by the error bound stated there."""
import ctypes as C
import subprocess

import numpy as np
import pytest
import torch

from monc_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "reciprocal.cuh"
template <typename T>
__global__ void k(const T* x, T* a, T* b, long long n) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  a[t] = mgpu::rcp_newton(x[t]);
  b[t] = (T)1.0 / x[t];
}
template <typename T>
static int run(const T* x, T* a, T* b, long long n) {
  k<T><<<(unsigned)((n + 255) / 256), 256>>>(x, a, b, n);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run64(const double* x, double* a, double* b, long long n) { return run<double>(x, a, b, n); }
extern "C" int run32(const float* x, float* a, float* b, long long n) { return run<float>(x, a, b, n); }
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("reciprocal")
    src, so = d / "probe.cu", d / "probe.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "-I", build.CSRC, "-shared", "-o", str(so), str(src),
                    "-lcudart"], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("dtype", [np.float64, np.float32], ids=["fp64", "fp32"])
def test_within_one_unit_of_the_rounded_reciprocal(probe, dtype):
    rng = np.random.default_rng(3)
    powers = np.ldexp(1.0, np.arange(-99, 100)).astype(dtype)
    x = np.concatenate([np.array([1e-30, 1.0, 3.0, 1e30], dtype), powers, np.nextafter(powers, dtype(0)),
                        np.nextafter(powers, dtype(np.inf)), (10.0 ** rng.uniform(-29.9, 29.9, 4_000_000)).astype(dtype),
                        rng.uniform(1.0, 2.0, 4_000_000).astype(dtype)])  # every mantissa region densely
    tx = torch.from_numpy(x).cuda()
    a, b = torch.empty_like(tx), torch.empty_like(tx)
    f = probe.run64 if dtype == np.float64 else probe.run32
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_longlong]
    torch.cuda.synchronize()
    assert f(tx.data_ptr(), a.data_ptr(), b.data_ptr(), x.size) == 0
    it = torch.int64 if dtype == np.float64 else torch.int32
    ulps = (a.view(it) - b.view(it)).abs().max().item()  # positive values: units in the last place
    assert ulps <= 1
