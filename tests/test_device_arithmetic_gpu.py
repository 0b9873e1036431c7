"""Device functions of the headers themselves, compiled into a library of their
own: the division by the speed of light bit for bit against x / C, and the
sines of the complex folds against float64."""

from __future__ import annotations

import ctypes as C
import subprocess
from fractions import Fraction

import numpy as np
import pytest
import torch

from pyloki_gb300 import build

pytestmark = pytest.mark.gpu

CVAL = 299792458.0

SOURCE = r"""
#include "loki_common.cuh"
#include "sincos.cuh"
using namespace loki;
__global__ void div_kernel(const double* x, int n, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = div_c(x[i]);
}
__global__ void sincos_kernel(const float* a, int n, int way, float* s, float* c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (way == 0) sincos_small(a[i], s + i, c + i);
  else if (way == 1) sincos_mid(a[i], s + i, c + i);
  else sincos_reduced(a[i], s + i, c + i);
}
extern "C" int div_run(const double* x, int n, double* out) {
  div_kernel<<<(n + 255) / 256, 256>>>(x, n, out);
  return (int)cudaDeviceSynchronize();
}
extern "C" int sincos_run(const float* a, int n, int way, float* s, float* c) {
  sincos_kernel<<<(n + 255) / 256, 256>>>(a, n, way, s, c);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("device")
    (d / "arith.cu").write_text(SOURCE)
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-I", str(build.CSRC), "-shared",
                    str(d / "arith.cu"), "-o", str(d / "arith.so"), "-lcudart"], check=True)
    lib = C.CDLL(str(d / "arith.so"))
    lib.div_run.argtypes = [C.c_void_p, C.c_int, C.c_void_p]
    lib.sincos_run.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    return lib


def _divisors():
    """Random doubles of every exponent, those whose quotients lie next to a
    midpoint of two doubles, both ends of the window in which the division takes
    two operations, and what it leaves to the division itself."""
    rng = np.random.default_rng(1)
    mant = rng.uniform(1.0, 2.0, 200_000)
    x = [np.ldexp(mant, rng.integers(-1074, 1024, mant.size))]
    mid = np.array([float(Fraction(2 * k + 1, 1 << 53) * 299792458)
                    for k in rng.integers(1 << 52, 1 << 53, 2000).tolist()])
    for e in (-1040, -860, -850, -300, 0, 300, 700, 740, 750):
        y = np.ldexp(mid, e)
        x += [y, np.nextafter(y, np.inf), np.nextafter(y, 0.0)]
    edge = np.ldexp(1.0, np.array([-1074, -1023, -1022, -824, -823, -822, 775, 776, 777, 1023]))
    x += [edge, np.nextafter(edge, np.inf), np.nextafter(edge, 0.0),
          np.array([0.0, np.inf, np.nan, 5e-324, np.finfo(np.float64).max, CVAL, 3 * CVAL])]
    x = np.concatenate(x)
    return np.concatenate([x, -x])


def test_div_c_is_the_division(cuda_device, lib):
    x = _divisors()
    t = torch.from_numpy(x).to(cuda_device)
    out = torch.zeros_like(t)
    torch.cuda.synchronize(cuda_device)
    assert lib.div_run(t.data_ptr(), t.numel(), out.data_ptr()) == 0
    with np.errstate(over="ignore", under="ignore"):
        want = x / CVAL
    got = out.cpu().numpy()
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.int64), want[~nan].view(np.int64))


@pytest.mark.parametrize(("way", "top"), [(0, 1.9e5), (1, 1.6e6), (2, 2.05e5), (2, 1e8)])
def test_sines_against_float64(cuda_device, lib, way, top):
    """Within 1.6 x 2^-24; where sincosf is called, within its 2 x 2^-24 and half a
    unit, 2 x 2^-24, of an angle reduced to [-pi, pi]."""
    rng = np.random.default_rng(way)
    a = np.concatenate([rng.uniform(-top, top, 1_000_000), rng.uniform(-2.0, 2.0, 100_000),
                        np.arange(-2000, 2000) * (np.pi / 4), [0.0, -0.0, top, -top]])
    a = a[np.abs(a) <= top].astype(np.float32)
    t = torch.from_numpy(a).to(cuda_device)
    s, c = torch.zeros_like(t), torch.zeros_like(t)
    torch.cuda.synchronize(cuda_device)
    assert lib.sincos_run(t.data_ptr(), t.numel(), way, s.data_ptr(), c.data_ptr()) == 0
    bound = (4.0 if way == 2 else 1.6) * 2.0**-24
    x = a.astype(np.float64)
    assert np.abs(s.cpu().numpy() - np.sin(x)).max() <= bound
    assert np.abs(c.cpu().numpy() - np.cos(x)).max() <= bound
