"""pangu_b200/csrc/exactdiv.h on the device: the error of the first approximation that
its proof (and the Newton step's convergence test) assumes, and quotients, reciprocals
and twelfths against the device's `/`."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from test_exactdiv import next_to_a_rounding_boundary  # noqa: E402

from pangu_b200 import build  # noqa: E402

pytestmark = pytest.mark.gpu

SRC = r"""
#include "exactdiv.h"
// |1 - b y0| over every value of the upper 20 mantissa bits, with the lowest, a middle
// and the highest accepted lower word, as bits ordered like the number.
__global__ void seed_error(int expo, unsigned long long *worst) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;  // 2^20 threads
  const unsigned low[4] = {0u, 1u, 0x7fffffffu, 0xfffffffeu};
  for (unsigned lo : low) {
    const double b = __hiloint2double((int)((unsigned)(1023 + expo) << 20 | i), (int)lo);
    const double e = fabs(__fma_rn(-b, xd::rcp_seed(b), 1.0));
    atomicMax(worst, (unsigned long long)__double_as_longlong(e));
  }
}
__global__ void divide(long n, const double *a, const double *b, double *o, int *ok) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  o[i] = xd::quot_s(a[i], xd::rcp(b[i]));
  o[n + i] = a[i] / b[i];
  o[2 * n + i] = xd::recip(b[i]);
  o[3 * n + i] = 1.0 / b[i];
  o[4 * n + i] = xd::div12(a[i]);
  o[5 * n + i] = a[i] / 12.0;
  ok[i] = (xd::in_range0(a[i]) ? 1 : 0) | (xd::in_range_den(b[i]) ? 2 : 0);
}
extern "C" int run_seed_error(int expo, unsigned long long *worst) {
  seed_error<<<1 << 12, 256>>>(expo, worst);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run_divide(long n, const double *a, const double *b, double *o, int *ok) {
  divide<<<(unsigned)((n + 127) / 128), 128>>>(n, a, b, o, ok);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("exactdiv")
    src, so = d / "t.cu", d / "t.so"
    src.write_text(SRC)
    subprocess.check_call([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false",
                           "-shared", "-Xcompiler", "-fPIC", "-I", build.CSRC, str(src), "-o",
                           str(so)])
    return C.CDLL(str(so))


@pytest.mark.parametrize("expo", [-400, -1, 0, 1, 59])
def test_first_approximation(lib, expo):
    worst = torch.zeros(1, dtype=torch.int64, device="cuda")
    assert lib.run_seed_error(expo, C.c_void_p(worst.data_ptr())) == 0
    assert 0.0 < worst.cpu().numpy().view(np.float64)[0] < 2.0 ** -19


@pytest.mark.parametrize("kind", ["wide", "narrow", "boundary", "twelfths"])
def test_same_bits_as_division(lib, kind):
    rng = np.random.default_rng(21)
    n = 1 << 20
    sign = rng.choice([-1.0, 1.0], n)
    b = np.ldexp(rng.uniform(1, 2, n), rng.integers(-400, 60, n))
    if kind == "wide":
        a = sign * np.ldexp(rng.uniform(1, 2, n), rng.integers(-960, 400, n))
        a[:64], a[64:128] = 0.0, -0.0
    elif kind == "narrow":
        a, b = sign * rng.uniform(1, 2, n), rng.uniform(1, 2, n)
    elif kind == "boundary":
        a, b = next_to_a_rounding_boundary(rng)
    else:  # 12 (2 M + 1) / 2 and its neighbours
        m = rng.integers(2 ** 48, 2 ** 49, n)
        a = ((12 * (2 * m + 1)) // 2 + rng.integers(-2, 3, n)).astype(float)
    n = a.size
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    out = torch.empty((6, n), dtype=torch.float64, device="cuda")
    ok = torch.empty(n, dtype=torch.int32, device="cuda")
    ptr = [C.c_void_p(t.data_ptr()) for t in (ta, tb, out, ok)]
    assert lib.run_divide(C.c_long(n), *ptr) == 0
    bits, ok = out.cpu().numpy().view(np.int64), ok.cpu().numpy()
    assert (ok == 3).mean() > 0.99
    assert np.array_equal(bits[0][ok == 3], bits[1][ok == 3])
    assert np.array_equal(bits[2][ok & 2 != 0], bits[3][ok & 2 != 0])
    assert np.array_equal(bits[4][ok & 1 != 0], bits[5][ok & 1 != 0])
