"""The branch-free quotients of pangu_b200/csrc/exactdiv.h against `/`, compiled
for the host (the same operations, with std::fma; test_gpu_exactdiv.py has the
device): random operands of the whole range, reciprocals from first approximations
as poor as allowed, zero numerators, and quotients built to lie next to a rounding
boundary."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cmath>
#include "exactdiv.h"
extern "C" void quotients(long n, const double *a, const double *b, const double *rel,
                          double *q, double *q0, int *ok) {
  for (long i = 0; i < n; ++i) {
    const xd::Rcp r = xd::rcp_from(b[i], (1.0 / b[i]) * (1.0 + rel[i]));
    q[i] = xd::quot_s(a[i], r);
    q0[i] = a[i] / b[i];
    ok[i] = xd::in_range_den(b[i]) && xd::in_range0(a[i]) ? 1 : 0;
  }
}
extern "C" void twelfths(long n, const double *a, double *q, double *q0, int *ok) {
  for (long i = 0; i < n; ++i) {
    q[i] = xd::div12(a[i]);
    q0[i] = a[i] / 12.0;
    ok[i] = xd::in_range0(a[i]) ? 1 : 0;
  }
}
"""
_D, _I = C.POINTER(C.c_double), C.POINTER(C.c_int)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("exactdiv")
    src, so = d / "t.cc", d / "t.so"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-shared",
                           "-fPIC", "-I", os.path.join(ROOT, "pangu_b200", "csrc"), str(src),
                           "-o", str(so)])
    return C.CDLL(str(so))


def _same(lib, a, b, rng):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    rel = rng.uniform(-2.0 ** -19, 2.0 ** -19, a.size)
    q, q0, ok = np.empty_like(a), np.empty_like(a), np.empty(a.size, np.int32)
    p = lambda x, t=_D: x.ctypes.data_as(t)  # noqa: E731
    lib.quotients(C.c_long(a.size), p(a), p(b), p(rel), p(q), p(q0), p(ok, _I))
    ok = ok.astype(bool)
    assert np.array_equal(q[ok].view(np.int64), q0[ok].view(np.int64))
    return ok


@pytest.mark.parametrize("ea,eb", [((-1, 1), (-1, 1)), ((-960, 400), (-400, 60)),
                                   ((-1074, -950), (-10, 10)), ((390, 1000), (-420, 70))])
def test_random_operands(lib, ea, eb):
    rng = np.random.default_rng(1)
    n = 300000
    a = rng.choice([-1.0, 1.0], n) * np.ldexp(rng.uniform(1, 2, n), rng.integers(*ea, n))
    b = np.ldexp(rng.uniform(1, 2, n), rng.integers(*eb, n))
    a[:50], a[50:100] = 0.0, -0.0
    ok = _same(lib, a, b, rng)
    if ea[0] >= -960 and ea[1] <= 400:
        assert ok.mean() > 0.999


def next_to_a_rounding_boundary(rng):
    """Operands with A 2^k - M B = K for small K: A / B is within |K| units of the
    midpoint M."""
    a, b = [], []
    for _ in range(20000):
        B = int(rng.integers(2 ** 52, 2 ** 53)) | 1
        for k in (53, 54):
            inv = pow(1 << k, -1, B)
            for K in (-3, -2, -1, 1, 2, 3):
                A = K * inv % B
                if k == 53:
                    A += B if A + B < 2 ** 53 else 0
                if 2 ** 52 <= A < 2 ** 53:
                    a.append(float(A))
                    b.append(float(B))
    assert len(a) > 20000
    return np.array(a), np.array(b)


def test_quotients_next_to_a_rounding_boundary(lib):
    rng = np.random.default_rng(2)
    a, b = next_to_a_rounding_boundary(rng)
    assert _same(lib, a, b, rng).all()


def test_mantissas_of_ones_are_refused_or_right(lib):
    rng = np.random.default_rng(3)
    ones = (np.array([0x3FEFFFFFFFFFFFFF, 0x3FEFFFFFFFFFFFFE, 0x3FF0000000000001,
                      0x3FF0000000000000]).view(np.float64))
    a = rng.uniform(1, 2, 40000)
    b = np.tile(ones, 10000)
    ok = _same(lib, a, b, rng)
    assert not ok[0::4].any() and ok[1::4].all()


def test_division_by_twelve(lib):
    rng = np.random.default_rng(4)
    n = 600000
    a = rng.choice([-1.0, 1.0], n) * np.ldexp(rng.uniform(1, 2, n), rng.integers(-1074, 420, n))
    a[:3] = 0.0, -0.0, np.inf
    m = rng.integers(2 ** 52, 2 ** 53, n // 2)  # next to midpoints: 12 (2 M + 1) / 2 +- 1, +- 2
    a[n // 2:] = ((12 * (2 * (m % 2 ** 49) + 1)) // 2 + rng.integers(-2, 3, n // 2)).astype(float)
    q, q0, ok = np.empty_like(a), np.empty_like(a), np.empty(n, np.int32)
    p = lambda x, t=_D: x.ctypes.data_as(t)  # noqa: E731
    lib.twelfths(C.c_long(n), p(a), p(q), p(q0), p(ok, _I))
    ok = ok.astype(bool)
    assert not ok[2] and ok[:2].all() and ok.mean() > 0.9
    assert np.array_equal(q[ok].view(np.int64), q0[ok].view(np.int64))
