"""The strip solve's division by a stored reciprocal (div_by, tl_device.cuh)
against the division operator.  The header is compiled for the host, whose
fma() and arithmetic are IEEE's as the GPU's are, so the bits are the same."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = """
#include <math.h>
#include <stdint.h>
#include <string.h>
#define __device__
#define __noinline__
#define __forceinline__ inline
static inline int __double2hiint(double x) {
    uint64_t b;
    memcpy(&b, &x, 8);
    return (int)(uint32_t)(b >> 32);
}
#include "tl_device.cuh"
extern "C" void quotients(const double *x, const double *b, double *q, double *ref, long long n) {
    for (long long k = 0; k < n; ++k) {
        const double y = 1.0 / b[k];
        q[k] = tl::div_by(x[k], b[k], y);
        ref[k] = x[k] / b[k];
    }
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    src, so = str(d / "q.cpp"), str(d / "q.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "tealeaf_cuda_gb300", "csrc"), src, "-o", so], check=True)
    lib = C.CDLL(so)
    lib.quotients.argtypes = [C.c_void_p] * 4 + [C.c_longlong]

    def run(x, b):
        x, b = (np.ascontiguousarray(a, dtype=np.float64) for a in np.broadcast_arrays(x, b))
        q, ref = np.empty_like(x), np.empty_like(x)
        lib.quotients(x.ctypes.data, b.ctypes.data, q.ctypes.data, ref.ctypes.data, x.size)
        return q, ref

    return run


def _equal(q, ref):
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(q), nan)
    bad = np.flatnonzero(q.view(np.uint64)[~nan] != ref.view(np.uint64)[~nan])
    assert bad.size == 0, (bad.size, q[~nan][bad[:4]], ref[~nan][bad[:4]])


def _mantissas(rng, n):
    """1 + k ulps and 2 - k ulps (ties and all-ones lie there), and any"""
    near = rng.integers(0, 64, n).astype(np.uint64)
    kind = rng.integers(0, 3, n)
    frac = np.where(kind == 0, near, np.where(kind == 1, np.uint64((1 << 52) - 1) - near,
                                              rng.integers(0, 1 << 52, n).astype(np.uint64)))
    return (frac | np.uint64(1023 << 52)).view(np.float64)


@pytest.mark.parametrize("x_exponents", [(-60, 60), (-1022, 1000), (-1074, -840)])
@pytest.mark.parametrize("b_exponents", [(0, 40), (-30, 150)])
def test_finite_quotients(quotients, x_exponents, b_exponents):
    rng = np.random.default_rng(11)
    n = 200_000
    with np.errstate(over="ignore"):
        x = np.ldexp(_mantissas(rng, n), rng.integers(*x_exponents, n)) * rng.choice([-1.0, 1.0], n)
    b = np.ldexp(_mantissas(rng, n), rng.integers(*b_exponents, n))
    _equal(*quotients(x, b))
    _equal(*quotients(x, -b))


def test_zeros_infinities_and_nan(quotients):
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1.0, -3.0, 1.7976931348623157e308])
    b = np.array([1.0, 1.5, 3.0, 1e10, 0.3, -2.0, 0.0, -0.0, np.inf, -np.inf, np.nan])
    with np.errstate(all="ignore"):
        _equal(*quotients(x[:, None], b[None, :]))
