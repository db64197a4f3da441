"""Arithmetic that stands in for CUDA's divide, square root and exponential in
the hot kernels, against those functions and against long double (at least 64
bits of mantissa on both hosts).

Bounds, in units in the last place of the exact value:
  - rcp64: the step's own error is below 2^-57 of the value (0.1 ulp) and the
    last operation rounds once: below 1 ulp; sqrt64 and root64: the rounding of
    x y enters too, with half its size: below 1.1 ulp.  A correctly rounded
    result is then at most one ulp away;
  - expm64: exp(-x) has the rounding of the table's entry and of the product
    behind it, 2 ulp; 1 - exp(-x) adds an entry and a product of like size that
    may have opposite signs (a factor of two), 4 ulp;
  - tbl_index64 is the index of the FP64 expression it replaces, for every x;
  - quot is the approximate division of the FP32 form's flags, bit for bit, for
    |a|, |b| in 2^-100 .. 2^100.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
dp, fp = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_float)


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    from rrtmg_sw_gb300 import build
    d = tmp_path_factory.mktemp("arith")
    jobs, out = [], []
    for name, unit in (("arith64", "solve_fp64.cu"), ("arith32", "solve_fp32.cu")):
        so = str(d / (name + ".so"))
        jobs.append(subprocess.Popen([build.nvcc(), *build.ARCH, *build.COMMON, *build.UNITS[unit], "-I", build.CSRC, "-shared",
                                      os.path.join(HERE, "cuda", name + ".cu"), "-o", so],
                                     stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True))
        out.append(so)
    for j in jobs:
        log = j.communicate()[0]
        assert j.returncode == 0, log[-3000:]
    return [ctypes.CDLL(so) for so in out]


def run64(lib, what, x, nres):
    x = np.ascontiguousarray(x)
    own, cuda = np.zeros((nres, x.size)), np.zeros((nres, x.size))
    p = lambda a: a.ctypes.data_as(dp)
    assert lib.arith64(ctypes.c_int(what), ctypes.c_int(x.size), p(x), p(own), p(cuda)) == 0
    return own, cuda


def ulps(v, exact):
    """|v - exact| in units of the spacing of doubles at exact (a long double)."""
    return np.abs(v.astype(np.longdouble) - exact) / np.spacing(np.abs(exact.astype(np.float64))).astype(np.longdouble)


def positive(rng, n, lo, hi):
    x = 2.0 ** rng.uniform(lo, hi, n) * rng.uniform(1.0, 2.0, n)
    # powers of two and their neighbours, where the spacing changes
    p = 2.0 ** np.arange(lo, hi)
    return np.concatenate([x, p, np.nextafter(p, 0.0), np.nextafter(p, np.inf)])


def test_reciprocal_and_roots(libs):
    x = positive(np.random.default_rng(1), 2_000_000, -1000, 1000)
    own, cuda = run64(libs[0], 0, x, 4)
    X = x.astype(np.longdouble)
    root = np.sqrt(X)
    for k, exact in enumerate((1.0 / X, root, root, 1.0 / root)):
        assert np.max(ulps(own[k], exact)) < (1.0 if k == 0 else 1.1), k
        if k < 3:  # CUDA's are correctly rounded
            assert np.max(np.abs(own[k].view(np.int64) - cuda[k].view(np.int64))) <= 1, k


def test_exponential(libs):
    rng = np.random.default_rng(2)
    step = np.log(2.0) / 1024.0
    near = (np.arange(0, 4096)[:, None] * 0.5 + rng.uniform(-1e-9, 1e-9, (4096, 8))).ravel() * step  # entries, midpoints
    x = np.concatenate([10.0 ** rng.uniform(-18.0, np.log10(500.0), 2_000_000), rng.uniform(0.0, 500.0, 500_000),
                        np.abs(near), [0.0, 500.0, np.nextafter(500.0, 0.0)]])
    own, cuda = run64(libs[0], 1, x, 2)
    X = x.astype(np.longdouble)
    assert np.max(ulps(own[0], np.exp(-X))) < 2.0
    om = -np.expm1(-X)
    some = x > 0.0
    assert np.max(ulps(own[1][some], om[some])) < 4.0
    assert np.all(own[1][~some] == 0.0) and np.all(own[0][~some] == 1.0)
    np.testing.assert_allclose(own, cuda, rtol=1.2e-15, atol=0.0)  # 4 ulp and CUDA's own one


def test_table_index(libs):
    rng = np.random.default_rng(3)
    b = 1.0 / 0.278
    t = (np.arange(165, 9929) + 0.5) / 10000.0  # edges between entries
    edge = b * t / (1.0 - t)
    x = np.concatenate([rng.uniform(0.06, 500.0, 1_000_000), 10.0 ** rng.uniform(np.log10(0.06), np.log10(500.0), 1_000_000)] +
                       [edge * (1.0 + d) for d in (0.0, 1e-16, -1e-16, 1e-13, -1e-13, 1e-10, -1e-10, 1e-7, -1e-7, 1e-6, -1e-6)])
    x = x[(x > 0.06) & (x <= 500.0)]
    own, cuda = run64(libs[0], 2, x, 1)
    np.testing.assert_array_equal(own, cuda)


def test_fp32_quotient(libs):
    rng = np.random.default_rng(4)
    n = 4_000_000
    a, b = (np.ascontiguousarray((2.0 ** rng.uniform(-100, 100, n) * rng.choice([-1.0, 1.0], n)).astype(np.float32))
            for _ in range(2))
    own, cuda = np.zeros(n, np.float32), np.zeros(n, np.float32)
    p = lambda v: v.ctypes.data_as(fp)
    assert libs[1].arith32(ctypes.c_int(n), p(a), p(b), p(own), p(cuda)) == 0
    np.testing.assert_array_equal(own.view(np.int32), cuda.view(np.int32))
