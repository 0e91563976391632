"""The FP64 reciprocals, roots and quotients that the kernels build from the
MUFU seeds (amuse_gb300/csrc/fp64_approx.cuh, g6_div_const of g6_dev.h),
element by element against CUDA's own operators and extended precision.

Derived bounds (u = 2^-53): rcp64 1.07 u and rsqrt64 1.7 u relative; div64, Div's
inverse and sqrt64 half an ulp and 2^-49 of one; div_by with the rounded
reciprocal and g6_div_const are the rounded quotient (Markstein 1990, theorem 3).
Outside the seeds' range they are CUDA's operators."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from amuse_gb300 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
RCP, RSQRT, SQRT, DIV, DIVBY, INV, DIV3, DIV12, DIV20 = range(9)
U = 2.0 ** -53


@pytest.fixture(scope="module")
def ops(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fp64") / "libfp64ops.so")
    nvcc = os.path.join(build.cuda_home(), "bin", "nvcc")
    subprocess.run([nvcc, *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", build.CSRC, "-I", build.INCLUDE, "-o", so,
                    os.path.join(HERE, "fp64_ops.cu")], check=True)
    lib = ctypes.CDLL(so)
    pd = ctypes.POINTER(ctypes.c_double)

    def run(op, a, b=None):
        a = np.ascontiguousarray(a)
        b = np.ones_like(a) if b is None else np.ascontiguousarray(b)
        got, want = np.empty_like(a), np.empty_like(a)
        rc = lib.fp64_ops(op, len(a), *(q.ctypes.data_as(pd) for q in (a, b, got, want)))
        assert rc == 0
        return got, want
    return run


def operands(seed, n=1 << 21, lo=-299, hi=299, signed=True):
    """Random mantissas, half of them within 1024 ulps of either end of the
    mantissa range, at exponents lo .. hi."""
    r = np.random.RandomState(seed)
    bits = r.randint(0, 1 << 52, size=n, dtype=np.int64)
    near = r.randint(0, 1024, size=n)
    bits = np.where(r.rand(n) < 0.25, near, np.where(r.rand(n) < 1 / 3, (1 << 52) - 1 - near, bits))
    x = (bits + (1 << 52)).astype(np.float64) * 2.0 ** -52
    x = np.ldexp(x, r.randint(lo, hi + 1, size=n))
    return np.where(r.rand(n) < 0.5, -x, x) if signed else x


EDGES = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** -1022, 1e-310, 1e308,
                  -1e308, 2.0 ** -300, np.nextafter(2.0 ** -300, 0), 2.0 ** 300,
                  np.nextafter(2.0 ** 300, 0), 2.0 ** -961, 2.0 ** -959, 2.0 ** 961, 2.0 ** 993, 1.0,
                  -1.0, 3.0, 1 / 3])


LONG = np.longdouble
# half an ulp is to be told from half an ulp and 2^-49 of one
quad = pytest.mark.skipif(np.finfo(LONG).eps > 2.0 ** -105, reason="no 128-bit long double")


@quad
def test_reciprocal_and_root_bounds(ops):
    for seed in range(2):
        x = operands(seed)
        got, _ = ops(RCP, x)
        assert np.abs(got * x.astype(LONG) - 1).max() <= 1.07 * U
        x = np.abs(x)
        got, _ = ops(RSQRT, x)
        assert np.abs(got * np.sqrt(x.astype(LONG)) - 1).max() <= 1.7 * U


@quad
@pytest.mark.parametrize("op", [DIV, INV, SQRT], ids=["div64", "inv", "sqrt"])
def test_half_an_ulp(ops, op):
    for seed in range(2):
        x, y = operands(10 + seed, signed=op != SQRT), operands(20 + seed)
        got, _ = ops(op, x, y)
        x, y = x.astype(LONG), y.astype(LONG)
        true = x / y if op == DIV else 1 / x if op == INV else np.sqrt(x)
        err = np.abs(got - true) / np.spacing(np.abs(got))
        assert err.max() <= 0.5 + 2.0 ** -49


@pytest.mark.parametrize("op", [DIVBY, DIV3, DIV12, DIV20], ids=["div_by", "3", "12", "20"])
def test_rounded_as_the_operator(ops, op):
    for seed in range(2):
        got, want = ops(op, operands(30 + seed), operands(40 + seed))
        assert np.array_equal(got, want)


def test_outside_the_range(ops):
    """Zeros, infinities, NaN, subnormals and the limits: as the operators
    (to the bounds above where the seeds are used)."""
    pairs = np.array([(a, b) for a in EDGES for b in EDGES]).T
    for op in (RCP, RSQRT, SQRT, DIV, DIVBY, INV, DIV3, DIV12, DIV20):
        a, b = pairs if op in (DIV, DIVBY) else (EDGES, EDGES)
        got, want = ops(op, a, b)
        # 1.7 u, and two roundings in what RSQRT is compared with
        fin = np.isfinite(want) & (want != 0)
        assert (np.abs(got[fin] / want[fin] - 1) <= 4 * U).all(), op
        got, want = got[~fin], want[~fin]
        assert np.array_equal(got, want, equal_nan=True), op
        num = ~np.isnan(want)
        assert np.array_equal(np.signbit(got[num]), np.signbit(want[num])), op
