"""The FP64 device arithmetic of mo-dmft_gb300/csrc/math64.cuh against 80-bit (or
longer) host arithmetic, over random significands and at both ends of the ranges
beyond which the functions take the IEEE operations, zero, denormals,
infinities and NaN.

Bounds in units of the last place of the exact value.  rcp_pos: the last FMA
rounds once (1/2); the terms before it are below 2^-19 of the result, so their
few roundings and the truncated series add less than 1/100.  rsqrt_pos: the
rounding of d y0, half an ulp of e at most, adds another half.  sqrt_by, rsqrt_by,
div_by: the correction terms are below 2^-50 of the result; 1/2 and 1/100.  widen
is exact."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "math64.cuh"
using namespace moed;
__global__ void k(int f, int n, const double *a, const double *b, double *o)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (f == 0) o[i] = rcp_pos(a[i]);
    if (f == 1) o[i] = rsqrt_pos(a[i]);
    if (f == 2) o[i] = sqrt_by(a[i], rsqrt_pos(a[i]));
    if (f == 8) o[i] = rsqrt_by(a[i], rsqrt_pos(a[i]));
    if (f == 3) o[i] = div_by(b[i], a[i], rcp_pos(a[i]));
    if (f == 4) o[i] = div_by(b[i], a[i], 1.0 / a[i]);
    if (f == 5) o[i] = widen((float)a[i]);
    if (f == 6) o[i] = (double)(float)a[i];
    if (f == 7) {
        double d[4], y[4];
        for (int q = 0; q < 4; ++q) d[q] = a[(i + q) % n];
        rcp_pos_n<4>(d, y);
        o[i] = y[0];
    }
}
extern "C" int run(int f, int n, const double *a, const double *b, double *o)
{
    double *d = nullptr;
    if (cudaMalloc(&d, 3 * sizeof(double) * (size_t)n)) return 1;
    cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(f, n, d, d + n, d + 2 * (size_t)n);
    cudaMemcpy(o, d + 2 * (size_t)n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from __graft_entry__ import PKG_DIR
    sys.path.insert(0, PKG_DIR)
    try:
        import build as b
    finally:
        sys.path.remove(PKG_DIR)
    d = tmp_path_factory.mktemp("math64")
    src, lib = d / "m.cu", d / "m.so"
    src.write_text(SRC)
    subprocess.run([b.nvcc()] + b.ARCH + b.FLAGS + ["-shared", "-I", b.CSRC, "-o", str(lib), str(src)], check=True)
    L = C.CDLL(str(lib))
    dp = C.POINTER(C.c_double)

    def f(which, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = a if b is None else np.ascontiguousarray(b, dtype=np.float64)
        o = np.full(a.size, -7.0)
        assert L.run(which, a.size, a.ctypes.data_as(dp), b.ctypes.data_as(dp), o.ctypes.data_as(dp)) == 0
        return o
    return f


def ulps(got, exact):
    return np.abs((got.astype(np.longdouble) - exact) / np.spacing(np.abs(exact.astype(np.float64))).astype(np.longdouble)).max()


def numbers(lo, hi, n=200_000):
    r = np.random.default_rng(n + hi)
    x = np.ldexp(r.uniform(1.0, 2.0, n), r.integers(lo, hi, n))
    edge = np.array([np.ldexp(s, e) for e in range(lo, hi + 1) for s in (1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52)])
    return np.concatenate([x, edge])


def test_reciprocal(run):
    for lo, hi in ((-2, 2), (-130, 130), (-900, 900)):   # the FP32 seed's range ends at 2^-125 and 2^126
        x = numbers(lo, hi)
        assert ulps(run(0, x), 1 / x.astype(np.longdouble)) < 0.51
        assert (run(7, x) == run(0, x)).all()


def test_reciprocal_square_root(run):
    for lo, hi in ((-2, 2), (-104, 104), (-900, 900)):   # 2^-100, 2^100
        x = numbers(lo, hi)
        inside = (x >= 2.0 ** -100) & (x < 2.0 ** 101)
        y, exact = run(1, x), 1 / np.sqrt(x.astype(np.longdouble))
        assert ulps(y[inside], exact[inside]) < 1.01
        assert (y[~inside] == 1.0 / np.sqrt(x[~inside])).all()
        far = np.abs(np.log2(x)) < 500
        assert ulps(run(2, x)[far], np.sqrt(x.astype(np.longdouble))[far]) < 0.51
        assert ulps(run(8, x)[far], exact[far]) < 0.51


def test_division(run):
    r = np.random.default_rng(3)
    x = numbers(-120, 120)
    s = np.ldexp(r.uniform(1.0, 2.0, x.size), r.integers(-300, 300, x.size)) * r.choice([-1.0, 1.0], x.size)
    exact = s.astype(np.longdouble) / x.astype(np.longdouble)
    assert ulps(run(3, x, s), exact) < 0.51
    # divisors of up to 24 bits (norb^2 nw of a fit): the division itself
    d = r.integers(1, 1 << 24, 400_000).astype(np.float64)
    s = np.ldexp(r.uniform(1.0, 2.0, d.size), r.integers(-60, 60, d.size))
    assert (run(4, d, s) == s / d).all()
    far = np.array([0.0, -0.0, 1e-300, 1e300, np.inf, np.nan])
    assert np.array_equal(run(4, np.full(6, 3.0), far), far / 3.0, equal_nan=True)


def test_special_values(run):
    x = np.array([0.0, 5e-324, 1e-310, 2.0 ** -1022, 1.7e308, np.inf, np.nan])
    with np.errstate(divide="ignore", over="ignore"):
        assert np.array_equal(run(0, x), 1.0 / x, equal_nan=True)
        assert np.array_equal(run(1, x), 1.0 / np.sqrt(x), equal_nan=True)
        assert np.array_equal(run(0, -x[1:5]), -1.0 / x[1:5])


def test_widen(run):
    r = np.random.default_rng(4)
    bits = np.concatenate([r.integers(0, 1 << 32, 300_000, dtype=np.uint32),
                           np.array([0, 1, 2, 0x7fffff, 0x800000, 0x7f7fffff, 0x7f800000, 0x80000000, 0x80000001, 0xff800000],
                                    dtype=np.uint32)])
    f = bits.view(np.float32)
    f = f[~np.isnan(f)].astype(np.float64)
    a, b = run(5, f), run(6, f)
    assert (a.view(np.int64) == b.view(np.int64)).all()
    assert np.isnan(run(5, np.array([np.nan])))
