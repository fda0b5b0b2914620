"""The host routines of the long Lanczos runs and of the final Rayleigh-Ritz
(mo-dmft_gb300/csrc/symeig.h: lowest eigenvalues of a tridiagonal matrix by
bisection, its eigenvectors and those of a Hessenberg matrix by inverse
iteration, a generalised symmetric problem by Cholesky) against numpy, for one
to 488 rows, with clusters, equal values in separate blocks, zero off-diagonals.

Bounds: bisection ends within 2 eps of the scale and its counts are those of a
matrix within a few eps; numpy's own errors are n eps: n 1e-15 of the scale, 1e-14
at least.  Inverse iteration from such a value leaves a residual of the same order
divided by the growth it starts with (the start vector's share of the eigenvector,
at least 1 / (100 n) in the models here): 1e-12 n."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include <vector>
#include "symeig.h"
using namespace moed;
extern "C" {
void lowest(int n, const double *d, const double *e, int k, double *w) { tri_lowest(n, d, e, k, w); }
// eigenvectors of k values, each orthogonal to those before it within `same`
void vectors(int n, const double *d, const double *e, int k, const double *w, double same, double *y)
{
    std::vector<const double *> prev;
    for (int i = 0; i < k; ++i) {
        if (i && w[i] - w[i - 1] > same) prev.clear();
        tri_eigvec(n, d, e, w[i], y + (size_t)i * n, prev.data(), (int)prev.size());
        prev.push_back(y + (size_t)i * n);
    }
}
void hess(int n, const double *h, double theta, double scale, double *y) { hess_eigvec(n, h, n, theta, scale, y); }
int gen(int n, const double *p, const double *s, double *w, double *c)
{
    std::vector<double> P(p, p + (size_t)n * n), S(s, s + (size_t)n * n);
    return gen_sym_eig(n, P, S, w, c) ? 0 : 1;
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("symeig_tri")
    src, so = d / "shim.cpp", d / "lib.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mo-dmft_gb300", "csrc"),
                    "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))


def p(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def matrices(n):
    rng = np.random.default_rng(n)
    yield rng.standard_normal(n), rng.uniform(0.1, 1.0, max(n - 1, 1))           # a Lanczos run
    yield 20.0 * rng.standard_normal(n), 1e-6 * rng.uniform(0.1, 1.0, max(n - 1, 1))   # nearly decoupled
    e = rng.uniform(0.1, 1.0, max(n - 1, 1))
    e[::3] = 0.0
    yield rng.standard_normal(n), e                                              # blocks of three
    d = np.tile(rng.standard_normal((n + 3) // 4), 4)[:n]
    e = np.tile(np.append(rng.uniform(0.1, 1.0, (n + 3) // 4 - 1), 0.0), 4)[:max(n - 1, 1)]
    yield d, e                                                                   # four equal blocks: copies of every value
    yield np.zeros(n), np.zeros(max(n - 1, 1))


@pytest.mark.parametrize("n", [1, 2, 3, 8, 40, 130, 488])
def test_tridiagonal(lib, n):
    for d, e in matrices(n):
        d, e = np.ascontiguousarray(d), np.ascontiguousarray(e)
        T = np.diag(d) + (np.diag(e, 1) + np.diag(e, -1) if n > 1 else 0.0)
        exact = np.linalg.eigvalsh(T)
        scale = max(np.abs(T).sum(1).max(), 1e-300)
        k = min(n, 12)
        w = np.zeros(k)
        lib.lowest(n, p(d), p(e), k, p(w))
        assert np.abs(w - exact[:k]).max() <= max(n * 1e-15, 1e-14) * scale
        assert (np.diff(w) >= -1e-14 * scale).all()
        y = np.zeros((k, n))
        lib.vectors(n, p(d), p(e), k, p(w), C.c_double(1e-9 * scale), p(y))
        assert np.abs(np.linalg.norm(y, axis=1) - 1).max() < 1e-12
        assert np.abs(T @ y.T - y.T * w).max() <= 1e-12 * n * scale
        assert np.abs(y @ y.T - np.eye(k)).max() < 1e-5           # the closest values here are 1e-9 and more apart


@pytest.mark.parametrize("n", [1, 2, 5, 40, 200])
def test_hessenberg(lib, n):
    """T + h with h as large as orthogonality is allowed to be off."""
    rng = np.random.default_rng(n)
    d, e = rng.standard_normal(n), rng.uniform(0.1, 1.0, max(n - 1, 1))
    H = np.diag(d) + (np.diag(e, 1) + np.diag(e, -1) if n > 1 else 0.0) + 1e-3 * np.triu(rng.standard_normal((n, n)), 2)
    ev = np.linalg.eigvals(H)
    theta = np.sort(ev[np.abs(ev.imag) < 1e-14].real)[0]
    y, scale = np.zeros(n), np.abs(H).sum(1).max()
    h = np.ascontiguousarray(H.T)      # column-major
    lib.hess(n, p(h), C.c_double(theta), C.c_double(scale), p(y))
    assert abs(np.linalg.norm(y) - 1) < 1e-12
    assert np.abs(H @ y - theta * y).max() <= 1e-12 * n * scale


@pytest.mark.parametrize("n", [1, 2, 6, 20, 60])
def test_generalised(lib, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    P = A + A.T
    Q = np.eye(n) + 1e-3 * rng.standard_normal((n, n))
    S = Q @ Q.T
    w, c = np.zeros(n), np.zeros((n, n))
    P, S = np.ascontiguousarray(P), np.ascontiguousarray(S)
    assert lib.gen(n, p(P), p(S), p(w), p(c)) == 0
    sc = np.abs(P).sum(1).max()
    assert np.abs(P @ c.T - S @ c.T * w).max() <= 1e-13 * n * sc
    assert np.abs(c @ S @ c.T - np.eye(n)).max() <= 1e-13 * n
    assert (np.diff(w) >= 0).all()
    S[0, 0] = -1.0
    assert lib.gen(n, p(P), p(S), p(w), p(c)) == 1     # not positive definite
