"""The host side of the eigensolver's Lanczos run (mo-dmft_gb300/csrc/kryhost.h)
on its own, without a GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "kryhost.h"
#include "symeig.h"
using namespace moed;
extern "C" {
// judges n reorthogonalisations one after the other; returns the last verdict
int judge(int f32, int n, const int *j, const int *gap, const double *c, int *period, int *good, double *hmax)
{
    KryPeriod p(f32 != 0, 1 << 20);
    int v = KryPeriod::kept;
    for (int i = 0; i < n && v == KryPeriod::kept; ++i) v = p.judge(KryClean{j[i], gap[i]}, c[i], false);
    *period = p.period;
    *good = p.good;
    *hmax = p.hmax;
    return v;
}
// hp: [m][m] columns, then the right eigenvectors y[n][m] of the eigenvalues th
void projected(int m, const double *al, const double *be, const double *inv, int nre, const int *j, const double *h,
               int ldh, double *hp, int n, const double *th, double scale, double *y)
{
    std::vector<KryClean> re;
    for (int i = 0; i < nre; ++i) re.push_back(KryClean{j[i], 0});
    std::vector<double> H;
    kry_projected(m, al, be, inv, re, h, ldh, H);
    std::copy(H.begin(), H.end(), hp);
    std::vector<const double *> prev;
    for (int i = 0; i < n; ++i) {
        hess_eigvec(m, H.data(), m, th[i], scale, y + (size_t)i * m, prev.data(), (int)prev.size());
        prev.push_back(y + (size_t)i * m);
    }
}
double limit(int f32, double tol, double anorm) { return kry_residual_limit(f32 != 0, tol, anorm); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("kryhost")
    src, so = d / "shim.cpp", d / "lib.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mo-dmft_gb300", "csrc"),
                    "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))


def judge(lib, f32, rounds):
    n = len(rounds)
    j, gap = (C.c_int * n)(*[r[0] for r in rounds]), (C.c_int * n)(*[r[1] for r in rounds])
    c = (C.c_double * n)(*[r[2] for r in rounds])
    period, good, hmax = C.c_int(), C.c_int(), C.c_double()
    v = lib.judge(f32, n, j, gap, c, C.byref(period), C.byref(good), C.byref(hmax))
    return ("kept", "back", "lost")[v], period.value, good.value, hmax.value


@pytest.mark.parametrize("f32,little,much", [(1, 4e-7, 0.2), (0, 1e-15, 1e-3)])
def test_every_reorthogonalisation_counts(lib, f32, little, much):
    """Components that grew too large are found wherever they are among the
    reorthogonalisations of one read, not in the last of them alone."""
    fine = [(6, 6, little), (12, 6, little), (18, 6, little)]
    v, p0, good, hmax = judge(lib, f32, fine)
    assert v == "kept" and good == 18 and hmax == little
    v, p1, good, hmax = judge(lib, f32, fine[:2] + [(18, 6, 100 * little), (24, 6, little)])
    assert v == "kept" and good == 24 and hmax == 100 * little and p1 < p0
    v, p, good, _ = judge(lib, f32, fine + [(24, 6, much), (30, 6, little)])
    assert v == "back" and good == 18 and p == 3
    assert judge(lib, f32, fine + [(24, 6, np.nan)])[0] == "back"
    assert judge(lib, f32, fine + [(20, 2, much)])[0] == "lost"
    assert judge(lib, f32, [(6, 6, much)])[0] == "lost"
    assert judge(lib, f32, [(6, 6, 0.0)])[0] == "kept"


def run(A, v0, m, period, noise, rng):
    """The device's recurrence (vectors stored unnormalised, the last two of them
    reorthogonalised together every `period` steps) with random errors of the
    relative size `noise`: al, be, inv, h, steps and the unit vectors q_0 .. q_m."""
    n = len(v0)
    U, al, be, inv = [v0], np.zeros(m + 1), np.zeros(m + 1), np.zeros(m + 1)
    h, steps = np.zeros((m + 2, m + 2)), []
    for j in range(m + 1):
        if j:
            u = inv[j - 1] * (w - al[j - 1] * U[j - 1])
            if j >= 2:
                u = u - be[j - 1] * inv[j - 2] * U[j - 2]
            U.append(u + noise * np.linalg.norm(u) * rng.standard_normal(n) / np.sqrt(n))
            if j >= 3 and (j % period == 0 or j == m):
                for x in (j - 1, j):
                    g = np.array([U[l] @ U[x] * inv[l] for l in range(j - 1)])
                    h[x, :j - 1] = g
                    U[x] = U[x] - sum(g[l] * inv[l] * U[l] for l in range(j - 1))
                steps.append(j)
        n2 = U[j] @ U[j]
        w = A @ U[j]
        inv[j], be[j], al[j] = 1 / np.sqrt(n2), np.sqrt(n2), U[j] @ w / n2
    return al, be, inv, h, steps, np.stack([u * i for u, i in zip(U, inv)], 1)


@pytest.mark.parametrize("m,period", [(33, 12), (35, 12), (36, 12)])
def test_projected_matrix(lib, m, period):
    """H Q = Q hp + be[m] q_m e^T, with a reorthogonalisation of the last pair
    among the others.  Every step brings an error of `noise` ||H|| at most and
    what a reorthogonalisation takes out squared; without the components of the
    last one the last two columns are off by their size."""
    rng = np.random.default_rng(m)
    n, noise = 200, 1e-11
    A = np.diag(np.concatenate([[-1.8, -1.5], rng.uniform(-1, 1, n - 2)]))
    al, be, inv, h, steps, Q = run(A, rng.standard_normal(n), m, period, noise, rng)
    assert steps[-1] == m
    big = max(np.abs(h[j]).max() * inv[j] for j in steps)
    last = np.abs(h[m]).max() * inv[m]
    assert big < 1e-2 and last > 1e3 * noise, "the run does not show what this test is about"
    hp, y = np.zeros(m * m), np.zeros(m)
    d = lambda a: np.ascontiguousarray(a, dtype=np.float64).ctypes.data_as(C.POINTER(C.c_double))
    js = (C.c_int * len(steps))(*steps)
    al_, be_, inv_, h_, th = (np.ascontiguousarray(a, dtype=np.float64) for a in (al, be, inv, h, [-1.8]))
    lib.projected(m, d(al_), d(be_), d(inv_), len(steps), js, d(h_), h.shape[1], d(hp), 1, d(th), C.c_double(1.8), d(y))
    HP = hp.reshape(m, m).T
    R = A @ Q[:, :m] - Q[:, :m] @ HP
    R[:, m - 1] -= be[m] * Q[:, m]
    tol = 1.8 * (10 * noise + 4 * big * big)
    assert np.linalg.norm(R, axis=0).max() < tol
    x = Q[:, :m] @ y
    assert np.linalg.norm(A @ x + 1.8 * x) / np.linalg.norm(x) < abs(be[m] * y[m - 1]) + 3 * tol


def test_copies_of_a_level(lib):
    """Two Ritz values that agree: two independent vectors of T + h."""
    rng = np.random.default_rng(0)
    m = 12
    Z = np.linalg.qr(rng.standard_normal((m, m)))[0]
    lam = np.concatenate([[-5.0, -5.0], np.linspace(-1, 1, m - 2)])
    T = Z @ np.diag(lam) @ Z.T
    # Householder to tridiagonal splits at the copy; a Hessenberg matrix of the
    # same spectrum with both copies: two tridiagonal blocks
    H = np.zeros((m, m))
    for s, e, lo in ((0, m // 2, lam[:1]), (m // 2, m, lam[1:2])):
        k = e - s
        B = np.diag(np.concatenate([lo, np.linspace(-1, 1, k - 1)]))
        q = np.linalg.qr(rng.standard_normal((k, k)))[0]
        from scipy.linalg import hessenberg
        H[s:e, s:e] = hessenberg(q @ B @ q.T)
    H[:m // 2, m // 2:] = 0.0
    be, al, inv = np.zeros(m + 1), np.zeros(m + 1), np.ones(m + 1)
    al[:m] = np.diag(H)
    be[1:m] = np.diag(H, 1)
    th, hp, y = np.array([-5.0, -5.0]), np.zeros(m * m), np.zeros(2 * m)
    d = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    lib.projected(m, d(al), d(be), d(inv), 0, (C.c_int * 1)(), d(np.zeros(1)), 1, d(hp), 2, d(th), C.c_double(5.0), d(y))
    Y = y.reshape(2, m)
    assert np.abs(Y @ Y.T - np.eye(2)).max() < 1e-12
    assert np.abs(H @ Y.T + 5.0 * Y.T).max() < 1e-12 * 5 * m


def test_residual_limit(lib):
    lib.limit.restype = C.c_double
    f = lambda f32, tol, an: lib.limit(f32, C.c_double(tol), C.c_double(an))
    assert f(1, 1e-7, 10.0) == 10 * 1e-7 * 10
    assert f(1, 1e-12, 10.0) == 1e-6 * 10        # the vectors' own rounding
    assert f(0, 1e-11, 20.0) == 10 * 1e-11 * 20
    assert f(0, 1e-11, 0.1) == 10 * 1e-11 and f(0, 1e-4, 1.0) == 1e-3
