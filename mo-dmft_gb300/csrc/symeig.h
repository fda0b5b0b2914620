// symeig.h -- eigenvalues and eigenvectors of small matrices on the host: the
// projected (Rayleigh-Ritz) problems of the eigensolvers, dense for the thick
// restarts, tridiagonal or Hessenberg for the long runs (below).  The reference's eigensolver (PARPACK) also solves
// its projected problem on the host (LAPACK); on GB300 a one-CTA FP64
// Jacobi of an m = 40 matrix takes ~1.4 ms per call, the host a few tens of
// microseconds.
//
// Method (Golub & Van Loan, Matrix Computations, 4th ed., 8.3):
//   1. Householder reduction to tridiagonal form, T = Q^T A Q, with Q
//      accumulated;
//   2. implicit symmetric QR steps with the Wilkinson shift on T, chasing the
//      bulge with Givens rotations that are accumulated into Q, deflating
//      off-diagonal entries below eps (|d_i| + |d_i+1|);
//   3. eigenpairs sorted by ascending eigenvalue.
#pragma once

#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

namespace moed {

// Implicit symmetric QR steps with the Wilkinson shift on the tridiagonal
// matrix of diagonal d[n] and off-diagonal e[i] = T(i+1, i), deflating from
// the bottom.  On return d holds the eigenvalues (unordered); the rotations
// are applied to the columns of Q, `rows` x n row-major.  Returns false if
// the iteration did not converge.
inline bool tri_qr(int n, double *d, double *e, int rows, double *Q)
{
    const double eps = 2.220446049250313e-16;
    int hi = n - 1, iters = 0;
    while (hi > 0) {
        if (std::fabs(e[hi - 1]) <= eps * (std::fabs(d[hi - 1]) + std::fabs(d[hi]))) {
            e[hi - 1] = 0.0;
            --hi;
            continue;
        }
        if (++iters > 60 * n) return false;
        int lo = hi - 1;
        while (lo > 0 && std::fabs(e[lo - 1]) > eps * (std::fabs(d[lo - 1]) + std::fabs(d[lo]))) --lo;
        // shift: the eigenvalue of the trailing 2 x 2 closer to d[hi]
        const double delta = 0.5 * (d[hi - 1] - d[hi]), b = e[hi - 1];
        const double mu = delta == 0.0 ? d[hi] - std::fabs(b)
                                       : d[hi] - b * b / (delta + std::copysign(std::hypot(delta, b), delta));
        double x = d[lo] - mu, y = e[lo];
        for (int k = lo; k < hi; ++k) {
            // rotation R = [c s; -s c] on rows / columns k, k+1 that zeroes y
            // (the shifted first column, then the bulge at (k+1, k-1))
            const double r = std::hypot(x, y);
            const double c = r == 0.0 ? 1.0 : x / r, s = r == 0.0 ? 0.0 : y / r;
            if (k > lo) e[k - 1] = r;
            const double dk = d[k], dk1 = d[k + 1], ek = e[k];
            d[k] = c * c * dk + 2.0 * c * s * ek + s * s * dk1;
            d[k + 1] = s * s * dk - 2.0 * c * s * ek + c * c * dk1;
            e[k] = c * s * (dk1 - dk) + (c * c - s * s) * ek;
            if (k + 1 < hi) {
                y = s * e[k + 1];                          // the bulge at (k+2, k)
                e[k + 1] *= c;
                x = e[k];
            }
            for (int rr = 0; rr < rows; ++rr) {            // Q <- Q R^T
                const double qk = Q[(size_t)rr * n + k], qk1 = Q[(size_t)rr * n + k + 1];
                Q[(size_t)rr * n + k] = c * qk + s * qk1;
                Q[(size_t)rr * n + k + 1] = -s * qk + c * qk1;
            }
        }
    }
    return true;
}

// a: n x n symmetric, row-major (only read).  w[n]: ascending eigenvalues.
// z[n * n]: column j (z[j * n + i], i = 0..n-1) is the unit eigenvector of
// w[j].  Returns false if the QR iteration did not converge.
inline bool sym_eig(int n, const std::vector<double> &a, double *w, double *z)
{
    if (n <= 0) return true;
    std::vector<double> A(a.begin(), a.begin() + (size_t)n * n);
    std::vector<double> Q((size_t)n * n, 0.0);   // row-major, Q[r * n + c]
    for (int i = 0; i < n; ++i) Q[(size_t)i * n + i] = 1.0;
    std::vector<double> v(n), p(n);
    // 1. Householder: zero column k below the subdiagonal, k = 0 .. n-3
    for (int k = 0; k + 2 < n; ++k) {
        double s2 = 0.0;
        for (int i = k + 1; i < n; ++i) s2 += A[(size_t)i * n + k] * A[(size_t)i * n + k];
        const double tail = s2 - A[(size_t)(k + 1) * n + k] * A[(size_t)(k + 1) * n + k];
        if (tail == 0.0) continue;                        // already tridiagonal in this column
        const double x0 = A[(size_t)(k + 1) * n + k];
        const double alpha = x0 >= 0.0 ? -std::sqrt(s2) : std::sqrt(s2);
        for (int i = 0; i < n; ++i) v[i] = 0.0;
        for (int i = k + 1; i < n; ++i) v[i] = A[(size_t)i * n + k];
        v[k + 1] = x0 - alpha;
        double vv = 0.0;
        for (int i = k + 1; i < n; ++i) vv += v[i] * v[i];
        if (vv == 0.0) continue;
        const double beta = 2.0 / vv;                     // H = I - beta v v^T
        // H A H on the trailing block: A - v q^T - q v^T, p = beta A v,
        // q = p - (beta v^T p / 2) v
        double vp = 0.0;
        for (int i = k + 1; i < n; ++i) {
            double t = 0.0;
            for (int j = k + 1; j < n; ++j) t += A[(size_t)i * n + j] * v[j];
            p[i] = beta * t;
            vp += v[i] * p[i];
        }
        const double K = 0.5 * beta * vp;
        for (int i = k + 1; i < n; ++i) p[i] -= K * v[i];
        for (int i = k + 1; i < n; ++i)
            for (int j = k + 1; j < n; ++j) A[(size_t)i * n + j] -= v[i] * p[j] + p[i] * v[j];
        A[(size_t)(k + 1) * n + k] = A[(size_t)k * n + k + 1] = alpha;
        for (int i = k + 2; i < n; ++i) A[(size_t)i * n + k] = A[(size_t)k * n + i] = 0.0;
        // Q <- Q H
        for (int r = 0; r < n; ++r) {
            double t = 0.0;
            for (int j = k + 1; j < n; ++j) t += Q[(size_t)r * n + j] * v[j];
            t *= beta;
            for (int j = k + 1; j < n; ++j) Q[(size_t)r * n + j] -= t * v[j];
        }
    }
    std::vector<double> d(n), e(n, 0.0);                  // e[i] = T(i+1, i)
    for (int i = 0; i < n; ++i) d[i] = A[(size_t)i * n + i];
    for (int i = 0; i + 1 < n; ++i) e[i] = A[(size_t)(i + 1) * n + i];
    // 2. implicit QR with the Wilkinson shift
    if (!tri_qr(n, d.data(), e.data(), n, Q.data())) return false;
    // 3. ascending order
    std::vector<int> ord(n);
    std::iota(ord.begin(), ord.end(), 0);
    std::stable_sort(ord.begin(), ord.end(), [&](int i, int j) { return d[i] < d[j]; });
    for (int j = 0; j < n; ++j) {
        w[j] = d[ord[j]];
        for (int i = 0; i < n; ++i) z[(size_t)j * n + i] = Q[(size_t)i * n + ord[j]];
    }
    return true;
}

// The k lowest eigenvalues (ascending) of the symmetric tridiagonal matrix
// of diagonal d[n] and off-diagonal e[n - 1]: bisection on the Sturm counts,
// all k intervals together so that their divisions overlap.
inline void tri_lowest(int n, const double *d, const double *e, int k, double *w)
{
    double lo0 = d[0], hi0 = d[0], scale = 0.0;
    for (int i = 0; i < n; ++i) {
        const double r = (i > 0 ? std::fabs(e[i - 1]) : 0.0) + (i + 1 < n ? std::fabs(e[i]) : 0.0);
        lo0 = std::min(lo0, d[i] - r);
        hi0 = std::max(hi0, d[i] + r);
        scale = std::max(scale, std::fabs(d[i]) + r);
    }
    const double eps = 2.220446049250313e-16, tiny = eps * eps * (scale + 1e-300);
    lo0 -= 2 * eps * scale;
    hi0 += 2 * eps * scale;
    std::vector<double> lo(k, lo0), hi(k, hi0), x(k), q(k);
    std::vector<int> cnt(k);
    for (int round = 0; round < 64; ++round) {
        double width = 0.0;
        for (int c = 0; c < k; ++c) {
            x[c] = 0.5 * (lo[c] + hi[c]);
            q[c] = 1.0;
            cnt[c] = 0;
            width = std::max(width, hi[c] - lo[c]);
        }
        if (width <= 2 * eps * scale) break;
        for (int i = 0; i < n; ++i) {
            const double e2 = i > 0 ? e[i - 1] * e[i - 1] : 0.0, di = d[i];
            for (int c = 0; c < k; ++c) {
                double v = di - x[c] - e2 / q[c];
                if (std::fabs(v) < tiny) v = -tiny;
                cnt[c] += v < 0.0;
                q[c] = v;
            }
        }
        for (int c = 0; c < k; ++c) (cnt[c] > c ? hi[c] : lo[c]) = x[c];   // cnt eigenvalues lie below x
    }
    for (int c = 0; c < k; ++c) w[c] = 0.5 * (lo[c] + hi[c]);
}

// Unit eigenvector y[n] of that matrix for its eigenvalue theta: three steps
// of inverse iteration on LU factors with partial pivoting (a second
// superdiagonal holds the fill of the row exchanges).  prev[0 .. nprev): unit
// vectors of (nearly) the same eigenvalue that y has to be orthogonal to.
inline void tri_eigvec(int n, const double *d, const double *e, double theta, double *y,
                       const double *const *prev = nullptr, int nprev = 0)
{
    double scale = std::fabs(theta);
    for (int i = 0; i < n; ++i) scale = std::max(scale, std::fabs(d[i]) + (i + 1 < n ? std::fabs(e[i]) : 0.0));
    const double tiny = 2.220446049250313e-16 * scale + 1e-290;
    std::vector<double> u0(n), u1(n, 0.0), u2(n, 0.0), l(n, 0.0);
    std::vector<char> swp(n, 0);
    double a = d[0] - theta, b = n > 1 ? e[0] : 0.0;     // the row being eliminated: a at k, b at k + 1
    for (int k = 0; k + 1 < n; ++k) {
        const double sub = e[k], nd = d[k + 1] - theta, ne = k + 2 < n ? e[k + 1] : 0.0;
        if (std::fabs(sub) > std::fabs(a)) {             // rows k and k + 1 change places
            swp[k] = 1;
            u0[k] = sub;
            u1[k] = nd;
            u2[k] = ne;
            l[k] = a / sub;
            a = b - l[k] * nd;
            b = -l[k] * ne;
        } else {
            u0[k] = std::fabs(a) < tiny ? tiny : a;
            u1[k] = b;
            l[k] = sub / u0[k];
            a = nd - l[k] * b;
            b = ne;
        }
    }
    u0[n - 1] = std::fabs(a) < tiny ? tiny : a;
    for (int i = 0; i < n; ++i) y[i] = 1.0 + 0.37 * ((i + 3 * nprev * (i % 5)) % 7);   // no structure in common with an eigenvector
    for (int it = 0; it < 3; ++it) {
        for (int k = 0; k + 1 < n; ++k) {
            if (swp[k]) std::swap(y[k], y[k + 1]);
            y[k + 1] -= l[k] * y[k];
        }
        for (int i = n - 1; i >= 0; --i) {
            double t = y[i];
            if (i + 1 < n) t -= u1[i] * y[i + 1];
            if (i + 2 < n) t -= u2[i] * y[i + 2];
            y[i] = t / u0[i];
        }
        double s = 0.0;
        for (int i = 0; i < n; ++i) s = std::max(s, std::fabs(y[i]));
        for (int i = 0; i < n; ++i) y[i] /= s;
        double q = 0.0;
        for (int pass = 0; pass < 2; ++pass)
            for (int k = 0; k < nprev; ++k) {
                double c = 0.0;
                for (int i = 0; i < n; ++i) c += y[i] * prev[k][i];
                for (int i = 0; i < n; ++i) y[i] -= c * prev[k][i];
            }
        for (int i = 0; i < n; ++i) q += y[i] * y[i];
        q = 1.0 / std::sqrt(q);
        for (int i = 0; i < n; ++i) y[i] *= q;
    }
}

// Unit right eigenvector y[n] of the upper Hessenberg matrix h (column-major,
// leading dimension ld) for its eigenvalue theta: two steps of inverse
// iteration with the LU factors of h - theta I (partial pivoting between
// neighbouring rows, the only ones that can hold the pivot).  scale: a norm
// of h; a pivot below 2^-52 scale is replaced by that.  prev[0 .. nprev): unit
// vectors of (nearly) the same eigenvalue that y has to be orthogonal to.
inline void hess_eigvec(int n, const double *h, int ld, double theta, double scale, double *y,
                        const double *const *prev = nullptr, int nprev = 0)
{
    const double tiny = 2.220446049250313e-16 * scale + 1e-290;
    std::vector<double> u((size_t)n * n, 0.0), l(n, 0.0);   // u row-major
    std::vector<char> swp(n, 0);
    auto U = [&](int i, int j) -> double & { return u[(size_t)i * n + j]; };
    for (int j = 0; j < n; ++j)
        for (int i = 0; i <= std::min(j + 1, n - 1); ++i) U(i, j) = h[(size_t)j * ld + i] - (i == j ? theta : 0.0);
    for (int k = 0; k + 1 < n; ++k) {
        if (std::fabs(U(k + 1, k)) > std::fabs(U(k, k))) {
            swp[k] = 1;
            for (int j = k; j < n; ++j) std::swap(U(k, j), U(k + 1, j));
        }
        if (std::fabs(U(k, k)) < tiny) U(k, k) = tiny;
        l[k] = U(k + 1, k) / U(k, k);
        U(k + 1, k) = 0.0;
        for (int j = k + 1; j < n; ++j) U(k + 1, j) -= l[k] * U(k, j);
    }
    if (std::fabs(U(n - 1, n - 1)) < tiny) U(n - 1, n - 1) = tiny;
    for (int i = 0; i < n; ++i) y[i] = 1.0 + 0.37 * ((i + 3 * nprev * (i % 5)) % 7);   // no structure in common with an eigenvector
    for (int it = 0; it < (nprev ? 3 : 2); ++it) {
        for (int k = 0; k + 1 < n; ++k) {
            if (swp[k]) std::swap(y[k], y[k + 1]);
            y[k + 1] -= l[k] * y[k];
        }
        for (int i = n - 1; i >= 0; --i) {
            double t = y[i];
            for (int j = i + 1; j < n; ++j) t -= U(i, j) * y[j];
            y[i] = t / U(i, i);
        }
        double s = 0.0;
        for (int i = 0; i < n; ++i) s = std::max(s, std::fabs(y[i]));
        double q = 0.0;
        for (int i = 0; i < n; ++i) y[i] /= s;
        for (int pass = 0; pass < 2; ++pass)
            for (int k = 0; k < nprev; ++k) {
                double c = 0.0;
                for (int i = 0; i < n; ++i) c += y[i] * prev[k][i];
                for (int i = 0; i < n; ++i) y[i] -= c * prev[k][i];
            }
        for (int i = 0; i < n; ++i) q += y[i] * y[i];
        q = 1.0 / std::sqrt(q);
        for (int i = 0; i < n; ++i) y[i] *= q;
    }
}

// Generalized symmetric problem P c = lambda S c (n x n row-major, symmetric,
// S positive definite): S = L L^T, then the eigenpairs of L^-1 P L^-T.  w[n]
// ascending, c[j * n + i] the column of w[j], S-orthonormal.  Returns false
// if S is not positive definite or the iteration did not converge.
inline bool gen_sym_eig(int n, const std::vector<double> &P, const std::vector<double> &S, double *w, double *c)
{
    std::vector<double> L((size_t)n * n, 0.0), A(P);
    for (int j = 0; j < n; ++j) {
        double d = S[(size_t)j * n + j];
        for (int t = 0; t < j; ++t) d -= L[(size_t)j * n + t] * L[(size_t)j * n + t];
        if (!(d > 0.0)) return false;
        L[(size_t)j * n + j] = std::sqrt(d);
        for (int i = j + 1; i < n; ++i) {
            double v = S[(size_t)i * n + j];
            for (int t = 0; t < j; ++t) v -= L[(size_t)i * n + t] * L[(size_t)j * n + t];
            L[(size_t)i * n + j] = v / L[(size_t)j * n + j];
        }
    }
    for (int pass = 0; pass < 2; ++pass) {   // A <- (L^-1 A)^T, twice
        for (int col = 0; col < n; ++col)
            for (int i = 0; i < n; ++i) {
                double v = A[(size_t)i * n + col];
                for (int t = 0; t < i; ++t) v -= L[(size_t)i * n + t] * A[(size_t)t * n + col];
                A[(size_t)i * n + col] = v / L[(size_t)i * n + i];
            }
        for (int i = 0; i < n; ++i)
            for (int j = i + 1; j < n; ++j) std::swap(A[(size_t)i * n + j], A[(size_t)j * n + i]);
    }
    for (int i = 0; i < n; ++i)
        for (int j = i + 1; j < n; ++j)
            A[(size_t)i * n + j] = A[(size_t)j * n + i] = 0.5 * (A[(size_t)i * n + j] + A[(size_t)j * n + i]);
    if (!sym_eig(n, A, w, c)) return false;
    for (int j = 0; j < n; ++j)   // c <- L^-T c
        for (int i = n - 1; i >= 0; --i) {
            double v = c[(size_t)j * n + i];
            for (int t = i + 1; t < n; ++t) v -= L[(size_t)t * n + i] * c[(size_t)j * n + t];
            c[(size_t)j * n + i] = v / L[(size_t)i * n + i];
        }
    return true;
}

}  // namespace moed
