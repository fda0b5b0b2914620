// kryhost.h -- the host side of the eigensolver's Lanczos run (eigs.cu): when it
// reorthogonalises, and the projected matrix with what that takes out.  Host
// code only.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

namespace moed {

// One reorthogonalisation: of the pair U_{j-1}, U_j against all earlier vectors,
// `gap` steps after the one before.
struct KryClean {
    int j, gap;
};

// When to reorthogonalise.  Rounding errors grow by the ratio at which Ritz
// values converge; the period follows the components that each reorthogonalisation
// has found, so that they stay near `target`.
struct KryPeriod {
    double unit, target, most;
    int pmax, ptop, period;
    int good = -1;            // step of the last reorthogonalisation that found little
    double grow = 0.0;        // largest growth per step seen
    double hmax = 0.0;        // largest component seen since the last restart
    enum Verdict { kept, back, lost };

    // The longest period rises while little is found.  In small sectors, where
    // a reorthogonalisation costs about a step, it does not: one that comes
    // too late costs a period's steps.  9 million FP32 elements: 79 -> 65 ms.
    KryPeriod(bool f32, long long D)
        : unit(f32 ? 6e-8 : 1.1e-16), target(f32 ? 2e-5 : 1e-11), most(f32 ? 1e-2 : 1e-4), pmax(f32 ? 16 : 24),
          ptop(D < (1 << 19) ? pmax : 2 * pmax), period(f32 ? 6 : 10)
    {
    }

    // A reorthogonalisation found components of up to c.  back: orthogonality
    // was lost before it; the run has to go back to step `good`, with shorter
    // periods.  lost: there is nothing to go back to.  To be called for every
    // one, in order.
    Verdict judge(const KryClean &r, double c, bool restarted)
    {
        if (!(c < most)) {
            if (good < 0 || r.gap <= 2) return lost;
            ptop = pmax = period = std::max(2, std::min(r.gap, pmax) / 2);
            return back;
        }
        good = r.j;
        // Components c taken out once leave c^2 in every vector to come (the
        // earlier vectors are orthogonal to c only), which does not grow.
        grow = std::max(grow, std::max(std::log(c / std::max(2 * unit, hmax * hmax)), 0.3) / r.gap);
        hmax = std::max(hmax, c);
        if (c < target) pmax = std::max(pmax, std::min(ptop, r.gap + r.gap / 4 + 1));
        period = std::max(2, std::min(restarted ? std::min(5, pmax) : pmax, (int)(std::log(target / (2 * unit)) / grow)));
        return kept;
    }

    void restart()
    {
        good = -1;
        hmax = 0.0;
        period = std::min(period, 4);
    }
};

// The projected matrix hp (m x m, column-major) of the vectors q_0 .. q_{m-1}
// of a run with reorthogonalisations `re` (those of steps up to m): the
// tridiagonal T of al and be, and what the reorthogonalisations took out, so that
// H Q = Q hp + be[m] q_m e^T to rounding.  inv: reciprocal norms of the stored
// vectors; h: column j (leading dimension ldh) the components taken out of U_j
// along q_0, q_1, ...
//
// Cleaning q_{j-1} = q'_{j-1} + Q g1 and q_j = q'_j + Q g2 (Q the earlier vectors)
// changes H q_{j-2} and H q'_{j-1}:
//   column j-2 gains beta_{j-1} g1,
//   column j-1 gains beta_j g2 + alpha_{j-1} g1 - T g1.
// Both columns are there for j = m as well, where q_m is the residual vector.
inline void kry_projected(int m, const double *al, const double *be, const double *inv, const std::vector<KryClean> &re,
                          const double *h, int ldh, std::vector<double> &hp)
{
    hp.assign((size_t)m * m, 0.0);
    for (int i = 0; i < m; ++i) {
        hp[(size_t)i * m + i] = al[i];
        if (i + 1 < m) hp[(size_t)i * m + i + 1] = hp[(size_t)(i + 1) * m + i] = be[i + 1];
    }
    for (const KryClean &cl : re) {
        const int j = cl.j;
        if (j > m) continue;
        const double *g1 = h + (size_t)(j - 1) * ldh, *g2 = h + (size_t)j * ldh;
        const double s1 = inv[j - 1], s2 = inv[j];
        double *c2 = j >= 2 ? &hp[(size_t)(j - 2) * m] : nullptr, *c1 = &hp[(size_t)(j - 1) * m];
        for (int l = 0; l < j - 1; ++l) {
            if (c2) c2[l] += be[j - 1] * s1 * g1[l];
            double tg = al[l] * g1[l];
            if (l > 0) tg += be[l] * g1[l - 1];
            if (l + 1 < j - 1) tg += be[l + 1] * g1[l + 1];
            c1[l] += be[j] * s2 * g2[l] + s1 * (al[j - 1] * g1[l] - tg);
        }
        if (j >= 2) c1[j - 1] -= be[j - 1] * s1 * g1[j - 2];
    }
}

// Largest true residual ||H x - E x|| of the returned unit vectors that a run
// is accepted with.  Convergence is judged on T's estimate; what a run lost
// beyond it shows only here.  Ten times the tolerance, as the estimate of a sound run
// is within a few times the residual; 1e-6 and 1e-12 of the norm are ten times
// the rounding of the vectors themselves (measured: 1.4e-7 with FP32 vectors of
// up to 41 million elements).
inline double kry_residual_limit(bool f32, double tol, double anorm)
{
    return std::max(10 * tol, f32 ? 1e-6 : 1e-12) * std::max(anorm, 1.0);
}

}  // namespace moed
