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

}  // namespace moed
