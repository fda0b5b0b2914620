// degeneracy.h -- whether a model can have exactly degenerate levels within one
// (Nup, Ndown) sector, beyond accidents of its parameters.  Host code only.
//
// A Krylov space holds one vector of each eigenspace, so the eigensolver looks
// for further members of a level where this says that there can be some.
// Levels are degenerate where symmetries of H within the sector do not commute:
//
//   * spin rotation: its multiplets have one member per sector, no reason;
//   * spins that rotate separately: one orbital with U = 0, or several with
//     J = 0, where an orbital with bath levels of its own keeps its spin;
//   * rotations of bath levels among themselves: two levels of one energy, or
//     levels that couple to nothing;
//   * rotations of orbitals, under which the Kanamori terms are invariant.  With
//     all bath energies different the bath has to stay as it is, so the generator
//     A, antisymmetric and not zero, needs A V = 0: V has at most norb - 2
//     independent rows.  With norb - 1 or norb of them every symmetry multiplies
//     each column of V by +1 or -1, and those commute;
//   * a particle-hole transformation that exchanges orbitals (two orbitals or
//     more): it does not commute with the electron parities of the orbitals.  It
//     needs bath energies that are their own mirror image about some level.  With
//     one orbital it commutes with the rest.
//
// "Zero", "equal" and "independent" allow for values that split levels by less
// than an eigensolve resolves; a model that is named here without need costs one
// more Lanczos run.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

namespace moed {

// ebath: [nbath] bath energies; vk: [nbath][norb] couplings (orbital fastest)
inline bool can_be_degenerate(int norb, int nbath, double U, double J, const double *ebath, const double *vk)
{
    constexpr double small = 1e-2;        // of U, J and couplings
    constexpr double near = 1e-3;         // of differences between bath energies
    if (norb > 1 ? std::fabs(J) < small : std::fabs(U) < small) return true;
    std::vector<double> e(ebath, ebath + nbath);
    std::sort(e.begin(), e.end());
    for (int k = 0; k + 1 < nbath; ++k)
        if (!(e[k + 1] - e[k] > near * std::max(1.0, std::fabs(e[k])))) return true;
    for (int k = 0; k < nbath; ++k) {
        double v = 0.0;
        for (int i = 0; i < norb; ++i) v = std::max(v, std::fabs(vk[(size_t)k * norb + i]));
        if (!(v > small)) return true;
    }
    if (norb < 2) return false;
    // independent rows of V: Gram-Schmidt, longest remaining row first
    std::vector<double> r(vk, vk + (size_t)nbath * norb);
    std::vector<char> used(norb, 0);
    int rank = 0;
    for (; rank < norb; ++rank) {
        int p = -1;
        double most = small;
        for (int i = 0; i < norb; ++i) {
            double s = 0.0;
            for (int k = 0; k < nbath; ++k) s += r[(size_t)k * norb + i] * r[(size_t)k * norb + i];
            if (!used[i] && std::sqrt(s) > most) {
                most = std::sqrt(s);
                p = i;
            }
        }
        if (p < 0) break;
        used[p] = 1;
        for (int i = 0; i < norb; ++i) {
            if (used[i]) continue;
            double c = 0.0;
            for (int k = 0; k < nbath; ++k) c += r[(size_t)k * norb + i] * r[(size_t)k * norb + p];
            for (int k = 0; k < nbath; ++k) r[(size_t)k * norb + i] -= c / (most * most) * r[(size_t)k * norb + p];
        }
    }
    if (rank <= norb - 2) return true;
    for (int k = 0; k < nbath; ++k)
        if (std::fabs(e[k] + e[nbath - 1 - k] - (e[0] + e[nbath - 1])) > near * std::max(1.0, std::fabs(e[k]))) return false;
    return true;
}

}  // namespace moed
