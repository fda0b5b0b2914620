"""can_be_degenerate (mo-dmft_gb300/csrc/degeneracy.h) against the spectra of
small models by dense diagonalisation of the oracle's H: it is true for every
model with a degenerate level in a sector, whatever the symmetry behind it, and
false for models with random parameters, whose eigensolves would only pay for
a search that finds nothing."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "degeneracy.h"
extern "C" int f(int norb, int nbath, double U, double J, const double *e, const double *v)
{
    return moed::can_be_degenerate(norb, nbath, U, J, e, v) ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def can(tmp_path_factory):
    d = tmp_path_factory.mktemp("degeneracy")
    src, lib = d / "shim.cpp", d / "lib.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mo-dmft_gb300", "csrc"),
                    "-o", str(lib), str(src)], check=True)
    L = C.CDLL(str(lib))
    dp = C.POINTER(C.c_double)

    def run(U, J, ek, vk):
        norb, nbath = vk.shape
        e, v = np.ascontiguousarray(ek[norb:]), np.ascontiguousarray(vk.T)
        return bool(L.f(norb, nbath, C.c_double(U), C.c_double(J), e.ctypes.data_as(dp), v.ctypes.data_as(dp)))
    return run


def levels(norb, U, J, shift=0.0):
    return np.full(norb, shift - 0.5 * (U + (norb - 1) * (2 * (U - 2 * J) - J)))


def blocks(v):
    return np.kron(np.eye(v.shape[0]), np.ones((1, v.shape[1]))) * np.tile(v.ravel(), (v.shape[0], 1))


def models():
    r = np.random.default_rng(5)
    u = lambda *s: r.uniform(0.1, 0.5, s)
    e = lambda n: r.uniform(-1, 1, n)
    out = []

    def add(name, U, J, eb, vk, shift=0.0):
        out.append((name, U, J, np.concatenate([levels(vk.shape[0], U, J, shift), eb]), vk))

    add("free_spins_1x4", 0.0, 0.0, e(4), u(1, 4), 0.3)
    add("free_spins_1x5", 0.0, 0.5, e(5), u(1, 5), 0.1)
    add("no_J_2x4", 2.0, 0.0, e(4), blocks(u(2, 2)), 0.1)
    add("equal_baths_2x4", 4.0, 1.0, np.tile(e(2), 2), blocks(np.tile(u(1, 2), (2, 1))))
    add("two_equal_levels_1x4", 2.0, 0.0, np.array([0.3, -0.7, 0.3, 0.1]), u(1, 4))
    add("loose_level_1x4", 2.0, 0.0, e(4), np.array([[0.3, 0.0, 0.2, 0.4]]))
    add("equal_rows_3x3", 3.0, 0.5, e(3), np.tile(u(1, 3), (3, 1)))
    add("proportional_rows_3x2", 3.0, 0.5, e(2), np.outer([0.4, 0.9, -0.7], u(2)))
    add("four_on_two_4x2", 3.0, 0.5, e(2), u(4, 2))
    add("three_on_one_3x1", 3.0, 0.5, e(1), u(3, 1))
    eb, v = e(2), u(1, 2)
    add("mirrored_2x4", 4.0, 1.0, np.concatenate([eb, -eb]), blocks(np.tile(v, (2, 1))))
    add("mirrored_about_a_level_2x4", 4.0, 1.0, 0.4 + np.concatenate([eb, -eb]), blocks(np.tile(v, (2, 1))), 0.4)
    for k in range(4):
        add(f"random_dense_2x4_{k}", 4.0, 1.0, e(4), u(2, 4), 0.1 * k)
        add(f"random_blocks_2x4_{k}", 4.0, 1.0, e(4), blocks(u(2, 2)), 0.1 * k)
        add(f"random_1x5_{k}", 2.0, 0.0, e(5), u(1, 5), 0.1 * k)
        add(f"random_dense_3x3_{k}", 3.0, 0.5, e(3), u(3, 3))
        add(f"random_mirrored_1x4_{k}", 2.0, 0.0, np.concatenate([eb, -eb]) * (k + 1) / 4, u(1, 4))
    return out


@pytest.mark.parametrize("name,U,J,ek,vk", models(), ids=[m[0] for m in models()])
def test_against_spectra(can, oracle, name, U, J, ek, vk):
    norb, nbath = vk.shape
    m = oracle.Model(norb, nbath, U, J, ek, vk)
    n, found = norb + nbath, False
    for nu in range(1, n // 2 + 1):
        for nd in {nu, nu + 1, n - nu} & set(range(1, n)):
            w = np.linalg.eigvalsh(oracle.dense_H(m, oracle.Basis(n, nu, nd)))
            found |= bool((np.diff(w) < 1e-9).any())
    assert found == (not name.startswith("random")), "the model is not what its name says"
    assert can(U, J, ek, vk) == found


def test_tolerances(can):
    """Values that split levels by next to nothing count as equal or zero."""
    e, v = np.array([0.2, -0.6, 0.2 + 5e-4, 0.9]), np.full((1, 4), 0.3)
    assert can(2.0, 0.0, np.concatenate([[-1.0], e]), v)
    assert can(5e-3, 0.0, np.concatenate([[-1.0], [0.2, -0.6, 0.4, 0.9]]), v)
    assert not can(2.0, 0.0, np.concatenate([[-1.0], [0.2, -0.6, 0.4, 0.9]]), v)
    v[0, 2] = 1e-3
    assert can(2.0, 0.0, np.concatenate([[-1.0], [0.2, -0.6, 0.4, 0.9]]), v)
    row = np.array([[0.3, 0.2, 0.4, 0.25]])
    V = np.concatenate([row, row, row + 1e-3 * np.array([[1, -1, 1, -1]])])
    assert can(3.0, 0.5, np.concatenate([np.zeros(3), [0.2, -0.6, 0.4, 0.8]]), V)
