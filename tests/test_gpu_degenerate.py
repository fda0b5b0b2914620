"""Eigensolves of models with exactly degenerate levels, where a single Krylov
space holds one member of each level: equal baths, spins that rotate
separately (U = 0), orbitals that couple alike or in fewer combinations than
there are orbitals, baths that are each other's mirror image.
The lowest levels with their multiplicities against sums of one-spin levels
(U = 0) or dense diagonalisation of the oracle's H.  Bounds: those of the other
eigensolver tests (1e-9 FP64, 1e-8 FP32)."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-9, "fp32": 1e-8}


def levels(norb, U, J):
    return np.full(norb, -0.5 * (U + (norb - 1) * (2 * (U - 2 * J) - J)))


def dense(oracle, norb, nbath, U, J, ek, vk, nu, nd):
    m = oracle.Model(norb, nbath, U, J, ek, vk)
    return np.linalg.eigvalsh(oracle.dense_H(m, oracle.Basis(m.nsite, nu, nd)))


def check(solver, precision, norb, nbath, U, J, ek, vk, nu, nd, w, nevs):
    for nev in nevs:
        solver.set_options(precision=precision, nev=nev, green_fp64=False)
        solver.set_model(norb, nbath, U, J, ek, vk)
        ev, _ = solver.diag(nu, nd, nev, vectors=False)
        assert np.abs(ev - w[:nev]).max() < TOL[precision], (nev, ev, w[:nev], solver.diag_stats())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("sym", [False, True])
@pytest.mark.parametrize("norb,nbath,secs", [(3, 3, ((3, 3), (2, 3), (4, 3))), (2, 4, ((3, 3), (2, 3), (4, 3)))])
def test_equal_baths(solver, oracle, precision, sym, norb, nbath, secs):
    """Many members of a level, found by one search run each, in sectors of a few
    hundred states, where runs fill their space and give up."""
    per, (U, J) = nbath // norb, (4.0, 1.0) if norb == 2 else (3.0, 0.5)
    rng = np.random.default_rng(1)
    e, v = (np.linspace(-0.8, 0.8, per), np.full(per, 0.35)) if sym else (rng.uniform(-1, 1, per), rng.uniform(0.1, 0.5, per))
    ek = np.concatenate([levels(norb, U, J), np.tile(e, norb)])
    vk = np.kron(np.eye(norb), v[None, :])
    for nu, nd in secs:
        w = dense(oracle, norb, nbath, U, J, ek, vk, nu, nd)
        check(solver, precision, norb, nbath, U, J, ek, vk, nu, nd, w, (3, 4, 6, 12, 20))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_thick_restarts(solver, oracle, precision):
    """Sectors of 90 to 225 states, below the line of the unrestarted solver, and
    a given Krylov dimension."""
    norb, nbath, U, J = 3, 3, 3.0, 0.5
    rng = np.random.default_rng(1)
    ek = np.concatenate([levels(norb, U, J), np.full(3, rng.uniform(-1, 1))])
    vk = np.eye(3) * rng.uniform(0.1, 0.5)
    try:
        for nu, nd, nevs, ncv in ((1, 3, (3, 6, 12), 0), (2, 1, (3, 6, 12), 0), (2, 2, (20,), 0), (3, 3, (3, 6, 12), 30)):
            w = dense(oracle, norb, nbath, U, J, ek, vk, nu, nd)
            solver.set_options(gs_ncv=ncv)
            check(solver, precision, norb, nbath, U, J, ek, vk, nu, nd, w, nevs)
    finally:
        solver.set_options(gs_ncv=0)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("seed", range(4))
def test_free_spins(solver, precision, seed):
    rng = np.random.default_rng(seed)
    nbath, nu, nd = 7, 4, 4
    ek = np.concatenate([[rng.uniform(-0.5, 0.5)], rng.uniform(-1, 1, nbath)])
    vk = rng.uniform(0.1, 0.6, (1, nbath))
    h = np.diag(ek)
    h[0, 1:] = h[1:, 0] = vk[0]
    one = np.array([sum(c) for c in itertools.combinations(np.linalg.eigvalsh(h), nu)])
    w = np.sort((one[:, None] + one[None, :]).ravel())
    check(solver, precision, 1, nbath, 0.0, 0.0, ek, vk, nu, nd, w, (3, 4, 8))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("seed", range(200, 203))
def test_dependent_couplings(solver, oracle, precision, seed):
    rng = np.random.default_rng(seed)
    U, J = 3.0, 0.5
    for norb, nbath in ((3, 3), (3, 4), (4, 2), (4, 3)):
        vk = np.tile(rng.uniform(0.1, 0.5, nbath), (3, 1)) if norb == 3 else \
            rng.uniform(-1, 1, (norb, 2)) @ rng.uniform(0.1, 0.5, (2, nbath))
        ek = np.concatenate([levels(norb, U, J), rng.uniform(-1, 1, nbath)])
        n = norb + nbath
        for nu, nd in ((n // 2, n // 2), (n // 2 - 1, n // 2)):
            w = dense(oracle, norb, nbath, U, J, ek, vk, nu, nd)
            check(solver, precision, norb, nbath, U, J, ek, vk, nu, nd, w, (3, 4, 6, 12, 20))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("seed", range(3))
def test_mirrored_baths(solver, oracle, precision, seed):
    rng = np.random.default_rng(seed)
    e, v = rng.uniform(-1, 1, 2), rng.uniform(0.1, 0.5, 2)
    U, J = 4.0, 1.0
    ek = np.concatenate([levels(2, U, J), e, -e])
    vk = np.kron(np.eye(2), v[None, :])
    for nu, nd in ((3, 3), (2, 4)):
        w = dense(oracle, 2, 4, U, J, ek, vk, nu, nd)
        check(solver, precision, 2, 4, U, J, ek, vk, nu, nd, w, (3, 4, 6, 12))
