"""Eigensolves of models with exactly degenerate levels, where a single Krylov
space holds one member of each level.  The lowest levels with their
multiplicities against dense diagonalisation of the oracle's H.  Bounds: those of the other
eigensolver tests (1e-9 FP64, 1e-8 FP32)."""
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
