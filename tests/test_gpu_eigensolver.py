"""The unrestarted eigensolver and the thick restarts on both sides of the line
between them (D = 4 (2 nev + 24), 128), with Krylov spaces that fill up and go
on from the kept vectors, and on models whose levels are exactly degenerate,
where a Krylov space holds one vector of each eigenspace: the lowest nev levels
with their multiplicities against dense diagonalisation of the oracle's H.
Bounds: the eigenvalues' of the other eigensolver tests (1e-9 FP64, 1e-8 FP32);
the vectors are orthonormal and eigenvectors to the residual tolerances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(solver, oracle, norb, nbath, U, J, ek, vk, nu, nd, nev, precision):
    solver.set_options(precision=precision, nev=nev, green_fp64=False)
    solver.set_model(norb, nbath, U, J, ek, vk)
    m = oracle.Model(norb, nbath, U, J, ek, vk)
    H = oracle.dense_H(m, oracle.Basis(m.nsite, nu, nd))
    w = np.linalg.eigvalsh(H)
    ev, vec = solver.diag(nu, nd, nev)
    assert np.abs(ev - w[:nev]).max() < (1e-9 if precision == "fp64" else 1e-8), (ev, w[:nev], solver.diag_stats())
    assert np.abs(vec.T @ vec - np.eye(nev)).max() < (1e-9 if precision == "fp64" else 1e-5)
    r = H @ vec - vec * ev
    assert np.linalg.norm(r, axis=0).max() < (1e-7 if precision == "fp64" else 1e-4)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("norb,nbath,nu,nd,nev", [
    (1, 5, 3, 2, 3),    # 300: a run of at most 225 vectors
    (1, 5, 2, 2, 6),    # 225
    (2, 3, 2, 3, 1),    # 100: thick restarts
    (2, 4, 2, 1, 2),    # 90
    (2, 4, 3, 3, 6),    # 400
    (3, 4, 3, 3, 12),   # 1,225
    (2, 6, 3, 4, 20),   # 3,920: more states than one output tile
    (4, 3, 3, 4, 5),    # 1,225, four orbitals
])
def test_generic_models(solver, oracle, precision, norb, nbath, nu, nd, nev):
    rng = np.random.default_rng(norb * 100 + nbath * 10 + nev)
    ek = np.concatenate([rng.uniform(-2, -1, norb), rng.uniform(-1, 1, nbath)])
    vk = rng.uniform(0.1, 0.6, (norb, nbath))
    run(solver, oracle, norb, nbath, 3.0, 0.5, ek, vk, nu, nd, nev, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("norb,nbath,nu,nd,nev", [(2, 6, 4, 4, 4), (2, 6, 3, 3, 4), (2, 6, 3, 4, 6), (3, 6, 3, 4, 3)])
def test_equivalent_orbitals(solver, oracle, precision, norb, nbath, nu, nd, nev):
    """Identical baths per orbital: the Kanamori interaction is invariant under
    rotations among the orbitals."""
    per = nbath // norb
    rng = np.random.default_rng(3)
    eps, v = np.tile(rng.uniform(-1, 1, per), norb), rng.uniform(0.1, 0.5, per)
    vk = np.kron(np.eye(norb), v[None, :])
    U, J = (4.0, 1.0) if norb == 2 else (3.0, 0.5)
    mu = 0.5 * (U + (norb - 1) * (2 * (U - 2 * J) - J))
    if (norb, nbath) == (3, 6):   # dense diagonalisation of 10,584 states is too long: multiplicity alone
        solver.set_options(precision=precision, nev=nev)
        solver.set_model(norb, nbath, U, J, np.concatenate([np.full(norb, -mu), eps]), vk)
        ev, _ = solver.diag(nu, nd, nev, vectors=False)
        assert np.ptp(ev) < (1e-9 if precision == "fp64" else 1e-8)   # the ground triplet
        return
    run(solver, oracle, norb, nbath, U, J, np.concatenate([np.full(norb, -mu), eps]), vk, nu, nd, nev, precision)
