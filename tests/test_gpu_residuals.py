"""The eigenvectors' true residual ||H x - E x|| of small random models, whose
Krylov runs come near the sector's whole space and lose orthogonality on the
way: a run that steps back judges convergence by the steps it keeps.  Bound:
10 tolerances of the largest |alpha| + beta of the run, which is at most
2 ||H||; 1e-7 is the FP32, 1e-11 the FP64 tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bound(precision, w):
    return 20 * (1e-7 if precision == "fp32" else 1e-11) * max(1.0, np.abs(w).max())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("seed", [5, 6, 17, 21, 1, 2])
def test_random_models(solver, oracle, precision, seed):
    rng = np.random.default_rng(seed)
    norb, nbath, U, J = 2, 4, 4.0, 1.0
    ek = np.concatenate([np.full(norb, -0.5 * (U + (2 * (U - 2 * J) - J))), rng.uniform(-1, 1, nbath)])
    vk = rng.uniform(0.1, 0.5, (norb, nbath))
    m = oracle.Model(norb, nbath, U, J, ek, vk)
    for nu, nd in ((2, 2), (2, 3), (3, 3)):
        H = oracle.dense_H(m, oracle.Basis(m.nsite, nu, nd))
        w = np.linalg.eigvalsh(H)
        for nev in (3, 6, 12):
            solver.set_options(precision=precision, nev=nev, green_fp64=False)
            solver.set_model(norb, nbath, U, J, ek, vk)
            ev, vec = solver.diag(nu, nd, nev)
            st = solver.diag_stats()
            assert st["res_true"] <= bound(precision, w), (nu, nd, nev, st)
            assert np.linalg.norm(H @ vec - vec * ev, axis=0).max() <= 1.01 * bound(precision, w)
            assert np.abs(ev - w[:nev]).max() < (1e-9 if precision == "fp64" else 1e-8)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("sym", [False, True])
def test_copies_of_levels(solver, oracle, precision, sym):
    """Identical baths: rounding brings further members of a level into a run,
    whose vectors have to be as good as the others'."""
    norb, nbath, U, J = 3, 3, 3.0, 0.5
    rng = np.random.default_rng(1)
    e, v = (np.zeros(1), np.full(1, 0.35)) if sym else (rng.uniform(-1, 1, 1), rng.uniform(0.1, 0.5, 1))
    ek = np.concatenate([np.full(norb, -0.5 * (U + 2 * (2 * (U - 2 * J) - J))), np.tile(e, norb)])
    vk = np.kron(np.eye(norb), v[None, :])
    m = oracle.Model(norb, nbath, U, J, ek, vk)
    for nu, nd in ((3, 3), (2, 3), (2, 2), (4, 3)):
        H = oracle.dense_H(m, oracle.Basis(m.nsite, nu, nd))
        w = np.linalg.eigvalsh(H)
        for nev in (3, 6, 12, 20):
            solver.set_options(precision=precision, nev=nev, green_fp64=False)
            solver.set_model(norb, nbath, U, J, ek, vk)
            ev, vec = solver.diag(nu, nd, nev)
            st = solver.diag_stats()
            assert st["res_true"] <= bound(precision, w), (nu, nd, nev, st)
            assert np.linalg.norm(H @ vec - vec * ev, axis=0).max() <= 1.01 * bound(precision, w)
