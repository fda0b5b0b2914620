"""k_hv_wide and k_hv_row at the edges of their packings: one to three orbitals
(bath groups of 1, 2 and 3 rows), dense and block V, sectors with only single
rows, one row, fewer rows than an item and column counts on both sides of the
64-column unit; against the oracle's H*v with the FP32 and FP64 bounds of the
other H*v tests (2e-6, 1e-13 relative).  Models with four orbitals refuse the
wide shapes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def model(norb, nbath, dense):
    rng = np.random.default_rng(10 * norb + nbath)
    ek = np.concatenate([rng.uniform(-2, 0, norb), rng.uniform(-1, 1, nbath)])
    vk = rng.uniform(0.1, 0.6, (norb, nbath))
    if not dense:
        vk *= np.kron(np.eye(norb), np.ones((1, nbath // norb)))
    return 3.0, 0.6, ek, vk


@pytest.mark.parametrize("norb,nbath,dense", [(1, 5, True), (1, 7, True), (2, 4, False), (2, 5, True), (3, 3, False),
                                              (3, 4, True), (3, 6, False)])
def test_every_sector_shape(solver, oracle, pkg, norb, nbath, dense):
    U, J, ek, vk = model(norb, nbath, dense)
    solver.set_model(norb, nbath, U, J, ek, vk)
    m = oracle.Model(norb, nbath, U, J, ek, vk)
    n = norb + nbath
    rng = np.random.default_rng(7)
    secs = {(n // 2, n // 2), (n // 2, n // 2 + 1), (2, n - 2), (1, 1), (0, n // 2), (n // 2, 0), (n, 1), (n - 1, n), (1, n // 2)}
    for nu, nd in sorted(secs):
        b = oracle.Basis(n, nu, nd)
        x = rng.standard_normal(b.ntot).astype(np.float32)
        ref = oracle.multiply_H(m, b, x.astype(np.float64))
        for dt, xx, tol in ((pkg.FP32, x, 2e-6), (pkg.FP64, x.astype(np.float64), 1e-13)):
            shapes, _ = solver.hv_tuning(nu, nd, dt)
            for v, (shape, _) in enumerate(shapes):
                try:
                    solver.hv_set_variant(nu, nd, v, dt)
                except pkg.EDError as e:
                    assert e.code == 1
                    continue
                assert rel(solver.multiply_H(nu, nd, xx), ref) < tol, (nu, nd, dt, v, shape)


def test_four_orbitals_refused(solver, pkg):
    U, J, ek, vk = model(4, 4, True)
    solver.set_model(4, 4, U, J, ek, vk)
    with pytest.raises(pkg.EDError) as e:
        solver.hv_set_variant(4, 4, 0, pkg.FP32)
    assert e.value.code == 1
