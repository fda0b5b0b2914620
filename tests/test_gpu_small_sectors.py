"""Eigensolves of small sectors whose steps run inside one launch: k_trl_steps
(one CTA, thick restarts) down to a single state, with fewer states than a
cycle and with restarts, and k_kry_cluster with 1 to 8 CTAs and 1, 2 and 4
elements per thread, row pads of 0 and 31 elements among them.  Eigenvalues
against dense diagonalisation of the oracle's H, or for the larger sectors
against the launch-per-step path (another H*v variant).  Bounds: those of the
other eigensolver tests (1e-9 FP64, 1e-8 FP32; residuals 1e-7, 1e-4)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def model(solver, precision, norb, nbath, nev, gs_ncv=0):
    rng = np.random.default_rng(norb * 100 + nbath)
    ek = np.concatenate([rng.uniform(-2, -1, norb), rng.uniform(-1, 1, nbath)])
    vk = rng.uniform(0.1, 0.6, (norb, nbath))
    solver.set_options(precision=precision, nev=nev, green_fp64=False, gs_ncv=gs_ncv)
    solver.set_model(norb, nbath, 3.0, 0.5, ek, vk)
    return ek, vk


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("norb,nbath,nu,nd,nev,gs_ncv", [
    (2, 4, 0, 0, 1, 0), (2, 4, 6, 1, 3, 0), (1, 3, 1, 1, 6, 0), (2, 6, 0, 4, 6, 0), (2, 6, 4, 8, 8, 0),
    (2, 6, 1, 1, 8, 0), (3, 3, 1, 2, 5, 0), (2, 6, 2, 2, 4, 20), (3, 4, 3, 2, 3, 30), (1, 6, 3, 3, 4, 30),
    (2, 4, 2, 3, 6, 0), (5, 2, 2, 3, 4, 24)])
def test_against_dense(solver, oracle, precision, norb, nbath, nu, nd, nev, gs_ncv):
    try:
        ek, vk = model(solver, precision, norb, nbath, nev, gs_ncv)
        m = oracle.Model(norb, nbath, 3.0, 0.5, ek, vk)
        H = oracle.dense_H(m, oracle.Basis(m.nsite, nu, nd))
        w = np.linalg.eigvalsh(H)
        ev, vec = solver.diag(nu, nd, nev)
    finally:
        solver.set_options(gs_ncv=0)
    assert np.abs(ev[:nev] - w[:nev]).max() < (1e-9 if precision == "fp64" else 1e-8)
    assert np.abs(vec.T @ vec - np.eye(nev)).max() < (1e-9 if precision == "fp64" else 1e-5)
    assert np.linalg.norm(H @ vec - vec * ev, axis=0).max() < (1e-7 if precision == "fp64" else 1e-4)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("norb,nbath,nu,nd,nev", [
    (2, 6, 1, 4, 3), (1, 9, 9, 5, 3), (2, 6, 3, 3, 4), (1, 8, 4, 2, 3), (3, 6, 3, 3, 2), (3, 6, 5, 3, 5),
    (2, 7, 4, 4, 3)])
def test_against_launches(solver, precision, norb, nbath, nu, nd, nev):
    D = math.comb(norb + nbath, nu) * math.comb(norb + nbath, nd)
    dt = 1 if precision == "fp32" else 0
    model(solver, precision, norb, nbath, nev)
    ev, vec = solver.diag(nu, nd, nev)
    _, chosen = solver.hv_tuning(nu, nd, dt)
    other = 0 if chosen else 1
    try:
        solver.hv_set_variant(nu, nd, other, dt)
        ref, _ = solver.diag(nu, nd, nev, vectors=False)
    finally:
        solver.hv_set_variant(nu, nd, chosen, dt)
    assert vec.shape[0] == D
    assert np.abs(ev - ref).max() < (1e-9 if precision == "fp64" else 1e-8)
    assert np.abs(vec.T @ vec - np.eye(nev)).max() < (1e-9 if precision == "fp64" else 1e-5)
    hx = np.stack([solver.multiply_H(nu, nd, np.ascontiguousarray(vec[:, i])) for i in range(nev)], 1)
    assert np.linalg.norm(hx - vec * ev, axis=0).max() < (1e-7 if precision == "fp64" else 1e-4)
