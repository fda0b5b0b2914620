"""k_delta_new at the edges of its range: grids whose points have weights 1, 2, 4
and 8 in every mixture (odd and even sqrt(Nq), down to one point), output
counts on both sides of the lines between its thread groups, and a Green's
function without imaginary part (the term-by-term division).

Gksum: both sides sum at most 10,000 terms of relative error a few 2^-53 whose
moduli add up to less than 100 times the sum's, so 1e-12 relative bounds the
difference.  D_ev = 1/Gr - 1/Gksum + D_ev cancels (|1/Gr| grows with w_n while
D_ev does not), so it is checked as what it is, that formula on the device's
own Gksum: two divisions and two sums, each within 8 x 2^-53 of the moduli."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def check(solver, oracle, hk, mu, gr, dev):
    dn, gk = solver.delta_new(gr, dev, mu)
    _, gk_o = oracle.delta_new(hk, mu, gr, dev)
    assert rel(gk, gk_o) < 1e-12
    scale = np.abs(1.0 / gr) + np.abs(1.0 / gk) + np.abs(dev)
    assert (np.abs(dn - (1.0 / gr - 1.0 / gk + dev)) <= 8 * 2.0 ** -53 * scale).all()


@pytest.mark.parametrize("norb,nw,nk", [(1, 1, 1), (1, 5, 2), (2, 7, 3), (1, 304, 4), (1, 305, 5), (3, 811, 16),
                                        (2, 1216, 17), (3, 1111, 31), (3, 4096, 100)])
def test_delta_new_grids(solver, oracle, norb, nw, nk):
    rng = np.random.default_rng(100 * nk + nw)
    solver.set_model(norb, 1, 1.0, 0.0, np.zeros(norb + 1), np.full((norb, 1), 0.3))
    solver.set_band_structure(nk * nk)
    hk, _ = oracle.set_band_structure(norb, nk * nk)
    om = (2.0 * np.arange(nw) + 1.0) * np.pi / 50.0
    gr = 1.0 / (1j * om[None, :] + 0.3 * rng.standard_normal((norb, 1)))
    dev = 0.2 * (rng.standard_normal((norb, nw)) - 1j * rng.random((norb, nw)))
    check(solver, oracle, hk, 0.4, gr, dev)


def test_delta_new_real_axis(solver, oracle):
    """Im z = 0: outside the band every term is real and finite."""
    solver.set_model(1, 1, 1.0, 0.0, np.zeros(2), np.full((1, 1), 0.3))
    solver.set_band_structure(81)
    hk, _ = oracle.set_band_structure(1, 81)
    gr = np.array([[0.25, 0.2, -0.3]], dtype=np.complex128)
    check(solver, oracle, hk, 0.1, gr, np.zeros((1, 3), dtype=np.complex128))
