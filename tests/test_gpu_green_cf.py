"""k_green_cf at the edges of its blocks of 32 frequencies: G against the
records' continued fractions in the oracle's term-by-term division, for 1 and 2
orbitals.

Tolerance: with 1/w = conj(w) / |w|^2 each level carries a few roundings of its
|E| + |a| + |g| (below 64 here), and the error of a level reaches G multiplied
by at most |G| / w_0 (on the Matsubara axis the product of the b / |w|^2 down
the fraction telescopes to that): 2 sides x 100 levels x 4 x 64 x 2^-53 / w_0 =
1e-10 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,nw", [("C1", 1), ("C1", 31), ("C1", 33), ("C1", 1000), ("C2", 64), ("C2", 97)])
def test_green_of_records(solver, oracle, pkg, name, nw):
    cfg = pkg.configs.config(name)
    ek, vk = cfg.model()
    om = (2.0 * np.arange(nw) + 1.0) * np.pi / 50.0
    solver.set_options(precision="fp64", nstep=min(cfg.nstep, 100), nev=8, beta=cfg.beta, fortran_cmplx=True)
    solver.set_model(cfg.norb, cfg.nbath, cfg.U, cfg.J, ek, vk)
    solver.set_sectors([n for n, _ in cfg.sectors], [u for _, u in cfg.sectors])
    solver.set_omega(om)
    st = solver.ed_solve()
    G = solver.ed_calc_green_ftn()
    recs = iter(solver.green_coeffs())
    Go = np.zeros_like(G)
    for e in st:
        nelec, nup = cfg.sectors[e["sector"] - 1]
        even = nelec == 2 * nup
        for _ in range(1 if even else 2):
            for a in range(cfg.norb):
                r, g = next(recs), np.zeros(nw, complex)
                for sgn, n, ca, cb in ((1, r["np"], r["ap"], r["bp"]), (-1, r["nn"], r["an"], r["bn"])):
                    if n >= 0:
                        oracle.green_cf(sgn, e["val"], e["prob"], 1.0 if even else 0.5, n, ca, cb, om, g)
                Go[a] += g
    assert next(recs, None) is None
    assert (np.abs(G - Go) <= 1e-10 * np.abs(Go).max()).all()
