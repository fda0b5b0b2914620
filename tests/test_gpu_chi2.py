"""k_chi2 at the edges of its range: fewer frequencies than threads, counts
around a CTA's 128 and around the lines where a parameter set is split over 2,
4 and 8 CTAs, batches on both sides of the split, no bath, couplings that are
zero, the largest tables.

Reference: the formulas of func.f90 in 80-bit arithmetic (64-bit significand or
more).  Tolerance: every sum's terms carry at most nbath + 24 roundings (the
level sums, the residual, the weights) on quantities bounded by the same
formula with absolute values, and a thread's sum, its 16 + 8 segment sums, the
CTAs' 8 and the 5 orbitals' at most nw / 128 + 40 more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def reference(x, om, dev, nbath, norb):
    """chi^2, its gradient and both with absolute values (fortran_cmplx rounds the w_n of z alone)."""
    L = np.longdouble
    e, V, ef = x[:nbath].astype(L), x[nbath:nbath * (1 + norb)].reshape(norb, nbath).astype(L), x[x.size - norb:].astype(L)
    w, wz = om.astype(L)[None], om.astype(np.float32).astype(L)[None]
    y = 1 / (wz ** 2 + e[:, None] ** 2)                       # [nbath][nw]
    zr, zi = -e[:, None] * y, -wz * y
    rr = V ** 2 @ zr + ef[:, None] - dev.real
    ri = V ** 2 @ zi - dev.imag
    ra = V ** 2 @ abs(zr) + abs(ef)[:, None] + abs(dev.real)
    ia = V ** 2 @ abs(zi) + abs(dev.imag)
    nw = om.size
    c = L(norb * norb)
    out = []
    for R, I, s in ((rr, ri, 1), (ra, ia, 0)):
        Rw, Iw = R / w, I / w
        f = ((R * Rw + I * Iw).sum()) / (c * nw)
        if s:
            gv = 4 * V * (Rw @ zr.T + Iw @ zi.T) / c / nw
            ge = 2 * ((V ** 2)[:, :, None] * (Rw[:, None] * (zr ** 2 - zi ** 2) + 2 * Iw[:, None] * zr * zi)).sum((0, 2)) / c / nw
            gf = 2 * Rw.sum(1) / c / nw
        else:
            gv = 4 * abs(V) * (Rw @ abs(zr).T + Iw @ abs(zi).T) / c / nw
            ge = 2 * ((V ** 2)[:, :, None] * (Rw[:, None] * (2 * zr ** 2 + y) + 2 * Iw[:, None] * abs(zr * zi))).sum((0, 2)) / c / nw
            gf = 2 * Rw.sum(1) / c / nw
        out.append((f, np.concatenate([ge, gv.ravel(), gf])))
    return out


@pytest.mark.parametrize("norb,nbath,nw,nbatch,zeros", [
    (1, 0, 33, 2, False), (1, 1, 1, 1, False), (1, 29, 127, 3, False), (2, 4, 128, 5, True), (3, 12, 129, 1, True),
    (3, 9, 511, 152, True), (3, 9, 512, 152, True), (2, 12, 1023, 76, False), (2, 12, 1024, 77, False),
    (3, 14, 2048, 38, False), (5, 9, 2050, 2, False), (4, 11, 4096, 1, True), (3, 12, 512, 400, True)])
def test_chi2_batches(solver, norb, nbath, nw, nbatch, zeros):
    import torch

    rng = np.random.default_rng(1000 * nbath + nw)
    om = (2.0 * np.arange(nw) + 1.0) * np.pi / 100.0
    dev = 0.3 * (rng.standard_normal((norb, nw)) - 1j * rng.random((norb, nw)))
    X = np.concatenate([rng.uniform(-2, 2, (nbatch, nbath)), rng.uniform(-0.6, 0.6, (nbatch, norb * nbath)),
                        rng.uniform(-0.5, 0.5, (nbatch, norb))], 1)
    if zeros:
        X[:, nbath:nbath * (1 + norb)] *= rng.random(norb * nbath) < 0.4
    nx = X.shape[1]
    solver.set_options(fortran_cmplx=True)
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")
    x, o, d = t(X), t(om), t(np.ascontiguousarray(dev.T).view(np.float64))
    f, g, f0 = (torch.full(s, np.nan, dtype=torch.float64, device="cuda") for s in ((nbatch,), (nbatch, nx), (nbatch,)))
    torch.cuda.synchronize()
    solver.chi2_grad_dev(nbatch, x.data_ptr(), nw, nx, o.data_ptr(), d.data_ptr(), nbath, norb, f.data_ptr(), g.data_ptr())
    solver.chi2_grad_dev(nbatch, x.data_ptr(), nw, nx, o.data_ptr(), d.data_ptr(), nbath, norb, f0.data_ptr(), 0)
    torch.cuda.synchronize()
    f, g, f0 = f.cpu().numpy(), g.cpu().numpy(), f0.cpu().numpy()
    tol = (nbath + 24 + nw / 128 + 40) * U
    assert (f == f0).all()
    for b in sorted({0, 1, nbatch // 2, nbatch - 1} & set(range(nbatch))):
        (fr, gr), (fa, ga) = reference(X[b], om, dev, nbath, norb)
        assert abs(f[b] - fr) <= tol * fa
        assert (abs(g[b] - gr) <= tol * ga).all()


@pytest.mark.parametrize("norb,nbath,nw", [(1, 1, 40), (1, 2, 255), (1, 3, 256), (1, 5, 300), (2, 6, 1024), (1, 7, 2049),
                                           (3, 6, 4096), (1, 4, 5200), (2, 4, 130)])
def test_fit_function(solver, oracle, norb, nbath, nw):
    """FUNC inside a fit (fit_func_sum): levels in groups of 4, 2 and 1, one
    CTA and clusters, grids with more w_n per thread than are laid out
    beforehand.  The value a fit returns is FUNC at the x it returns, which the
    oracle sums in another order: 1e-12 as for FUNC itself."""
    rng = np.random.default_rng(nbath * 100 + nw)
    om = (2.0 * np.arange(nw) + 1.0) * np.pi / 50.0
    solver.set_options(fortran_cmplx=True)
    e, v = rng.uniform(-1.5, 1.5, nbath), rng.uniform(0.2, 0.5, (norb, nbath))
    dev = (v[:, None, :] ** 2 / (1j * om[None, :, None] - e)).sum(-1) + 0.1
    dev = dev + 1e-3 * (rng.standard_normal(dev.shape) + 1j * rng.standard_normal(dev.shape))
    X = np.stack([np.concatenate([e + 0.02 * s, v.ravel() * (1 + 0.03 * s), np.full(norb, 0.1)]) for s in (1, -1)])
    if norb == 2:
        X[1, nbath] = 0.0   # a coupling that a fit keeps at zero or not, as the gradient says
    x, f, _, _ = solver.fit_batch(X, om, dev, nbath, norb, ftol=1e-3)
    for b in range(2):
        fo = oracle.func(x[b], norb + nbath, om, dev, nbath, norb)
        assert abs(f[b] - fo) < 1e-12 * fo
