"""Performance cases of the exact-diagonalization impurity solver.

Each case is one call (or the solve + Green's function pair of calls) that a
DMFT program makes through the public entry points of ``EDSolver``:

  hv       y = H x on device vectors (``multiply_H_dev`` / ``_mixed_dev``)
  lanczos  the Green's-function recurrence from a host vector
  diag     the lowest eigenvalues of one sector
  solve    ``ed_solve`` over a sector list, then ``ed_calc_green_ftn``
  chi2     chi^2 and its gradient for a batch of bath parameter sets on the device
  delta    the k-summed hybridisation update of the self-consistency loop
  fit      conjugate-gradient bath fits

``listed`` names the sizes, ``draw`` makes more of the same ranges, ``prepare``
makes the inputs, ``run`` is one pass, ``work`` counts what the pass cannot do
without and ``exact`` is a plain 64-bit restatement in torch / numpy.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
from __graft_entry__ import load_package  # noqa: E402

_STREAM = None


def _stream():
    """The program's compute stream: the solver's kernels and torch share it."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _hv(name, dtype, norb, nbath, dense, nu, nd):
    return dict(name=name, kind="hv", dtype=dtype, norb=norb, nbath=nbath, dense=dense, nu=nu, nd=nd)


def listed():
    return [
        # one application of H on the half-filled ground sector of the largest model, 3 orbitals x 4 bath
        # levels: the FP32 eigensolver's and the FP32 Green's function's operator
        _hv("hv_f32_3x4_ground", "f32", 3, 12, False, 7, 8),
        # the same model in double precision, on the sector a hole excitation of the ground state lives in
        _hv("hv_f64_3x4_hole", "f64", 3, 12, False, 6, 8),
        # the middle-sized model, 3 orbitals x 3 bath levels, half filling
        _hv("hv_f32_3x3", "f32", 3, 9, False, 6, 6),
        # the reference's general input: every orbital couples to every level of one shared bath; FP32 vector in,
        # FP64 product out, as the Rayleigh quotients of an FP32 eigensolve take it
        _hv("hv_mixed_dense_2x11", "mixed", 2, 11, True, 6, 7),
        # the smallest call: the largest sector of the 2-orbital x 3-level model, bound by the launch
        _hv("hv_f64_2x3", "f64", 2, 6, False, 4, 4),
        # the Green's-function recurrence of one excitation with the default 50 continued-fraction steps, FP64
        dict(name="lanczos_f64_3x3", kind="lanczos", dtype="f64", norb=3, nbath=9, dense=False, nu=7, nd=6, nstep=50),
        # the lowest states of a large sector in the default FP32-mixed precision
        dict(name="diag_f32_3x4", kind="diag", dtype="f32", norb=3, nbath=12, dense=False, nu=5, nd=6, nev=6),
        # the lowest states of the middle-sized model's ground sector in FP64
        dict(name="diag_f64_3x3", kind="diag", dtype="f64", norb=3, nbath=9, dense=False, nu=6, nd=6, nev=6),
        # the impurity solver's whole call in one DMFT iteration: all 81 sectors of the 2-orbital x 3-level model,
        # then G(i w_n) on 2048 frequencies
        dict(name="solve_f32_2x3", kind="solve", dtype="f32", norb=2, nbath=6, nev=6, nw=2048, nstep=100),
        # chi^2 and gradient of 256 candidate baths of the 3-orbital x 4-level fit on 512 frequencies
        dict(name="chi2_256x512", kind="chi2", norb=3, nbath=12, dense=False, nw=512, nbatch=256),
        # the k-summed hybridisation of 3 orbitals on the large frequency grid with the default 10,000 k points
        dict(name="delta_4096x10000", kind="delta", norb=3, nw=4096, nk=100),
        # the bath fit of the single-band DMFT loop, from 8 starts
        dict(name="fit_1x4", kind="fit", norb=1, nbath=4, nw=1024, nbatch=8),
    ]


def _binom(n, k):
    return math.comb(n, k) if 0 <= k <= n else 0


def _dim(c):
    n = c["norb"] + c["nbath"]
    return _binom(n, c["nu"]) * _binom(n, c["nd"])


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_sector(rng, lo, hi):
    """A model and sector whose dimension is near a target drawn over [lo, hi] in its logarithm."""
    target = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    best = None
    for _ in range(400):
        norb = rng.choice([1, 2, 2, 3, 3, 3, 4])
        dense = rng.random() < 0.35
        nbath = rng.randint(2, 15 - norb) if dense else norb * rng.randint(1, (15 - norb) // norb)
        n = norb + nbath
        if n < 4:
            continue
        nu = n // 2 + rng.randint(-1, 1)
        nd = n // 2 + rng.randint(-2, 2)
        if not (1 <= nu < n and 1 <= nd < n):
            continue
        c = dict(norb=norb, nbath=nbath, dense=dense, nu=nu, nd=nd)
        d = _dim(c)
        if not (lo <= d <= hi):
            continue
        off = abs(math.log(d / target))
        if best is None or off < best[0]:
            best = (off, c)
        if off < 0.25:
            break
    return best[1]


def draw(rng):
    kind = rng.choice(["hv", "hv", "hv", "hv", "lanczos", "diag", "diag", "solve", "chi2", "delta", "fit"])
    if kind == "hv":
        dtype = rng.choice(["f32", "f32", "f64", "mixed"])
        hi = 41_409_225 if dtype == "f32" else 32_207_175
        return dict(kind=kind, dtype=dtype, **_draw_sector(rng, 1_000, hi))
    if kind == "lanczos":
        return dict(kind=kind, dtype="f64", nstep=rng.randint(20, 50), **_draw_sector(rng, 100_000, 2_000_000))
    if kind == "diag":
        dtype = rng.choice(["f32", "f64"])
        hi = 15_030_015 if dtype == "f32" else 1_500_000
        return dict(kind=kind, dtype=dtype, nev=rng.randint(2, 6), **_draw_sector(rng, 20_000, hi))
    if kind == "solve":
        norb, nbath = rng.choice([(1, 3), (1, 4), (1, 5), (2, 2), (2, 4), (2, 6)])
        return dict(kind=kind, dtype=rng.choice(["f32", "f64"]), norb=norb, nbath=nbath, nev=rng.randint(3, 8),
                    nw=_log_int(rng, 100, 2048), nstep=rng.randint(40, 100))
    if kind == "chi2":
        dense = rng.random() < 0.4
        norb = rng.randint(1, 3)
        nbath = rng.randint(1, 12 if norb < 3 else 10) if dense else norb * rng.randint(1, 4)
        return dict(kind=kind, norb=norb, nbath=nbath, dense=dense, nw=_log_int(rng, 64, 1024),
                    nbatch=_log_int(rng, 1, 256))
    if kind == "delta":
        return dict(kind=kind, norb=rng.randint(1, 3), nw=_log_int(rng, 64, 4096), nk=_log_int(rng, 8, 100))
    return dict(kind="fit", norb=1, nbath=rng.randint(3, 4), nw=_log_int(rng, 200, 1024), nbatch=rng.randint(1, 8))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _model(case, seed):
    """(U, J, ek, vk) of the case's impurity: bath energies in [-1, 1], couplings in [0.1, 0.5] (block-diagonal per
    orbital, or dense), impurity levels at particle-hole symmetry, as the benchmark configurations draw them."""
    norb, nbath = case["norb"], case["nbath"]
    rng = np.random.default_rng(7_000_003 + seed)
    U, J = (2.0, 0.0) if norb == 1 else (4.0, 1.0) if norb == 2 else (3.0, 0.5)
    eps = rng.uniform(-1.0, 1.0, nbath)
    vk = rng.uniform(0.1, 0.5, (norb, nbath))
    if not case.get("dense", False):
        per = nbath // norb
        vk *= np.kron(np.eye(norb), np.ones((1, per)))
    mu = 0.5 * (U + (norb - 1) * (2 * (U - 2 * J) - J))
    return U, J, np.concatenate([np.full(norb, -mu), eps]), vk


def _omega(nw, beta):
    return (2.0 * np.arange(nw) + 1.0) * np.pi / beta


def _start_vector(case, seed, dtype, device):
    g = torch.Generator(device=device)
    g.manual_seed(11 + seed)
    x = torch.randn(_binom(case["norb"] + case["nbath"], case["nd"]), _binom(case["norb"] + case["nbath"], case["nu"]),
                    generator=g, device=device, dtype=dtype)
    return x / x.norm()


def _bath_target(case, seed):
    """The hybridisation function of a hidden bath plus noise, and starting parameter sets near it."""
    norb, nbath, nw, nb = case["norb"], case["nbath"], case["nw"], case["nbatch"]
    rng = np.random.default_rng(400_009 + seed)
    mask = np.ones((norb, nbath)) if case.get("dense", False) else np.kron(np.eye(norb), np.ones((1, nbath // norb)))
    omega = _omega(nw, 200.0 if case["kind"] == "chi2" else 50.0)

    def params():
        return rng.uniform(-2.0, 2.0, nbath), rng.uniform(0.1, 0.6, (norb, nbath)) * mask, rng.uniform(-0.5, 0.5, norb)

    e, v, f = params()
    dev = (v[:, None, :] ** 2 / (1j * omega[None, :, None] - e)).sum(-1) + f[:, None]
    dev = dev + 1e-4 * (rng.standard_normal(dev.shape) + 1j * rng.standard_normal(dev.shape))
    X = np.zeros((nb, nbath + nbath * norb + norb))
    for b in range(nb):
        e, v, f = params()
        X[b] = np.concatenate([e, v.ravel(), f])
    return omega, dev, X


def _green_and_bath(case, seed):
    """A local Green's function and hybridisation as the loop has them between the solver and the k sum."""
    norb, nw = case["norb"], case["nw"]
    rng = np.random.default_rng(900_001 + seed)
    omega = _omega(nw, 200.0)
    e = rng.uniform(-1.0, 1.0, (norb, 4))
    v = rng.uniform(0.1, 0.5, (norb, 4))
    D = (v[:, None, :] ** 2 / (1j * omega[None, :, None] - e[:, None, :])).sum(-1)
    shift = rng.uniform(-0.3, 0.3, norb)[:, None]
    self_energy = 0.6 / (1j * omega[None, :] + rng.uniform(-0.5, 0.5, norb)[:, None])
    G = 1.0 / (1j * omega[None, :] + shift - D - self_energy)
    return G, D, float(rng.uniform(-0.2, 0.2))


class _State:
    pass


def prepare(case, seed):
    pkg = load_package()
    s = _State()
    s.case = case
    kind = case["kind"]
    st = _stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        s.solver = pkg.EDSolver(torch.cuda.current_device(), st.cuda_stream)
        if kind in ("hv", "lanczos", "diag", "solve"):
            U, J, ek, vk = _model(case, seed)
            prec = "fp32" if case["dtype"] == "f32" else "fp64"
            s.solver.set_options(precision=prec, nev=case.get("nev", 6), nstep=case.get("nstep", 50), beta=100.0)
            s.solver.set_model(case["norb"], case["nbath"], U, J, ek, vk)
        if kind == "hv":
            ld, _ = s.solver.vector_layout(case["nu"], case["nd"])
            tx = torch.float64 if case["dtype"] == "f64" else torch.float32
            ty = torch.float32 if case["dtype"] == "f32" else torch.float64
            x = _start_vector(case, seed, tx, "cuda")
            s.x = torch.zeros(x.shape[0], ld, dtype=tx, device="cuda")
            s.x[:, :x.shape[1]] = x
            s.y = torch.empty(x.shape[0], ld, dtype=ty, device="cuda")
            s.dtype = pkg.FP64 if case["dtype"] == "f64" else pkg.FP32
            if case["dtype"] == "mixed":   # the plan of the sector: its tables and tile shape
                s.solver.multiply_H_mixed_dev(case["nu"], case["nd"], s.x.data_ptr(), s.y.data_ptr())
            else:
                s.solver.hv_tuning(case["nu"], case["nd"], s.dtype)
        elif kind == "lanczos":
            s.x = _start_vector(case, seed, torch.float64, "cuda").cpu().numpy().ravel()
            s.solver.hv_tuning(case["nu"], case["nd"], pkg.FP64)
        elif kind == "diag":
            s.solver.hv_tuning(case["nu"], case["nd"], pkg.FP32 if case["dtype"] == "f32" else pkg.FP64)
        elif kind == "solve":
            n = case["norb"] + case["nbath"]
            s.solver.set_sectors([a + b for a in range(n + 1) for b in range(n + 1)],
                                 [a for a in range(n + 1) for b in range(n + 1)])
            s.solver.set_omega(_omega(case["nw"], 100.0))
        elif kind == "chi2":
            omega, dev, X = _bath_target(case, seed)
            s.X = torch.from_numpy(X).cuda()
            s.omega = torch.from_numpy(omega).cuda()
            s.dev = torch.from_numpy(np.ascontiguousarray(dev.T)).cuda()
            s.f = torch.empty(case["nbatch"], dtype=torch.float64, device="cuda")
            s.g = torch.empty(case["nbatch"], X.shape[1], dtype=torch.float64, device="cuda")
        elif kind == "delta":
            s.G, s.D, s.mu = _green_and_bath(case, seed)
            s.solver.set_model(case["norb"], 1, 1.0, 0.0, np.zeros(case["norb"] + 1), np.full((case["norb"], 1), 0.3))
            s.solver.set_band_structure(case["nk"] ** 2)
        elif kind == "fit":
            s.omega, s.dev, s.X = _bath_target(case, seed)
    torch.cuda.current_stream().wait_stream(st)
    return s


def run(s):
    c, e = s.case, s.solver
    kind = c["kind"]
    if kind == "hv":
        if c["dtype"] == "mixed":
            e.multiply_H_mixed_dev(c["nu"], c["nd"], s.x.data_ptr(), s.y.data_ptr())
        else:
            e.multiply_H_dev(c["nu"], c["nd"], s.x.data_ptr(), s.y.data_ptr(), s.dtype)
        return s.y
    if kind == "lanczos":
        return e.lanczos_iteration(c["nu"], c["nd"], s.x)
    if kind == "diag":
        return e.diag(c["nu"], c["nd"], c["nev"], vectors=False)[0]
    if kind == "solve":
        states = e.ed_solve()
        G = e.ed_calc_green_ftn()
        val, prob = np.zeros(c["nev"]), np.zeros(c["nev"])   # the states kept, in room for all
        for i, t in enumerate(states):
            val[i], prob[i] = t["val"], t["prob"]
        # an FP32 recurrence gives G to single precision: kept as such
        return val, prob, G.astype(np.complex64) if c["dtype"] == "f32" else G
    if kind == "chi2":
        e.chi2_grad_dev(c["nbatch"], s.X.data_ptr(), c["nw"], s.X.shape[1], s.omega.data_ptr(), s.dev.data_ptr(),
                        c["nbath"], c["norb"], s.f.data_ptr(), s.g.data_ptr())
        return s.f, s.g
    if kind == "delta":
        return e.delta_new(s.G, s.D, s.mu)
    return e.fit_batch(s.X, s.omega, s.dev, c["nbath"], c["norb"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _hv_flops(c):
    """2 per coupling term and element, 2 for the diagonal (4-operator terms are under one per element: left out)."""
    n = c["norb"] + c["nbath"]
    ncpl = c["norb"] * c["nbath"] if c.get("dense", False) else c["nbath"]
    up, dn = (2.0 * ncpl * _binom(n - 2, k - 1) / _binom(n, k) for k in (c["nu"], c["nd"]))
    return _dim(c) * 2.0 * (up + dn + 1.0)


def work(case):
    kind = case["kind"]
    if kind == "hv":
        b = {"f32": 8, "f64": 16, "mixed": 12}[case["dtype"]]
        return {"bytes": b * _dim(case), "flops": _hv_flops(case)}
    if kind == "lanczos":
        # per step: read the two last vectors, write the next; the product's terms and two dots
        d, n = _dim(case), case["nstep"]
        return {"bytes": 8.0 * d * (1 + 3 * n), "flops": n * (_hv_flops(case) + 8.0 * d)}
    if kind == "diag":
        # one Krylov space of 40 vectors: per step read the two last vectors, write the next (more steps are
        # needed; how many depends on the spectrum)
        d = _dim(case)
        return {"bytes": 40 * 3.0 * (4 if case["dtype"] == "f32" else 8) * d, "flops": 40 * (_hv_flops(case) + 8.0 * d)}
    if kind == "solve":
        # one Krylov space per sector, as above, and the continued fractions of one kept state
        n, es = case["norb"] + case["nbath"], 4 if case["dtype"] == "f32" else 8
        b = f = 0.0
        for nu in range(n + 1):
            for nd in range(n + 1):
                c = dict(case, nu=nu, nd=nd)
                if 0 < nu < n and 0 < nd < n:
                    k = min(40, _dim(c))
                    b += k * 3.0 * es * _dim(c)
                    f += k * (_hv_flops(c) + 8.0 * _dim(c))
        cf = case["norb"] * case["nw"] * 2.0 * case["nstep"]
        return {"bytes": b + 16.0 * case["norb"] * case["nw"], "flops": f + 12.0 * cf}
    if kind in ("chi2", "fit"):
        norb, nbath, nw, nb = case["norb"], case["nbath"], case["nw"], case["nbatch"]
        ncpl = norb * nbath if case.get("dense", False) else nbath
        nx = nbath + nbath * norb + norb
        # per frequency: the poles (8 per level), the residuals (4 per coupling), the gradients (16 per coupling)
        per = nw * (8.0 * nbath + 20.0 * ncpl + 10.0 * norb)
        # a fit: some 100 conjugate-gradient iterations of some 20 evaluations
        times = 1 if kind == "chi2" else 2000
        return {"bytes": 8.0 * (2 * nb * nx + nb + nw + 2 * norb * nw), "flops": nb * per * times}
    n = case["norb"] * case["nw"]
    # per k point and frequency: one difference, one squared modulus, one reciprocal, two sums
    return {"bytes": 64.0 * n + 8.0 * case["nk"] ** 2, "flops": 8.0 * n * case["nk"] ** 2}


# ---------------------------------------------------------------------------
# 64-bit restatement
# ---------------------------------------------------------------------------
class _H:
    """H on one sector in FP64: dense index arithmetic over the two spins' words, no code of this package."""

    def __init__(self, case, seed, device):
        U, J, ek, vk = _model(case, seed)
        norb, n = case["norb"], case["norb"] + case["nbath"]
        self.J = J
        side = []
        for ne in (case["nu"], case["nd"]):
            w = np.array([b for b in range(1 << n) if bin(b).count("1") == ne], dtype=np.int64)
            occ = (w[:, None] >> np.arange(n)) & 1
            rank = np.full(1 << n, -1, dtype=np.int64)
            rank[w] = np.arange(len(w))

            def transfer(dst, src):
                """(reachable, rank of c+_dst c_src w, sign); elsewhere the word itself with sign 0"""
                ok = (occ[:, src] == 1) & (occ[:, dst] == 0)
                w1 = w ^ (1 << src)
                par = self._parity(w, src) ^ self._parity(w1, dst)
                t = np.where(ok, rank[np.where(ok, w1 ^ (1 << dst), w)], np.arange(len(w)))
                return t, np.where(ok, 1.0 - 2.0 * par, 0.0)

            hops = []
            for o in range(norb):
                for k in range(norb, n):
                    v = vk[o, k - norb]
                    if v != 0.0:
                        (ta, sa), (tb, sb) = transfer(o, k), transfer(k, o)
                        hops.append((np.where(sa != 0, ta, tb), v * (sa + sb)))
            four = {(i, j): transfer(i, j) for i in range(norb) for j in range(norb) if i != j}
            imp = occ[:, :norb].astype(np.float64)
            cnt = imp.sum(1)
            diag = occ @ ek + (U - 3 * J) * 0.5 * cnt * (cnt - 1)

            def put(a):
                return torch.from_numpy(np.ascontiguousarray(a)).to(device)

            side.append(dict(diag=put(diag), imp=put(imp), hops=[(put(t), put(c)) for t, c in hops],
                             four={k: (put(t), put(c)) for k, (t, c) in four.items()}))
        self.up, self.dn = side
        m = np.full((norb, norb), U - 2 * J)
        np.fill_diagonal(m, U)
        self.cross = torch.from_numpy(m).to(device)

    @staticmethod
    def _parity(w, bit):
        p = w & ((1 << bit) - 1)
        for s in (8, 4, 2, 1):
            p = p ^ (p >> s)
        return p & 1

    def __call__(self, x):
        up, dn = self.up, self.dn
        y = (dn["imp"] @ self.cross @ up["imp"].T + up["diag"][None, :] + dn["diag"][:, None]) * x
        for t, c in up["hops"]:
            y.addcmul_(x.index_select(1, t), c[None, :].expand_as(x))
        for t, c in dn["hops"]:
            y.addcmul_(x.index_select(0, t), c[:, None].expand_as(x))
        for (i, j), (tu, cu) in up["four"].items():
            live_u = torch.nonzero(cu)[:, 0]
            for td, cd in (dn["four"][(j, i)], dn["four"][(i, j)]):   # spin flip, pair hopping
                live_d = torch.nonzero(cd)[:, 0]
                if len(live_u) and len(live_d):
                    g = x[td[live_d][:, None], tu[live_u][None, :]] * (self.J * cd[live_d][:, None] * cu[live_u][None, :])
                    y[live_d[:, None], live_u[None, :]] += g
        return y


def _lowest(h, shape, nev, device, most=400):
    """The nev lowest eigenvalues by a Lanczos run with full reorthogonalisation; None if not converged."""
    g = torch.Generator(device=device)
    g.manual_seed(3)
    d = shape[0] * shape[1]
    V = torch.empty(most + 1, d, dtype=torch.float64, device=device)
    v = torch.randn(d, generator=g, device=device, dtype=torch.float64)
    V[0] = v / v.norm()
    a, b = [], []
    for j in range(most):
        w = h(V[j].view(shape)).reshape(-1)
        a.append(float(w @ V[j]))
        for _ in range(2):
            w = w - V[: j + 1].T @ (V[: j + 1] @ w)
        b.append(float(w.norm()))
        V[j + 1] = w / b[-1]
        if j >= 40 and j % 10 == 0:
            T = np.diag(a) + np.diag(b[:-1], 1) + np.diag(b[:-1], -1)
            e, z = np.linalg.eigh(T)
            if np.all(b[-1] * np.abs(z[-1, :nev]) < 1e-7 * max(1.0, abs(e[0]))):
                return e[:nev]
    return None


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "hv":
        x = _start_vector(case, seed, torch.float64 if case["dtype"] == "f64" else torch.float32, dev).double()
        y = _H(case, seed, dev)(x)
        out = torch.zeros(y.shape[0], (y.shape[1] + 31) // 32 * 32, dtype=torch.float64, device=dev)   # row pads are zero
        out[:, :y.shape[1]] = y
        return out
    if kind == "lanczos":
        h = _H(case, seed, dev)
        v = _start_vector(case, seed, torch.float64, dev)
        n = case["nstep"]
        a, b = np.zeros(n + 1), np.zeros(n + 1)
        nrm, last = v.norm(), torch.zeros_like(v)
        v = v / nrm
        for j in range(n + 1):
            w = h(v)
            a[j] = float((w * v).sum())
            if j == n:
                break
            w = w - a[j] * v - math.sqrt(b[j]) * last
            b[j + 1] = float((w * w).sum())
            last, v = v, w / math.sqrt(b[j + 1])
        return None, a, b
    if kind == "diag":
        n = case["norb"] + case["nbath"]
        shape = (_binom(n, case["nd"]), _binom(n, case["nu"]))
        return _lowest(_H(case, seed, dev), shape, case["nev"], dev)
    if kind == "chi2":
        omega, D, X = _bath_target(case, seed)
        norb, nbath, nw = case["norb"], case["nbath"], case["nw"]
        w = torch.from_numpy(omega).to(dev)
        x = torch.from_numpy(X).to(dev)
        e, v, f = x[:, :nbath], x[:, nbath:nbath + norb * nbath].reshape(-1, norb, nbath), x[:, -norb:]
        z = 1.0 / (1j * w.float().double()[None, :, None] - e[:, None, :])         # the poles: CMPLX rounds w_n
        r = torch.einsum("bak,bnk->ban", (v * v).to(z.dtype), z) + f[:, :, None] - torch.from_numpy(D).to(dev)[None]
        chi = (r.abs() ** 2 / w).sum((1, 2)) / (norb * norb * nw)
        rw = r.conj() / w
        ge = torch.einsum("ban,bak,bnk->bk", rw, (v * v).to(z.dtype), z * z).real
        gv = 2 * torch.einsum("ban,bnk->bak", rw, z).real * v
        gf = rw.real.sum(2)
        return chi, 2.0 * torch.cat([ge, gv.reshape(len(x), -1), gf], 1) / (norb * norb * nw)
    if kind == "delta":
        G, D, mu = _green_and_bath(case, seed)
        q = 2.0 * math.pi / case["nk"] * torch.arange(case["nk"], dtype=torch.float64, device=dev)
        hk = (-0.5 * (torch.cos(q)[:, None] + torch.cos(q)[None, :])).reshape(-1)
        gi, d = 1.0 / torch.from_numpy(G).to(dev), torch.from_numpy(D).to(dev)
        base = (gi + d + mu).reshape(-1)
        ks = torch.cat([(1.0 / (p[:, None] - hk[None, :])).sum(1) for p in base.split(1024)]).view(d.shape) / len(hk)
        return gi - 1.0 / ks + d, ks
    # solve: 81 sectors' spectra and the excitations' fractions; fit: a trajectory of line searches, which ends
    # where its stop test first holds and not at a point that 64-bit arithmetic fixes
    return None
