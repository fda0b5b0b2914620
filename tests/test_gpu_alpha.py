"""alpha_0 = x . H x of an FP32 recurrence with the shapes of k_hv_wide: the shares
of a long row are added in FP64 after every unit of 64 columns.  H is the
identity here (energies that add up to one, couplings of 1e-30) and x is 1 in
the first 1,024 columns, 16 units, and 2^-13 in the others, whose squares vanish
in an FP32 sum that has reached 4 but not in one of their own: alpha_0 is 1 up
to FP64 roundings (below 1e-12), while shares that run over the row in FP32
miss some 1e-9."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_shares_in_fp64(solver, pkg):
    norb, nbath, nu, nd = 1, 12, 6, 2
    solver.set_options(precision="fp32", nstep=1)
    seen = 0
    try:
        solver.set_model(norb, nbath, 0.0, 0.0, np.full(13, 0.125), np.full((1, 12), 1e-30))
        x = np.full((math.comb(13, nd), math.comb(13, nu)), 2.0 ** -13)
        x[:, :1024] = 1.0
        shapes, _ = solver.hv_tuning(nu, nd, pkg.FP32)
        for v, (shape, _) in enumerate(shapes):
            if shape[0] != 8 and shape[:3] != (4, 512, 2):
                continue
            solver.hv_set_variant(nu, nd, v, pkg.FP32)
            seen += 1
            assert np.array_equal(solver.multiply_H(nu, nd, x.astype(np.float32).ravel()), x.astype(np.float32).ravel())
            _, a, _ = solver.lanczos_iteration(nu, nd, x.ravel())
            assert abs(a[0] - 1.0) < 1e-12, (v, shape, a[0] - 1.0)
        assert seen == 3
    finally:
        solver.set_options(nstep=50)
