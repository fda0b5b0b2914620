"""What a context keeps between calls is there for the rest of the process: after
an eigensolve with 20 GB of Krylov vectors, all of the device's free memory but
a few GB can be allocated by something else, and the context still works."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_workspace_is_given_back(pkg):
    import torch

    torch.zeros(1, device="cuda")
    rt = C.CDLL("libcudart.so")
    norb, nbath = 3, 12
    rng = np.random.default_rng(0)
    ek = np.concatenate([np.full(norb, -3.75), rng.uniform(-1, 1, nbath)])
    vk = rng.uniform(0.1, 0.5, (norb, nbath)) * np.kron(np.eye(norb), np.ones((1, nbath // norb)))
    s = pkg.EDSolver(0)
    try:
        s.set_options(precision="fp32", nev=6)
        s.set_model(norb, nbath, 3.0, 0.5, ek, vk)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        first, _ = s.diag(5, 6, 6, vectors=False)
        size = free - (6 << 30)     # other workspaces stay: 4 GB at most
        p = C.c_void_p()
        rc = rt.cudaMalloc(C.byref(p), C.c_size_t(size))
        rt.cudaGetLastError()
        assert rc == 0, f"{size >> 30} of {free >> 30} GB that were free before the solve"
        # with what is left, the solve still runs
        again, _ = s.diag(3, 4, 6, vectors=False)
        assert np.isfinite(again).all()
        assert rt.cudaFree(p) == 0
        assert np.abs(s.diag(5, 6, 6, vectors=False)[0] - first).max() < 1e-8
    finally:
        s.close()
