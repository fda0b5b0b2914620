"""The host side of the eigensolver's Lanczos run (mo-dmft_gb300/csrc/kryhost.h)
on its own, without a GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "kryhost.h"
using namespace moed;
extern "C" {
// judges n reorthogonalisations one after the other; returns the last verdict
int judge(int f32, int n, const int *j, const int *gap, const double *c, int *period, int *good, double *hmax)
{
    KryPeriod p(f32 != 0, 1 << 20);
    int v = KryPeriod::kept;
    for (int i = 0; i < n && v == KryPeriod::kept; ++i) v = p.judge(KryClean{j[i], gap[i]}, c[i], false);
    *period = p.period;
    *good = p.good;
    *hmax = p.hmax;
    return v;
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("kryhost")
    src, so = d / "shim.cpp", d / "lib.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "mo-dmft_gb300", "csrc"),
                    "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))


def judge(lib, f32, rounds):
    n = len(rounds)
    j, gap = (C.c_int * n)(*[r[0] for r in rounds]), (C.c_int * n)(*[r[1] for r in rounds])
    c = (C.c_double * n)(*[r[2] for r in rounds])
    period, good, hmax = C.c_int(), C.c_int(), C.c_double()
    v = lib.judge(f32, n, j, gap, c, C.byref(period), C.byref(good), C.byref(hmax))
    return ("kept", "back", "lost")[v], period.value, good.value, hmax.value


@pytest.mark.parametrize("f32,little,much", [(1, 4e-7, 0.2), (0, 1e-15, 1e-3)])
def test_every_reorthogonalisation_counts(lib, f32, little, much):
    """Components that grew too large are found wherever they are among the
    reorthogonalisations of one read, not in the last of them alone."""
    fine = [(6, 6, little), (12, 6, little), (18, 6, little)]
    v, p0, good, hmax = judge(lib, f32, fine)
    assert v == "kept" and good == 18 and hmax == little
    v, p1, good, hmax = judge(lib, f32, fine[:2] + [(18, 6, 100 * little), (24, 6, little)])
    assert v == "kept" and good == 24 and hmax == 100 * little and p1 < p0
    v, p, good, _ = judge(lib, f32, fine + [(24, 6, much), (30, 6, little)])
    assert v == "back" and good == 18 and p == 3
    assert judge(lib, f32, fine + [(24, 6, np.nan)])[0] == "back"
    assert judge(lib, f32, fine + [(20, 2, much)])[0] == "lost"
    assert judge(lib, f32, [(6, 6, much)])[0] == "lost"
    assert judge(lib, f32, [(6, 6, 0.0)])[0] == "kept"
