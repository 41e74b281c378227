"""Which materials keep the FP64 form of the stencil.  On a grid of one tile it agrees
bit for bit with e3d_apply_noalloc, which has no other; the fixed-point form rounds
differently."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import elas3d_xtal_gb300 as e3d
from elas3d_xtal_gb300 import workloads as W

CSRC = os.path.join(os.path.dirname(os.path.abspath(e3d.__file__)), "csrc")


def test_condition(tmp_path):
    (tmp_path / "m.cpp").write_text("""
#include "e3d_material.h"
extern "C" int iso(double k, double g) { return e3d::semidefinite(k, g); }
extern "C" int cubic(double a, double b, double c) { return e3d::semidefinite_cubic(a, b, c); }
""")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(tmp_path / "m.cpp"), "-o",
                    str(tmp_path / "m.so")], check=True)
    lib = C.CDLL(str(tmp_path / "m.so"))
    lib.iso.argtypes, lib.cubic.argtypes = [C.c_double] * 2, [C.c_double] * 3
    rng = np.random.default_rng(1)
    for c11, c12, c44 in rng.uniform(-1, 1, (200, 3)):
        m = np.diag([c44] * 6) * 1.0
        m[:3, :3] = c12
        m[:3, :3] += np.eye(3) * (c11 - c12)
        assert bool(lib.cubic(c11, c12, c44)) == (np.linalg.eigvalsh(m).min() >= 0)
    for k, g in rng.uniform(-1, 1, (50, 2)):
        assert bool(lib.iso(k, g)) == (min(k, g) >= 0)
    assert lib.iso(0, 0) and lib.cubic(0, 0, 0)
    nan = float("nan")
    assert not (lib.iso(nan, 1) or lib.iso(1, nan) or lib.cubic(nan, 0, 1) or lib.cubic(1, nan, 1) or lib.cubic(1, 0, nan))


@pytest.mark.gpu
@pytest.mark.parametrize("c,fixed", [((240e9, 150e9, 90e9), True), ((240e9, -100e9, 90e9), True),
                                     ((240e9, 150e9, -1e9), False), ((100e9, 150e9, 90e9), False),
                                     ((100e9, -60e9, 90e9), False)],
                         ids=["steel", "auxetic", "c44", "c11-c12", "c11+2c12"])
def test_form(c, fixed):
    torch = pytest.importorskip("torch")
    ng = 4
    pix, rod = e3d.micro_grains(20, 6, 5, ng, 5)
    p = e3d.Problem(20, 6, 5, ng + 1, c11=c[0], c12=c[1], c44=c[2])
    x = W.random_field(p.ns, seed=1)
    with e3d.Elas3D(p) as g:
        y = g.upload(pix, rod).femat().apply(x)
        cmod = np.empty(36 * p.nphase)
        assert g.L.e3d_get_cmod(g.handle, e3d._dp(cmod)) == e3d.E3D_OK
        d = [torch.from_numpy(a).cuda() for a in (pix, cmod, x, np.zeros_like(x))]
        torch.cuda.synchronize()
        assert g.L.e3d_apply_noalloc(p.nx, p.ny, p.nz, p.nphase, *(C.c_void_p(t.data_ptr()) for t in d), None) == e3d.E3D_OK
    assert np.array_equal(d[3].cpu().numpy(), y) != fixed
