"""Volume averages of stress and strain at the edges of their 32 x 4 tiles, on grids
one and two nodes thick, with every jump, one phase and many, and at values inside,
beyond and off the range of the fixed-point sums."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as E
import oracle as O
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# The oracle adds the voxels in 64 bits: at most ns * 1.1e-16 of the largest voxel,
# 5e-12 for the largest grid here.
TOL = 1e-11
STRAIN = (1e-3, -2e-3, 5e-4, 7e-4, -3e-4, 4e-4)


def _case(shape, ngrains, strain):
    nx, ny, nz = shape
    pix, rod = E.micro_grains(nx, ny, nz, ngrains, 5)
    pix[:: 7 * 13] = ngrains + 1
    k = dict(c11=240e9, c12=150e9, c44=90e9)
    p = E.Problem(nx, ny, nz, ngrains + 1, strain=strain, **k)
    exx, eyy, ezz, exz, eyz, exy = strain
    o = O.Oracle(O.Problem(nx, ny, nz, ngrains + 1, exx=exx, eyy=eyy, ezz=ezz, exz=exz, eyz=eyz, exy=exy, **k), pix, rod)
    return p, pix, rod, o.femat()


@pytest.mark.parametrize("shape,ngrains", [((1, 1, 1), 1), ((1, 3, 2), 2), ((2, 1, 3), 1), ((31, 3, 5), 4), ((32, 4, 16), 40),
                                           ((33, 5, 17), 300), ((64, 8, 33), 1), ((65, 9, 2), 5), ((7, 13, 40), 9)])
def test_tile_edges(shape, ngrains):
    p, pix, rod, o = _case(shape, ngrains, STRAIN)
    u = o.affine_u() + 1e-3 * W.random_field(p.ns, 11)
    with E.Elas3D(p) as g:
        g.upload(pix, rod).femat().set_u(u)
        s, e = g.stress()
    s_ref, e_ref = o.stress(u)
    peak = 4 * np.abs(u).max() + np.abs(STRAIN).max() * max(shape)  # of a voxel's strain
    assert np.abs(e - e_ref).max() <= TOL * peak
    assert np.abs(s - s_ref).max() <= TOL * peak * 3 * 240e9


def test_range():
    """A power of two commutes with the sums: inside the range exactly, and beyond it
    in the FP64 form; what is not finite stays so."""
    p, pix, rod, o = _case((33, 5, 17), 6, (0.0,) * 6)
    u = W.random_field(p.ns, 12)
    with E.Elas3D(p) as g:
        g.upload(pix, rod).femat()
        get = lambda k: (g.set_u(np.ldexp(u, k)), g.stress())[1]
        s, e = get(0)
        for k in (-380, -60, 60, 300):
            sk, ek = get(k)
            assert np.array_equal(sk, np.ldexp(s, k)) and np.array_equal(ek, np.ldexp(e, k)), k
        for k in (-480, 480):
            sk, ek = get(k)
            assert np.abs(np.ldexp(sk, -k) - s).max() <= TOL * 4 * np.abs(u).max() * 3 * 240e9, k
            assert np.abs(np.ldexp(ek, -k) - e).max() <= TOL * 4 * np.abs(u).max(), k
        g.set_u(np.zeros(3 * p.ns))
        assert not np.any(g.stress()[0])
        u[5] = np.nan
        g.set_u(u)
        assert np.isnan(g.stress()[0]).any()
