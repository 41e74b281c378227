"""Volume averages where one component of the displacement is much larger than the others,
and with phases that no voxel has."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as E
import oracle as O
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu
MATERIAL = dict(c11=240e9, c12=150e9, c44=90e9)
# The oracle adds the voxels in 64 bits: at most ns * 1.1e-16 of the largest voxel.
TOL = 1e-11


@pytest.mark.parametrize("shape", [(33, 5, 17), (64, 8, 33), (1, 3, 2)])
@pytest.mark.parametrize("component", range(3))
@pytest.mark.parametrize("size", [2.0 ** 40, 2.0 ** -40])
def test_offset(shape, component, size):
    ng = 6
    pix, rod = E.micro_grains(*shape, ng, 5)
    zero = dict(exx=0.0, eyy=0.0, ezz=0.0, exz=0.0, eyz=0.0, exy=0.0)
    o = O.Oracle(O.Problem(*shape, ng + 1, **zero, **MATERIAL), pix, rod).femat()
    u = W.random_field(pix.size, 11).reshape(3, -1)
    u *= size if size < 1 else 1.0
    u[component] = 0.0  # the oracle adds values, not differences: it would round the constant's
    s_ref, e_ref = o.stress(u.ravel())
    u[component] = 1.0 if size < 1 else size
    with E.Elas3D(E.Problem(*shape, ng + 1, strain=(0.0,) * 6, **MATERIAL)) as g:
        g.upload(pix, rod).femat().set_u(u.ravel())
        s, e = g.stress()
    peak = 4 * np.abs(np.delete(u, component, 0)).max()  # of a voxel's strain
    assert np.abs(e - e_ref).max() <= TOL * peak
    assert np.abs(s - s_ref).max() <= TOL * peak * 3 * 240e9


def test_phase_without_voxels():
    shape, ng = (20, 9, 7), 5
    pix, rod = E.micro_grains(*shape, ng, 5)
    pix[pix == 3] = 2
    rod = np.array(rod, dtype=np.float64)
    u = W.random_field(pix.size, 12)
    got = []
    for r in (0.25, np.inf):
        rod.reshape(-1, 3)[2] = r  # of the phase that is not there
        with E.Elas3D(E.Problem(*shape, ng + 1, strain=(1e-3, 0, 0, 0, 0, 0), **MATERIAL)) as g:
            g.upload(pix, rod).femat().set_u(u)
            got.append(np.concatenate(g.stress()))
    assert np.isfinite(got[1]).all()
    assert np.array_equal(*got)
