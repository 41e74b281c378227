"""Block-Jacobi inverses where the blocks of the kernel end, with one grain (every
node takes its phase's inverse), with grains of a few nodes (hardly one does), and
from the size on where a block serves four times as many nodes."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as E
import oracle as O

pytestmark = pytest.mark.gpu

# the same 73 operations a node as the oracle's, on blocks of condition below 1e2
TOL = 1e-12


@pytest.mark.parametrize("shape,ngrains", [((1, 1, 1), 1), ((1, 3, 2), 2), ((255, 1, 1), 3), ((16, 16, 1), 1), ((257, 1, 1), 40),
                                           ((9, 10, 11), 300), ((128, 98, 100), 60), ((109, 108, 107), 1)])
def test_inverse(shape, ngrains):
    nx, ny, nz = shape
    pix, rod = E.micro_grains(nx, ny, nz, ngrains, 7)
    pix[:: 7 * 13] = ngrains + 1
    p = E.Problem(nx, ny, nz, ngrains + 1, c11=240e9, c12=150e9, c44=90e9, strain=(1e-3, 0, 0, 0, 0, 0))
    with E.Elas3D(p) as g:
        g.upload(pix, rod).femat().init_affine()
        g.energy()
        g.solve_begin()
        minv = np.asarray(g.get_minv())
    o = O.Oracle(O.Problem(nx, ny, nz, ngrains + 1, c11=p.c11, c12=p.c12, c44=p.c44), pix, rod)
    ref = o.femat().block_jacobi().reshape(3, 3, p.ns).transpose(2, 1, 0)
    assert np.abs(minv.ravel() - ref.ravel()).max() <= TOL * np.abs(ref).max()
