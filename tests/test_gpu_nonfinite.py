"""Material data that is not finite: it has to show in what depends on it, and only there."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as E
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu
MATERIAL = dict(c11=240e9, c12=150e9, c44=90e9)


def _nodes_of(pix, shape, phase):
    """Nodes with an element of the phase around them (an element's corners are its node and the next ones)."""
    nx, ny, nz = shape
    e = (pix == phase).reshape(nz, ny, nx)
    for axis in range(3):
        e = e | np.roll(e, 1, axis)
    return np.broadcast_to(e.ravel(), (3, e.size)).ravel()


@pytest.mark.parametrize("ngrains", [3, 40, 120])  # fewer phases than the table's reduction has threads, and more
@pytest.mark.parametrize("bad", [1e200, np.inf])  # its square overflows (a NaN gives the identity, as in the reference)
@pytest.mark.parametrize("where", ["first", "middle", "last"])
def test_orientation(ngrains, bad, where):
    shape = (36, 9, 14)
    pix, rod = E.micro_grains(*shape, ngrains, 5)
    g = {"first": 0, "middle": ngrains // 2, "last": ngrains - 1}[where]
    pix[17] = g + 1  # it has a voxel at least
    p = E.Problem(*shape, ngrains + 1, strain=(1e-3, 0, 0, 0, 0, 0), **MATERIAL)
    x = W.random_field(p.ns, 3)
    with E.Elas3D(p) as s:
        clean = s.upload(pix, rod).femat().apply(x)
        rod = np.array(rod, dtype=np.float64)
        rod.reshape(-1, 3)[g, 1] = bad
        y = s.upload(pix, rod).femat().apply(x)
        u, gg = s.init_affine().energy()
    hit = _nodes_of(pix, shape, g + 1)
    assert not np.isfinite(y[hit]).any()
    # two orders of summation of the same products (a node has 192 of them)
    assert np.linalg.norm((y - clean)[~hit]) <= 1e-12 * np.linalg.norm(clean)
    assert np.isnan(u) and np.isnan(gg)


def test_inclusion():
    shape, ngrains = (20, 9, 7), 4
    pix, rod = E.micro_grains(*shape, ngrains, 5)
    pix[400:403] = ngrains + 1
    x = W.random_field(pix.size, 3)
    y = []
    for e1 in (1e11, np.nan):
        with E.Elas3D(E.Problem(*shape, ngrains + 1, e1=e1, nu1=0.3, **MATERIAL)) as s:
            y.append(s.upload(pix, rod).femat().apply(x))
    hit = _nodes_of(pix, shape, ngrains + 1)
    assert not np.isfinite(y[1][hit]).any()
    assert np.linalg.norm((y[1] - y[0])[~hit]) <= 1e-12 * np.linalg.norm(y[0])


@pytest.mark.parametrize("component", range(6))
def test_strain(component):
    pix, rod = E.micro_grains(20, 9, 7, 4, 5)
    strain = [1e-3] * 6
    strain[component] = np.nan
    p = E.Problem(20, 9, 7, 5, strain=tuple(strain), **MATERIAL)
    with E.Elas3D(p) as s:
        s.upload(pix, rod).femat().set_u(W.random_field(p.ns, 4))
        sig, eps = s.stress()
    assert np.isnan(eps[component])
    assert np.isnan(sig).all()
