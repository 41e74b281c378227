"""Vectors whose values differ by many powers of two from place to place: entry by entry,
K.x is as exact as the values around the entry, not as the largest of the grid."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as E
import oracle as O
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# 192 products a node, each rounded at 1.1e-16 of sum |K||x| over the 27 nodes around it,
# in each of two codes.  D, the largest row sum of |K|, is eight elements' of |k|.
TOL = 2 * 192 * 1.1e-16
MATERIAL = dict(c11=240e9, c12=150e9, c44=90e9)


def _case(shape, ngrains=5):
    pix, rod = E.micro_grains(*shape, ngrains, 3)
    pix[:: 7 * 13] = ngrains + 1
    p = E.Problem(*shape, ngrains + 1, strain=(0.0,) * 6, **MATERIAL)
    o = O.Oracle(O.Problem(*shape, ngrains + 1, exx=0.0, eyy=0.0, ezz=0.0, exz=0.0, eyz=0.0, exy=0.0, **MATERIAL), pix,
                 rod).femat()
    return p, pix, rod, o


def _row_sum(o):
    return 8 * np.abs(o.dk_array().reshape(-1, 24, 24)).sum(2).max()


def _around(x, shape):
    """Largest |value| of the 27 nodes around each node, of all components."""
    m = np.abs(x).reshape(3, *shape[::-1]).max(0)
    for axis in range(3):
        m = np.max([np.roll(m, s, axis) for s in (-1, 0, 1)], 0)
    return m


@pytest.mark.parametrize("shape", [(40, 12, 40), (33, 5, 17), (64, 8, 33), (7, 4, 70), (96, 2, 5)])
@pytest.mark.parametrize("pattern", ["entry", "plane", "far", "denormal"])
def test_apply(shape, pattern):
    p, pix, rod, o = _case(shape)
    nx, ny, nz = shape
    x = 1e-9 * W.random_field(p.ns, 7)
    v = x.reshape(3, nz, ny, nx)
    if pattern == "entry":
        v[1, nz // 2, ny // 2, nx // 2] = 1.0
    elif pattern == "plane":  # every row of every tile along x and y has values of both sizes
        v[:, nz // 2] *= 1e9
    elif pattern == "far":
        v *= 2.0 ** -np.arange(nx)[None, None, None, :] * 2.0 ** (-3.0 * np.arange(nz)[None, :, None, None])
    else:
        v *= 2.0 ** -1030
    with E.Elas3D(p) as g:
        y = g.upload(pix, rod).femat().apply(x).reshape(v.shape)
    ref = o.apply(x).reshape(v.shape)
    limit = TOL * _row_sum(o) * _around(x, shape) + 64 * 5e-324
    assert np.abs(ref).max() > 0
    assert (np.abs(y - ref) <= limit).all()


def test_offset():
    """A constant in one component adds nothing to K.x, and takes nothing from the others."""
    shape = (40, 12, 40)
    p, pix, rod, o = _case(shape)
    x = W.random_field(p.ns, 8).reshape(3, -1)
    x[1] = 0.0
    ref = o.apply(x).reshape(3, -1)
    limit = TOL * _row_sum(o) * np.abs(x).max()
    x[1] = 2.0 ** 40
    with E.Elas3D(p) as g:
        y = g.upload(pix, rod).femat().apply(x.ravel()).reshape(3, -1)
    assert np.abs(y - ref).max() <= limit


@pytest.mark.parametrize("shape", [(40, 12, 40), (33, 5, 17), (65, 9, 30)])
def test_solve_steps(shape):
    """The residual after one and after ten iterations from a start field of one large
    value among small ones: small where it was small, to the accuracy of the values there."""
    p, pix, rod, o = _case(shape)
    nx, ny, nz = shape
    u = 1e-9 * W.random_field(p.ns, 7)
    at = (nz // 2, ny // 2, nx // 2)
    u.reshape(3, nz, ny, nx)[(0, *at)] = 1.0
    g0, _ = o.energy(u)
    far = np.ones((nz, ny, nx), bool)  # three nodes off: two of K and one of the preconditioner's element
    near = [np.arange(c - 3, c + 4) % n for c, n in zip(at, (nz, ny, nx))]
    far[np.ix_(*near)] = False
    s = o.pcg(u, g0, float(g0 @ g0))
    with E.Elas3D(p) as e:
        e.upload(pix, rod).femat().set_u(u)
        e.energy()
        e.solve_begin()
        s.iterate(1)
        e.iterate(1)
        r, ref = e.get_g().reshape(3, nz, ny, nx), s.g.reshape(3, nz, ny, nx)
        # the step length comes from sums over the grid in another order
        limit = TOL * _row_sum(o) * 1e-9 * np.abs(W.random_field(p.ns, 7)).max() * 4
        assert far.any()
        assert np.abs(r - ref)[:, far].max() <= limit
        s.iterate(9)
        e.iterate(9)
        assert np.linalg.norm(e.get_g() - s.g) <= 1e-9 * np.linalg.norm(s.g)
    s.close()


def test_split_iterations_and_checkpoint(tmp_path):
    """The forms for even and uneven directions take over from each other at the same
    iterations, in whatever steps the caller goes and across a checkpoint."""
    shape = (40, 12, 40)
    p, pix, rod, o = _case(shape)
    u = 1e-9 * W.random_field(p.ns, 7)
    u[5000] = 1.0

    def start(e):
        e.upload(pix, rod).femat().set_u(u)
        e.energy()
        e.solve_begin()
        return e

    with E.Elas3D(p) as a, E.Elas3D(p) as b, E.Elas3D(p) as c:
        start(a).iterate(30)
        start(b)
        for n in (1, 2, 4, 1):
            b.iterate(n)
        b.checkpoint_save(str(tmp_path / "c"))
        b.iterate(22)
        c.upload(pix, rod).femat().checkpoint_load(str(tmp_path / "c"))
        c.iterate(22)
        assert np.array_equal(a.get_u(), b.get_u())
        assert np.array_equal(a.get_u(), c.get_u())
