"""The fixed-point form of the FP64 stencil (csrc/e3d_fixed.cuh) at the sizes
and values where it can go wrong: edges of its 32 x 4 tiles, grids one and two
nodes thick, the range of its exponents, values that are not finite, phases too
different for one table exponent."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as E
import oracle as O
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# K.x of two FP64 codes that sum in different orders: 192 products a node, each
# rounded at 1.1e-16, give at most 2.1e-14 of sum |K||x|, which is within 50 of
# |K x| for random x
TOL = 1e-12


def _problem(shape, ngrains=5, seed=3, e1=0.0, nu1=0.0, pores=True):
    nx, ny, nz = shape
    pix, rod = E.micro_grains(nx, ny, nz, ngrains, seed)
    if pores:
        pix[:: 7 * 13] = ngrains + 1
    p = E.Problem(nx, ny, nz, ngrains + 1, c11=240e9, c12=150e9, c44=90e9, e1=e1, nu1=nu1, strain=(1e-3, 0, 0, 0, 0, 0))
    return p, pix, rod


def _oracle_apply(p, pix, rod, x):
    op = O.Problem(p.nx, p.ny, p.nz, p.nphase, flag_m=p.flag_m, c11=p.c11, c12=p.c12, c44=p.c44, e1=p.e1, nu1=p.nu1)
    return O.Oracle(op, pix, rod).femat().apply(x)


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("shape", [(1, 3, 2), (2, 1, 3), (3, 4, 1), (31, 3, 5), (32, 4, 16), (33, 5, 17), (64, 8, 33),
                                   (65, 9, 2), (7, 13, 40)])
def test_tile_edges(shape):
    p, pix, rod = _problem(shape)
    x = W.random_field(p.ns, 11)
    with E.Elas3D(p) as g:
        g.upload(pix, rod).femat()
        y = g.apply(x)
    assert _rel(y, _oracle_apply(p, pix, rod, x)) < TOL


def test_exponent_range_and_zero():
    """A power of two commutes with K exactly, inside the fixed-point range and,
    in the FP64 form, beyond it; zero gives zero."""
    p, pix, rod = _problem((35, 6, 9))
    x = W.random_field(p.ns, 12)
    with E.Elas3D(p) as g:
        g.upload(pix, rod).femat()
        y = g.apply(x)
        for k in (-380, -60, 60, 300):
            assert np.array_equal(g.apply(np.ldexp(x, k)), np.ldexp(y, k)), k
        for k in (-480, 480):
            assert _rel(np.ldexp(g.apply(np.ldexp(x, k)), -k), y) < TOL, k
        assert not g.apply(np.zeros_like(x)).any()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_not_finite_stay_where_they_are(bad):
    p, pix, rod = _problem((40, 10, 24), pores=False)
    x = W.random_field(p.ns, 13)
    with E.Elas3D(p) as g:
        g.upload(pix, rod).femat()
        clean = g.apply(x)
        x[5 + 40 * (4 + 10 * 7)] = bad
        y = g.apply(x).reshape(3, 24, 10, 40)
    hit = np.zeros(y.shape, bool)
    hit[:, 6:9, 3:6, 4:7] = True
    assert not np.isfinite(y[hit]).any()
    assert _rel(y[~hit], clean.reshape(y.shape)[~hit]) < TOL


@pytest.mark.parametrize("e1", [2.0e9, 70.0e9, 3.0e14])
def test_stiffness_contrast(e1):
    """An inclusion within the contrast of one table exponent and two beyond it
    (the FP64 form)."""
    p, pix, rod = _problem((37, 7, 12), e1=e1, nu1=0.3)
    x = W.random_field(p.ns, 14)
    with E.Elas3D(p) as g:
        g.upload(pix, rod).femat()
        y = g.apply(x)
    assert _rel(y, _oracle_apply(p, pix, rod, x)) < TOL


def test_solve_leaves_the_range():
    """Directions beyond the fixed-point range: the solve goes on in the FP64
    form, through the same iterations."""
    p, pix, rod = _problem((24, 18, 16))
    with E.Elas3D(p) as g:
        g.upload(pix, rod)
        ref = g.run()
    s = 2.0 ** 440
    p.strain = tuple(v * s for v in p.strain)
    with E.Elas3D(p) as g:
        g.upload(pix, rod)
        big = g.run()
    assert big["exit_reason"] == ref["exit_reason"] == E.EXIT_CONVERGED
    assert abs(big["iterations"] - ref["iterations"]) <= 2
    assert abs(big["utot"] / s / s - ref["utot"]) <= 1e-9 * abs(ref["utot"])
