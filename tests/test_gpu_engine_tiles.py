"""The batch engine's tiles at the sizes where they can go wrong: edges of its
32 x 8 tiles, rows of every alignment (nodes of a row are read one, two or four
at a time), odd y (two rows to a thread), more groups of threads than tiles, and
phases too far apart for the fixed-point stencil's table."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as e3d
import oracle as O
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# At |z.g| <= 1e-9 |z0.g0| the energy is off by about 1e-18 of the first change and
# the stress by 1e-9 of its scale; the oracle's iterate, in 64 bits and other
# orders, stops within as much of the solution.  Two decades for both.
ENERGY_TOL = 1e-8
STRESS_TOL = 1e-7


@pytest.mark.parametrize("shape,parts,e1", [((31, 7, 9), 1, 0.0), ((32, 8, 16), 3, 0.0), ((33, 9, 17), 5, 0.0),
                                            ((34, 15, 6), 2, 0.0), ((36, 16, 5), 40, 0.0), ((65, 17, 3), 7, 0.0),
                                            ((30, 11, 21), 4, 9e12)])
def test_tile_edges(shape, parts, e1):
    rve = W.rve(0, 5, 60 + parts, A=2.5, shape=shape, pore_frac=0.02)
    nu1 = 0.3 if e1 else 0.0
    with e3d.Batch([rve], criterion=e3d.CRIT_PRECOND_REL, tol=1e-9, parts=parts, load_cases=0b010001, e1=e1,
                   nu1=nu1) as b:
        b.solve()
        res = b.results()
    assert [r["load_case"] for r in res] == [0, 4] and {r["parts"] for r in res} == {parts}
    nx, ny, nz = shape
    for r in res:
        assert r["status"] == e3d.EXIT_CONVERGED, r
        s = [0.0] * 6
        s[r["load_case"]] = 1e-3 if r["load_case"] < 3 else 0.5e-3
        p = O.Problem(nx, ny, nz, rve["ngrains"] + 1, c11=rve["c11"], c12=rve["c12"], c44=rve["c44"], exx=s[0],
                      eyy=s[1], ezz=s[2], exz=s[3], eyz=s[4], exy=s[5], tol=1e-9, criterion=1, e1=e1, nu1=nu1)
        ref = O.run(p, rve["pix"], rve["rodrigues"])
        assert ref["exit_reason"] == 0
        assert abs(r["utot0"] - ref["utot0"]) <= 1e-12 * abs(ref["utot0"])
        assert abs(r["utot"] - ref["utot"]) <= ENERGY_TOL * abs(ref["utot"])
        assert np.linalg.norm(r["strav"] - ref["strav"]) <= STRESS_TOL * np.linalg.norm(ref["strav"])
