"""The batch engine's FP64 residual where tiles read displacements of very different
size: the lowest chunk of a long RVE under zz strain has the top plane below it."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as e3d
import oracle as O
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# As in the test of the engine's tile edges: two decades above what a solution at this
# tolerance may be off by.
ENERGY_TOL = 1e-8
STRESS_TOL = 1e-7


# chunks of two planes of 200 (one tile in a hundred uneven), of all planes (none), and
# tiles of partly filled rows
@pytest.mark.parametrize("shape,parts", [((20, 12, 200), 152), ((20, 12, 200), 1), ((5, 3, 150), 100), ((33, 6, 90), 152)])
def test_long_rve(shape, parts):
    rve = W.rve(0, 5, 60 + parts, A=2.5, shape=shape, pore_frac=0.02)
    with e3d.Batch([rve], criterion=e3d.CRIT_PRECOND_REL, tol=1e-9, parts=parts, load_cases=0b000100) as b:
        b.solve()
        r = b.results()[0]
    p = O.Problem(*shape, rve["ngrains"] + 1, c11=rve["c11"], c12=rve["c12"], c44=rve["c44"], exx=0.0, eyy=0.0, ezz=1e-3,
                  exz=0.0, eyz=0.0, exy=0.0, tol=1e-9, criterion=1)
    ref = O.run(p, rve["pix"], rve["rodrigues"])
    assert r["status"] == e3d.EXIT_CONVERGED and ref["exit_reason"] == 0
    assert r["refinements"] > 0
    assert abs(r["utot"] - ref["utot"]) <= ENERGY_TOL * abs(ref["utot"])
    assert np.linalg.norm(r["strav"] - ref["strav"]) <= STRESS_TOL * np.linalg.norm(ref["strav"])
