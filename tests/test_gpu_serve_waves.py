"""Serving rounds of whole waves: requests that together ask for more blocks than
the device has take turns, and each result is bit for bit the one it has alone."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as e3d
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# 152 blocks: two waves and a rest, one wave and a rest of one request, exactly one wave
@pytest.mark.parametrize("count,parts", [(9, 40), (8, 20), (8, 19)])
def test_same_results_as_alone(count, parts):
    rng = np.random.default_rng(count)
    reqs = [(W.rve(int(rng.integers(10, 20)), 5, 40 + i, A=2.0, pore_frac=0.01), rng.normal(size=6) * 1e-3)
            for i in range(count)]
    with e3d.Server(round_iters=7, parts=parts) as srv:
        ids = [srv.submit(*r) for r in reqs]
        while srv.step():
            pass
        together = [srv.result(i) for i in ids]
    for req, r in zip(reqs, together):
        with e3d.Server(round_iters=7, parts=parts) as srv:
            i = srv.submit(*req)
            while srv.step():
                pass
            a = srv.result(i)
        assert r["status"] == a["status"] == e3d.EXIT_CONVERGED
        assert (r["iterations"], r["parts"], r["utot"]) == (a["iterations"], a["parts"], a["utot"])
        assert np.array_equal(r["strav"], a["strav"])
