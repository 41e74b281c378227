"""Serving rounds of whole waves under a stream of arrivals (the choice itself:
test_rounds.py)."""
import numpy as np
import pytest

import elas3d_xtal_gb300 as e3d
from elas3d_xtal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_long_request_among_arrivals():
    """Two slots of 100 blocks, so that a round holds one of them, and a request of a few
    rounds after every step: the long one gets every second round."""
    long = (W.rve(14, 6, 3, A=3.0, pore_frac=0.01), np.array([1e-3, 0, 0, 0, 0, 0]))
    short = (W.rve(8, 2, 4, A=1.5, pore_frac=0.0), np.array([1e-3, 0, 0, 0, 0, 0]))

    def steps(arrivals):
        with e3d.Server(round_iters=3, parts=100, max_active=2) as srv:
            i = srv.submit(*long)
            for n in range(1, 200):
                if arrivals:
                    srv.submit(*short)
                srv.step()
                r = srv.result(i)
                if r:
                    return n, r
        return None, None

    alone, a = steps(False)
    busy, b = steps(True)
    assert alone >= 6
    assert busy is not None and busy <= 2 * alone
    assert (a["iterations"], a["utot"]) == (b["iterations"], b["utot"])
