"""The choice of a serving round's requests (csrc/e3d_rounds.h), replayed on the host
with requests that keep arriving."""
import ctypes as C
import os
import random
import subprocess

import pytest

import elas3d_xtal_gb300 as e3d

CSRC = os.path.join(os.path.dirname(os.path.abspath(e3d.__file__)), "csrc")
SOURCE = """
#include "e3d_rounds.h"
extern "C" int pick(int n, const int* parts, const long long* last, int blocks, int* out) {
  const std::vector<int> t = e3d::round_requests({parts, parts + n}, {last, last + n}, blocks);
  std::copy(t.begin(), t.end(), out);
  return (int)t.size();
}
"""


@pytest.fixture(scope="module")
def pick(tmp_path_factory):
    d = tmp_path_factory.mktemp("rounds")
    (d / "r.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "r.cpp"), "-o", str(d / "r.so")],
                   check=True)
    f = C.CDLL(str(d / "r.so")).pick

    def call(parts, last, blocks):
        n = len(parts)
        out = (C.c_int * n)()
        k = f(n, (C.c_int * n)(*parts), (C.c_longlong * n)(*last), blocks, out)
        return list(out[:k])

    return call


@pytest.mark.parametrize("blocks,slots,parts", [(152, 2, "half"), (152, 9, "mixed"), (152, 9, "full"), (152, 32, "mixed"),
                                                (152, 64, "small"), (7, 5, "mixed")])
def test_stream(pick, blocks, slots, parts):
    """Every slot that falls free is taken by a request of a few rounds: nobody waits
    twice in a row, and a round never runs fewer parts a wave than everything would."""
    rng = random.Random(slots)
    draw = {"half": lambda: blocks // 2 + 10, "mixed": lambda: rng.randint(1, blocks),
            "full": lambda: blocks if rng.random() < 0.3 else rng.randint(1, 20), "small": lambda: rng.randint(1, 9)}[parts]
    active = [dict(parts=draw(), last=-1, need=200, waits=0)]
    for rnd in range(600):
        while len(active) < slots:
            active.append(dict(parts=draw(), last=rnd - 1, need=rng.randint(1, 6), waits=0))
        p = [a["parts"] for a in active]
        take = pick(p, [a["last"] for a in active], blocks)
        assert take == sorted(set(take)) and take
        ran, every = sum(p[i] for i in take), sum(p)
        assert ran * -(-every // blocks) >= every * -(-ran // blocks)
        for i, a in enumerate(active):
            if i in take:
                a.update(last=rnd, need=a["need"] - 1, waits=0)
            else:
                a["waits"] += 1
                assert a["waits"] == 1
        if active[0]["need"] == 0:  # the long one
            assert rnd < 2 * 200
            break
        active = [a for a in active if a["need"] > 0]
    else:
        pytest.fail("the long request did not finish")


def test_all_that_fit_run(pick):
    assert pick([60, 60, 32], [0, 0, 0], 152) == [0, 1, 2]
    assert pick([152, 100, 52], [0, 0, 0], 152) == [0, 1, 2]  # two whole waves
    assert pick([80, 60, 32], [0, 0, 0], 152) == [0, 1]  # one whole wave: 140 parts in it, 86 a wave with the third
    assert pick([80, 60, 32], [1, 1, 0], 152) == [0, 2]  # the third waited
    assert pick([152, 20], [1, 0], 152) == [0, 1]  # the short one waited, and 20 parts are no wave
