"""The batch autotuner's choice (csrc/e3d_autotune.h) with times that a host model makes."""
import ctypes as C
import os
import subprocess

import pytest

import elas3d_xtal_gb300 as e3d

CSRC = os.path.join(os.path.dirname(os.path.abspath(e3d.__file__)), "csrc")
# A solve of k blocks takes nodes / k + 200 k; solves fill the blocks in whole waves.
# `cold`: added to the first run's time; calls: runs made.
SOURCE = """
#include "e3d_autotune.h"
extern "C" double pick(int n, const long long* nodes, int blocks, double cold, int fail_at, int* plan, int* calls) {
  *calls = 0;
  auto model = [&](const std::vector<int>& p) {
    double longest = 0.0, work = 0.0;
    for (int j = 0; j < n; ++j) {
      const double t = (double)nodes[j] / p[j] + 200.0 * p[j];
      longest = std::max(longest, t);
      work += t * p[j];
    }
    return std::max(longest, work / blocks);
  };
  std::vector<int> best(n, 1);
  const int rc = e3d::pick_parts(
      n, blocks, 152, [](size_t, int k) { return k; }, [&](size_t j) { return nodes[j]; },
      [&](const std::vector<int>&) { return ++*calls == fail_at ? 7 : 0; },
      [&](const std::vector<int>& p, double* ms) {
        *ms = model(p) + (*calls == 0 ? cold : 0.0);
        return ++*calls == fail_at ? 7 : 0;
      },
      best);
  std::copy(best.begin(), best.end(), plan);
  return rc ? -rc : model(best);
}
"""


@pytest.fixture(scope="module")
def pick(tmp_path_factory):
    d = tmp_path_factory.mktemp("autotune")
    (d / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "a.cpp"), "-o", str(d / "a.so")],
                   check=True)
    f = C.CDLL(str(d / "a.so")).pick
    f.restype = C.c_double

    def call(nodes, cold=0.0, fail_at=-1, blocks=152):
        n = len(nodes)
        plan, calls = (C.c_int * n)(), C.c_int()
        t = f(n, (C.c_longlong * n)(*nodes), blocks, C.c_double(cold), fail_at, plan, C.byref(calls))
        return t, list(plan), calls.value

    return call


@pytest.mark.parametrize("nodes", [[64 ** 3] * 6, [32 ** 3, 48 ** 3, 88 ** 3] * 20, [20 ** 3] * 2, [128 ** 3], [40 ** 3] * 700])
@pytest.mark.parametrize("cold", [1e9, -1e9])  # the first run much longer; its difference of two runs negative
def test_first_run_does_not_count(pick, nodes, cold):
    t, plan, calls = pick(nodes)
    assert (t, plan, calls) == pick(nodes, cold)
    assert calls <= 13


def test_few_solves_share_the_blocks(pick):
    _, plan, _ = pick([64 ** 3] * 6)
    assert plan == [25] * 6


def test_failure_is_passed_on(pick):
    assert pick([64 ** 3] * 6, fail_at=1)[0] == -7
    assert pick([64 ** 3] * 6, fail_at=4)[0] == -7
