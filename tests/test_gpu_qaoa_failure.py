"""Waits of the batched passes that run out, made on the host: the test hook sets their limit to zero.

The launches then end early with a status that the call returns, nothing is left in flight, and the context
stays usable."""
import ctypes as C

import numpy as np
import pytest

import orkan_b200
from oracle import restate as R
from orkan_b200 import OrkanError
from orkan_b200.batch import QaoaBatch, random_regular_graph

pytestmark = pytest.mark.gpu

TOL = 1e-12
TIMEOUT = 702                               # cudaErrorLaunchTimeout


def make(f64_costs, p=3):
    ork = orkan_b200.load(5)
    ork.lib.orkan_qaoa_test_expire.argtypes = [C.c_void_p, C.c_int]
    rng = np.random.default_rng(3)
    ns = [20] * 4 + [16] * 8 + [14, 9]
    edges = [random_regular_graph(n, 3, rng) for n in ns]
    g, b = rng.uniform(0, np.pi, (len(ns), p)), rng.uniform(0, np.pi / 2, (len(ns), p))
    want = {i: R.qaoa_mean(ns[i], R.maxcut_cost(ns[i], edges[i]), g[i], b[i]) for i in (4, 12, 13)}
    return QaoaBatch(ork, ns, edges, None, p, f64_costs=f64_costs), g, b, want


def expire(bt, on):
    assert bt.lib.orkan_qaoa_test_expire(bt.h, on) == 0


def check(bt, g, b, want):
    means = bt.run(g, b)
    for i, m in want.items():
        assert abs(means[i] - m) < TOL


@pytest.mark.parametrize("f64_costs", [False, True])
def test_expired_waits_are_reported_and_leave_the_context_usable(f64_costs):
    bt, g, b, want = make(f64_costs)
    with bt:
        expire(bt, 1)
        with pytest.raises(OrkanError, match=str(TIMEOUT)):
            bt.run(g, b)
    fresh, g, b, want = make(f64_costs)
    with fresh:
        check(fresh, g, b, want)


def test_the_next_run_of_the_batch_is_good_again():
    bt, g, b, want = make(False)
    with bt:
        check(bt, g, b, want)
        expire(bt, 1)
        for _ in range(2):
            with pytest.raises(OrkanError, match=str(TIMEOUT)):
                bt.run(g, b)
        expire(bt, 0)
        check(bt, g, b, want)


def test_tuning_takes_no_time_of_an_expired_candidate(tmp_path):
    bt, g, b, want = make(False)
    with bt:
        before = {n: bt.config(n) for n in (9, 14, 16, 20)}
        expire(bt, 1)
        path = tmp_path / "tune.json"
        bt.tune(g, b, str(path))
        assert {n: bt.config(n) for n in before} == before          # the defaults: nothing was timed
        recorded = path.read_text() if path.exists() else ""
        assert "|n20|" not in recorded and "|n16|" not in recorded
        expire(bt, 0)
        check(bt, g, b, want)
