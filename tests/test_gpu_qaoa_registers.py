"""The pass kernels' form without a register split, which serves builds whose compiler gave the kernels other
register counts, against the plain composition and the default form."""
import ctypes as C

import numpy as np
import pytest

import orkan_b200
from oracle import restate as R
from orkan_b200.batch import QaoaBatch, random_regular_graph

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("f64_costs", [False, True])
def test_passes_without_the_register_split(f64_costs):
    ork = orkan_b200.load(5)
    ork.lib.orkan_qaoa_test_plain_registers.argtypes = [C.c_void_p]
    rng = np.random.default_rng(8)
    ns, p = [13, 14, 15, 16, 17, 20, 24, 25], 3          # every number of mixed bits up to 12, chunks of 2^12 and 2^13
    edges = [random_regular_graph(n, 3, rng) for n in ns]
    g, b = rng.uniform(0, np.pi, (len(ns), p)), rng.uniform(0, np.pi / 2, (len(ns), p))
    with QaoaBatch(ork, ns, edges, None, p, f64_costs=f64_costs) as bt:
        want = bt.run(g, b)
        assert bt.lib.orkan_qaoa_test_plain_registers(bt.h) == 0
        got = bt.run(g, b)
    assert np.abs(got - want).max() < TOL
    for i in range(5):
        assert abs(got[i] - R.qaoa_mean(ns[i], R.maxcut_cost(ns[i], edges[i]), g[i], b[i])) < TOL
