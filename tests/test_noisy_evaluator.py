"""NoisyEvaluator's attributes between calls: what a caller sets is what the next call evaluates."""
import numpy as np
import pytest

from oracle import restate as R
from orkan_b200.surrogate import NoisyEvaluator

EDGES = [(0, 1), (1, 2), (2, 3), (0, 3), (1, 4)]
WEIGHTS = [0.3, 0.9, 0.4, 0.7, 0.2]
PROB = 0.03
TOL = 1e-12


def oracle(kind, n, cost, gs, bs):
    sop = R.kraus_to_superop(R.depolarizing_kraus(PROB))
    out = []
    for g, b in zip(gs, bs):
        rho = R.plus_state(kind, n)
        for gk, bk in zip(g, b):
            rho = R.exp_diag(kind, rho, cost, gk)
            for q in range(n):
                rho = R.apply_superop1(R.apply_gate(kind, rho, "rx", [q], 2 * bk), sop, q)
        out.append(R.mean(kind, rho, cost))
    return np.array(out)


def angles(count, p, seed=1):
    rng = np.random.default_rng(seed)
    return rng.uniform(0, np.pi, (count, p)), rng.uniform(0, np.pi / 2, (count, p))


def test_construction_needs_no_device():
    ev = NoisyEvaluator(None, 5, EDGES, WEIGHTS, 2, PROB)
    assert np.array_equal(ev.cost, R.maxcut_cost(5, EDGES, np.array(WEIGHTS)))


@pytest.mark.gpu
def test_costs_changed_in_place_and_replaced(ork5):
    ev = NoisyEvaluator(ork5, 5, EDGES, WEIGHTS, 2, PROB)
    g, b = angles(3, 2)
    ev(g, b)
    ev.cost *= -2.5
    assert np.abs(ev(g, b) - oracle("tiled", 5, ev.cost, g, b)).max() < TOL
    ev.cost = [float(x % 7) for x in range(32)]            # a list, as exp_diag and mean take one
    assert np.abs(ev(g, b) - oracle("tiled", 5, np.array(ev.cost), g, b)).max() < TOL
    assert abs(ev.one(g[1], b[1]) - ev(g, b)[1]) < TOL


@pytest.mark.gpu
def test_layout_and_qubit_count_changed_between_calls(ork5):
    ev = NoisyEvaluator(ork5, 5, EDGES, WEIGHTS, 2, PROB)
    g, b = angles(2, 2)
    ev(g, b)
    ev.kind = "packed"
    assert np.abs(ev(g, b) - oracle("packed", 5, ev.cost, g, b)).max() < TOL
    ev.n, ev.cost = 7, R.maxcut_cost(7, EDGES + [(5, 6), (0, 6)])
    assert np.abs(ev(g, b) - oracle("packed", 7, ev.cost, g, b)).max() < TOL
    ev.close()
    assert np.abs(ev(g, b) - oracle("packed", 7, ev.cost, g, b)).max() < TOL


@pytest.mark.gpu
def test_angle_sets_are_paired_and_a_failed_call_keeps_no_state(ork5):
    ev = NoisyEvaluator(ork5, 5, EDGES, WEIGHTS, 2, PROB)
    g, b = angles(3, 2)
    want = oracle("tiled", 5, ev.cost, g, b)
    assert np.abs(ev(g, b[:2]) - want[:2]).max() < TOL     # as zip(gammas, betas)
    assert np.abs(ev(g[:1], b) - want[:1]).max() < TOL
    assert type(ev.one(g[2], b[2])) is float
    assert len(ev(g[:0], b[:0])) == 0
    with pytest.raises(IndexError):
        ev(g[:, :1], b)                                    # too few angles for two layers
    assert np.abs(ev(g, b) - want).max() < TOL
    ev.close()
    assert not ev._states
