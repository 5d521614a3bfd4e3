"""Fused statevector runs whose first stage reads device memory and whose last stage writes it
(orkan_b200/csrc/cuda/pure_fused.cuh): a stage does so where its group leaves the lowest three qubits
alone.  Runs that begin and end on low or high qubits, with one stage and several, at the smallest
chunks that have direct stages and one below, equal the gates applied one by one bit for bit."""
import numpy as np
import pytest

from orkan_b200 import workloads as W
import kemu

LOW = [("h", (0,), None), ("cx", (2, 1), None)]
HIGH = [("ry", (-1,), 0.7), ("swap", (-2, -3), None), ("p", (0,), 1.1)]
MID = [("h", (3,), None), ("hy", (1,), None), ("rx", (-2,), 0.4), ("ccx", (-1, 2, 3), None), ("h", (0,), None)]
RUNS = {"high": HIGH, "low": LOW, "high-high": HIGH + MID + HIGH, "high-low": HIGH + MID + LOW,
        "low-high": LOW + MID + HIGH, "low-low": LOW + MID + LOW, "diagonal": [("rz", (1,), 0.3), ("cz", (0, -1), None)]}


def gates_of(run, n):
    return [(g, tuple(q % n for q in qs), th) for g, qs, th in RUNS[run]]


@pytest.mark.parametrize("run", list(RUNS))
@pytest.mark.parametrize("n,log_chunk", [(5, 5), (6, 6), (7, 7), (9, 6), (9, 7), (9, 8), (12, 11)])
def test_emulated(n, log_chunk, run):
    gates = gates_of(run, n)
    need = 7
    for g, qs, _ in gates:
        need |= kemu.fused_need(g, qs)
    if bin(need).count("1") > log_chunk:
        pytest.skip("mixes more qubits than the chunk has")
    psi = W.gaussian_pure(n, 11)
    r = kemu.pure_fused(psi, n, log_chunk, gates, 3)
    assert r.oob == 0
    assert (r.reads == 1).all() and (r.writes == 1).all()
    want = psi
    for g, qs, th in gates:
        want = kemu.pure_gate(want, n, g, qs, th).out
    assert np.array_equal(r.out, want)


@pytest.mark.gpu
@pytest.mark.parametrize("run", list(RUNS))
@pytest.mark.parametrize("n", [5, 7, 12, 13, 20])
def test_on_the_gpu(ork5, n, run):
    outs = []
    for fusion in (48, 0):
        ork5.set_gate_fusion(fusion)
        try:
            st = ork5.plus("pure", n)
            for part in (W.random_circuit(n, 8, seed=2), gates_of(run, n)):
                for g, qs, th in part:
                    ork5.gate(st, g, qs, th)
                ork5.flush()
            outs.append(ork5.storage(st))
            ork5.free(st)
        finally:
            ork5.set_gate_fusion(48)
    assert np.array_equal(*outs)
