"""The staged engine's 1-qubit operations, controlled flips and SWAP at small sizes.

The library gives most of these to the direct kernels and keeps the engine for large tiled matrices; the engine's
test hook, at its default limit, asks for the engine everywhere.  Every qubit tuple against the oracle."""
import ctypes as C
import itertools

import numpy as np
import pytest

from oracle import restate as R
from orkan_b200 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-12
GATES = ("x", "y", "h", "hy", "rx", "ry", "cx", "cy", "swap", "ccx")


@pytest.mark.parametrize("lt", [3, 5])
@pytest.mark.parametrize("kind", ["packed", "tiled"])
@pytest.mark.parametrize("n", [1, 2, 4, 6, 7])
def test_engine_forms(request, lt, kind, n):
    ork = request.getfixturevalue(f"ork{lt}")
    hook = ork.lib.orkan_cu_engine_test_wait
    hook.argtypes, hook.restype = [C.c_ulonglong, C.c_int], None
    ork.lib.orkan_cu_engine_status.restype = C.c_uint
    rng = np.random.default_rng(n)
    a = rng.standard_normal((1 << n, 3)) + 1j * rng.standard_normal((1 << n, 3))
    full = a @ a.conj().T
    full /= np.trace(full).real
    start = R.to_storage(kind, full, lt)
    st = ork.state(kind, n, start)
    sop = R.kraus_to_superop(R.depolarizing_kraus(0.05))
    hook(1 << 24, 0)                        # the default limit of the engine's waits
    try:
        for g in GATES:
            for qs in itertools.permutations(range(n), W.gate_arity(g)):
                th = float(rng.uniform(0, 2 * np.pi)) if g in W.GATES_ROT else None
                ork.upload(st, start)
                ork.gate(st, g, qs, th)
                want = R.to_storage(kind, R.apply_gate(kind, full, g, qs, th), lt)
                assert np.abs(ork.storage(st) - want).max() <= TOL, (g, qs)
        for q in range(n):
            ork.upload(st, start)
            ork.channel_1q(st, sop, q)
            want = R.to_storage(kind, R.apply_superop1(full, sop, q), lt)
            assert np.abs(ork.storage(st) - want).max() <= TOL, ("channel", q)
    finally:
        hook(0, 0)
    assert ork.lib.orkan_cu_engine_status() == 0
    ork.free(st)


@pytest.mark.parametrize("kind", ["packed", "tiled"])
def test_engine_blocks_of_many_items(ork5, kind):
    """12 qubits are 2080 blocks of 64 x 64 for at most 444 resident ones: each takes several in turn.  Against the
    direct kernels on the same state."""
    hook = ork5.lib.orkan_cu_engine_test_wait
    hook.argtypes, hook.restype = [C.c_ulonglong, C.c_int], None
    ork5.lib.orkan_cu_engine_status.restype = C.c_uint
    n = 12
    st = ork5.plus(kind, n)
    for q in range(n):
        ork5.gate(st, "ry", [q], 0.3 + 0.2 * q)
        ork5.gate(st, "rz", [q], 0.7 - 0.1 * q)
    sop = R.kraus_to_superop(R.depolarizing_kraus(0.05))
    ops = [lambda s, q=q, g=g: ork5.gate(s, g, [(q + 7) % n, q] if g[0] == "c" else [q], 0.9 if g == "rx" else None)
           for g in ("h", "rx", "x", "y", "cx", "cy") for q in (0, 5, 11)]
    ops += [lambda s, q=q: ork5.channel_1q(s, sop, q) for q in (0, 5, 11)]
    for op in ops:
        want, got = ork5.copy(st), ork5.copy(st)
        op(want)
        hook(1 << 24, 0)
        try:
            op(got)
            ork5.sync()
        finally:
            hook(0, 0)
        assert np.abs(ork5.storage(got) - ork5.storage(want)).max() <= TOL
        ork5.free(want)
        ork5.free(got)
    assert ork5.lib.orkan_cu_engine_status() == 0
    ork5.free(st)
