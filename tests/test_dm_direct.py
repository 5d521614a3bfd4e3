"""The direct density-matrix kernels (dm_direct.cuh) on the CPU emulator: every access in range, every
stored element that changes read and written once, mirrors of diagonal tiles written and never read, and the
oracle's result."""
import itertools

import numpy as np
import pytest

import kemu
from oracle import restate as R
from test_emu_kernels import check_engine_counts, rand_rho

TOL = 1e-12
LAYOUTS = [("packed", 5), ("tiled", 3), ("tiled", 5), ("tiled", 6)]
FLIP = {"x": (1, 1), "y": (-1j, 1j), "cx": (1, 1), "cy": (-1j, 1j), "ccx": (1, 1)}


def rand_u(rng):
    q, _ = np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))
    return q


# one thread per group below 6 qubits, and both forms at 6 (one tile), 7 and 8 qubits, where the tiles of group
# rows and columns meet every case: on the diagonal, partner stored, partner transposed
@pytest.mark.parametrize("kind,lt", LAYOUTS)
@pytest.mark.parametrize("n,tile", [(1, False), (2, False), (4, False), (6, False), (6, True), (7, False), (7, True),
                                    (8, True)])
def test_one_qubit_operations(kind, lt, n, tile):
    rng = np.random.default_rng(n)
    rho = rand_rho(n, n)
    st = R.to_storage(kind, rho, lt)
    for q in range(n):
        u = rand_u(rng)
        res = kemu.dm_direct(kind, lt, st, n, "unitary", [q], u, tile)
        check_engine_counts(kind, n, lt, res)
        assert np.abs(res.out - R.to_storage(kind, R.conjugate_by(rho, u, [q], n), lt)).max() < TOL
        iso, _ = np.linalg.qr(rng.standard_normal((8, 2)) + 1j * rng.standard_normal((8, 2)))
        sop = R.kraus_to_superop([iso[2 * i:2 * i + 2] for i in range(4)])
        res = kemu.dm_direct(kind, lt, st, n, "super", [q], sop, tile)
        check_engine_counts(kind, n, lt, res)
        assert np.abs(res.out - R.to_storage(kind, R.apply_superop1(rho, sop, q), lt)).max() < TOL


@pytest.mark.parametrize("kind,lt", LAYOUTS)
@pytest.mark.parametrize("n,tile", [(3, False), (5, False), (7, True), (8, True)])
def test_flips(kind, lt, n, tile):
    rho = rand_rho(n, n)
    st = R.to_storage(kind, rho, lt)
    some = [0, n // 2, n - 1] if n > 5 else range(n)
    for name, k in (("x", 1), ("y", 1), ("cx", 2), ("cy", 2), ("ccx", 3)):
        for qs in itertools.permutations(some, k):
            res = kemu.dm_direct(kind, lt, st, n, "flip", qs, FLIP[name], tile)
            check_engine_counts(kind, n, lt, res, name, qs)
            assert np.abs(res.out - R.to_storage(kind, R.apply_gate(kind, rho, name, list(qs)), lt)).max() < TOL


@pytest.mark.parametrize("kind,lt", LAYOUTS)
@pytest.mark.parametrize("n", [2, 3, 6])
def test_swap_and_phase(kind, lt, n):
    rho = rand_rho(n, n)
    st = R.to_storage(kind, rho, lt)
    for qs in itertools.permutations(range(n), 2):
        res = kemu.dm_direct(kind, lt, st, n, "swap", qs, [])
        check_engine_counts(kind, n, lt, res, "swap", qs)
        assert np.abs(res.out - R.to_storage(kind, R.apply_gate(kind, rho, "swap", list(qs)), lt)).max() < TOL
        res = kemu.dm_direct(kind, lt, st, n, "ctrlphase", qs, [-1.0])
        assert res.oob == 0 and res.reads.max() <= 1 and res.writes.max() <= 1
        assert np.abs(res.out - R.to_storage(kind, R.apply_gate(kind, rho, "cz", list(qs)), lt)).max() < TOL
