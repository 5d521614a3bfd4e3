"""channel_1q with superoperators that do not map Hermitian matrices to Hermitian ones: every stored element is what
the oracle's update of the whole matrix gives for it, wherever its group lies."""
import numpy as np
import pytest

import kemu
from oracle import restate as R
from test_emu_kernels import rand_rho

TOL = 1e-12


def rand_sop(rng):
    return (rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))) / 4


def stored(kind, full, lt):
    """Storage of the lower triangle of full (diagonal tiles hold its mirror image)."""
    low = np.tril(full)
    return R.to_storage(kind, low + np.tril(full, -1).conj().T, lt)


@pytest.mark.parametrize("kind,lt", [("packed", 5), ("tiled", 3), ("tiled", 5), ("tiled", 6)])
@pytest.mark.parametrize("n,tile", [(1, False), (4, False), (7, False), (6, True), (7, True), (8, True)])
def test_emulated(kind, lt, n, tile):
    rng = np.random.default_rng(n)
    rho = rand_rho(n, n)
    st = R.to_storage(kind, rho, lt)
    for q in range(n):
        sop = rand_sop(rng)
        res = kemu.dm_direct(kind, lt, st, n, "super", [q], sop, tile)
        assert np.abs(res.out - stored(kind, R.apply_superop1(rho, sop, q), lt)).max() < TOL, q


@pytest.mark.gpu
@pytest.mark.parametrize("lt", [5, 3])
@pytest.mark.parametrize("kind", ["packed", "tiled"])
@pytest.mark.parametrize("n", [1, 4, 6, 8, 11])
def test_on_the_gpu(request, kind, n, lt):
    ork = request.getfixturevalue(f"ork{lt}")
    rng = np.random.default_rng(n)
    rho = rand_rho(n, n)
    st = ork.state(kind, n)
    for q in range(n) if n < 11 else (0, 5, 10):           # below, on and above a tile of 32 groups
        sop = rand_sop(rng)
        ork.upload(st, R.to_storage(kind, rho, lt))
        ork.channel_1q(st, sop, q)
        assert np.abs(ork.storage(st) - stored(kind, R.apply_superop1(rho, sop, q), lt)).max() < TOL, q
    ork.free(st)
