"""Half-state QAOA passes on the CPU emulator: the launch shapes of the pass kernel.

The passes keep psi(y) for y with the top bit clear, in an order that puts columns c and ~c of
a row side by side, and groups 0 and 1 of an item exchange data within half-warps only.
"""
import numpy as np
import pytest

import kemu
from oracle import restate as R


@pytest.mark.parametrize("n,C", [(n, C) for C in (11, 12, 13) for n in range(C + 1, min(26, 2 * C) + 1)])
def test_half_warps_keep_to_their_slots(n, C):
    for kind in (1, 2):                                    # low, high
        closed = kemu.lib().emu_qaoa_half_warp_closed(n, C, kind)
        high_bits = n - C
        assert closed == (1 if kind == 1 or high_bits >= 8 else -1)


@pytest.mark.parametrize("n,p", [(13, 1), (13, 2), (16, 3), (17, 2), (20, 1), (21, 2)])
@pytest.mark.parametrize("byte_cost", [True, False])
def test_launch_shape_means(n, p, byte_cost):
    """Chunks of 2^12 slots (high items of 1 to 9 mixed bits, so every register set from one
    mixer up) and 2^11 (10 mixed bits), each thread count as launched."""
    rng = np.random.default_rng(n + p)
    edges = [(u, v) for u in range(n) for v in range(u + 1, n) if rng.random() < 0.3]
    w = None if byte_cost else rng.uniform(0.0, 1.0, len(edges))
    cost = R.maxcut_cost(n, edges, w)
    g, b = rng.uniform(0, np.pi, p), rng.uniform(0, np.pi / 2, p)
    C, nthr = (11, 128) if n == 21 else (12, 256)
    res, m = kemu.qaoa(n, cost, p, g, b, log_chunk=C, nthr=nthr, byte_cost=byte_cost)
    assert res.oob == 0
    assert np.all(res.writes == p) and np.all(res.reads == p)
    assert abs(m - R.qaoa_mean(n, cost, g, b)) < 1e-12
