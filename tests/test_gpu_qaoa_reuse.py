"""Batches large enough that every block of a pass stages several instances into one buffer.

At n = C + 4 one stage of the middle high passes holds the phase and the stores, and byte costs take the phase from
a table staged with the item: the next instance's table must not arrive before the last thread has read this
one's.  Every mean is compared with the same batch on FP64 costs (no table) and with a repeated run."""
import json

import numpy as np
import pytest

import orkan_b200
from orkan_b200.batch import QaoaBatch, random_regular_graph

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("n,log_chunk", [(16, 12), (15, 11), (17, 13)])
@pytest.mark.parametrize("p", [2, 3])
def test_buffers_shared_by_many_instances(n, log_chunk, p, tmp_path):
    import torch
    ork = orkan_b200.load(5)
    rng = np.random.default_rng(100 * n + p)
    count = 256                             # 8 items each: 2048 for 148 blocks of 1 to 6 buffers
    edges = [random_regular_graph(n, 3, rng) for _ in range(count)]
    g, b = rng.uniform(0, np.pi, (count, p)), rng.uniform(0, np.pi / 2, (count, p))
    path = tmp_path / "chunks.json"
    path.write_text(json.dumps({f"{torch.cuda.get_device_name()}|n{n}|p{p}|u8|v3":
                                {"C": log_chunk, "threads": 256, "ring": 1}}) + "\n")
    with QaoaBatch(ork, [n] * count, edges, None, p) as b8, QaoaBatch(ork, [n] * count, edges, None, p, f64_costs=True) as b64:
        b8.tune(g, b, str(path))            # takes the chunk from the file
        assert b8.config(n)[0] == log_chunk
        want = b64.run(g, b)
        first = b8.run(g, b)
        assert np.abs(first - want).max() < TOL
        for _ in range(5):
            assert np.array_equal(b8.run(g, b), first)
