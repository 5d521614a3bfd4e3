"""Row-tile kernels of the 256-unit surrogate network at the edges of their tiles and rules,
against the float64 oracle."""
import numpy as np
import pytest

import orkan_b200
from oracle import mlp as M

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


# 8-row tiles up to 2368 rows, 32-row tiles above, 64-row tiles (forward) from 18944
@pytest.mark.parametrize("n_in,rows,max_batch", [(1, 1, 1), (12, 7, 8), (12, 9, 64), (64, 65, 65), (12, 2368, 2400),
                                                 (3, 2369, 2400), (12, 18943, 64), (12, 18945, 64)])
def test_tiles_match_oracle(n_in, rows, max_batch):
    import torch
    from orkan_b200.surrogate import Mlp
    ork = orkan_b200.load(5)
    rng = np.random.default_rng(n_in + rows)
    net = Mlp(ork, n_in, 256, max_batch, seed=3)
    p = (rng.normal(0, 1, net.param_count) / 16.0).astype(np.float32)
    net.set_params(p)
    x = rng.uniform(-1, 1, (rows, n_in)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    y = net.forward(xd).cpu().numpy()
    pick = np.unique(np.concatenate([np.arange(min(rows, 40)), np.arange(max(0, rows - 40), rows)]))
    y_ref, _ = M.forward(p, x[pick], n_in, 256)
    assert rel(y[pick], y_ref) < 1e-5
    if rows <= max_batch:
        t = rng.normal(0, 1, rows).astype(np.float32)
        loss, g, gx = net.gradients(xd, torch.from_numpy(t).cuda(), want_x=True)
        loss_ref, g_ref, gx_ref = M.gradients(p, x, t, n_in, 256)
        assert abs(loss - loss_ref) < 1e-5 * max(1.0, loss_ref)
        g, o = g.cpu().numpy(), 0
        for size in (n_in * 256, 256, 256 * 256, 256, 256, 1):
            assert rel(g[o:o + size], g_ref[o:o + size]) < 1e-4, f"block at {o}"
            o += size
        assert rel(gx.cpu().numpy(), gx_ref) < 1e-4
    net.close()


@pytest.mark.parametrize("h", [255, 257])
def test_other_widths_keep_the_general_kernels(h):
    import torch
    from orkan_b200.surrogate import Mlp
    ork = orkan_b200.load(5)
    rng = np.random.default_rng(h)
    net = Mlp(ork, 5, h, 40, seed=1)
    p = (rng.normal(0, 1, net.param_count) / 16.0).astype(np.float32)
    net.set_params(p)
    x = rng.uniform(-1, 1, (101, 5)).astype(np.float32)
    y_ref, _ = M.forward(p, x, 5, h)
    assert rel(net.forward(torch.from_numpy(x).cuda()).cpu().numpy(), y_ref) < 1e-5
    t = rng.normal(0, 1, 33).astype(np.float32)
    loss, g, gx = net.gradients(torch.from_numpy(x[:33]).cuda(), torch.from_numpy(t).cuda(), want_x=True)
    loss_ref, g_ref, gx_ref = M.gradients(p, x[:33], t, 5, h)
    assert rel(g.cpu().numpy(), g_ref) < 1e-4 and rel(gx.cpu().numpy(), gx_ref) < 1e-4
    net.close()
