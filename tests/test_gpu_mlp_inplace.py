"""Results of the surrogate network that lie on its inputs (the C entry points take any device pointers)."""
import ctypes as C

import pytest

import orkan_b200
from orkan_b200.surrogate import Mlp

pytestmark = pytest.mark.gpu


def ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("hidden,n_in,rows,max_batch", [(256, 12, 3000, 3000), (256, 1, 5000, 600), (256, 64, 900, 900),
                                                        (64, 12, 500, 500)])
def test_results_on_the_inputs(hidden, n_in, rows, max_batch):
    import torch
    net = Mlp(orkan_b200.load(5), n_in, hidden, max_batch, seed=2)
    lib, h = net.lib, net.h
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows)
    x = torch.rand(rows, n_in, generator=gen, device="cuda") * 2 - 1
    k = min(rows, max_batch)
    t = torch.randn(k, generator=gen, device="cuda")
    want = torch.cat([net.forward(x[c:c + max_batch]) for c in range(0, rows, max_batch)])     # the same pieces
    loss, grad, gx = net.gradients(x[:k].contiguous(), t, want_x=True)
    for _ in range(3):
        a = x.clone()
        assert lib.orkan_mlp_predict(h, ptr(a), rows, ptr(a), None) == 0             # y over x
        torch.cuda.synchronize()
        assert torch.equal(a.reshape(-1)[:rows], want)
    a = x[:k].clone()
    assert lib.orkan_mlp_forward(h, ptr(a), k, ptr(a), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(a.reshape(-1)[:k], want[:k])
    a, g = x[:k].clone(), torch.empty_like(grad)
    one = torch.empty(1, device="cuda")
    assert lib.orkan_mlp_gradients(h, ptr(a), ptr(t), k, ptr(one), ptr(g), ptr(a), None) == 0        # dL/dx over x
    torch.cuda.synchronize()
    assert torch.equal(a, gx) and torch.equal(g, grad) and float(one) == loss
    net.close()
