"""Surrogate training takes its batches as slices of one gather per epoch, at addresses that need not be
16-byte aligned: the parameters are bit for bit those of batches gathered one by one."""
import ctypes

import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian import Surrogate
from altar_gb300.device import ptr, stream_handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,batch", [((5, 64, 24), 33), ((3, 72, 40, 8), 17), ((10, 300, 64), 21), ((7, 5, 3), 9)])
def test_slices_of_the_epoch(cuda, sizes, batch):
    n, epochs = 5 * batch + 3, 2
    g = torch.Generator("cuda").manual_seed(batch)
    x = torch.rand(n, sizes[0], device="cuda", generator=g) * 2 - 1
    y = torch.randn(n, sizes[-1], device="cuda", generator=g)
    sur = [Surrogate(sizes=sizes, seed=4, batch=batch).init_params() for _ in range(2)]
    for s in sur:
        s.reserve(n, sizes[0])
        s.add(x, y)
    losses = sur[0].train(epochs=epochs)

    # the same, batch by batch
    ref, lib, st = sur[1], _native.load(), stream_handle()
    net = ctypes.byref(ref.net)
    new = lambda *shape: torch.empty(*shape, dtype=torch.float32, device="cuda")
    acts, out, dout = new(lib.ag_mlp_activation_floats(net, batch)), new(batch, ref.k), new(batch, ref.k)
    scratch, loss = new(2 * batch * max(sizes)), new(batch)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(ref.seed)
    step = 0
    for ep in range(epochs):
        perm = torch.randperm(n, device="cuda", generator=gen)
        total = 0.0
        for b0 in range(0, n - batch + 1, batch):
            xb, yb = x[perm[b0:b0 + batch]].contiguous(), y[perm[b0:b0 + batch]].contiguous()
            _native.call("ag_mlp_forward", net, ptr(ref.params), ptr(ref.pbf), ptr(xb), batch, ptr(out), ptr(acts), st)
            _native.call("ag_mse_grad", batch, ref.k, ptr(out), ptr(yb), ptr(dout), ptr(loss), st)
            _native.call("ag_mlp_backward", net, ptr(ref.params), ptr(ref.pbf), ptr(xb), batch, ptr(acts), ptr(dout),
                         ptr(ref.grads), ptr(scratch), st)
            step += 1
            _native.call("ag_adam_step", ref.params.numel(), ptr(ref.params), ptr(ref.grads), ptr(ref.m), ptr(ref.v),
                         step, ref.lr, 0.9, 0.999, 1e-8, ptr(ref.pbf), st)
            total += float(loss.double().mean())
        assert abs(losses[ep] - total / (n // batch)) <= 1e-12 * abs(losses[ep])
    assert torch.equal(sur[0].params, ref.params) and torch.equal(sur[0].pbf, ref.pbf)
