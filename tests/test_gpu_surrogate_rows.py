"""Training kernels of narrow networks (one launch forward, one per layer backward) at the edges of
their tiles, against the FP64 oracle: rows beside a multiple of the row block, fewer rows than parts
of the row split, layers of 8 to 256 outputs, inputs that are no multiple of 8, and networks just
outside the rule (a width above 256, an output count that is no multiple of 8).

The row-wise kernels also give the tiled products' values bit for bit.

Tolerance: network outputs and gradients within 1e-4 of the oracle, normwise.  A chain of at most 256
FP32 products is off by at most 256 u = 1.5e-5 of the sum of its terms' sizes, and random signs leave a
few u of it; up to five layers in sequence."""

import ctypes

import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian.surrogate import Surrogate
from altar_gb300.device import ptr, stream_handle
from oracle import mlp

from gpu_helpers import dev

pytestmark = pytest.mark.gpu

NETS = [(10, 256, 256, 256, 256, 64), (1, 8), (13, 40, 72, 136, 256), (256, 256, 8), (7, 32, 64, 128, 24),
        (200, 8, 248, 16), (9, 264, 32), (5, 40, 12), (64, 33, 8)]
ROWS = [1, 7, 9, 513, 1300]


@pytest.mark.parametrize("sizes", NETS)
@pytest.mark.parametrize("n", ROWS)
def test_forward_and_backward(cuda, sizes, n):
    sur = Surrogate(sizes, seed=5).init_params()
    rng = np.random.default_rng(n)
    sur.set_params(sur.params + dev(0.1 * rng.normal(size=sur.params.numel()), torch.float32))  # biases too
    flat = sur.params.double().cpu().numpy()
    W16 = sur.params.to(torch.bfloat16).double().cpu().numpy()
    P, o = [], 0
    for fi, fo in zip(sizes[:-1], sizes[1:]):
        P.append((W16[o:o + fo * fi].reshape(fo, fi), flat[o + fo * fi:o + fo * fi + fo]))
        o += fo * fi + fo
    xd = dev(rng.uniform(-1, 1, (n, sizes[0])), torch.float32)
    yd = dev(rng.normal(size=(n, sizes[-1])), torch.float32)
    net, s = ctypes.byref(sur.net), stream_handle()
    acts = torch.empty(_native.load().ag_mlp_activation_floats(net, n), dtype=torch.float32, device="cuda")
    guard = 64
    out = torch.full((n * sizes[-1] + guard,), 7.0, dtype=torch.float32, device="cuda")
    scratch = torch.full((2 * n * max(sizes) + guard,), 7.0, dtype=torch.float32, device="cuda")
    dout, loss = torch.empty(n, sizes[-1], dtype=torch.float32, device="cuda"), torch.empty(n, device="cuda")
    _native.call("ag_mlp_forward", net, ptr(sur.params), ptr(sur.pbf), ptr(xd), n, ptr(out), ptr(acts), s)
    _native.call("ag_mse_grad", n, sizes[-1], ptr(out), ptr(yd), ptr(dout), ptr(loss), s)
    sur.grads.fill_(float("nan"))
    _native.call("ag_mlp_backward", net, ptr(sur.params), ptr(sur.pbf), ptr(xd), n, ptr(acts), ptr(dout),
                 ptr(sur.grads), ptr(scratch), s)
    torch.cuda.synchronize()
    x, y = xd.double().cpu().numpy(), yd.double().cpu().numpy()
    ref, _ = mlp.forward(P, x)
    got = out[:-guard].double().cpu().numpy().reshape(n, -1)
    assert np.max(np.abs(got - ref)) <= 1e-4 * np.max(np.abs(ref))
    row = 0.5 * ((got - y) ** 2).sum(axis=1)
    np.testing.assert_allclose(loss.double().cpu().numpy(), row, rtol=1e-4)
    g_ref = np.concatenate([np.concatenate([gW.ravel(), gb]) for gW, gb in mlp.backward(P, x, y)])
    g = sur.grads.double().cpu().numpy()
    assert np.linalg.norm(g - g_ref) <= 1e-4 * np.linalg.norm(g_ref)
    assert torch.all(out[-guard:] == 7.0) and torch.all(scratch[-guard:] == 7.0)


@pytest.mark.parametrize("sizes", NETS)
@pytest.mark.parametrize("n", ROWS + [450, 2050])
def test_rows_and_tiles_agree_bit_for_bit(cuda, sizes, n):
    """The row-wise kernels add in the tiled products' order.  Weights that do not start on a 16-byte
    boundary take the tiled products, so both run on the same values."""
    sur = Surrogate(sizes, seed=6).init_params()
    rng = np.random.default_rng(n + 1)
    net, s = ctypes.byref(sur.net), stream_handle()
    odd = torch.empty(sur.pbf.numel() + 1, dtype=torch.int16, device="cuda")[1:]
    odd.copy_(sur.pbf)
    x = dev(rng.uniform(-1, 1, (n, sizes[0])), torch.float32)
    y = dev(rng.normal(size=(n, sizes[-1])), torch.float32)
    results = []
    for weights in (sur.pbf, odd):
        acts = torch.zeros(_native.load().ag_mlp_activation_floats(net, n), dtype=torch.float32, device="cuda")
        out, dout, loss = torch.empty_like(y), torch.empty_like(y), torch.empty(n, device="cuda")
        scratch, grads = torch.empty(2 * n * max(sizes), device="cuda"), torch.empty_like(sur.grads)
        _native.call("ag_mlp_forward", net, ptr(sur.params), ptr(weights), ptr(x), n, ptr(out), ptr(acts), s)
        _native.call("ag_mse_grad", n, sizes[-1], ptr(out), ptr(y), ptr(dout), ptr(loss), s)
        _native.call("ag_mlp_backward", net, ptr(sur.params), ptr(weights), ptr(x), n, ptr(acts), ptr(dout),
                     ptr(grads), ptr(scratch), s)
        results.append((out, acts, loss, grads))
    torch.cuda.synchronize()
    for a, b in zip(*results):
        assert torch.equal(a, b)
