"""The surrogate log-likelihood and the network layers at the edges of their tiles.

Likelihood: 128 chains per block, 8 coefficients per group, up to 96; the FP32 products G c̃ are the
sequential sums over b, the rest exact: against FP64 the bound is k 2^-24 of Σ |c̃_a| Σ_b |G_ab c̃_b|.
Layers on the tensor cores against the FP32 layers of training at row counts around the 128-row
tile: each is held to 1e-4 of the largest FP64 output by its own test, so the two agree within 2e-4."""
import ctypes

import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian import Surrogate
from altar_gb300.device import ptr, stream_handle

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 8, 9, 64, 96])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_llk_tiles(cuda, k, n):
    rng = np.random.default_rng(100 * k + n)
    f32 = lambda a: dev(a, dtype=torch.float32)
    c, scale, h = f32(rng.normal(size=(n, k))), f32(rng.uniform(0.5, 2, k)), f32(rng.normal(size=k))
    A = rng.normal(size=(k, k + 3))
    G = f32(A @ A.T)
    llk = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    _native.call("ag_surrogate_llk", n, k, ptr(c), ptr(scale), ptr(G), ptr(h), 3.5, -2.0, ptr(llk), stream_handle())
    cs = (c * scale).double()
    ref = -2.0 - 0.5 * (3.5 - 2.0 * cs @ h.double() + ((cs @ G.double().T) * cs).sum(1))
    bound = k * 2.0 ** -24 * ((cs.abs() @ G.double().abs().T) * cs.abs()).sum(1) + 1e-12
    assert bool(((llk - ref).abs() <= bound).all())


@pytest.mark.parametrize("n", [1, 127, 129, 20000])
def test_layer_tiles(cuda, n):
    sur = Surrogate(sizes=(10, 256, 64, 320, 64), seed=3).init_params()
    lib, net, s = _native.load(), ctypes.byref(sur.net), stream_handle()
    x = torch.rand(n, 10, device="cuda", generator=torch.Generator("cuda").manual_seed(n)) * 2 - 1
    a, b = (torch.empty(n, 64, device="cuda") for _ in range(2))
    acts = torch.empty(lib.ag_mlp_activation_floats(net, n), device="cuda")
    ws = torch.empty(lib.ag_mlp_tc_workspace_bytes(net, n), dtype=torch.uint8, device="cuda")
    flags = torch.zeros(1, dtype=torch.int32, device="cuda")
    _native.call("ag_mlp_forward", net, ptr(sur.params), ptr(sur.pbf), ptr(x), n, ptr(a), ptr(acts), s)
    _native.call("ag_mlp_forward_tc", net, ptr(sur.params), ptr(sur.wpack), ptr(x), n, ptr(b), None, ptr(ws),
                 ws.numel(), ptr(flags), s)
    assert int(flags.item()) == 0
    assert float((a - b).abs().max()) <= 2e-4 * float(a.abs().max())
