"""Tensor-core layers where their division changes: weights held for up to 256 inputs or streamed with
the rows, one to eight blocks of columns, fewer row tiles than CTAs and several per CTA, a last tile
of one row.

Tolerance: outputs within 1e-4 of the FP64 oracle, normwise.  The activations' two BF16 parts leave
2^-17 of them per layer and FP32 adds at most 1,024 products, 1,024 2^-24 = 6e-5 of the sum of their sizes
at worst and, with random signs, 32 2^-24; three layers in sequence."""
import ctypes

import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian.surrogate import Surrogate
from altar_gb300.device import ptr, stream_handle, workspace
from oracle import mlp

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(3, 64), (10, 256, 64), (70, 128, 320, 64), (12, 512, 192, 128)])
@pytest.mark.parametrize("n", [1, 129, 5000, 40001])
def test_layers(cuda, sizes, n):
    sur = Surrogate(sizes, seed=9).init_params()
    flat = sur.params.cpu().numpy().astype(np.float64)
    W16 = sur.params.to(torch.bfloat16).double().cpu().numpy()
    P, o = [], 0
    for fi, fo in zip(sizes[:-1], sizes[1:]):
        P.append((W16[o:o + fo * fi].reshape(fo, fi), flat[o + fo * fi:o + fo * fi + fo]))
        o += fo * fi + fo
    lib, net, s = _native.load(), ctypes.byref(sur.net), stream_handle()
    x = dev(np.random.default_rng(n).uniform(-1, 1, (n, sizes[0])), torch.float32)
    out = torch.full((n + 1, sizes[-1]), 5.0, dtype=torch.float32, device="cuda")
    ws = workspace(lib.ag_mlp_tc_workspace_bytes(net, n))
    for _ in range(2):                          # a second evaluation in the same workspace
        _native.call("ag_mlp_forward_tc", net, ptr(sur.params), ptr(sur.wpack), ptr(x), n, ptr(out), None, ptr(ws),
                     ws.numel(), ptr(sur._tc_flags), s)
    torch.cuda.synchronize()
    assert int(sur._tc_flags.item()) == 0 and bool((out[n] == 5.0).all())
    ref, _ = mlp.forward(P, x.double().cpu().numpy())
    assert np.max(np.abs(out[:n].double().cpu().numpy() - ref)) <= 1e-4 * np.max(np.abs(ref))
