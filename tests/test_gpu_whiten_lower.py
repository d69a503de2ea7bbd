"""The tensor-core evaluations at the edges of their tiles.

The triangular whitening leaves out products with zeros only, so it equals the general one bit for
bit.  Both against FP64 within the split products' own error: with z = W (r - r̄) + W r̄, each factor's
two BF16 parts leave 2^-17 of it, the dropped product of the low parts 2^-18, and FP32 adds 3 m
terms, so |dz| <= (3 2^-17 + 3 m 2^-24) |W| |r - r̄| + 2^-23 |W r̄|, and the misfit moves by at most
Σ 2 |z| |dz| + dz².  128 chains, 256 observations and 64
columns per tile, two rows per thread of the split, rows that are not 16-byte aligned."""
import ctypes

import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.device import ptr, stream_handle, workspace

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 63, 64, 255, 256, 257, 700])
@pytest.mark.parametrize("n", [1, 7, 128, 129, 1500])
def test_lower_whitening(cuda, m, n):
    rng = np.random.default_rng(1000 * m + n)
    lib = _native.load()
    W = dev(np.tril(rng.normal(size=(m, m))) / np.sqrt(m) + np.eye(m))
    col0, ldr = (m % 3), m + 5 + (m % 2)
    r = dev(rng.normal(0.3, 1.0, (n, ldr)), dtype=torch.float32)
    split = torch.empty(m * 3 * lib.ag_linear_kpad(m), dtype=torch.int16, device="cuda")
    _native.call("ag_linear_prepare", ptr(W), m, m, ptr(split), stream_handle())
    block = _native.WhitenBlock(W.data_ptr(), split.data_ptr(), col0, m)
    ws = workspace(lib.ag_whiten_workspace_bytes(m, n))
    flags = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = {}
    for name in ("ag_whiten_llk", "ag_whiten_llk_lower"):
        llk = torch.full((n,), 3.0, dtype=torch.float64, device="cuda")
        for _ in range(2):                      # a second evaluation in the same workspace
            _native.call(name, ctypes.byref(block), ptr(r), ldr, n, ptr(llk), ptr(ws), ws.numel(), ptr(flags),
                         stream_handle())
        got[name] = llk.cpu().numpy()
    assert int(flags.item()) == 0
    np.testing.assert_array_equal(got["ag_whiten_llk_lower"], got["ag_whiten_llk"])
    x = r[:, col0:col0 + m].double()
    rows = min(n, 256)
    centre = x[:: n // rows][:rows].mean(0)
    z = x @ W.T
    dz = (3 * 2.0 ** -17 + 3 * m * 2.0 ** -24) * ((x - centre).abs() @ W.abs().T) + 2.0 ** -23 * (W @ centre).abs()
    miss = (torch.from_numpy(3.0 - got["ag_whiten_llk"]).cuda() - (z * z).sum(1)).abs()
    assert bool((miss <= (2 * z.abs() * dz + dz * dz).sum(1) + 1e-14).all())


@pytest.mark.parametrize("m,n", [(3000, 9000), (700, 20001), (600, 9473)])
def test_lower_whitening_tile_order(cuda, m, n):
    """Several rounds of tiles, in two groups (3,000) and in one, forwards and backwards."""
    lib = _native.load()
    g = torch.Generator(device="cuda").manual_seed(m)
    W = torch.tril(torch.randn(m, m, generator=g, device="cuda", dtype=torch.float64)) / m ** 0.5
    r = torch.randn(n, m, generator=g, device="cuda")
    split = torch.empty(m * 3 * lib.ag_linear_kpad(m), dtype=torch.int16, device="cuda")
    _native.call("ag_linear_prepare", ptr(W), m, m, ptr(split), stream_handle())
    block = _native.WhitenBlock(W.data_ptr(), split.data_ptr(), 0, m)
    ws = workspace(lib.ag_whiten_workspace_bytes(m, n))
    flags = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = []
    for name in ("ag_whiten_llk", "ag_whiten_llk_lower"):
        llk = torch.zeros(n, dtype=torch.float64, device="cuda")
        _native.call(name, ctypes.byref(block), ptr(r), m, n, ptr(llk), ptr(ws), ws.numel(), ptr(flags),
                     stream_handle())
        got.append(llk)
    assert int(flags.item()) == 0 and bool((got[0] < 0).all())
    assert torch.equal(got[0], got[1])
