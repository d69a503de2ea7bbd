"""Triangular whitening with anything above the diagonal of W, as a packed factor's other half has it.

ag_whiten_prepare_lower leaves it out, so the log-likelihood is that of the lower triangle alone, bit for
bit, within a tile of 256 columns and over several, with residuals far from zero (W r̄ in FP64 reads
the same triangle) and with entries that are not finite."""
import ctypes

import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.device import ptr, stream_handle, workspace

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 64, 255, 257, 700])
@pytest.mark.parametrize("junk", [1.0, 1e30, np.nan])
def test_upper_triangle_does_not_count(cuda, m, junk):
    n, lib = 150, _native.load()
    rng = np.random.default_rng(m)
    lower = np.tril(rng.normal(size=(m, m))) / np.sqrt(m) + np.eye(m)
    r = dev(rng.normal(2.0, 1.0, (n, m)), dtype=torch.float32)
    ws = workspace(lib.ag_whiten_workspace_bytes(m, n))
    flags = torch.zeros(1, dtype=torch.int32, device="cuda")

    def llk(W, prepare, *shape):
        split = torch.empty(m * 3 * lib.ag_linear_kpad(m), dtype=torch.int16, device="cuda")
        _native.call(prepare, ptr(W), *shape, ptr(split), stream_handle())
        block = _native.WhitenBlock(W.data_ptr(), split.data_ptr(), 0, m)
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        _native.call("ag_whiten_llk_lower", ctypes.byref(block), ptr(r), m, n, ptr(out), ptr(ws), ws.numel(),
                     ptr(flags), stream_handle())
        return out

    clean = dev(lower)
    want = llk(clean, "ag_linear_prepare", m, m)
    z = r.double() @ clean.T
    assert torch.allclose(want, -0.5 * (z * z).sum(1), rtol=1e-4, atol=0.0)
    assert torch.equal(llk(clean, "ag_whiten_prepare_lower", m), want)
    full = dev(lower + np.triu(np.full((m, m), junk), 1))
    assert torch.equal(llk(full, "ag_whiten_prepare_lower", m), want)
    assert int(flags.item()) == 0
