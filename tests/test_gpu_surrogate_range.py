"""The surrogate log-likelihood where its terms leave FP32's range.

A coefficient far outside the training range makes products beyond 3.4e38; the log-likelihood is the FP64
one (the chain is rejected), never NaN (which the accept test lets through).  Bound as for ordinary
coefficients: k 2^-24 of Σ |c̃_a| Σ_b |G_ab c̃_b|, and a coefficient that is not finite stays not finite."""
import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.device import ptr, stream_handle

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 9, 64, 96])
@pytest.mark.parametrize("amp", [1e16, 1e18, 1e19])
def test_llk_beyond_fp32(cuda, k, amp):
    n = 200
    rng = np.random.default_rng(k)
    f32 = lambda a: dev(a, dtype=torch.float32)
    x = rng.normal(size=(n, k))
    x[::2] *= amp                                        # ordinary chains between them
    c, scale, h = f32(x), f32(rng.uniform(0.5, 2, k)), f32(rng.normal(size=k))
    A = rng.normal(size=(k, 400))
    G = f32(A @ A.T)
    llk = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    args = [ptr(scale), ptr(G), ptr(h), 3.5, -2.0, ptr(llk), stream_handle()]
    _native.call("ag_surrogate_llk", n, k, ptr(c), *args)
    cs = (c * scale).double()
    ref = -2.0 - 0.5 * (3.5 - 2.0 * cs @ h.double() + ((cs @ G.double().T) * cs).sum(1))
    bound = k * 2.0 ** -24 * ((cs.abs() @ G.double().abs().T) * cs.abs()).sum(1) + 1e-12
    assert bool(((llk - ref).abs() <= bound).all())
    c[3, k - 1], c[4, 0] = float("nan"), float("inf")
    _native.call("ag_surrogate_llk", n, k, ptr(c), *args)
    assert not bool(torch.isfinite(llk[3:5]).any()) and bool(torch.isfinite(llk[5:]).all())
