"""FP64 linear likelihood where its work division changes: fewer chains than a group of eight, groups
for 1 to 8 CTAs each, several CTAs per SM, observations that are no multiple of a round or fewer than
the CTAs, the smallest products and more parameters than the staged kernel holds.

Tolerance, from FP64 rounding alone (u = 2^-53): a residual is off by at most e = (p + 2) u (Σ|a θ| + |b|),
the sum of squares by Σ(2|ρ| e + e²) and, added in any order of m terms, by (m + 1) u Σρ²; the
result by u (|norm| + |llk|).  The reference is off by as much at most: twice the sum."""

import ctypes

import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.device import ptr, stream_handle

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 9, 305, 1000, 1217, 2003, 4900])
@pytest.mark.parametrize("m,p", [(1, 1), (31, 5), (37, 11), (33, 61), (997, 61), (96, 128), (40, 600), (20, 601)])
def test_exact_likelihood(cuda, n, m, p):
    rng = np.random.default_rng(n + 7 * m)
    A, b, theta = rng.normal(size=(m, p)), rng.normal(size=m), rng.normal(size=(n, p))
    Ad, bd, td = dev(A), dev(b), dev(theta)
    model = _native.LinearModel(ptr(Ad), ptr(bd), None, m, p)
    llk = torch.full((n + 8,), 3.0, dtype=torch.float64, device="cuda")
    _native.call("ag_linear_llk_fp64", ctypes.byref(model), ptr(td), n, -12.5, ptr(llk), stream_handle())
    torch.cuda.synchronize()
    rho = theta @ A.T - b
    ref = -12.5 - 0.5 * (rho ** 2).sum(axis=1)
    u = 2.0 ** -53
    e = (p + 2) * u * (np.abs(theta) @ np.abs(A.T) + np.abs(b))
    off = 0.5 * ((2 * np.abs(rho) * e + e ** 2).sum(axis=1) + (m + 1) * u * (rho ** 2).sum(axis=1)) \
        + u * (12.5 + np.abs(ref))
    got = llk.cpu().numpy()
    assert np.all(np.abs(got[:n] - ref) <= 2 * off)
    assert np.all(got[n:] == 3.0)
