"""The Mogi likelihood's misfit sums against FP64 sums of the residual rows it writes.

Each of 256 lanes adds w r² of its stations in float-float, then the lanes are added as exactly as FP64
does.  With w a power of two:
* 256 stations: a lane's one term, the square of an FP32 number, is exact in two FP32 parts, and an
  FP64 summation over the lanes takes at most 5 additions in the warp and 8 over the warps:
  13 units of 2^-53 relative.
* 4,096 stations per lane: an addition of float-float leaves at most 2^-46 of the sum (a unit of the
  low part's last place for each of its three rounded additions), 4,096 of them 2^-34 = 5.8e-11; equal
  small terms behind a large one leave the same rounding error in each addition, which a sum
  that does not carry the low parts' own errors collects to 1e-9."""
import numpy as np
import pytest
import torch

from gpu_helpers import dev, mogi_strategy

pytestmark = pytest.mark.gpu


def _misfits(X, Y, d, theta, variant, nsources=1):
    m = X.size
    strat, _ = mogi_strategy(X, Y, np.tile([0.38, -0.08, 0.92], (m, 1)), d, np.full(m, 2.0 ** -15), log_strength=True,
                             nparams=theta.shape[1], nsources=nsources, stride=4 if nsources > 1 else 0)
    strat.norm = 0.0
    strat.layout.variant = variant
    out = torch.empty(theta.shape[0], dtype=torch.float64, device="cuda")
    res = torch.zeros(theta.shape[0], strat.stations.m_padded, device="cuda")
    strat.forward(dev(theta), out, residuals=res)
    r = res[:, :m].double().cpu().numpy().astype(np.longdouble)
    ref = -0.5 * 2.0 ** 15 * (r * r).sum(1)
    return np.abs((out.cpu().numpy() - ref) / ref).astype(np.float64)


def _theta(n, rng):
    return np.stack([rng.uniform(-1e4, 1e4, n), rng.uniform(-1e4, 1e4, n), rng.uniform(1e3, 8e3, n),
                     rng.uniform(5, 7, n)], 1)


@pytest.mark.parametrize("n,variant", [(64, 0), (3001, 0), (5000, 0), (100, 1), (100, 2)])
@pytest.mark.parametrize("nsources", [1, 2])
def test_lanes_add_as_fp64(cuda, n, variant, nsources):
    rng = np.random.default_rng(n + variant)
    X, Y = rng.uniform(-2e4, 2e4, 256), rng.uniform(-2e4, 2e4, 256)
    th = _theta(n, rng)
    err = _misfits(X, Y, rng.normal(0, 5e-3, 256), np.concatenate([th] * nsources, 1), variant, nsources)
    assert err.max() <= 13 * 2.0 ** -53


@pytest.mark.parametrize("variant", [0, 1, 2])
def test_many_equal_terms(cuda, variant):
    rng = np.random.default_rng(7)
    m = 4096 * 256
    d = np.full(m, 7e-3)
    d[:256] = 40.0                                     # a lane's first term: 1 / 3e7 of it is each other
    err = _misfits(np.full(m, 3e3), np.full(m, -2e3), d, _theta(64, rng), variant)
    assert err.max() <= 2.0 ** -34


def test_sum_beyond_fp32(cuda):
    """Every lane's sum is an FP32 number, the 256 of them together are not."""
    rng = np.random.default_rng(1)
    X, Y = rng.uniform(-2e4, 2e4, 256), rng.uniform(-2e4, 2e4, 256)
    err = _misfits(X, Y, np.full(256, 1e17), _theta(8, rng), 0)      # w r² = 3.3e38, Σ = 8.4e40
    assert err.max() <= 13 * 2.0 ** -53
