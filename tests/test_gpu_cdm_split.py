"""The CDM likelihood with the stations of a chain split over CTAs (few chains, default launch).

A chain's log-likelihood, residuals, status and early rejection are the same bits whatever the
number of chains in the call: few (split over up to 32 CTAs), more than the split takes (one CTA
per chain, slots ordered by cost), and another launch variant.  Station counts around the tile
(128), the number of parts (32 tiles) and one tile more."""
import numpy as np
import pytest
import torch

from gpu_helpers import LOS, cdm_prior_rows, cdm_strategy, dev

pytestmark = pytest.mark.gpu


def _run(strat, theta, floor=None, residuals=False):
    n = theta.shape[0]
    out = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    status = torch.zeros(n, dtype=torch.int32, device="cuda")
    status[n // 2] = 1                                   # one proposal outside the support
    res = torch.zeros(n, strat.stations.m_padded, device="cuda") if residuals else None
    strat.forward(theta, out, mask=status, status=status, residuals=res, floor=floor)
    return [t.cpu().numpy() for t in (out, status)] + ([res.cpu().numpy()] if residuals else [])


@pytest.mark.parametrize("m", [1, 129, 577, 4096, 4097, 6000])
@pytest.mark.parametrize("n", [1, 9, 700])
def test_split_keeps_the_bits(cuda, m, n):
    rng = np.random.default_rng(m + n)
    X, Y = rng.uniform(-2e4, 2e4, m), rng.uniform(-2e4, 2e4, m)
    los = np.tile(LOS, (m, 1))
    rows = cdm_prior_rows(8, seed=m)
    rows = np.concatenate([rows, rows[:1]])
    rows[8, 2], rows[8, 4:7] = 200.0, 2000.0             # above the surface
    d = rng.normal(0, 3e-3, m)
    few = dev(rows[np.arange(n) % 9])
    many = dev(rows[np.arange(9000) % 9])
    base, _ = cdm_strategy(X, Y, los, d, np.full(m, 9e-6))
    other, _ = cdm_strategy(X, Y, los, d, np.full(m, 9e-6), variant=11)
    a, st_a, res = _run(base, few, residuals=True)
    b, st_b, res_b = _run(other, few, residuals=True)
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(st_a, st_b)
    np.testing.assert_array_equal(res, res_b)
    big, st_big = _run(base, many)
    keep = np.arange(n) != n // 2
    np.testing.assert_array_equal(a[keep], big[:n][keep])
    np.testing.assert_array_equal(st_a[keep], st_big[:n][keep])
    # early rejection: -inf exactly where the log-likelihood lies below its floor
    alive = (st_a == 0)
    if alive.any():
        floor = dev(np.where(np.arange(n) % 2 == 0, a * (1 - 1e-6) - 1.0, a * (1 + 1e-6) + 1.0))
        f, _ = _run(base, few, floor=floor)
        g, _ = _run(other, few, floor=floor)
        want = np.where(alive & (a < floor.cpu().numpy()), -np.inf, a)
        np.testing.assert_array_equal(f, want)
        np.testing.assert_array_equal(g, want)
