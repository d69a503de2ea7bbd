"""The Mogi likelihood's chains per CTA: the default takes 4, 8 or 16 by the number of chains.

A chain's log-likelihood and residuals are the same bits in calls of every size and launch variant (a
population may be split across ranks), for one and two sources, with and without dataset offsets,
odd numbers of chains and stations, and chains left out by the mask."""
import numpy as np
import pytest
import torch

from gpu_helpers import dev, mogi_strategy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 257, 1000])
@pytest.mark.parametrize("nsources,datasets", [(1, 0), (1, 3), (2, 0)])
def test_chains_per_cta_keep_the_bits(cuda, m, nsources, datasets):
    rng = np.random.default_rng(m + 10 * nsources + datasets)
    X, Y = rng.uniform(-25e3, 25e3, m), rng.uniform(-25e3, 25e3, m)
    los = np.tile([0.38, -0.08, 0.92], (m, 1))
    n = 6001
    cols = [rng.uniform(-1e4, 1e4, n), rng.uniform(-1e4, 1e4, n), rng.uniform(1e3, 8e3, n), rng.uniform(5, 7, n)]
    theta = np.stack(cols * nsources + [rng.normal(0, 0.01, n) for _ in range(datasets)], 1)
    oid = rng.integers(0, datasets, m) if datasets else None
    strat, _ = mogi_strategy(X, Y, los, rng.normal(0, 5e-3, m), np.full(m, 2.5e-5), log_strength=True,
                             nparams=theta.shape[1], nsources=nsources, stride=4 if nsources > 1 else 0, oid=oid,
                             offset_idx=4 * nsources if datasets else -1)
    th = dev(theta)

    def run(rows, variant=0, mask=None):
        strat.layout.variant = variant
        out = torch.full((rows.shape[0],), 7.0, dtype=torch.float64, device="cuda")
        res = torch.zeros(rows.shape[0], strat.stations.m_padded, device="cuda")
        strat.forward(rows.contiguous(), out, residuals=res, mask=mask)
        return out, res

    whole, res = run(th)
    assert bool(torch.isfinite(whole).all())
    for first, count in ((0, 1), (5, 3), (100, 2431), (1, 2500), (17, 4865)):
        out, r = run(th[first:first + count])
        assert torch.equal(out, whole[first:first + count]) and torch.equal(r, res[first:first + count])
    for variant in (1, 2):
        out, r = run(th[:999], variant)
        assert torch.equal(out, whole[:999]) and torch.equal(r, res[:999])
    mask = torch.zeros(999, dtype=torch.int32, device="cuda")
    mask[::4] = 1
    out, _ = run(th[:999], mask=mask)
    assert torch.equal(out[mask == 0], whole[:999][mask == 0]) and bool((out[mask != 0] == 7.0).all())
