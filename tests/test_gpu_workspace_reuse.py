"""A strategy's workspace, made for its largest population, serves every smaller call in place.

The CDM's split launch (up to 3,072 chains) keeps counters and partial misfits that larger calls do not use:
a workspace for 3,100 chains has them all the same, the buffer stays where captured graphs expect
it, and the log-likelihoods are those of a workspace made for the call."""
import numpy as np
import pytest
import torch

from altar_gb300 import _native

from gpu_helpers import LOS, cdm_prior_rows, cdm_strategy, dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large", [3073, 3100, 3364])
def test_smaller_call_in_a_larger_workspace(cuda, large):
    rng = np.random.default_rng(large)
    m = 300
    X, Y = rng.uniform(-2e4, 2e4, m), rng.uniform(-2e4, 2e4, m)
    args = (X, Y, np.tile(LOS, (m, 1)), rng.normal(0, 3e-3, m), np.full(m, 9e-6))
    rows = dev(cdm_prior_rows(64, seed=large)[np.arange(large) % 64])
    strat, _ = cdm_strategy(*args)
    strat.reserve(large)
    address = strat._ws.data_ptr()
    for n in (large, 3072, 3000, 2806, 17):
        fresh, _ = cdm_strategy(*args)
        got, want = (torch.full((n,), np.nan, dtype=torch.float64, device="cuda") for _ in "ab")
        strat.forward(rows[:n], got)
        fresh.forward(rows[:n], want)
        assert strat._ws.data_ptr() == address
        assert bool(torch.isfinite(want).all()) and torch.equal(got, want)
        assert _native.load().ag_forward_workspace_bytes(_native.AG_MODEL_CDM, n) <= strat._ws_bytes
