"""The δβ search and its median where their partitions change, against the oracle's grid solver.

Block and chunk edges (256 chains per block, 152 blocks, 1,024 chains per chunk, 1,024 keys
ranked directly by the median), log-likelihoods with ties, with one outlier, over many
decades, and all equal.  β and δβ to 1e-12 relative and the weights to 1e-10, as the schedule's own tests.
"""
import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian.coolingstep import StageState
from altar_gb300.device import ptr, stream_handle, workspace
from oracle import catmip

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


def _llk(kind, n, rng):
    if kind == "normal":
        return rng.normal(-3e4, 1e3, n)
    if kind == "ties":
        return np.round(rng.normal(-300.0, 40.0, n))
    if kind == "outlier":
        llk = rng.normal(-500.0, 20.0, n)
        llk[rng.integers(n)] = -1e300
        return llk
    if kind == "decades":
        return -np.exp(rng.uniform(-3.0, 16.0, n))
    return np.full(n, -7.25)


@pytest.mark.parametrize("kind", ["normal", "ties", "outlier", "decades", "equal"])
@pytest.mark.parametrize("n", [2, 3, 255, 257, 1025, 4096, 38912, 38913, 60001])
def test_grid_schedule_partitions(cuda, kind, n):
    llk = _llk(kind, n, np.random.default_rng(n))
    st = StageState(n, 1)
    ws = workspace(_native.load().ag_cov_workspace_bytes(n))
    dllk = dev(llk)
    _native.call("ag_cov_schedule", st.struct, ptr(dllk), n, 1.0, 0.01, ptr(ws), ws.numel(), stream_handle())
    torch.cuda.synchronize()
    b_ref, db_ref, cov_ref, w_ref = catmip.dbeta_grid(llk, 0.0, 1.0, 0.01)
    # the median is the first word of the schedule's state
    assert ws[:8].view(torch.float64).item() == np.median(llk)
    b, db, cov = st.scalars.cpu().numpy()[:3]
    assert abs(db - db_ref) <= 1e-12 * abs(db_ref) and abs(b - b_ref) <= 1e-12
    assert abs(cov - cov_ref) <= 1e-9 * max(1.0, cov_ref)
    np.testing.assert_allclose(st.w.cpu().numpy(), w_ref, rtol=1e-10, atol=1e-300)


@pytest.mark.parametrize("kind", ["normal", "ties"])
@pytest.mark.parametrize("n", [2, 128, 129, 897, 1024, 1025, 2048, 2049])
def test_grid_schedule_in_a_cluster(cuda, kind, n):
    """One to eight blocks of one cluster (128 chains per block, then 256), and the first size beyond;
    the bounds of the test above, twice in the same workspace."""
    llk = _llk(kind, n, np.random.default_rng(7 * n))
    b_ref, db_ref, _, w_ref = catmip.dbeta_grid(llk, 0.0, 1.0, 0.01)
    ws = workspace(_native.load().ag_cov_workspace_bytes(n))
    dllk = dev(llk)
    for _ in range(2):
        st = StageState(n, 1)
        _native.call("ag_cov_schedule", st.struct, ptr(dllk), n, 1.0, 0.01, ptr(ws), ws.numel(), stream_handle())
        torch.cuda.synchronize()
        b, db, _ = st.scalars.cpu().numpy()[:3]
        assert abs(db - db_ref) <= 1e-12 * abs(db_ref) and abs(b - b_ref) <= 1e-12
        np.testing.assert_allclose(st.w.cpu().numpy(), w_ref, rtol=1e-10, atol=1e-300)
        assert int(st.flags.item()) == 0


@pytest.mark.parametrize("p", [1, 2, 10, 21, 22, 33])
@pytest.mark.parametrize("n", [1, 16, 17, 2433, 39000])
def test_weighted_cov_partitions(cuda, p, n):
    """Σ where its partition changes: one to many groups of threads per block (22 parameters on, a
    thread takes several entries), fewer chains than a block's, several chunks per block."""
    rng = np.random.default_rng(100 * n + p)
    theta = rng.normal(size=(n, p)) * np.logspace(0, 2, p) + 5.0
    w = rng.random(n) + 1e-3
    w /= w.sum()
    st = StageState(n, p)
    st.w.copy_(dev(w))
    ws = workspace(_native.load().ag_sigma_workspace_bytes(n, p))
    dth = dev(theta)
    _native.call("ag_weighted_cov", st.struct, ptr(dth), n, p, ptr(ws), ws.numel(), stream_handle())
    torch.cuda.synchronize()
    # E[θθ] and the mean's square cancel: the bound is relative to the moments, not to their difference
    np.testing.assert_allclose(st.sigma.cpu().numpy(), catmip.weighted_cov(theta, w), rtol=0,
                               atol=1e-13 * np.max(theta ** 2))
