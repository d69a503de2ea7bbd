"""The δβ search where its median and Brent's launch change, against the oracle.

Median: up to 128 keys are ranked against each other, more are first narrowed to one bucket by counting.
Brent: up to 4,096 chains (two points of four chunks) the blocks are one cluster, one to eight of them, more
meet at the grid's barrier.  The median exactly; Brent as its own test: δβ within 1e-8 relative, COV within
1e-6, and a second call in the same workspace with the same bits."""
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
        return np.round(rng.normal(-30.0, 3.0, n))
    if kind == "outlier":                        # one bucket takes nearly all keys, again and again
        llk = rng.normal(-500.0, 20.0, n)
        llk[rng.integers(n)] = -1e300
        return llk
    if kind == "signs":
        return rng.normal(0.0, 1.0, n) * 10.0 ** rng.integers(-300, 3, n)
    return np.full(n, -7.25)


@pytest.mark.parametrize("kind", ["normal", "ties", "outlier", "signs", "equal"])
@pytest.mark.parametrize("n", [126, 127, 128, 129, 130, 255, 256, 257, 258, 1023, 1024])
def test_median(cuda, kind, n):
    llk = _llk(kind, n, np.random.default_rng(n))
    st = StageState(n, 1)
    ws = workspace(_native.load().ag_cov_workspace_bytes(n))
    dllk = dev(llk)
    _native.call("ag_cov_schedule", st.struct, ptr(dllk), n, 1.0, 0.01, ptr(ws), ws.numel(), stream_handle())
    torch.cuda.synchronize()
    # the first word of the schedule's state
    assert ws[:8].view(torch.float64).item() == np.median(llk)


@pytest.mark.parametrize("n", [2, 1023, 1024, 1025, 2048, 2049, 3073, 4096, 4097])
def test_brent(cuda, n):
    llk = np.random.default_rng(3 * n).normal(-3e4, 1e3, n)
    _, db_ref, cov_ref, w_ref = catmip.dbeta_brent(llk, 0.0, 1.0, 0.01, 1000)
    ws = workspace(_native.load().ag_cov_workspace_bytes(n))
    dllk = dev(llk)
    got = []
    for _ in range(2):
        st = StageState(n, 1)
        _native.call("ag_cov_schedule_brent", st.struct, ptr(dllk), n, 1.0, 0.01, 1000, ptr(ws), ws.numel(),
                     stream_handle())
        torch.cuda.synchronize()
        _, db, cov = st.scalars.cpu().numpy()[:3]
        assert abs(db - db_ref) <= 1e-8 * abs(db_ref) and abs(cov - cov_ref) <= 1e-6 * max(1.0, cov_ref)
        np.testing.assert_allclose(st.w.cpu().numpy(), w_ref, rtol=1e-6, atol=1e-300)
        assert int(st.flags.item()) == 0
        got.append(torch.cat([st.scalars, st.w]))
    assert torch.equal(got[0], got[1])
