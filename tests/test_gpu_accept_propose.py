"""The accept of one step with the proposal and floor of the next, in one launch: bit for bit what the
three calls in a row give, for blocks of 32 chains with and without a rest, odd and even numbers of
parameters, the most that a block takes and one more, masked chains, and a launch without floors."""
import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian.coolingstep import StageState
from altar_gb300.device import ptr, stream_handle

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 6, 11, 32, 33])
@pytest.mark.parametrize("n", [1, 31, 33, 1000])
@pytest.mark.parametrize("floors", [False, True])
@pytest.mark.parametrize("beta", [0.0, 0.3])
def test_one_launch_equals_three(cuda, p, n, floors, beta):
    rng = np.random.default_rng(100 * p + n)
    seed, step, s = 77, 4, stream_handle()
    lo, hi = dev(np.full(p, -1.0)), dev(np.full(p, 1.5))
    L = np.linalg.cholesky(np.eye(p) + 0.1) * 0.25
    start = dict(theta=rng.uniform(-0.9, 1.4, (n, p)), prior=np.full(n, -0.5), data=rng.normal(-10, 3, n),
                 post=rng.normal(-4, 2, n), cand=rng.uniform(-1, 1.5, (n, p)), cprior=np.full(n, -0.25),
                 cdata=rng.normal(-10, 4, n))
    mask0 = (rng.random(n) < 0.3).astype(np.int32)
    results = []
    for fused in (False, True):
        st = StageState(n, p)
        st.chol.copy_(dev(L))
        st.epoch.fill_(5)
        st.beta.fill_(beta)
        t = {k: dev(v) for k, v in start.items()}
        mask = torch.tensor(mask0, device="cuda")
        floor = torch.full((n,), 9.0, dtype=torch.float64, device="cuda")
        if fused:
            _native.call("ag_accept_propose", st.struct, n, p, ptr(lo), ptr(hi), seed, step, ptr(mask), ptr(t["cand"]),
                         ptr(t["cprior"]), ptr(t["cdata"]), ptr(t["theta"]), ptr(t["prior"]), ptr(t["data"]),
                         ptr(t["post"]), ptr(floor) if floors else None, s)
        else:
            _native.call("ag_accept", st.struct, n, p, seed, step, ptr(mask), ptr(t["cand"]), ptr(t["cprior"]),
                         ptr(t["cdata"]), ptr(t["theta"]), ptr(t["prior"]), ptr(t["data"]), ptr(t["post"]), s)
            _native.call("ag_propose", st.struct, ptr(t["theta"]), n, p, ptr(lo), ptr(hi), seed, step + 1,
                         ptr(t["cand"]), ptr(mask), ptr(t["cprior"]), s)
            if floors:
                _native.call("ag_accept_floor", st.struct, n, seed, step + 1, ptr(mask), ptr(t["cprior"]),
                             ptr(t["post"]), ptr(floor), s)
        torch.cuda.synchronize()
        results.append({**t, "mask": mask, "floor": floor, "counters": st.counters.clone()})
    for k, v in results[0].items():
        assert torch.equal(v, results[1][k]), k
    assert int(results[0]["counters"].sum()) == n
