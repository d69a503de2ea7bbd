"""The weighted covariance where its launch changes, and its time at sizes on both sides.

Entries shared by groups of threads (up to 21 parameters) or several per thread, one chain to several blocks
of 16 and more rows, with the blocks' partial sums read 16 at a time: against longdouble sums, n 2^-52
of Σ w |θ_a θ_b| (each product and addition rounds once, Σ w = 1) and the same of the means' product.
With one thread per entry and 32 rows per block these sizes took 8.3 µs (two chains of one parameter),
1,343 (2,400 of 200) and 6,422 (1,000 of 512): the limits are those and a quarter, or the launch's own spread."""
import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian.coolingstep import StageState
from altar_gb300.device import ptr, stream_handle, workspace

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


def _sigma(n, p):
    rng = np.random.default_rng(100 * n + p)
    theta, w = rng.normal(0.5, 2.0, (n, p)), rng.uniform(0.1, 1.0, n)
    w /= w.sum()
    st = StageState(n, p)
    st.w.copy_(dev(w))
    th = dev(theta)
    ws = workspace(_native.load().ag_sigma_workspace_bytes(n, p))

    def run():
        _native.call("ag_weighted_cov", st.struct, ptr(th), n, p, ptr(ws), ws.numel(), stream_handle())
    return theta, w, st, run


@pytest.mark.parametrize("n", [1, 2, 15, 17, 33, 255, 2432, 2433, 5000])
@pytest.mark.parametrize("p", [1, 2, 15, 21, 22, 40])
def test_against_longdouble(cuda, n, p):
    theta, w, st, run = _sigma(n, p)
    run()
    t, v = theta.astype(np.longdouble), w.astype(np.longdouble)
    mean = (v @ t) / v.sum()
    ref = (v[:, None] * t).T @ t - np.outer(mean, mean)
    size = (v[:, None] * np.abs(t)).T @ np.abs(t) + np.outer(v @ np.abs(t), v @ np.abs(t))
    assert np.all(np.abs(st.sigma.cpu().numpy() - ref) <= (n + 8) * 2.0 ** -52 * size)


@pytest.mark.parametrize("n,p,limit", [(2, 1, 12.0), (16, 1, 12.0), (2400, 200, 1680.0), (1000, 512, 6422.0)])
def test_time(cuda, n, p, limit):
    _, _, _, run = _sigma(n, p)
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    graph = torch.cuda.CUDAGraph()
    run()
    reps = 20 if n <= 16 else 1
    with torch.cuda.graph(graph):
        for _ in range(reps):
            run()
    times = []
    for _ in range(10):
        a.record()
        graph.replay()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 1e3 / reps)
    assert min(times) < limit, times
