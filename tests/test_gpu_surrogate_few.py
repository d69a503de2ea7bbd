"""The surrogate log-likelihood of few chains: two chains per thread up to 64 per SM, eight beyond.

A chain's log-likelihood is the same bits in calls of every size (the same sums in the same order),
around both tiles (32 and 128 chains) and the number of chains where the launch changes.  And few chains do not
wait for a tile made for many: 1,000 x 64 took 10.4 µs with a warp per chain and 13.4 in tiles of 128."""
import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.device import ptr, stream_handle

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


def _problem(n, k):
    rng = np.random.default_rng(k)
    f32 = lambda a: dev(a, dtype=torch.float32)
    A = rng.normal(size=(k, k + 3))
    c, rest = f32(rng.normal(size=(n, k))), [f32(rng.uniform(0.5, 2, k)), f32(A @ A.T), f32(rng.normal(size=k))]

    def run(first, count, out):
        rows = c[first:first + count].contiguous()
        _native.call("ag_surrogate_llk", count, k, ptr(rows), *[ptr(t) for t in rest], 3.5, -2.0, ptr(out),
                     stream_handle())
        return out
    return run


@pytest.mark.parametrize("k", [1, 8, 9, 64, 96])
def test_few_and_many_keep_the_bits(cuda, k):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 64 * sms + 200
    run = _problem(n, k)
    whole = run(0, n, torch.full((n,), np.nan, dtype=torch.float64, device="cuda"))
    assert bool(torch.isfinite(whole).all())
    for first, count in ((0, 1), (3, 31), (0, 32), (64, 33), (7, 1000), (1, 64 * sms), (1, 64 * sms + 1)):
        got = run(first, count, torch.full((count,), np.nan, dtype=torch.float64, device="cuda"))
        assert torch.equal(got, whole[first:first + count])


@pytest.mark.parametrize("n,k,limit", [(1000, 64, 10.4), (250, 96, 16.7)])
def test_few_chains_time(cuda, n, k, limit):
    run = _problem(n, k)
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    graph = torch.cuda.CUDAGraph()                        # the kernels alone, without the host's pace
    run(0, n, out)
    with torch.cuda.graph(graph):
        for _ in range(40):
            run(0, n, out)
    times = []
    for _ in range(10):
        a.record()
        graph.replay()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 1e3 / 40)
    assert min(times) < limit, times
