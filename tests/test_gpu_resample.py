"""The resampling's parallel partial sums and ranks where they change regime.

The edges must equal the sequential FP64 accumulation bit for bit (numpy's add.accumulate),
whatever the weights do to the running sum: many binades, ties between two representable sums,
zeros, subnormals, weights that dwarf the sum, non-finite ones.  Ranks must follow decreasing
count with ties by index on both sides of the kernel's chunk and of its small-count limit.
"""
import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian.coolingstep import StageState
from altar_gb300.device import ptr, stream_handle, workspace
from oracle import catmip, philox

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


def _weights(kind, n, rng):
    u = rng.random(n)
    if kind == "uniform":
        return u / u.sum()
    if kind == "equal":
        return np.full(n, 1.0 / n)
    if kind == "ties":
        return np.ldexp(rng.integers(0, 4096, n).astype(np.float64), -40) + np.ldexp(1.0, -30)
    if kind == "wide":
        return np.exp(-700.0 * u)
    if kind == "subnormal":
        return np.ldexp(u, -1074 + rng.integers(0, 60, n))
    if kind == "few":
        return np.where(u < 1e-3, u, 0.0)
    return np.where(u < 0.01, np.where(u < 0.005, -u, np.nan), u)


def _resample(w, seed=5, offset=0):
    n = w.size
    st = StageState(n, 1)
    st.w.copy_(dev(w))
    st.beta.fill_(0.5)
    z = lambda: torch.zeros(n, dtype=torch.float64, device="cuda")
    index = dev(np.arange(n, dtype=np.float64))
    out = z()
    counts = torch.zeros(n + 1, dtype=torch.int32, device="cuda")[offset:offset + n]
    ws = workspace(_native.load().ag_resample_workspace_bytes(n))
    _native.call("ag_resample", st.struct, n, 1, seed, ptr(index), ptr(z()), ptr(z()), ptr(out), ptr(z()), ptr(z()),
                 ptr(z()), ptr(counts), ptr(ws), ws.numel(), stream_handle())
    torch.cuda.synchronize()
    # the edges follow the 256-byte header of the workspace
    edges = ws[256:256 + 8 * (n + 1)].view(torch.float64).cpu().numpy()
    return edges, counts.cpu().numpy(), out.cpu().numpy()


@pytest.mark.parametrize("kind", ["uniform", "equal", "ties", "wide", "subnormal", "few", "bad"])
@pytest.mark.parametrize("n", [1, 63, 65, 4160, 4161, 40000])
def test_edges_equal_the_sequential_sum(cuda, kind, n):
    w = _weights(kind, n, np.random.default_rng(n))
    edges, _, _ = _resample(w)
    ref = np.concatenate([[0.0], np.add.accumulate(w)])
    np.testing.assert_array_equal(edges, ref)


@pytest.mark.parametrize("n", [31, 1024, 32767, 32769, 70001])
@pytest.mark.parametrize("heavy", [0.0, 0.3])
def test_ranks_across_chunks_and_large_counts(cuda, n, heavy):
    rng = np.random.default_rng(n)
    w = rng.gamma(0.2, size=n)
    if heavy:                                    # a few chains take most of the copies, many of them tied
        w[rng.random(n) < 40.0 / n] = w.sum() * heavy / 40.0
    w /= w.sum()
    # an odd offset: the caller's counts need not be 16-byte aligned
    _, counts, order = _resample(w, offset=int(heavy > 0))
    c_ref = catmip.multiplicities(w, philox.resample_uniforms(5, n, 0))
    assert np.array_equal(counts, c_ref)
    assert np.array_equal(order.astype(np.int64), catmip.rank_order(c_ref))
