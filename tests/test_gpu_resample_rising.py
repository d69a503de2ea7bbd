"""The resampling's partial sums for weights that rise over many decades.

Every few additions leave the running sum's binade, so the scan alternates with stretches of additions in a
row: the edges still equal the sequential accumulation bit for bit, in the warp's part (the first
1,024 weights) and the block's, where the rise ends and the tiles come back, and with a sum that
stops being finite.  And such weights do not restart a tile at each binade: 4,096 of them over 260
decades took 334 µs with all additions in a row and 2.6 ms with a tile per restart."""
import numpy as np
import pytest
import torch

from altar_gb300 import _native
from altar_gb300.bayesian.coolingstep import StageState
from altar_gb300.device import ptr, stream_handle, workspace

from gpu_helpers import dev

pytestmark = pytest.mark.gpu


class _Resample:
    def __init__(self, w):
        self.n = n = w.size
        self.st = StageState(n, 1)
        self.st.w.copy_(dev(w))
        self.arrays = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(7)]
        self.ws = workspace(_native.load().ag_resample_workspace_bytes(n))

    def __call__(self):
        _native.call("ag_resample", self.st.struct, self.n, 1, 5, *[ptr(a) for a in self.arrays], None, ptr(self.ws),
                     self.ws.numel(), stream_handle())

    def edges(self):
        self()
        torch.cuda.synchronize()
        return self.ws[256:256 + 8 * (self.n + 1)].view(torch.float64).cpu().numpy()   # behind the header


def _weights(kind, n, binades):
    rng = np.random.default_rng(n)
    i = np.arange(n)
    if kind == "rising":
        x = np.minimum(i * binades, 2000.0)
    elif kind == "teeth":                        # up to 900 weights at a time, every tooth above the last
        x = np.minimum((i % 900) * binades, 900.0) + 300.0 * (i // 900)
    elif kind == "late":                         # flat, then rising
        x = np.maximum(i - n // 2, 0) * binades
    else:                                        # past the largest double: inf, then NaN
        x = i * binades + 1000.0
    w = np.ldexp(rng.uniform(1.0, 2.0, n), (np.minimum(x, 2095.0) - 1072.0).astype(int))
    if kind == "overflow":
        w[n // 2], w[n // 2 + n // 4] = np.inf, np.nan
    return w


@pytest.mark.parametrize("kind", ["rising", "teeth", "late", "overflow"])
@pytest.mark.parametrize("binades", [0.01, 0.07, 0.5, 3.0])
@pytest.mark.parametrize("n", [17, 33, 1000, 1025, 1120, 4200, 30000])
def test_edges_of_rising_weights(cuda, kind, binades, n):
    w = _weights(kind, n, binades)
    with np.errstate(over="ignore", invalid="ignore"):
        ref = np.concatenate([[0.0], np.add.accumulate(w)])
    np.testing.assert_array_equal(_Resample(w).edges(), ref)


@pytest.mark.parametrize("n,limit", [(1000, 500.0), (4096, 1000.0)])
def test_rising_weights_time(cuda, n, limit):
    run = _Resample(np.exp(np.linspace(-600.0, 0.0, n)))
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(10):
        a.record()
        run()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 1e3)
    assert min(times) < limit, times
