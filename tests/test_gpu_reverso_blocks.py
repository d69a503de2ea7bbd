"""The Reverso likelihood where its partition changes: samples per block and tiles of points.

For one sample, fewer samples than SMs, ragged blocks and several tiles of 128 points: the
displacements against the FP64 oracle within 1e-12 of each sample's largest (the bound of the model's
own tests), the log-likelihood bit for bit that of the same sample evaluated in calls of other
sizes (a population may be split across ranks), and masked samples left alone."""
import numpy as np
import pytest
import torch

from oracle import reverso

from test_gpu_reverso import MATERIAL, PRIORS, _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [1, 35, 128, 129, 300])
@pytest.mark.parametrize("samples", [1, 100, 152, 4097, 5000])
def test_partitions(cuda, points, samples):
    rng = np.random.default_rng(points + samples)
    txy = np.stack([10.0 ** rng.uniform(1, 7.5, points), rng.uniform(-5e3, 5e3, points),
                    rng.uniform(-5e3, 5e3, points)], 1)
    d, var = rng.normal(0, 0.02, (points, 3)), rng.uniform(1e-4, 1e-3, (points, 3))
    theta = np.stack([rng.uniform(lo, hi, samples) for lo, hi in PRIORS], 1)
    m = _model(txy, d, var, "fast")
    th = torch.from_numpy(theta).cuda()

    def llk(rows, mask=None):
        out = torch.full((rows.shape[0],), 7.0, dtype=torch.float64, device="cuda")
        m.forward(rows.contiguous(), out, mask=mask)
        return out

    u = m.displacements(th).cpu().numpy()
    ref = np.stack([reverso.displacements(t, txy, east_cos=True, **MATERIAL) for t in theta[:64]])
    big = np.abs(ref).max((1, 2), keepdims=True)
    assert np.all(np.abs(u[:64] - ref) <= 1e-12 * big)
    whole = llk(th)
    k = samples // 3
    assert torch.equal(llk(th[k:]), whole[k:])
    assert torch.equal(llk(th[-1:]), whole[-1:])
    mask = torch.zeros(samples, dtype=torch.int32, device="cuda")
    mask[::3] = 2
    part = llk(th, mask)
    assert torch.equal(part[mask == 0], whole[mask == 0]) and bool((part[mask != 0] == 7.0).all())
