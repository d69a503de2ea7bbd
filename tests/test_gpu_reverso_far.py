"""The Reverso likelihood with a point so far away that its squared distance is infinite in FP64.

The displacement there is 0, so that a point of zero data adds nothing, and never NaN."""
import numpy as np
import pytest
import torch

from oracle import reverso

from test_gpu_reverso import PRIORS, _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e150, 1e160, 1e300])
@pytest.mark.parametrize("points", [1, 35, 130])
def test_far_point_adds_nothing(cuda, far, points):
    rng = np.random.default_rng(points)
    n = 300
    txy = np.stack([10.0 ** rng.uniform(1, 7.5, points), rng.uniform(-5e3, 5e3, points),
                    rng.uniform(-5e3, 5e3, points)], 1)
    d, var = rng.normal(0, 0.02, (points, 3)), np.full((points, 3), 1e-4)
    theta = torch.from_numpy(np.stack([rng.uniform(lo, hi, n) for lo, hi in PRIORS], 1)).cuda()
    d[0] = 0.0
    txy[0, 1:] = far
    with_far = _model(txy, d, var, "fast")
    u = with_far.displacements(theta).cpu().numpy().reshape(n, points, 3)
    assert np.all(u[:, 0] == 0.0) and np.isfinite(u).all()
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    with_far.forward(theta, out)
    ref = -0.5 * np.sum((u - d) ** 2 / 1e-4, axis=(1, 2))
    ref += reverso.normalization(var)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=1e-11, atol=1e-9)
