"""Cell-wise collision of device batches around the sizes of its 128-cell
tiles and 64-thread halves, against the oracle, with values past the batch
left alone."""
import numpy as np
import pytest
import torch

import lbm3_b200 as L
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 191, 193, 1000])
@pytest.mark.parametrize("limiter", [0.0, 0.05, 1e-39])
def test_matches_oracle_and_stays_inside(n, limiter):
    """Tolerance: about ten roundings of single-precision values, relative to
    the largest population (the bar of the collision's own parity test)."""
    rng = np.random.default_rng(n)
    dRho = rng.uniform(-0.02, 0.02, n).astype(np.float32)
    u = rng.uniform(-0.06, 0.06, (3, n)).astype(np.float32)
    f = np.stack([O.feq(dRho[c], u[0, c], u[1, c], u[2, c]) for c in range(n)], axis=1)
    f = (f * (1 + 0.05 * rng.standard_normal(f.shape))).astype(np.float32)
    ref = O.apply_collision_batch(f, nu=0.02, limiter=limiter, g=(1e-5, -2e-5, 0.0))
    d = torch.full((27 * n + 256,), 7.0, device="cuda")
    d[128:128 + 27 * n] = torch.from_numpy(f).cuda().reshape(-1)
    L.apply_collision_batch(d.data_ptr() + 4 * 128, n, 0.02, limiter, 1.0, (1e-5, -2e-5, 0.0))
    torch.cuda.synchronize()
    got = d.cpu().numpy()
    assert np.all(got[:128] == 7.0) and np.all(got[128 + 27 * n:] == 7.0)
    assert np.max(np.abs(got[128:128 + 27 * n].reshape(27, n) - ref)) / np.abs(ref).max() < 2e-6
