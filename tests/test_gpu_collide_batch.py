"""Cell-wise collision of device batches around the sizes of its 128-cell
tiles and 64-thread halves, against the oracle, with values past the batch
left alone."""
import math

import numpy as np
import pytest
import torch

import lbm3_b200 as L
from lbm3_b200 import _abi as A
import oracle as O
from helpers import FIELD_REL_L2, density_velocity_errors

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


def _noisy(f, rng):
    return (f * (1 + 0.05 * rng.standard_normal(f.shape))).astype(np.float32)


@pytest.mark.parametrize("limiter", [1e30, 1e38, 3.4028234e38, math.inf])
def test_unlimited_batch(limiter):
    """Limiters that leave every cumulant's relaxation at omega3..5 (same tolerance)."""
    rng = np.random.default_rng(2)
    f = _noisy(np.stack([O.feq(*rng.uniform(-0.06, 0.06, 4)) for _ in range(130)], axis=1), rng)
    ref = O.apply_collision_batch(f, nu=0.02, limiter=limiter)
    d = torch.from_numpy(f).cuda()
    L.apply_collision_batch(d.data_ptr(), f.shape[1], 0.02, limiter)
    torch.cuda.synchronize()
    assert np.max(np.abs(d.cpu().numpy() - ref)) / np.abs(ref).max() < 2e-6


@pytest.mark.parametrize("storage", [A.LBM_STORE_F32, A.LBM_STORE_F64])
@pytest.mark.parametrize("make", [lambda s: L.periodic_box(10, 8, 6, ux=0.03, storage=s),
                                  lambda s: L.open_channel(16, 8, 8, storage=s)], ids=["box", "channel"])
@pytest.mark.parametrize("limiter", [3.4028234e38, math.inf])
def test_unlimited_steps(make, storage, limiter):
    """The same through the step's kernels, at the field parity bar."""
    c = make(storage)
    c.collision_limiter = limiter
    o = O.OracleGrid(c)
    f = _noisy(o.populations(), np.random.default_rng(4))
    o.set_populations(f)
    with L.build_grids(c) as g:
        g.set_populations(f)
        g.update_all_grids(3)
        o.step(3)
        e_rho, e_u, _ = density_velocity_errors(g.macro(), o.macro())
        assert e_rho < FIELD_REL_L2 and e_u < FIELD_REL_L2, (e_rho, e_u)
    o.close()
