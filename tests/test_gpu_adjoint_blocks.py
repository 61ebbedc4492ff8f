"""The adjoint's passes at the edges of their 32 x 8 blocks: rasters one cell
smaller and larger than a block, and long boundary tables, against directional
derivatives of the frozen-dt forward."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# raster sizes include the one-cell no-data ring
@pytest.mark.parametrize("rows,cols", [(6, 30), (8, 32), (7, 31), (9, 33), (14, 66)])
def test_gradients_match_differences(cuda, rows, cols):
    from hipims_b200 import scenarios as S
    from hipims_b200.adjoint import GaugeMisfit

    rng = np.random.default_rng(100 * rows + cols)
    mask = np.full((rows, cols), 1, dtype=np.int32)
    mask[0, :] = mask[-1, :] = mask[:, 0] = mask[:, -1] = -9999
    mask[1, 1:-1], mask[-2, 1:-1], mask[2:-2, 1], mask[2:-2, -2] = 60, 50, 70, 40
    valid = mask > 0
    t = np.arange(70) * 0.05
    w = np.sin(np.arange(70))
    d = dict(mask=mask, z=np.where(valid, 0.2 * rng.uniform(0, 1, mask.shape), 0.0),
             h=np.where(valid, 0.4 + 0.1 * rng.uniform(0, 1, mask.shape), 0.0),
             qx=np.where(valid, 0.1 + 0.05 * rng.standard_normal(mask.shape), 0.0),
             qy=np.where(valid, -0.05 + 0.05 * rng.standard_normal(mask.shape), 0.0),
             landuse=rng.integers(0, 16, mask.shape).astype(np.uint8),
             manning=list(rng.uniform(0.03, 0.1, 16)), dx=2.0, cfl=0.5, first_dt=0.1,
             rain=np.array([[0.0, 1e-5], [100.0, 1e-5]]),
             given_depth=np.stack([t, 0.45 + 0.02 * w], 1),
             given_q=np.stack([t, 0.1 + 0.02 * w, 0.02 * w], 1), t_end=math.inf)
    rr, cc = np.nonzero(valid)
    pick = rng.choice(rr.size, size=min(6, rr.size), replace=False)
    nsteps = 20
    p = GaugeMisfit(S.catchment_from(d), rr[pick], cc[pick], nsteps, np.full(nsteps, 0.05),
                    every=5, checkpoint=7, obs=np.zeros((4, pick.size)), device=cuda)
    n0, eps = np.asarray(d["manning"]), 1e-5

    def J(n, r):
        return float(p.loss(p.simulate(list(n), r)))

    J(n0, 1.0)
    g = p.gradient()
    # a random direction through all zones, and the rain multiplier: central
    # differences with a relative step of 1e-5, to the 1e-4 of the largest
    # derivative that such quotients resolve on wet states
    v = rng.uniform(0.5, 1.0, 16) * n0
    fd = (J(n0 + eps * v, 1.0) - J(n0 - eps * v, 1.0)) / (2 * eps)
    fr = (J(n0, 1.0 + eps) - J(n0, 1.0 - eps)) / (2 * eps)
    scale = max(abs(fd), abs(fr))
    assert abs(float(g[:16] @ v) - fd) < 1e-4 * scale
    assert abs(float(g[16]) - fr) < 1e-4 * scale
