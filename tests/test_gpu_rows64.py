"""The FP64 step kernel: its 8-, 16- and 32-row blocks equal bit for bit, and
equal to the oracle up to the round-off of faces evaluated from one side."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

WHOLE = 8  # HB_FLAG_WHOLE_TILES


def _solver(cs, cuda, whole=False, **kw):
    from hipims_b200 import _lib
    from hipims_b200.fused import FusedSolver

    fs = FusedSolver(cs, dtype=torch.float64, device=cuda, **kw)
    if whole:
        fs.batch.flags |= WHOLE
        fs.prepare()  # whole tiles fit in the larger workspace
    return fs


# rows around the blocks' heights, columns around the tile's; the last two are
# on either side of the 148 tiles up to which blocks have 8 rows
@pytest.mark.parametrize("shape", [(1, 33), (7, 31), (8, 32), (17, 65), (33, 40), (350, 400),
                                   (400, 400)])
@pytest.mark.parametrize("order", [1, 2])
def test_blocks_equal_whole_tiles_and_the_oracle(cuda, shape, order):
    from hipims_b200 import scenarios as S
    from oracle.oracle import Sim

    d = S.urban_catchment(shape[1], n_rows=shape[0], seed=shape[0], rain_mm_h=150.0)
    rng = np.random.default_rng(shape[1])
    valid = d["mask"] > 0
    d["h"] = np.where(valid, rng.uniform(0.2, 0.4, valid.shape), 0.0)
    d["z"] = np.where(valid, 0.002 * d["z"], 0.0)
    d["wl"] = d["z"] + d["h"]
    d["first_dt"] = 0.1
    c = S.catchment_from(d)
    a, b = _solver(c, cuda, order=order), _solver(c, cuda, whole=True, order=order)
    loop = _solver(c, cuda, order=order, grid_blocks=3)
    sim = Sim(d, order=order)
    sim.step(10)
    for s in (a, b, loop):
        s.step(10)
    x, ca = a.compacted(0), a.controls()[0]
    for other in (b, loop):
        y, cb = other.compacted(0), other.controls()[0]
        for f in x:
            np.testing.assert_array_equal(x[f], y[f], err_msg=f)
        assert (ca.t, ca.dt, ca.step, ca.status) == (cb.t, cb.dt, cb.step, cb.status)
        assert ca.volume == pytest.approx(cb.volume, rel=1e-12)
    for f in ("h", "qx", "qy", "h_max"):
        np.testing.assert_allclose(x[f], sim.state()[f], rtol=0, atol=1e-10, err_msg=f)
    assert ca.t == pytest.approx(sim.t, rel=1e-10)


def test_dry_cells_and_limiter_follow_the_oracle(cuda):
    """Dry beds, thin films, still water and supercritical cells (the limiter's
    branch) of a walled box with every dry / wet pairing at a face."""
    from hipims_b200 import scenarios as S
    from oracle.oracle import Sim

    d = S.dam_break(48)
    rng = np.random.default_rng(0)
    valid = d["mask"] > 0
    pick = rng.integers(0, 4, valid.shape)
    d["h"] = np.where(valid, np.choose(pick, [0.0, 5e-7, 2e-6, 0.3]), 0.0)
    d["z"] = np.where(valid, rng.uniform(0.0, 0.4, valid.shape), 0.0)
    fast = rng.uniform(-1.0, 1.0, valid.shape)
    d["qx"] = np.where(d["h"] > 1e-6, 4.0 * fast, 0.0)
    d["qy"] = np.where(d["h"] > 0.1, 6.0 * fast[::-1], 0.0)
    d["wl"] = d["z"] + d["h"]
    sim = Sim(d, order=2)
    fs = _solver(S.catchment_from(d), cuda)
    sim.step(2)
    fs.step(2)
    got = fs.compacted(0)
    for f in ("h", "qx", "qy"):
        np.testing.assert_allclose(got[f], sim.state()[f], rtol=0, atol=1e-10, err_msg=f)


def test_tile_tasks_asked_for_after_prepare(cuda):
    """The other kernel's step on a batch prepared for this one: boundary
    values, maps and partial sums lie where both look for them."""
    from hipims_b200 import scenarios as S

    c = S.catchment_from(S.urban_catchment(200, n_rows=150, seed=4, rain_mm_h=150.0))
    a, b = _solver(c, cuda), _solver(c, cuda, kernel="tasks", tile=(32, 32))
    assert a.batch.tile_x == 32 and a.batch.tile_y == 32
    a.batch.flags |= 2  # HB_FLAG_TILE_TASKS
    for s in (a, b):
        s.step(10)
    x, y = a.compacted(0), b.compacted(0)
    for f in x:
        np.testing.assert_array_equal(x[f], y[f], err_msg=f)
    assert (a.controls()[0].t, a.controls()[0].step) == (b.controls()[0].t, 10)
