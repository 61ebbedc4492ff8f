"""Small batches step in 8- or 16-row blocks of their 32 x 64 tiles (one CTA each)
instead of whole tiles: the same arithmetic on every cell, so fields and
clocks are equal bit for bit to whole tiles (HB_FLAG_WHOLE_TILES); volumes are
summed in another order (FP32 per lane, then FP64): to 1e-6."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

WHOLE = 8  # HB_FLAG_WHOLE_TILES
SOIL = dict(infiltration=dict(ks=[2e-6, 1e-6], psi=[0.1, 0.2], dtheta=[0.3, 0.2]))


def _solver(cs, cuda, whole, **kw):
    from hipims_b200 import _lib
    from hipims_b200.fused import FusedSolver

    fs = FusedSolver(cs, dtype=torch.float32, device=cuda, **kw)
    if whole:
        divided = _lib.lib().hb_fused_workspace_size(ctypes.byref(fs.batch))
        fs.batch.flags |= WHOLE
        size = _lib.lib().hb_fused_workspace_size(ctypes.byref(fs.batch))
        assert size <= divided  # regions are 256-byte aligned
        fs.workspace = torch.zeros(size, dtype=torch.uint8, device=cuda)
        fs.batch.workspace = fs.workspace.data_ptr()
        fs.prepare()
    return fs


def _same(a, b):
    for k in range(len(a.inst)):
        x, y = a.compacted(k), b.compacted(k)
        for f in x:
            np.testing.assert_array_equal(x[f], y[f], err_msg=f"instance {k} {f}")
        ca, cb = a.controls()[k], b.controls()[k]
        assert (ca.t, ca.dt, ca.step, ca.cur) == (cb.t, cb.dt, cb.step, cb.cur)
        assert ca.status == cb.status == 0
        assert ca.volume == pytest.approx(cb.volume, rel=1e-6)
        assert ca.outflow_volume == pytest.approx(cb.outflow_volume, rel=1e-6, abs=1e-9)


# rows around the block height and the 64-row datum blocks; a single cell row;
# widths around the tile's; the last batch has more blocks than one sum group
@pytest.mark.parametrize("shapes", [((1, 40),), ((7, 63),), ((8, 64), (9, 65)), ((31, 130),),
                                    ((63, 200), (65, 33), (129, 70)), ((420, 390),)])
@pytest.mark.parametrize("order", [1, 2])
def test_blocks_equal_whole_tiles(cuda, shapes, order):
    from hipims_b200 import scenarios as S

    cs = [S.catchment_from(S.urban_catchment(c, n_rows=r, seed=k + 3, rain_mm_h=150.0))
          for k, (r, c) in enumerate(shapes)]
    a, b = _solver(cs, cuda, False, order=order), _solver(cs, cuda, True, order=order)
    a.step(30)
    b.step(30)
    _same(a, b)


def test_blocks_with_sources_strided_grid_and_persistent(cuda):
    """Infiltration; fewer CTAs than blocks (grid_blocks); the persistent step."""
    from hipims_b200 import scenarios as S

    cs = [S.catchment_from(S.urban_catchment(150, seed=11, rain_mm_h=150.0), **SOIL)]
    a, b = _solver(cs, cuda, False), _solver(cs, cuda, True)
    c = _solver(cs, cuda, False, grid_blocks=5)
    p = _solver(cs, cuda, False)
    for s in (a, b, c):
        s.step(25)
    p.run_persistent(25)
    _same(a, b)
    _same(a, c)
    _same(a, p)


def test_changed_division_without_prepare_is_refused(cuda):
    """The block height is prepare's: asking for another one afterwards raises
    instead of stepping on another list, and the solver steps on after it."""
    from hipims_b200 import scenarios as S
    from hipims_b200.fused import FusedSolver

    for dtype in (torch.float32, torch.float64):
        fs = FusedSolver(S.catchment_from(S.urban_catchment(100, seed=2)), dtype=dtype, device=cuda)
        fs.step(2)
        fs.batch.flags |= WHOLE
        with pytest.raises(RuntimeError, match="prepare"):
            fs.step(1)
        if dtype == torch.float32:
            with pytest.raises(RuntimeError, match="prepare"):
                fs.run_persistent(1)
        fs.batch.flags &= ~WHOLE
        fs.step(1)
        assert fs.controls()[0].step == 3 and fs.controls()[0].status == 0


# 16-row blocks: 297 to 592 tiles
@pytest.mark.parametrize("rows,cols,tiles,soil", [(860, 700, 297, False), (1180, 1020, 592, False),
                                                  (1180, 1020, 592, True)])
def test_sixteen_row_blocks_equal_whole_tiles(cuda, rows, cols, tiles, soil):
    from hipims_b200 import scenarios as S

    d = S.urban_catchment(cols, n_rows=rows, seed=3, rain_mm_h=150.0)
    c = S.catchment_from(d, **(SOIL if soil else {}))
    a, b = (_solver([c], cuda, w, origin=(0, 0)) for w in (False, True))
    assert a.n_tiles == tiles
    per = a.workspace.numel() / b.workspace.numel()
    assert per > 1.4  # divided
    a.step(12)
    b.step(12)
    _same(a, b)
    if not soil:
        p = _solver([c], cuda, False, origin=(0, 0))
        p.run_persistent(12)
        _same(a, p)
