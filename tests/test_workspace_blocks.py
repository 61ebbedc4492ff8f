"""The workspace a batch needs (pure host arithmetic): dividing tiles into
blocks is a matter of the batch record, and whole tiles keep the limits of the
fixed scratch (4 MiB: about 110,000 32-wide and 78,000 64-wide tiles)."""
import ctypes

import pytest

from hipims_b200 import _lib

WHOLE = 8  # HB_FLAG_WHOLE_TILES
MIB4 = 4 << 20


def _size(tiles, instances, tile, dtype, flags=0):
    b = _lib.HbFusedBatch()
    b.n_tiles, b.n_instances, b.dtype, b.flags = tiles, instances, dtype, flags
    b.tile_y, b.tile_x = tile
    return _lib.lib().hb_fused_workspace_size(ctypes.byref(b))


@pytest.mark.parametrize("tile,dtype,limit", [((32, 64), _lib.HB_F32, 78_000),
                                              ((32, 32), _lib.HB_F32, 110_000),
                                              ((32, 32), _lib.HB_F64, 110_000)])
def test_whole_tiles_keep_the_fixed_scratch_limits(tile, dtype, limit):
    assert _size(limit, 1, tile, dtype, WHOLE) <= MIB4
    assert _size(limit - 10_000, 256, tile, dtype, WHOLE) <= MIB4


@pytest.mark.parametrize("tile,dtype,tiles", [((32, 64), _lib.HB_F32, 592),
                                              ((32, 32), _lib.HB_F64, 148),
                                              ((32, 32), _lib.HB_F64, 5000)])
def test_divided_tiles_take_a_larger_workspace(tile, dtype, tiles):
    assert _size(tiles, 1, tile, dtype) > 2 * _size(tiles, 1, tile, dtype, WHOLE) - 64 * 1024
    assert _size(tiles, 1, tile, dtype) > _size(tiles, 1, tile, dtype, WHOLE)


def test_large_fp32_batches_are_not_divided():
    assert _size(593, 1, (32, 64), _lib.HB_F32) == _size(593, 1, (32, 64), _lib.HB_F32, WHOLE)


def test_size_does_not_depend_on_the_kernel_asked_for():
    tasks = 2  # HB_FLAG_TILE_TASKS: may be set or cleared after the workspace was sized
    assert _size(500, 3, (32, 32), _lib.HB_F64, tasks) == _size(500, 3, (32, 32), _lib.HB_F64)
