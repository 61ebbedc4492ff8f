"""The workspace holds every per-block region of a batch's blocks: a partial sum (32
bytes), an order entry (4), a class (1) and a list entry (16), on either side
of each line of the rule that divides tiles into blocks."""
import ctypes

import pytest

from hipims_b200 import _lib

PER_BLOCK = 32 + 4 + 1 + 16


@pytest.mark.parametrize("tile,dtype,tiles,blocks_per_tile", [
    ((32, 64), _lib.HB_F32, 1, 4), ((32, 64), _lib.HB_F32, 296, 4), ((32, 64), _lib.HB_F32, 297, 2),
    ((32, 64), _lib.HB_F32, 592, 2), ((32, 64), _lib.HB_F32, 593, 1),
    ((32, 32), _lib.HB_F64, 1, 4), ((32, 32), _lib.HB_F64, 148, 4), ((32, 32), _lib.HB_F64, 149, 2),
    ((32, 32), _lib.HB_F64, 5000, 2)])
@pytest.mark.parametrize("instances", [1, 7])
def test_size_covers_the_blocks(tile, dtype, tiles, blocks_per_tile, instances):
    b = _lib.HbFusedBatch()
    b.n_tiles, b.n_instances, b.dtype = tiles, instances, dtype
    b.tile_y, b.tile_x = tile
    n = tiles * blocks_per_tile
    size = _lib.lib().hb_fused_workspace_size(ctypes.byref(b))
    b.n_tiles = 0
    empty = _lib.lib().hb_fused_workspace_size(ctypes.byref(b))
    # beyond what an empty batch takes: the regions, and their groups' sums (a
    # partial and a counter for 128 blocks) and padding to 256 bytes
    assert size - empty >= n * PER_BLOCK - 6 * 256
    assert size - empty <= n * PER_BLOCK + (n // 128 + 1) * 36 + 6 * 256
