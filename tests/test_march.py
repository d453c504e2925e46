"""The 3D stage kernel's work list: marches shortened where few columns would leave SMs idle."""

import numpy as np
import pytest

from wellbalanced_b200.mesh import AMRHierarchy, Layout


def _covered(layout):
    """How often the tiles of a layout cover each computed cell / node plane of its patches."""
    counts = []
    ty, tz = layout.tile_shape
    for index, size in enumerate(layout._extents().tolist()):
        count = np.zeros(size, dtype=int)
        for t in layout.tiles[layout.tiles["patch"] == index]:
            x, y, z = int(t["x0"]), int(t["y0"]), int(t["z0"])
            count[x : x + layout.march, y : y + ty, z : z + tz] += 1
        counts.append(count)
    return counts


@pytest.mark.parametrize("shape", [(4, 4, 4), (7, 5, 33), (64, 64, 64), (150, 97, 75), (256, 256, 256)])
@pytest.mark.parametrize("lx", [3, 5, 32])
@pytest.mark.parametrize("precision, suit", [(32, False), (32, True), (64, True), (6432, True)])
def test_every_cell_lies_in_one_tile(shape, lx, precision, suit):
    layout = Layout(AMRHierarchy(shape, periodic=(True, False, True)), precision=precision, lx=lx, suit_tile=suit)
    assert 1 <= layout.march <= lx
    assert suit or layout.tile_shape == layout.default_tile
    for count in _covered(layout):
        assert np.all(count == 1)


def test_merged_parts_share_one_march():
    parts = [Layout(AMRHierarchy(s, periodic=(True,) * 3), precision=64) for s in ((24,) * 3, (64,) * 3, (160, 96, 96))]
    assert len({part.march for part in parts}) > 1
    merged = Layout.merge(parts)
    assert merged.march == min(part.march for part in parts)
    for count in _covered(merged):
        assert np.all(count == 1)


@pytest.mark.parametrize("precision", [32, 64, 6432])
@pytest.mark.parametrize("shape", [(4, 4), (33, 17), (64, 64), (200, 31), (501, 339), (2000, 1500)])
def test_the_suited_2d_tile_is_a_built_one_and_covers_the_patch(shape, precision):
    from wellbalanced_b200 import _lib

    layout = Layout(AMRHierarchy(shape, periodic=(True, False)), precision=precision)
    tile = layout.suited_tile()
    assert tile in _lib.tile_shapes(2, precision)
    layout.set_tile(tile)
    count = np.zeros(layout._extents()[0], dtype=int)
    for t in layout.tiles:
        count[int(t["x0"]) : int(t["x0"]) + tile[0], int(t["y0"]) : int(t["y0"]) + tile[1]] += 1
    assert np.all(count == 1)


def test_many_tiles_keep_the_default_shape():
    layout = Layout(AMRHierarchy((4096, 4096), periodic=(True, True)), precision=32)
    assert layout.suited_tile() == layout.default_tile
