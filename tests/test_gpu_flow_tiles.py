"""Flow accumulation over 64 x 64 tiles: sizes around the tiles' edges, signed and
unsigned water, long paths that cross many tiles and wind inside one, codes that lead
out of the raster or are no direction, and cycles inside a tile and across tiles;
bit-exact against the oracle, and with cycles against the whole-raster walks (the
plain launches)."""
import numpy as np
import pytest

from map_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DX, DY = (1, 1, 0, -1, -1, -1, 0, 1), (0, 1, 1, 1, 0, -1, -1, -1)


def accumulate(M, dirs, water):
    return M.to_numpy(M.flow_accumulation(M.from_numpy(water, bs=[128, 128]), M.from_numpy(dirs, bs=[128, 128])))


def check(M, dirs, water):
    ref, cyclic = O.flowacc_s32(water.astype(np.int32), dirs)
    assert not cyclic
    assert np.array_equal(accumulate(M, dirs, water).astype(np.int32), ref)


SIZES = [(1, 1), (1, 200), (200, 1), (2, 2), (63, 64), (64, 64), (64, 65), (65, 64), (66, 130), (129, 127), (300, 700)]


@pytest.mark.parametrize("shape", SIZES)
@pytest.mark.parametrize("dtype", [np.int32, np.uint32])
def test_tile_edges(M, shape, dtype):
    rng = np.random.default_rng(shape[0])
    dem = (rng.random(shape) * 100).astype(np.float32)   # short paths, pits everywhere
    dirs = M.to_numpy(M.flow_direction(M.from_numpy(dem, bs=[64, 64])))
    check(M, dirs, rng.integers(0, 1000, shape).astype(dtype))


def test_long_paths(M):
    # one river that crosses every tile row by row, back and forth
    h, w = 131, 260
    dirs = np.zeros((h, w), np.uint8)
    dirs[0::2, :-1], dirs[0::2, -1] = 1, 1 << 2
    dirs[1::2, 1:], dirs[1::2, 0] = 1 << 4, 1 << 2
    check(M, dirs, np.ones((h, w), np.int32))


def test_smooth_terrain_and_wrapping_sums(M):
    dem = synth.fbm_dem(700, 900, seed=4)
    dirs = M.to_numpy(M.flow_direction(M.from_numpy(dem, bs=[256, 256])))
    rng = np.random.default_rng(4)
    check(M, dirs, rng.integers(-2 ** 31, 2 ** 31, dem.shape).astype(np.int32))


def test_invalid_codes_and_edges(M):
    # acyclic random codes (each leads to a cell of higher index), codes that leave
    # the raster, and bytes that are no single direction
    rng = np.random.default_rng(8)
    h, w = 190, 333
    dirs = rng.choice(np.array([1, 2, 4, 8], np.uint8), (h, w))
    dirs[rng.random((h, w)) < 0.02] = 0
    dirs[rng.random((h, w)) < 0.02] = 3
    dirs[:, -1][rng.random(h) < 0.5] = 1
    check(M, dirs, rng.integers(0, 50, (h, w)).astype(np.int32))


@pytest.mark.parametrize("ring", [(5, 5, 9, 9), (60, 60, 70, 70), (30, 100, 30, 101), (10, 10, 180, 250)])
def test_cycles_leave_their_cells_empty(M, ring):
    # a ring of codes (clockwise) in terrain: its cells never complete and hold zero,
    # everything else is summed, as the walks do
    dem = synth.fbm_dem(200, 300, seed=12)
    dirs = M.to_numpy(M.flow_direction(M.from_numpy(dem, bs=[64, 64])))
    y0, x0, y1, x1 = ring
    if y0 == y1:
        dirs[y0, x0], dirs[y0, x1] = 1, 1 << 4
    else:
        dirs[y0, x0:x1], dirs[y0:y1, x1], dirs[y1, x0 + 1:x1 + 1], dirs[y0 + 1:y1 + 1, x0] = 1, 4, 16, 64
    water = np.ones(dem.shape, np.int32)
    got = accumulate(M, dirs, water)
    M.set_exec_mode(M.EXEC_PLAIN)
    try:
        ref = accumulate(M, dirs, water)
    finally:
        M.set_exec_mode(M.EXEC_FUSED)
    assert np.array_equal(got, ref)
    assert got[y0, x0] == 0
