"""Generations of a binary rule chained over rasters of other bytes than zero and one:
masks of 0 and 255, land-cover codes, noise, single cells, rules that keep such bytes
and rules that do not; over the tiles' and the raster's edges, the border rules and
small blocks. Bit-exact against the engine's one-cell form, a launch per generation."""
import numpy as np
import pytest

from map_b200 import synth
from map_b200 import workloads as W

pytestmark = pytest.mark.gpu

RING = [[1, 1, 1], [1, 0, 1], [1, 1, 1]]

RULES = {"life": lambda M, s: W.life_step(s),                        # keeps a byte whose neighbours sum to two
         "keep": lambda M, s: s * (M.convolve(s, RING) < 250),       # keeps every byte among small ones
         "erode": lambda M, s: M.convolve(s, [[1] * 3] * 3) == 9}    # zero or one from any bytes


def grids(shape):
    rng = np.random.default_rng(shape[0] * 7 + shape[1])
    sparse = synth.bernoulli_u8(shape[0], shape[1], 0.3, seed=5)
    for _ in range(3):
        sparse[rng.integers(shape[0]), rng.integers(shape[1])] = rng.integers(2, 256)
    return {"mask": (rng.random(shape) < 0.4).astype(np.uint8) * 255, "codes": rng.integers(0, 7, shape).astype(np.uint8),
            "noise": rng.integers(0, 256, shape).astype(np.uint8), "single": sparse}


def check(M, rule, grid, bs, gens):
    def run():
        s = M.from_numpy(grid, bs=list(bs))
        for _ in range(gens):
            s = rule(M, s)
        return M.to_numpy(s)
    got, launches = run(), M.last_launch_count()
    M.set_paired_cells(False)
    try:
        ref = run()
        alone = M.last_launch_count()
    finally:
        M.set_paired_cells(True)
    assert np.array_equal(got, ref)
    return launches, alone


SIZES = [(1, 1), (1, 40), (40, 1), (31, 33), (40, 992), (41, 993), (64, 1007), (65, 1010), (130, 1985)]


@pytest.mark.parametrize("shape", SIZES)
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("rule", list(RULES))
def test_sizes_and_borders(fresh, shape, mode, rule):
    M = fresh
    M.set_border(mode)
    for name, grid in grids(shape).items():
        for gens in (2, 14):
            launches, alone = check(M, RULES[rule], grid, (64, 48), gens)
            assert launches < alone == gens, name


@pytest.mark.parametrize("bs", [(1, 1), (7, 5), (16, 16), (300, 1)])
@pytest.mark.parametrize("rule", ["life", "keep"])
def test_block_mirror_blocks(fresh, bs, rule):
    M = fresh
    M.set_border(0)
    for grid in grids((150, 1100)).values():
        check(M, RULES[rule], grid, bs, 6)


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("gens", [3, 16, 33])
def test_large_tiles(fresh, mode, gens):
    M = fresh
    M.set_border(mode)
    for name, grid in grids((3100, 4300)).items():
        check(M, RULES["life"], grid, (512, 512), gens)


def test_scratch_given_back_between_programs(fresh):
    M = fresh
    M.set_border(2)
    for shape in ((90, 700), (1200, 1500), (90, 700)):
        check(M, RULES["life"], grids(shape)["mask"], (64, 48), 9)
        M.collect_garbage()   # releases the tiles' scratch too
