"""Generations of a binary neighbourhood rule chained in one launch, on tiles of
bits: sizes around the tiles' and words' edges, the three border rules over several
block sizes, chains shorter and longer than a launch, other rules than Life, cells
that are neither zero nor one, and in-place evaluation; bit-exact against the
oracle, or against the engine's one-cell form, which evaluates every generation by
itself."""
import numpy as np
import pytest

from map_b200 import synth
from map_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture
def border(M):
    yield lambda b: M.set_border(b)
    M.set_border(M.BORDER_BLOCK_MIRROR)


def rule(M, state, born, survive):
    # neighbours + 9 * centre tells every (centre, count) pair apart
    code = M.convolve(state, [[1, 1, 1], [1, 9, 1], [1, 1, 1]])
    hits = [code == c for c in list(born) + [9 + s for s in survive]]
    r = hits[0]
    for h in hits[1:]:
        r = r + h
    return r


SIZES = [(1, 1), (1, 40), (40, 1), (31, 33), (40, 992), (41, 993), (64, 1008), (65, 1009), (130, 2001), (400, 1985),
         (33, 8000), (3300, 1100)]


@pytest.mark.parametrize("shape", SIZES)
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_life_sizes_and_borders(M, border, shape, mode):
    border(mode)
    grid = synth.bernoulli_u8(shape[0], shape[1], 0.35, seed=shape[1])
    gens = 29
    got = M.to_numpy(W.life(M.from_numpy(grid, bs=[64, 48]), gens))
    assert M.last_launch_count() <= 3
    assert np.array_equal(got, O.life(grid, (64, 48), gens, border=mode))


@pytest.mark.parametrize("bs", [(1, 1), (7, 5), (16, 16), (300, 1), (5000, 5000)])
def test_block_mirror_blocks(M, border, bs):
    border(0)
    grid = synth.bernoulli_u8(150, 1100, 0.4, seed=3)
    got = M.to_numpy(W.life(M.from_numpy(grid, bs=list(bs)), 17))
    assert np.array_equal(got, O.life(grid, bs, 17, border=0))


@pytest.mark.parametrize("gens", [2, 11, 12, 13, 16, 17, 33])
@pytest.mark.parametrize("shape", [(70, 500), (3200, 4000)])   # small and large tiles
def test_generation_counts(M, border, gens, shape):
    border(2)
    grid = synth.bernoulli_u8(shape[0], shape[1], 0.3, seed=gens)
    got = M.to_numpy(W.life(M.from_numpy(grid, bs=[512, 512]), gens))
    assert np.array_equal(got, O.life(grid, (512, 512), gens, border=2))


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("born,survive", [((3, 6), (2, 3)), ((0, 3, 8), (0, 1, 4, 8)), ((1, 3, 5, 7), (1, 3, 5, 7))])
def test_other_rules(M, border, mode, born, survive):
    border(mode)
    grid = synth.bernoulli_u8(210, 1500, 0.5, seed=9)
    def run():
        s = M.from_numpy(grid, bs=[128, 96])
        for _ in range(14):
            s = rule(M, s, born, survive)
        return M.to_numpy(s)
    got, launches = run(), M.last_launch_count()
    M.set_paired_cells(False)
    try:
        ref = run()
        assert launches < M.last_launch_count() == 14
    finally:
        M.set_paired_cells(True)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("shape", [(90, 700), (3100, 4300)])
def test_cells_of_any_value(M, border, mode, shape):
    # tiles that hold other bytes than zero and one take the rule's own byte form
    border(mode)
    grid = synth.bernoulli_u8(shape[0], shape[1], 0.3, seed=5)
    rng = np.random.default_rng(5)
    for _ in range(6):
        grid[rng.integers(shape[0]), rng.integers(shape[1])] = rng.integers(2, 256)
    got = M.to_numpy(W.life(M.from_numpy(grid, bs=[256, 256]), 20))
    assert np.array_equal(got, O.life(grid, (256, 256), 20, border=mode))


def test_in_place_and_kept_generations(M, border):
    import torch
    border(2)
    grid = synth.bernoulli_u8(300, 1024, 0.3, seed=6)
    t = torch.from_numpy(grid).cuda()
    torch.cuda.synchronize()
    M.to_device(W.life(M.from_device(t.data_ptr(), 1024, [1024, 300], M.U8, [256, 256]), 5), t.data_ptr(), 1024)
    assert np.array_equal(t.cpu().numpy(), O.life(grid, (256, 256), 5, border=2))
    # a generation that is asked for too ends its chain
    src = M.from_numpy(grid, bs=[256, 256])
    mid = W.life(src, 4)
    end = W.life(mid, 6)
    a, b = M.materialize(mid, end)
    assert np.array_equal(M.to_numpy(a), O.life(grid, (256, 256), 4, border=2))
    assert np.array_equal(M.to_numpy(b), O.life(grid, (256, 256), 10, border=2))
