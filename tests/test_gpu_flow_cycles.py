"""Flow accumulation over tiles of directions full of cycles (random codes: two-cell
cycles almost everywhere, longer ones, trees of several tiles hanging off them), inside
tiles and across their edges; the same cells as the whole-raster walks, which complete
a cell only when all that flows into it has."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CODES = np.array([0, 1, 2, 4, 8, 16, 32, 64, 128, 5], np.uint8)


def both(M, dirs, water):
    def run():
        return M.to_numpy(M.flow_accumulation(M.from_numpy(water, bs=[128, 128]), M.from_numpy(dirs, bs=[128, 128])))
    got = run()
    M.set_exec_mode(M.EXEC_PLAIN)
    try:
        return got, run()
    finally:
        M.set_exec_mode(M.EXEC_FUSED)


@pytest.mark.parametrize("shape", [(1, 90), (64, 64), (65, 127), (200, 333), (700, 640)])
@pytest.mark.parametrize("picks", ["all", "no pits", "straight", "mostly east"])
def test_random_codes(M, shape, picks):
    rng = np.random.default_rng(shape[1])
    p = {"all": None, "no pits": [0] + [1 / 8] * 8 + [0], "straight": [0, .25, 0, .25, 0, .25, 0, .25, 0, 0],
         "mostly east": [0, .9, .02, .02, .01, .01, .01, .02, .01, 0]}[picks]
    dirs = rng.choice(CODES, shape, p=p)
    water = rng.integers(-2 ** 31, 2 ** 31, shape).astype(np.int32)
    got, ref = both(M, dirs, water)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("y0,x0,y1,x1", [(2, 2, 61, 61), (63, 63, 64, 64), (10, 10, 150, 300), (64, 64, 127, 127)])
def test_rivers_into_a_ring(M, y0, x0, y1, x1):
    # everything else drains east, or west past the ring: long trees end on its cells
    h, w = 170, 333
    dirs = np.full((h, w), 1, np.uint8)
    dirs[:, x1 + 1:] = 16
    dirs[y0, x0:x1], dirs[y0:y1, x1], dirs[y1, x0 + 1:x1 + 1], dirs[y0 + 1:y1 + 1, x0] = 1, 4, 16, 64
    got, ref = both(M, dirs, np.ones((h, w), np.int32))
    assert np.array_equal(got, ref)
    assert got[y0, x0] == 0 and (got != 0).any()
