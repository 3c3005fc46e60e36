"""Whole-raster reductions on the vector path of full tiles and the one-cell path of
the others: sizes around the 64 x 32 tiles, every element size, several inputs, and
inputs whose rows start on no 16-byte boundary; integers and extremes exact, float
sums within 2e-6 of float64. Squares and cubes of map_powf against float64."""
import numpy as np
import pytest

from map_b200 import map as MM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (31, 63), (32, 64), (33, 65), (64, 129), (257, 1000), (1500, 2300)])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.int32, np.int64, np.float32, np.float64])
def test_reductions_at_tile_edges(M, shape, dtype):
    rng = np.random.default_rng(shape[0])
    a = rng.integers(0, 100, shape).astype(dtype)
    if a.dtype.kind == "f":
        a = (a + rng.random(shape)).astype(dtype)
    r = M.from_numpy(a, bs=[128, 128])
    outs = [M.zmax(r), M.zmin(r), M.zsum(r)]
    M.eval(*outs)
    mx, mn, sm = [M.value(o) for o in outs]
    assert mx == a.max() and mn == a.min()
    if a.dtype.kind == "f":
        assert abs(sm - a.sum(dtype=np.float64)) <= 2e-6 * abs(a.sum(dtype=np.float64))
    else:
        assert dtype(sm) == a.sum(dtype=dtype)


def test_two_inputs_and_unaligned_rows(M):
    import torch
    w, h = 517, 300
    a = torch.rand((h, 520), device="cuda")
    b = torch.rand((h, 544), device="cuda")
    torch.cuda.synchronize()
    ra = M.from_device(a.data_ptr(), 520 * 4, [w, h], M.F32, [64, 64])
    rb = M.from_device(b.data_ptr() + 4, 544 * 4, [w, h], M.F32, [64, 64])   # realigned by the engine
    got = MM.value
    s = M.zsum(ra * rb)
    M.eval(s)
    ref = (a[:, :w].double() * b[:, 1:w + 1].double()).sum().item()
    assert abs(got(s) - ref) <= 2e-6 * ref


def test_squares_and_cubes(M):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-3000, 3000, 200000), 2.0 ** rng.uniform(-60, 60, 200000) * rng.choice([-1, 1], 200000)])
    special = [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-45, 3e38, -3e38, 7e12, 6.9e12, 1e-13, 5e-15, -5e-15, 1.0, -1.0]
    x = np.concatenate([x, special]).astype(np.float32)
    x = np.resize(x, (400, 1001))
    r = M.from_numpy(x)
    for k in (2, 3):
        got = M.to_numpy(r ** k)
        with np.errstate(over="ignore", invalid="ignore"):
            want = x.astype(np.float64) ** k
            near = want.astype(np.float32)
        assert np.array_equal(np.isnan(got), np.isnan(near)) and np.array_equal(np.isinf(got), np.isinf(near))
        assert np.array_equal(np.signbit(got[near == 0]), np.signbit(near[near == 0]))
        m = np.isfinite(near)
        # one rounding of the exact square; 0.51 ulp for the cube
        assert np.all(np.abs(got[m].astype(np.float64) - want[m]) <= 0.51 * np.spacing(np.abs(near[m])).astype(np.float64))
