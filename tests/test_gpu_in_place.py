"""Programs evaluated into memory of their own input: the result is the one of
separate buffers, whatever the kind of group, the launch mode and the place of the
output's rows in the input's memory (the same rows, other rows, aligned and not).
Element-wise programs write over their input directly; kernels that read other cells
than the ones they write (halos, scan fronts, a flow accumulation's water) must not."""
import numpy as np
import pytest

from map_b200 import synth
from map_b200 import workloads as W

pytestmark = pytest.mark.gpu

W3 = [[1, 2, 1], [2, 4, 2], [1, 2, 1]]


def _programs(M):
    """(name, type of the raster, program over it); results of the raster's own type."""
    return [("local", M.F32, lambda x: x * 3.0 + 1.0), ("conv", M.F32, lambda x: M.convolve(x, W3)),
            ("hillshade", M.F32, W.hillshade), ("read before", M.F32, lambda x: M.convolve(x * 2.0, W3) * 0.5),
            ("read after", M.F32, lambda x: M.convolve(M.convolve(x, W3), W3) + x),
            ("range", M.F32, lambda x: x - M.zmax(x) * 0.5), ("life", M.U8, W.life_step), ("life3", M.U8, lambda x: W.life(x, 3)),
            ("view", M.F32, lambda x: W.viewshed(x, [20, 30], 5.0)), ("rmax", M.F32, lambda x: M.rmax(x, [0, 64])),
            ("rsum64", M.F64, lambda x: M.rsum(x, [100, 7], 40.0))]


def _cells(M, shape, dt):
    if dt == M.U8:
        return synth.bernoulli_u8(shape[0], shape[1], 0.35, seed=4)
    a = synth.fbm_dem(shape[0], shape[1], seed=4)
    return a.astype(np.float64) if dt == M.F64 else a.astype(np.int32) if dt == M.S32 else a


def _check(M, a, dt, program, pitch, off, shift):
    """Evaluates program over the raster of cells a, held `off` bytes into a buffer at
    rows `pitch` bytes apart, into the rows `shift` bytes further on."""
    import torch
    h, w = a.shape
    row = a.itemsize * w
    want = M.to_numpy(program(M.from_numpy(a, bs=[64, 48])))
    raw = np.zeros((h, pitch), np.uint8)
    raw[:, :row] = np.ascontiguousarray(a).view(np.uint8).reshape(h, row)
    buf = torch.zeros(off + pitch * (h + 40), dtype=torch.uint8, device="cuda")
    buf[off:off + pitch * h].copy_(torch.from_numpy(raw.ravel()).cuda())
    torch.cuda.synchronize()
    x = M.from_device(buf.data_ptr() + off, pitch, [w, h], dt, [64, 48])
    M.to_device(program(x), buf.data_ptr() + off + shift, pitch)
    got = buf[off + shift:off + shift + pitch * h].cpu().numpy().reshape(h, pitch)[:, :row]
    got = np.ascontiguousarray(got).view(want.dtype)
    assert np.array_equal(got, want, equal_nan=want.dtype.kind == "f")


@pytest.mark.parametrize("shape", [(70, 129), (260, 333)])
@pytest.mark.parametrize("border,plain", [(0, False), (2, False), (1, True)])
@pytest.mark.parametrize("off,rows,bytes_", [(0, 0, 0), (0, 3, 0), (0, 0, 128), (8, 0, 0), (8, 3, 8)])
def test_into_the_input(fresh, shape, border, plain, off, rows, bytes_):
    M = fresh
    M.set_border(border)
    M.set_exec_mode(M.EXEC_PLAIN if plain else M.EXEC_FUSED)
    for name, dt, program in _programs(M):
        a = _cells(M, shape, dt)
        # rows of whole 128-byte pieces where the buffer starts on one, else of 8 bytes more
        pitch = (a.itemsize * shape[1] + 127) // 128 * 128 + (8 if off else 0)
        _check(M, a, dt, program, pitch, off, rows * pitch + bytes_)


@pytest.mark.parametrize("shape", [(50, 64), (200, 333)])
@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("dt", ["S32", "U32", "S64", "F32"])
def test_flow_into_its_water(fresh, shape, plain, dt):
    M = fresh
    M.set_exec_mode(M.EXEC_PLAIN if plain else M.EXEC_FUSED)
    dem = synth.fbm_dem(shape[0], shape[1], seed=8)
    rng = np.random.default_rng(8)
    np_dt = {"S32": np.int32, "U32": np.uint32, "S64": np.int64, "F32": np.float32}[dt]
    water = rng.integers(0, 50, shape).astype(np_dt)   # sums below 2^24: exact in float32 too
    d8 = M.materialize(M.flow_direction(M.from_numpy(dem, bs=[64, 48])))[0]
    pitch = (water.itemsize * shape[1] + 127) // 128 * 128
    for shift in (0, pitch, 128):
        _check(M, water, getattr(M, dt), lambda x: M.flow_accumulation(x, d8), pitch, 0, shift)


@pytest.mark.parametrize("shape,obs", [((700, 900), (300, 13)), ((2060, 2300), (700, 1050))])
def test_radial_into_its_raster(fresh, shape, obs):
    M = fresh
    dem = synth.fbm_dem(shape[0], shape[1], seed=12, hi=50.0)
    pitch = (4 * shape[1] + 127) // 128 * 128
    _check(M, dem, M.F32, lambda x: W.viewshed(x, list(obs), 5.0), pitch, 0, 0)
    _check(M, dem, M.F32, lambda x: M.rmin(x, list(obs)), pitch, 0, 128)


@pytest.mark.parametrize("border", [0, 2])
@pytest.mark.parametrize("band,shift", [(False, 0), (True, 0), (False, 2), (True, -1)])
def test_rows_into_the_input(fresh, border, band, shift):
    # rows [40, 90) evaluated into the rows `shift` further on of the raster, or of the
    # band of rows around them, that they are computed from
    import torch
    M = fresh
    M.set_border(border)
    h, w, y0, y1 = 150, 333, 40, 90
    dem = synth.fbm_dem(h, w, seed=14)
    pitch = (4 * w + 127) // 128 * 128
    for program in (W.hillshade, lambda x: x * 3.0 + 1.0, lambda x: M.convolve(M.convolve(x, W3), W3) + x):
        want = M.to_numpy(program(M.from_numpy(dem, bs=[64, 48])))[y0:y1]
        ra, rb = (y0 - 4, y1 + 4) if band else (0, h)
        raw = torch.zeros((rb - ra, pitch // 4), dtype=torch.float32, device="cuda")
        raw[:, :w].copy_(torch.from_numpy(dem[ra:rb]).cuda())
        torch.cuda.synchronize()
        x = (M.from_device_rows(raw.data_ptr(), pitch, [w, h], M.F32, ra, rb - ra, bs=[64, 48]) if band
             else M.from_device(raw.data_ptr(), pitch, [w, h], M.F32, [64, 48]))
        at = y0 - ra + shift
        M.eval_rows([program(x)], [(raw.data_ptr() + at * pitch, pitch)], y0, y1)
        assert np.array_equal(raw[at:at + y1 - y0, :w].cpu().numpy(), want)


@pytest.mark.parametrize("rows", [40, 257])
@pytest.mark.parametrize("shift", [0, 3])
def test_host_raster_into_its_own_memory(fresh, rows, shift):
    # streamed bands: a focal program into its input's rows runs whole, an element-wise
    # one on the very same rows in bands
    M = fresh
    h, w = 777, 523
    dem = synth.fbm_dem(h, w, seed=15)
    for program, bands in ((W.hillshade, 0), (lambda x: x * 2.0 + 1.0, 0 if shift else -(-h // rows))):
        M.set_stream_rows(-1)
        want = M.to_numpy(program(M.from_numpy(dem, bs=[128, 128])))
        mem = np.zeros((h + shift, w), np.float32)
        mem[:h] = dem
        M.set_stream_rows(rows)
        try:
            M.to_numpy(program(M.from_numpy(mem[:h], bs=[128, 128], copy=False)), out=mem[shift:])
            assert M.last_band_count() == bands
        finally:
            M.set_stream_rows(0)
        assert np.array_equal(mem[shift:], want)
