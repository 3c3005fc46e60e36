"""Scans whose tiles get no scratch memory: radial scans front by front (one CTA per
octant with the fronts in shared memory, clusters from 2048 cells across on, fronts too
long for either re-read from the output) and flow accumulations as sweeps and walks,
bit-exact against the oracle; and into their own input's memory, by way of a buffer."""
import numpy as np
import pytest

from map_b200 import synth
from map_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture
def bare(M, monkeypatch):
    monkeypatch.setenv("MAP_B200_SCAN_SCRATCH", "0")
    return M


@pytest.mark.parametrize("shape,obs", [((90, 133), (20, 30)), ((700, 900), (300, 13)), ((2047, 300), (299, 2046)),
                                       ((2100, 2300), (700, 1050)), ((2048, 2049), (2048, 2047)), ((3, 300000), (1, 2))])
def test_radial_front_by_front(bare, shape, obs):
    M = bare
    dem = synth.uniform_f32(shape[0], shape[1], seed=33)
    ref = O.radial_f32(dem, list(obs), 6)
    got = M.to_numpy(M.rmax(M.from_numpy(dem, bs=[512, 512]), list(obs)))
    assert np.array_equal(got, ref, equal_nan=True)


@pytest.mark.parametrize("shape,obs", [((90, 133), (20, 30)), ((2060, 2300), (700, 1050))])
def test_viewshed_whose_scan_is_not_kept(bare, monkeypatch, shape, obs):
    import torch
    M = bare
    dem = synth.fbm_dem(shape[0], shape[1], seed=5, hi=50.0)
    swept = M.to_numpy(W.viewshed(M.from_numpy(dem, bs=[64, 64]), list(obs), 10.0))
    limited = M.to_numpy(M.rmax(M.from_numpy(dem, bs=[64, 64]), list(obs), 41.0) * 2.0)
    # in the memory of its input
    pitch = (4 * shape[1] + 127) // 128 * 128
    buf = torch.zeros((shape[0], pitch // 4), dtype=torch.float32, device="cuda")
    buf[:, :shape[1]].copy_(torch.from_numpy(dem).cuda())
    torch.cuda.synchronize()
    x = M.from_device(buf.data_ptr(), pitch, [shape[1], shape[0]], M.F32, [64, 64])
    M.to_device(W.viewshed(x, list(obs), 10.0), buf.data_ptr(), pitch)
    monkeypatch.delenv("MAP_B200_SCAN_SCRATCH")
    tiled = M.to_numpy(W.viewshed(M.from_numpy(dem, bs=[64, 64]), list(obs), 10.0))
    assert np.array_equal(swept, tiled, equal_nan=True)
    assert np.array_equal(buf[:, :shape[1]].cpu().numpy(), tiled, equal_nan=True)
    assert np.array_equal(limited, M.to_numpy(M.rmax(M.from_numpy(dem, bs=[64, 64]), list(obs), 41.0) * 2.0), equal_nan=True)


@pytest.mark.parametrize("shape", [(40, 70), (300, 500), (3, 50000)])
def test_flow_walks(bare, shape):
    M = bare
    rng = np.random.default_rng(3)
    codes = np.array([0, 1, 2, 4, 8, 2, 4, 8, 3], np.uint8)   # no cycles
    d8 = codes[rng.integers(0, len(codes), shape)]
    water = rng.integers(-9, 99, shape).astype(np.int32)
    ref, cyclic = O.flowacc_s32(water, d8)
    assert not cyclic
    got = M.to_numpy(M.flow_accumulation(M.from_numpy(water, bs=[64, 64]), M.from_numpy(d8, bs=[64, 64])))
    assert np.array_equal(got, ref)
