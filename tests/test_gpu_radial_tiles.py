"""The tiled radial scan at the edges of its tiles: 32 fronts by 32 cells per tile,
observers on edges and corners, radius limits at strip ends, other reductions,
float64, and rasters whose scan is kept or not; bit-exact against the oracle or
the front-by-front recurrence in NumPy."""
import numpy as np
import pytest

from map_b200 import synth
from map_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

OCTANTS = ((0, -1, 1, 0), (1, 0, 0, -1), (1, 0, 0, 1), (0, 1, 1, 0), (0, 1, -1, 0), (-1, 0, 0, 1), (-1, 0, 0, -1),
           (0, -1, -1, 0))


def scan(a, start, fold, neutral, radius=None):
    """The recurrence front by front in a's own type."""
    h, w = a.shape
    one = a.dtype.type(1)
    out = np.full_like(a, np.nan)
    out[start[1], start[0]] = neutral
    for p0, p1, q0, q1 in OCTANTS:
        ep = w - 1 - start[0] if p0 > 0 else start[0] if p0 < 0 else h - 1 - start[1] if p1 > 0 else start[1]
        eq = w - 1 - start[0] if q0 > 0 else start[0] if q0 < 0 else h - 1 - start[1] if q1 > 0 else start[1]
        prev = np.array([neutral], a.dtype)
        for d0 in range(1, (ep if radius is None else min(ep, radius)) + 1):
            d1 = np.arange(min(d0, eq) + 1)
            ys, xs = start[1] + p1 * d0 + q1 * d1, start[0] + p0 * d0 + q0 * d1
            pa = np.zeros(d1.size, a.dtype)
            pb = np.zeros(d1.size, a.dtype)
            n = min(prev.size, d1.size)
            pa[:n] = prev[:n]
            pb[1:] = prev[:d1.size - 1]
            f0, f1 = a.dtype.type(d0), d1.astype(a.dtype)
            wt = f1 / f0 * (f0 - one) - (f1 - one)
            with np.errstate(invalid="ignore", over="ignore"):
                lit = pa * wt + pb * (one - wt)
            lit[0] = pa[0]
            if d1[-1] == d0:
                lit[-1] = pb[-1]
            v = a[ys, xs]
            with np.errstate(invalid="ignore", over="ignore"):
                prev = np.where(np.isfinite(v), fold(lit, v), lit)
            out[ys, xs] = prev
    return out


def same(got, ref):
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    m = ~np.isnan(ref)
    assert np.array_equal(got[m], ref[m])


@pytest.mark.parametrize("shape,obs", [((1, 1), (0, 0)), ((1, 200), (37, 0)), ((200, 1), (0, 199)), ((32, 33), (0, 0)),
                                       ((33, 32), (31, 32)), ((65, 66), (32, 33)), ((64, 129), (64, 63)),
                                       ((97, 161), (160, 0)), ((300, 700), (5, 290)), ((700, 300), (290, 5))])
def test_tile_edges_bit_exact(M, shape, obs):
    a = synth.fbm_dem(shape[0], shape[1], seed=7, hi=50.0) - np.float32(20)
    rng = np.random.default_rng(3)
    holes = rng.random(shape) < 0.01
    a[holes] = np.nan
    same(M.to_numpy(M.rmax(M.from_numpy(a), list(obs))), O.radial_f32(a, obs, 6))


@pytest.mark.parametrize("radius", [1, 31, 32, 33, 64, 65])
def test_radius_at_strip_ends(M, radius):
    a = synth.fbm_dem(150, 170, seed=8, hi=50.0)
    obs = (70, 90)
    same(M.to_numpy(M.rmax(M.from_numpy(a), list(obs), radius=radius)), scan(a, obs, np.fmax, -np.inf, radius))


@pytest.mark.parametrize("name,fold,neutral", [("rmin", np.fmin, np.inf), ("rsum", np.add, 0.0)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_reductions_and_types(M, name, fold, neutral, dtype):
    a = synth.fbm_dem(131, 203, seed=9, hi=2.0).astype(dtype)
    obs = (101, 33)
    same(M.to_numpy(getattr(M, name)(M.from_numpy(a), list(obs))), scan(a, obs, fold, dtype(neutral)))


def test_scan_kept_and_not_kept(M):
    # the line-of-sight raster alone leaves the scan unstored; asked for, it is the same scan
    dem_np = synth.fbm_dem(260, 333, seed=10, hi=80.0)
    dem, obs = M.from_numpy(dem_np), [200, 31]
    dist = W.distance(dem, obs)
    scan_r = M.rmax((dem - 10.0) / dist, obs)
    view = (scan_r * dist + 10.0) - dem
    alone = M.to_numpy(view)
    kept_view, kept_scan = M.materialize(view, scan_r)
    assert np.array_equal(M.to_numpy(kept_view), alone, equal_nan=True)
    same(M.to_numpy(kept_scan), M.to_numpy(scan_r))
