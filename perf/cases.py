"""Performance cases: the work a user has this framework do, through its public entry points.

`listed()` gives the fixed cases, `draw(rng)` one more of the same ranges,
`prepare(case, seed)` what a program holds before the call (rasters on the device
or the host, the expression, the batch or the server), `run(state)` one pass,
`work(case)` the bytes and operations a pass cannot do without and
`exact(case, seed)` the same outputs in 64 bits.

Kinds of case:
  hillshade  the hill.py composition on a resident elevation raster
  slope      the slope part of hill.py alone (atan of the gradient's length)
  host       the hill.py composition from pinned host memory to host memory
  life       generations of life.py on a byte grid
  overlay    the wsum.py weighted overlay of several float layers
  stats      the whole-raster statistics of stats.py
  zones      per-zone count / min / max / sum / mean over a Voronoi partition
  viewshed   view.py: the radial line-of-sight scan from one observer
  flow       D8 flow directions and the count of upstream cells
  batch      hillshade and overlay of many rasters of uneven size in one batch
  serving    a burst of mixed requests over windows of a resident elevation raster
"""
import math

import numpy as np
import torch

from map_b200 import map as M
from map_b200 import synth
from map_b200 import workloads as W

WEIGHTS = (0.1, 0.2, 0.3, 0.15, 0.15, 0.1, 0.25, 0.05)
BLOCK = 256
STATS = ("maxv", "minv", "rang", "mean", "geom", "harm", "quam", "cubm", "std", "nstd")


def listed():
    return [
        # one tile of a tiled elevation model: the smallest call, launch and host latency
        {"name": "hillshade_256", "kind": "hillshade", "w": 256, "h": 256, "border": 0, "dense": False},
        # the headline raster: one large elevation model kept on the device
        {"name": "hillshade_16384", "kind": "hillshade", "w": 16384, "h": 16384, "border": 0, "dense": False},
        # a raster of odd size straight from a dense array: rows that start on no 16-byte boundary
        {"name": "slope_odd_dense", "kind": "slope", "w": 3001, "h": 2203, "border": 0, "dense": True},
        # an elevation model in host memory, shaded and read back: the streamed path
        {"name": "hillshade_host", "kind": "host", "w": 6000, "h": 5000, "border": 0},
        # life.py: 100 generations on a grid that stays in L2, dead border
        {"name": "life_4096", "kind": "life", "w": 4096, "h": 4096, "gens": 100, "border": 2},
        # wsum.py: six layers of an odd size in one element-wise pass
        {"name": "overlay_6", "kind": "overlay", "w": 7001, "h": 5003, "layers": 6},
        # stats.py: the reductions of one raster, their scalars combined on the host
        {"name": "stats_8192", "kind": "stats", "w": 8192, "h": 8192},
        # statistics of 1024 parcels
        {"name": "zones_8192", "kind": "zones", "w": 8192, "h": 8192, "zones": 1024},
        # view.py: who sees the observer, over a whole raster
        {"name": "viewshed_4096", "kind": "viewshed", "w": 4096, "h": 4096, "ox": 0.45, "oy": 0.55, "radius": 0},
        # drainage of one catchment sheet: directions, then upstream counts
        {"name": "flow_2048", "kind": "flow", "w": 2048, "h": 2048},
        # many rasters of uneven size, two programs each, as one prepared batch
        {"name": "batch_128", "kind": "batch", "count": 128, "lo": 64, "hi": 2048},
        # a burst of requests to a server: windows of 256, 512 and 1024 cells, four programs
        {"name": "serving_32", "kind": "serving", "size": 4096, "requests": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """A raster of side log-uniform in [lo, hi] and aspect 0.5 to 2, sides of any remainder."""
    side, asp = math.exp(rng.uniform(math.log(lo), math.log(hi))), rng.uniform(0.5, 2.0)
    return max(16, int(round(side * math.sqrt(asp)))), max(16, int(round(side / math.sqrt(asp))))


def draw(rng):
    kind = rng.choice(("hillshade", "slope", "host", "life", "overlay", "stats", "zones", "viewshed", "flow", "batch",
                       "serving"))
    c = {"kind": kind}
    if kind in ("hillshade", "slope"):
        c["w"], c["h"] = _sides(rng, 100, 8000)
        c["border"] = rng.choice((0, 0, 1, 2))
        c["dense"] = rng.random() < 0.3
    elif kind == "host":
        c["w"], c["h"] = _sides(rng, 200, 6000)
        c["border"] = rng.choice((0, 1))
    elif kind == "life":
        c["w"], c["h"] = _sides(rng, 64, 2900)
        c["gens"] = rng.randint(1, 100)
        c["border"] = rng.choice((0, 2, 2))
    elif kind == "overlay":
        c["w"], c["h"] = _sides(rng, 200, 8000)
        c["layers"] = rng.randint(2, 8)
    elif kind == "stats":
        c["w"], c["h"] = _sides(rng, 200, 8000)
    elif kind == "zones":
        c["w"], c["h"] = _sides(rng, 200, 8000)
        c["zones"] = _log_int(rng, 16, 4096)
    elif kind == "viewshed":
        c["w"], c["h"] = _sides(rng, 200, 4000)
        c["ox"], c["oy"] = round(rng.uniform(0.02, 0.98), 3), round(rng.uniform(0.02, 0.98), 3)
        c["radius"] = rng.choice((0, 0, rng.randint(50, 500)))
    elif kind == "flow":
        c["w"], c["h"] = _sides(rng, 100, 3000)
    elif kind == "batch":
        c["count"], c["lo"], c["hi"] = rng.randint(8, 128), 64, rng.choice((512, 1024, 2048))
    else:
        c["size"], c["requests"] = rng.choice((2048, 3000, 4096)), rng.randint(4, 32)
    return c


# ------------------------------------------------------------------ inputs

def _seed(seed, k=0):
    return (int(seed) * 1000003 + k) % (2 ** 31 - 1)


def _gen(seed, k=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(_seed(seed, k))
    return g


def _pitched(h, w, dtype=torch.float32):
    """A zeroed device raster whose rows are padded to 128 bytes; its first w columns are the raster."""
    per = 128 // torch.empty((), dtype=dtype).element_size()
    return torch.zeros((h, (w + per - 1) // per * per), dtype=dtype, device="cuda")


def _pitch(t):
    return t.stride(0) * t.element_size()


def _dem(case, seed, k=0, lo=0.0):
    return synth.fbm_dem(case["h"], case["w"], _seed(seed, k), lo=lo, xp=torch, device="cuda")


def _held(cells, dense):
    """`cells` as a user holds it: rows padded, or a dense array."""
    if dense:
        return cells.contiguous()
    t = _pitched(cells.shape[0], cells.shape[1], cells.dtype)
    t[:, :cells.shape[1]] = cells
    return t


def _raster(t, w, dt):
    return M.from_device(t.data_ptr(), _pitch(t), [w, t.shape[0]], dt, [BLOCK, BLOCK])


def _batch_sides(case):
    """The rasters' sizes, log-uniform sides and aspect 0.5 to 2: the case's own, whatever the seed."""
    r = np.random.default_rng(case["count"] * 7919 + case["hi"])
    sides = []
    for _ in range(case["count"]):
        side, asp = float(np.exp(r.uniform(np.log(case["lo"]), np.log(case["hi"])))), float(r.uniform(0.5, 2.0))
        sides.append((max(8, int(round(side * math.sqrt(asp)))), max(8, int(round(side / math.sqrt(asp))))))
    return sides


def _batch_inputs(case, seed):
    """(w, h, padded width, elevation, layers) of each raster."""
    g, got = _gen(seed), []
    for i, (w, h) in enumerate(_batch_sides(case)):
        pw = (w + 31) // 32 * 32
        dem = torch.zeros((h, pw), dtype=torch.float32, device="cuda")
        dem[:, :w] = synth.fbm_dem(h, w, _seed(seed, i), xp=torch, device="cuda")
        got.append((w, h, pw, dem, [torch.rand((h, pw), generator=g, device="cuda") for _ in range(6)]))
    return got


def _requests(case, seed):
    """(program, x, y, side, observer) of each request: half hillshades, the rest slopes, viewsheds and flows."""
    r = np.random.default_rng(_seed(seed, 7))
    got = []
    for i in range(case["requests"]):
        side = (256, 512, 1024)[(i * 5 // 4) % 3]
        prog = (0, 1, 0, 2, 0, 3, 0, 1, 0, 2, 0, 3)[i % 12]
        x, y = int(r.integers(0, case["size"] - side + 1)), int(r.integers(0, case["size"] - side + 1))
        got.append((prog, x, y, side, (int(r.integers(0, side)), int(r.integers(0, side)))))
    return got


def _observer(case):
    return [min(case["w"] - 1, int(case["ox"] * case["w"])), min(case["h"] - 1, int(case["oy"] * case["h"]))]


# ------------------------------------------------------------------ the calls

def _border(case):
    """The border rule the script sets: block mirror unless the case has another; raster mirror for a batch."""
    return 1 if case["kind"] == "batch" else case.get("border", 0)


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    M.set_border(_border(case))
    if kind in ("hillshade", "slope"):
        s["dem"] = _held(_dem(case, seed), case["dense"])
        s["out"] = torch.zeros_like(s["dem"])
        s["expr"] = (W.hillshade if kind == "hillshade" else W.slope)(_raster(s["dem"], case["w"], M.F32))
    elif kind == "host":
        s["dem"] = torch.empty((case["h"], case["w"]), dtype=torch.float32, pin_memory=True)
        s["dem"].copy_(_dem(case, seed))
        s["out"] = torch.empty_like(s["dem"], pin_memory=True).numpy()
        s["expr"] = W.hillshade(M.from_numpy(s["dem"].numpy(), bs=[BLOCK, BLOCK], copy=False))
    elif kind == "life":
        grid = (torch.rand((case["h"], case["w"]), generator=_gen(seed), device="cuda") < 0.3).to(torch.uint8)
        s["grid"] = _held(grid, False)
        s["out"] = torch.zeros_like(s["grid"])
        s["expr"] = W.life(_raster(s["grid"], case["w"], M.U8), case["gens"])
    elif kind == "overlay":
        g = _gen(seed)
        s["layers"] = [_held(torch.rand((case["h"], case["w"]), generator=g, device="cuda"), False)
                       for _ in range(case["layers"])]
        s["out"] = torch.zeros_like(s["layers"][0])
        s["expr"] = W.wsum([_raster(t, case["w"], M.F32) for t in s["layers"]], WEIGHTS[:case["layers"]])
    elif kind == "stats":
        s["dem"] = _held(_dem(case, seed, lo=100.0), False)
        s["expr"] = W.stats(_raster(s["dem"], case["w"], M.F32))
    elif kind == "zones":
        w, h, n = case["w"], case["h"], case["zones"]
        val = torch.empty((h, w), dtype=torch.float32, device="cuda").log_normal_(0.0, 1.0, generator=_gen(seed))
        s["value"] = _held(val, False)
        s["zone"] = _held(synth.voronoi_s32(h, w, n, _seed(seed), xp=torch, device="cuda"), False)
        s["count"] = torch.zeros(n, dtype=torch.int64, device="cuda")
        s["f"] = [torch.zeros(n, dtype=torch.float32, device="cuda") for _ in range(4)]
    elif kind == "viewshed":
        s["dem"] = _held(_dem(case, seed), False)
        s["out"] = torch.zeros_like(s["dem"])
        dem = _raster(s["dem"], case["w"], M.F32)
        obs, height = _observer(case), 10.0
        if case["radius"]:
            dist = W.distance(dem, obs)
            seen = M.rmax((dem - height) / dist, obs, radius=case["radius"])
            s["expr"] = (seen * dist + height) - dem
        else:
            s["expr"] = W.viewshed(dem, obs, height)
    elif kind == "flow":
        s["dem"] = _held(_dem(case, seed), False)
        s["out"] = _pitched(case["h"], case["w"], torch.int32)
        dem = _raster(s["dem"], case["w"], M.F32)
        s["expr"] = M.flow_accumulation(M.ones_like(dem, M.S32), M.flow_direction(dem))
    elif kind == "batch":
        s["keep"] = _batch_inputs(case, seed)
        cells = sum(h * pw for _, h, pw, _, _ in s["keep"])
        s["out"] = torch.zeros(2 * cells, dtype=torch.float32, device="cuda")
        s["batch"], at = M.Batch(), s["out"].data_ptr()
        for w, h, pw, dem, layers in s["keep"]:
            outs = [W.hillshade(_raster(dem, w, M.F32)),
                    W.wsum([_raster(t, w, M.F32) for t in layers], WEIGHTS[:6])]
            s["batch"].add(outs, [(at, pw * 4), (at + h * pw * 4, pw * 4)])
            at += 2 * h * pw * 4
        torch.cuda.synchronize()   # the library's stream does not wait for torch's
        s["batch"].prepare()
    elif kind == "serving":
        n = case["size"]
        s["dem"] = synth.fbm_dem(n, n, _seed(seed), xp=torch, device="cuda").contiguous()
        s["requests"] = _requests(case, seed)
        torch.cuda.synchronize()
        s["server"] = M.Server(s["dem"].data_ptr(), n * 4, n, n, budget_bytes=2 << 30, max_batch=64)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    M.set_border(_border(case))
    if kind in ("hillshade", "slope", "life", "overlay", "viewshed", "flow"):
        M.to_device(s["expr"], s["out"].data_ptr(), _pitch(s["out"]), sync=False)
        return s["out"][:, :case["w"]]
    if kind == "host":
        return M.to_numpy(s["expr"], out=s["out"])
    if kind == "stats":
        M.eval(*s["expr"].values())
        return [float(M.value(s["expr"][k])) for k in STATS]
    if kind == "zones":
        f = [t.data_ptr() for t in s["f"]]
        M.zonal_stats_device(s["value"].data_ptr(), _pitch(s["value"]), s["zone"].data_ptr(), _pitch(s["zone"]),
                             case["w"], case["h"], case["zones"], s["count"].data_ptr(), f[0], f[1], f[2], f[3])
        return [s["count"]] + s["f"]
    if kind == "batch":
        s["batch"].run(sync=False)
        return s["out"]
    ids = [s["server"].submit(p, x, y, n, n, obs=obs, obs_h=10.0, radius=167.0 if p == 2 else 0.0)
           for p, x, y, n, obs in s["requests"]]
    got = []
    for i, (p, _, _, n, _) in zip(ids, s["requests"]):
        s["server"].wait(i)
        got.append(s["server"].result(i, (n, n), np.int32 if p == 3 else np.float32))
    return got


def work(case):
    kind = case["kind"]
    if kind == "batch":   # 7 rasters read and 2 written
        cells = float(sum(w * h for w, h in _batch_sides(case)))
        return {"bytes": 36.0 * cells, "flops": 61.0 * cells}
    if kind == "serving":   # a window read and a raster written per request
        cells = float(sum(n * n for _, _, _, n, _ in _requests(case, 0)))
        return {"bytes": 8.0 * cells, "flops": 40.0 * cells}
    cells = float(case["w"]) * case["h"]
    if kind == "viewshed" and case["radius"]:
        ox, oy = _observer(case)
        r = case["radius"]
        swept = float(min(case["w"], ox + r + 1) - max(0, ox - r)) * (min(case["h"], oy + r + 1) - max(0, oy - r))
        return {"bytes": 4.0 * swept + 4.0 * cells, "flops": 20.0 * swept}
    per = {"hillshade": (8, 50), "slope": (8, 40), "host": (8, 50), "life": (2, 12 * case.get("gens", 1)),
           "overlay": (4 * case.get("layers", 0) + 4, 2 * case.get("layers", 0)), "stats": (4, 25), "zones": (8, 4),
           "viewshed": (8, 20), "flow": (8, 20)}[kind]
    return {"bytes": per[0] * cells, "flops": per[1] * cells}


# ------------------------------------------------------------------ 64 bits

def _reflect(i, d):
    r = torch.where(i < 0, -i - 1, torch.where(i >= d, 2 * d - i - 1, i))
    return torch.minimum(torch.maximum(r, torch.zeros_like(r)), d - 1)


def _taps(a, dx, dy, border):
    """a[y + dy, x + dx] of every cell under the border rule (0 block mirror, 1 raster mirror, 2 zero)."""
    h, w = a.shape
    y, x = torch.arange(h, device=a.device), torch.arange(w, device=a.device)
    H, Wd = torch.full_like(y, h), torch.full_like(x, w)
    out = a[_reflect(y + dy, H)][:, _reflect(x + dx, Wd)]
    if border == 1:
        return out
    if border == 2:
        out[(y + dy < 0) | (y + dy >= h)] = 0.0
        out[:, (x + dx < 0) | (x + dx >= w)] = 0.0
        return out
    # a read outside the raster reflects both coordinates at the reading cell's block
    by, bx = y // BLOCK * BLOCK, x // BLOCK * BLOCK
    sy = by + _reflect(y + dy - by, torch.clamp(H - by, max=BLOCK))
    sx = bx + _reflect(x + dx - bx, torch.clamp(Wd - bx, max=BLOCK))
    for r in torch.nonzero((y + dy < 0) | (y + dy >= h)).flatten().tolist():
        out[r] = a[sy[r], sx]
    for c in torch.nonzero((x + dx < 0) | (x + dx >= w)).flatten().tolist():
        out[:, c] = a[sy, sx[c]]
    return out


def _gradient(dem, border):
    h, v = ((-1, 0, 1), (-2, 0, 2), (-1, 0, 1)), ((-1, -2, -1), (0, 0, 0), (1, 2, 1))
    x, y = torch.zeros_like(dem), torch.zeros_like(dem)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            a, b = h[dy + 1][dx + 1], v[dy + 1][dx + 1]
            if a or b:
                t = _taps(dem, dx, dy, border)
                if a:
                    x += a * t
                if b:
                    y += b * t
                del t
    return x.div_(8), y.div_(8)


def _slope64(dem, border):
    x, y = _gradient(dem.double(), border)
    return torch.atan(torch.sqrt(x * x + y * y))


def _hillshade64(dem, border):
    pi = W.PI
    x, y = _gradient(dem.double(), border)
    z = torch.atan2(y, -x)
    z += (z < 0) * (pi * 2)
    z = torch.where(x != 0, z, (y > 0) * (pi / 2) + (y < 0) * (pi * 2 - pi / 2))
    az, ar = 45 / 180 * pi, 90 / 180 * pi + 45 / 180 * pi
    sl = torch.atan(torch.sqrt(x.square_() + y.square_()))
    del x, y
    return math.cos(az) * torch.cos(sl) + math.sin(az) * torch.sin(sl) * torch.cos(ar - z)


def _viewshed64(dem, obs, height, radius):
    d = dem.double()
    h, w = d.shape
    ox, oy = obs
    ys, xs = torch.arange(h, device=d.device).double(), torch.arange(w, device=d.device).double()
    dist = torch.sqrt((ox - xs)[None, :] ** 2 + (oy - ys)[:, None] ** 2)
    slope = (d - height) / dist
    out = torch.full_like(d, float("nan"))
    out[oy, ox] = -math.inf
    P = torch.tensor([(0, -1, 1, 0), (1, 0, 0, -1), (1, 0, 0, 1), (0, 1, 1, 0), (0, 1, -1, 0), (-1, 0, 0, 1),
                      (-1, 0, 0, -1), (0, -1, -1, 0)], device=d.device)
    far = max(ox, w - 1 - ox, oy, h - 1 - oy)
    far = min(far, int(radius)) if radius else far
    prev = torch.full((8, 1), -math.inf, dtype=torch.float64, device=d.device)
    flat, oflat = slope.view(-1), out.view(-1)
    for d0 in range(1, far + 1):
        d1 = torch.arange(d0 + 1, device=d.device)
        cx, cy = ox + d0 * P[:, 0:1] + d1 * P[:, 2:3], oy + d0 * P[:, 1:2] + d1 * P[:, 3:4]
        ok = (cx >= 0) & (cx < w) & (cy >= 0) & (cy < h)
        at = torch.where(ok, cy * w + cx, 0)
        a, b = torch.cat([prev, prev[:, -1:]], 1), torch.cat([prev[:, :1], prev], 1)
        t = d1.double() / d0 * (d0 - 1.0) - (d1 - 1.0)
        lit = a * t + b * (1.0 - t)
        lit[:, 0], lit[:, -1] = prev[:, 0], prev[:, -1]
        v = flat[at]
        prev = torch.where(torch.isfinite(v), torch.maximum(lit, v), lit)
        oflat[at[ok]] = prev[ok]
        prev = torch.where(ok, prev, torch.zeros_like(prev))
    return (out * dist + height) - d


def exact(case, seed):
    kind = case["kind"]
    if kind in ("life", "flow"):
        return None   # whole numbers
    if kind in ("hillshade", "host"):
        return _hillshade64(_dem(case, seed), case["border"])
    if kind == "slope":
        return _slope64(_dem(case, seed), case["border"])
    if kind == "overlay":
        g, acc = _gen(seed), 0.0
        for wt in WEIGHTS[:case["layers"]]:
            acc = acc + float(np.float32(wt)) * torch.rand((case["h"], case["w"]), generator=g, device="cuda").double()
        return acc
    if kind == "stats":
        d = _dem(case, seed, lo=100.0).double()
        n, mx, mn, mean = d.numel(), d.max(), d.min(), d.mean()
        v = {"maxv": mx, "minv": mn, "rang": mx - mn, "mean": mean, "harm": n / (1.0 / d).sum(),
             "quam": torch.sqrt((d ** 2).sum() / n), "cubm": ((d ** 3).sum() / n) ** (1.0 / 3.0)}
        dev = (d - mean) ** 2
        v["std"] = torch.sqrt(dev.sum() / n)
        v["nstd"] = torch.sqrt(((dev - mn) / (mx - mn)).sum() / n)
        return [float(v[k]) if k in v else None for k in STATS]   # the product of all cells overflows
    if kind == "zones":
        w, h, n = case["w"], case["h"], case["zones"]
        val = torch.empty((h, w), dtype=torch.float32, device="cuda").log_normal_(0.0, 1.0, generator=_gen(seed))
        val = val.double().view(-1)
        z = synth.voronoi_s32(h, w, n, _seed(seed), xp=torch, device="cuda").long().view(-1)
        cnt = torch.bincount(z, minlength=n)
        sm = torch.bincount(z, weights=val, minlength=n)
        inf = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
        mn, mx = inf.scatter_reduce(0, z, val, "amin"), (-inf).scatter_reduce(0, z, val, "amax")
        return [cnt, mn, mx, sm, sm / cnt]
    if kind == "viewshed":
        return _viewshed64(_dem(case, seed), _observer(case), 10.0, case["radius"])
    if kind == "batch":
        parts = []
        for w, h, pw, dem, layers in _batch_inputs(case, seed):
            two = torch.zeros((2, h, pw), dtype=torch.float64, device="cuda")
            two[0, :, :w] = _hillshade64(dem[:, :w], 1)
            for t, wt in zip(layers, WEIGHTS[:6]):
                two[1, :, :w] += float(np.float32(wt)) * t[:, :w].double()
            parts.append(two.view(-1))
        return torch.cat(parts)
    n = case["size"]
    dem = synth.fbm_dem(n, n, _seed(seed), xp=torch, device="cuda")
    got = []
    for p, x, y, side, obs in _requests(case, seed):
        win = dem[y:y + side, x:x + side].contiguous()
        # a window is one block: its block mirror is the raster mirror
        got.append(_hillshade64(win, 1) if p == 0 else _slope64(win, 1) if p == 1 else
                   _viewshed64(win, obs, 10.0, 167.0) if p == 2 else None)
    return got
