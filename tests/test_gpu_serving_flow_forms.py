"""Flow accumulations in serving: the memory a request is charged is what its form
takes, and the forms that stand in for the tiles (MAP_B200_SERVE_PJ: pointer jumping
above 64 K cells, the one-CTA sweep below or alone) give the same cells. The variable
is read once, so each form runs in a process of its own."""
import ctypes as ct
import os
import subprocess
import sys

import numpy as np
import pytest

from map_b200 import synth

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes as ct, sys
import numpy as np
from map_b200 import map as M, synth
dem = synth.fbm_dem(700, 800, seed=21)
d = M._lib.ma_devAlloc(dem.nbytes)
M._lib.ma_memcpy(ct.c_void_p(d), dem.ctypes.data_as(ct.c_void_p), dem.nbytes, 1)
srv = M.Server(d, 800 * 4, 800, 700, budget_bytes=256 << 20, max_batch=16)
sizes = [(300, 260), (64, 64), (1, 90), (200, 300), (513, 400), (65, 3)]
ids = [srv.submit(M.Server.FLOW, 11 * k, 7 * k, w, h) for k, (w, h) in enumerate(sizes)]
for k, (i, (w, h)) in enumerate(zip(ids, sizes)):
    got = srv.result(i, (h, w), np.int32)
    win = M.from_numpy(np.ascontiguousarray(dem[7 * k:7 * k + h, 11 * k:11 * k + w]), bs=[w, h])
    want = M.to_numpy(M.flow_accumulation(M.ones_like(win, M.S32), M.flow_direction(win)))
    assert np.array_equal(got, want), (w, h)
srv.close()
print("same")
"""


@pytest.mark.parametrize("form", [None, "1", "0"])
def test_forms_agree(form):
    env = {k: v for k, v in os.environ.items() if k != "MAP_B200_SERVE_PJ"}
    if form is not None:
        env["MAP_B200_SERVE_PJ"] = form
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stderr[-2000:]


def test_charged_what_the_tiles_take(M):
    # two 512 x 512 flow windows: rasters and directions 2.3 MB each, the tiles' scratch 0.3 MB
    dem = synth.fbm_dem(600, 600, seed=5)
    d = M._lib.ma_devAlloc(dem.nbytes)
    M._lib.ma_memcpy(ct.c_void_p(d), dem.ctypes.data_as(ct.c_void_p), dem.nbytes, 1)
    budget = 6 << 20
    srv = M.Server(d, 600 * 4, 600, 600, budget_bytes=budget, max_batch=8)
    try:
        ids = [srv.submit(M.Server.FLOW, 8 * k, 4 * k, 512, 512) for k in range(5)]
        outs = [srv.result(i, (512, 512), np.int32) for i in ids]
        st = srv.stats()
        assert st["completed"] == 5 and 2 * 512 * 512 * 4 < st["peak_bytes"] <= budget
        win = M.from_numpy(np.ascontiguousarray(dem[8:520, 16:528]), bs=[512, 512])
        assert np.array_equal(outs[2], M.to_numpy(M.flow_accumulation(M.ones_like(win, M.S32), M.flow_direction(win))))
    finally:
        srv.close()
        M._lib.ma_devFree(ct.c_void_p(d))
