"""The recomputation of the block mirror's exceptional cells is part of the focal
kernel's own code: as a called function it took the kernel's registers with it, under
the border rules that never call it too."""
import numpy as np

from map_b200 import workloads as W


def test_no_calls_in_focal_kernels(M):
    x = M.from_numpy(np.zeros((64, 64), np.float32), bs=[32, 32])
    b = M.from_numpy(np.zeros((64, 64), np.uint8), bs=[32, 32])
    for prog in (W.hillshade(x), W.slope(x), M.convolve(x, [[1.0] * 5] * 5), M.flow_direction(x), W.life_step(b)):
        src = M.generated_source(prog)
        assert "focal_fix(a, t, smem)" in src and "__noinline__ void focal_fix" not in src
