"""Device rasters whose rows start on no 16-byte boundary, read and written in place:
every kind of group gives the bytes it gives on aligned rasters, under every border
rule and launch mode, and a program evaluated into its own input keeps working."""
import numpy as np
import pytest

from map_b200 import synth
from map_b200 import workloads as W

pytestmark = pytest.mark.gpu

W3 = [[1, 2, 1], [2, 4, 2], [1, 2, 1]]
W5 = [[1] * 5] * 5


def programs(M, f, b):
    """(name, raster) of programs over the float raster f and the byte raster b."""
    return [("hillshade", W.hillshade(f)), ("slope", W.slope(f)), ("conv5", M.convolve(f, W5)),
            ("chain", M.convolve(M.convolve(f, W3) * 0.0625, W3)), ("two reads", M.convolve(f, W3) + f * 2.0),
            ("local", f * 3.0 + 1.0), ("life", W.life_step(b)), ("life4", W.life(b, 4)), ("d8", M.flow_direction(f)),
            ("flow", M.flow_accumulation(M.ones_like(f, M.S32), M.flow_direction(f))),
            ("view", W.viewshed(f, [20, 30], 5.0)), ("mixed", M.convolve(b, W3) + M.convolve(f, W3))]


class Held:
    """A raster inside a larger allocation: `off` cells in, rows `pitch` cells apart."""

    def __init__(self, shape, dtype, off, pitch, cells=None):
        import torch
        self.h, self.w = shape
        self.off, self.pitch = off, pitch
        self.t = torch.full((off + pitch * self.h + 64,), 77, dtype=dtype, device="cuda")
        if cells is not None:
            self.view().copy_(torch.from_numpy(cells).cuda())

    def view(self):
        import torch
        return torch.as_strided(self.t, (self.h, self.w), (self.pitch, 1), self.off)

    def ptr(self):
        return self.t.data_ptr() + self.off * self.t.element_size()

    def bytes(self):
        return self.pitch * self.t.element_size()


def sources(M, shape, off, pitch):
    import torch
    h, w = shape
    f = Held(shape, torch.float32, off, pitch, synth.fbm_dem(h, w, seed=3))
    b = Held(shape, torch.uint8, off, pitch, synth.bernoulli_u8(h, w, 0.3, seed=3))
    torch.cuda.synchronize()
    return (f, b), [M.from_device(x.ptr(), x.bytes(), [w, h], dt, [64, 48]) for x, dt in ((f, M.F32), (b, M.U8))]


def torch_dtype(M, dt):
    import torch
    return {M.F32: torch.float32, M.U8: torch.uint8, M.S32: torch.int32, M.F64: torch.float64}[dt]


@pytest.mark.parametrize("shape", [(70, 129), (200, 333)])
@pytest.mark.parametrize("off,extra", [(0, 0), (1, 3), (3, 8)])
@pytest.mark.parametrize("border,plain", [(0, False), (1, False), (2, False), (0, True)])
def test_same_as_aligned(M, shape, off, extra, border, plain):
    import torch
    h, w = shape
    M.set_border(border)
    M.set_exec_mode(M.EXEC_PLAIN if plain else M.EXEC_FUSED)
    try:
        keep, (f, b) = sources(M, shape, off, w + extra)
        keep2, (fa, ba) = sources(M, shape, 0, (w + 127) // 128 * 128)
        for (name, got_r), (_, want_r) in zip(programs(M, f, b), programs(M, fa, ba)):
            out = Held(shape, torch_dtype(M, got_r.datatype()), off, w + extra)
            torch.cuda.synchronize()
            M.to_device(got_r, out.ptr(), out.bytes())
            want = M.to_numpy(want_r)
            assert np.array_equal(out.view().cpu().numpy(), want, equal_nan=want.dtype.kind == "f"), name
            # nothing outside the raster's cells was written
            out.view().fill_(77)
            assert bool((out.t == 77).all()), name
    finally:
        M.set_exec_mode(M.EXEC_FUSED)
        M.set_border(M.BORDER_BLOCK_MIRROR)


@pytest.mark.parametrize("shift", [0, 1, 400])
def test_into_memory_of_the_input(M, shift):
    # the output's rows start `shift` cells after the input's, in the same memory
    import torch
    h, w = 90, 333
    x = Held((h + 4, w), torch.float32, 1, w)
    src = synth.fbm_dem(h, w, seed=9)
    x.t[1:1 + h * w].copy_(torch.from_numpy(src).cuda().view(-1))
    torch.cuda.synchronize()
    r = M.from_device(x.ptr(), w * 4, [w, h], M.F32, [64, 64])
    M.to_device(M.convolve(r, W3), x.ptr() + 4 * shift, w * 4)
    want = M.to_numpy(M.convolve(M.from_numpy(src, bs=[64, 64]), W3))
    got = x.t[1 + shift:1 + shift + h * w].view(h, w).cpu().numpy()
    assert np.array_equal(got, want)
