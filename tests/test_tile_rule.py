"""Tiles of standalone focal kernels by raster size (CPU: read from the generated
source): flat hillshade tiles below six million cells whatever the raster's height, the
tiles of other focal kernels by the cells they cover, padding of narrow rasters included."""
import re

import numpy as np
import pytest

from map_b200 import workloads as W


def tile(M, program, w, h):
    x = M.from_numpy(np.zeros((h, w), np.float32), bs=[256, 256], copy=False)
    src = M.generated_source(program(M, x))
    found = re.findall(r"tile_interior<(\d+), (\d+)>", src)
    assert len(set(found)) == 1
    return tuple(map(int, found[0]))


@pytest.mark.parametrize("size,want", [((511, 512), (64, 16)), ((512, 511), (64, 16)), ((450, 520), (64, 16)), ((256, 1024), (64, 16)), ((64, 4000), (64, 16)),
                                       ((256, 256), (64, 16)), ((2400, 2499), (64, 16)), ((2400, 2501), (64, 64))])
def test_hillshade(M, size, want):
    assert tile(M, lambda M, x: W.hillshade(x), *size) == want


@pytest.mark.parametrize("size,want", [((1500, 1500), (64, 8)), ((20, 100000), (64, 16)), ((200, 14000), (64, 16)), ((100000, 20), (64, 8)),
                                       ((20, 40000), (64, 8)), ((64, 40000), (64, 8)), ((65, 24000), (64, 16)), ((2048, 2048), (64, 16)),
                                       ((3000, 3000), (64, 32))])
def test_correlation(M, size, want):
    assert tile(M, lambda M, x: M.convolve(x, [[1, 2, 1], [2, 4, 2], [1, 2, 1]]), *size) == want
