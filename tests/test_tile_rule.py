"""Tiles of standalone focal kernels by raster size (CPU: read from the generated
source): flat hillshade tiles below six million cells whatever the raster's height."""
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
