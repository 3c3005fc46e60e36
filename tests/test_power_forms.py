"""Powers of float32 cells: exponents written into the source take the products of
map_powf, exponents known only on the device CUDA's powf with no test per cell; both
forms compile one cell at a time and paired."""
import numpy as np
import pytest


@pytest.mark.parametrize("paired", [True, False])
def test_products_for_fixed_exponents_only(M, paired):
    x = M.from_numpy(np.ones((64, 64), np.float32), bs=[32, 32])
    y = M.from_numpy(np.ones((64, 64), np.float32), bs=[32, 32])
    box = M.convolve(x, [[1.0] * 3] * 3)
    M.set_paired_cells(paired)
    try:
        # (program, its exponent is in the source)
        for prog, fixed in ((x ** 2.0, True), (x ** 3, True), (x ** 2.5, True), (x ** y, False), (x ** M.zmax(y), False),
                            (2.0 ** x, False), (box ** 3.0, True), (box ** y, False), (M.zsum(x ** 3.0), True), (M.zsum(x ** y), False)):
            src = M.generated_source(prog)
            assert ("map_powf(" in src) == fixed
            assert any(f in src for f in (" powf(", "(powf(", "pr_powf(")) == (not fixed)
            assert M.compile_only(prog) >= 1
    finally:
        M.set_paired_cells(True)
