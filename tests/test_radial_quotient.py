"""The quotient of a radial scan's interpolation weight: the product with the
rounded reciprocal and one residual correction is the correctly rounded quotient
of every pair of cell numbers a front can hold below 2^20 (skeleton/scan.cuh
radial_weight). Both fused steps are replayed in float64: each product of two
floats is exact there, the residual too, and the corrected sum is off by less than
2^-53 of itself where no quotient lies within 2^-46 of a midpoint."""
import numpy as np


def quotient(d1, d0):
    f = np.float32
    a, b = d1.astype(f), d0.astype(f)
    rc = f(1) / b
    q = a * rc
    rem = (a.astype(np.float64) - q.astype(np.float64) * b.astype(np.float64)).astype(f)
    return (rem.astype(np.float64) * rc.astype(np.float64) + q.astype(np.float64)).astype(f)


def check(d1, d0):
    assert np.array_equal(quotient(d1, d0), d1.astype(np.float32) / d0.astype(np.float32))


def test_every_pair_of_small_fronts():
    for d0 in range(1, 2100):
        d1 = np.arange(d0 + 1)
        check(d1, np.full(d1.shape, d0))


def test_large_fronts():
    rng = np.random.default_rng(5)
    for d0 in np.unique(np.concatenate([2 ** np.arange(11, 20), 2 ** np.arange(11, 21) - 1,
                                        rng.integers(2100, 1 << 20, 200)])):
        d1 = np.unique(np.concatenate([np.arange(64), d0 - np.arange(64), rng.integers(0, d0 + 1, 20000)]))
        check(d1, np.full(d1.shape, d0))
