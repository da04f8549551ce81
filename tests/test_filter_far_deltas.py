"""Filter planes whose divisor 2 d^2 is a power of two outside the range of the
tile kernel's corrected quotient (a huge delta switches a plane off, a tiny one
keeps equal neighbours only), beside planes that need that quotient: the image
is the oracle's, word for word, infinite and NaN values in the guide planes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HUGE = [2.0 ** k for k in (19, 20, 59, 60, 61, 62)]
TINY = [2.0 ** -20, 2.0 ** -21, 2.0 ** -60]
DELTAS = ([(3.0, d, 0.3, 0.5) for d in HUGE + TINY] + [(d, 0.3, 0.7, 0.1) for d in HUGE + TINY] +
          [(3.0, 1.0, 1.0, d) for d in HUGE] + [(2.0 ** 61, 2.0 ** 60, 2.0 ** 62, 0.3), (50.0, 2.0 ** 61, 0.25, 0.5)])


@pytest.mark.parametrize("radius,emit", [(1, True), (4, False), (5, True), (9, False)])
def test_powers_of_two_outside_the_quotient(gbdev, orc, radius, emit):
    rng = np.random.Generator(np.random.PCG64(radius))
    W, H = 53, 39
    planes = [(rng.random(W * H * 3) * s).astype(np.float32) for s in (40.0, 3.0, 1.0, 2.0)]
    for k in range(4):
        planes[k][::7] = np.float32(0.5)  # equal neighbours
        for v in (np.inf, -np.inf, np.nan, 1e25) if k else (1e25, 1e-30):  # (a colour spreads to every neighbour)
            planes[k][rng.integers(0, W * H * 3, 2)] = np.float32(v)
    L = gbdev._native.load()
    g = np.zeros(64, np.float32)
    gbdev._native.check(L.gbpt_gaussian_table(0.5 * radius + 0.5, radius, g.ctypes.data))
    e = planes[3] if emit else None
    for deltas in DELTAS:
        out = np.zeros(W * H * 3, np.float32)
        gbdev._native.check(L.gbpt_bilateral(planes[0].ctypes.data, planes[1].ctypes.data, planes[2].ctypes.data,
                                             e.ctypes.data if emit else None, W, H, *deltas, radius, g.ctypes.data,
                                             out.ctypes.data, 0))
        want = orc.bilateral(planes[0], planes[1], planes[2], e, W, H, *deltas, radius,
                             orc.gaussian(0.5 * radius + 0.5, radius))
        assert np.array_equal(np.isnan(out), np.isnan(want)), deltas
        ok = ~np.isnan(want)
        assert ok.mean() > 0.1 and np.array_equal(out[ok].view(np.uint32), want[ok].view(np.uint32)), deltas
