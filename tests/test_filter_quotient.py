"""The bilateral tile kernel's quotients (product, Markstein's with one or two
corrections, division) against the oracle's division, word for word, over
divisors of every kind, equal and far neighbours, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,emit", [(1, False), (4, False), (5, True), (7, True), (9, False)])
@pytest.mark.parametrize("deltas", [(50.0, 1.0, 0.25, 0.5), (3.0, 0.7, 0.3, 0.1), (0.02, 1.0, 1.0, 0.5),
                                    (1.0, 1.0, 1.0, 1e-8), (1e-8, 0.3, 1e9, 0.5), (1.1, 2.0, 0.5, 4.0)])
def test_tile_kernel_quotients(gbdev, orc, radius, emit, deltas):
    rng = np.random.Generator(np.random.PCG64(radius * 10 + int(emit)))
    W, H = 53, 39
    planes = [(rng.random(W * H * 3) * s).astype(np.float32) for s in (40.0, 3.0, 1.0, 2.0)]
    planes[1] = np.round(planes[1], 1)  # equal neighbours
    for k, v in ((0, 1e25), (1, np.float32(np.inf)), (2, np.float32(np.nan)), (0, 1e-30)):
        planes[k][rng.integers(0, W * H * 3, 5)] = v
    L = gbdev._native.load()
    g = np.zeros(64, np.float32)
    gbdev._native.check(L.gbpt_gaussian_table(0.5 * radius + 0.5, radius, g.ctypes.data))
    out = np.zeros(W * H * 3, np.float32)
    e = planes[3] if emit else None
    gbdev._native.check(L.gbpt_bilateral(planes[0].ctypes.data, planes[1].ctypes.data, planes[2].ctypes.data,
                                         e.ctypes.data if emit else None, W, H, *deltas, radius, g.ctypes.data,
                                         out.ctypes.data, 0))
    want = orc.bilateral(planes[0], planes[1], planes[2], e, W, H, *deltas, radius, orc.gaussian(0.5 * radius + 0.5,
                                                                                                  radius))
    assert np.array_equal(np.isnan(out), np.isnan(want))
    ok = ~np.isnan(want)
    assert ok.any() and np.array_equal(out[ok].view(np.uint32), want[ok].view(np.uint32)), (radius, emit, deltas)
