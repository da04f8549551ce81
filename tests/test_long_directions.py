"""Rays whose directions are very long or very short: the ordered walk (the
default where nothing is counted) answers as the reference-order walk, word for
word, up to the largest float."""
import numpy as np
import pytest

from helpers import assert_bits_equal, random_rays, scene_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [2.0 ** -9, 1.0, 300.0])
@pytest.mark.parametrize("name", ["cornell", "interior"])
def test_directions_of_any_length(gbdev, name, scale):
    (v, t, m), _ = scene_arrays(name)
    v = v.copy()
    v["pos"] *= np.float32(scale)
    s = gbdev.RTScene(v, t, m).build_bvh()
    rays = np.tile(random_rays(v, 2000, 31, pad=0.1 * scale), (24, 1))
    rng = np.random.Generator(np.random.PCG64(32))
    exps = np.repeat([-60, -29, 0, 20, 38, 39, 40, 41, 42, 44, 48, 55, 62, 68, 74, 80, 86, 92, 98, 104, 110, 116, 122,
                      126], 2000)
    length = np.ldexp(1.0, exps)[:, None] * np.where(rng.random((len(rays), 3)) < 0.8, 1.0, 0.0)  # all axes, or some
    one = rng.random(len(rays)) < 0.5
    length[one] = np.ldexp(1.0, exps[one])[:, None]
    with np.errstate(over="ignore"):
        rays[:, 3:] = np.where(length > 0, rays[:, 3:] * length, rays[:, 3:]).astype(np.float32)
    hits = 0
    for kw in (dict(eps=0.0), dict(eps=0.0, max_dist=float("inf")), dict(eps=0.0, max_dist=1e-12), dict()):
        want, got = s.trace_rays(rays, counts=True, **kw), s.trace_rays(rays, **kw)
        hits += (want["tri"][exps >= 92] >= 0).sum()
        for k in ("tri", "t", "w", "u", "v"):
            assert_bits_equal(got[k], want[k], f"{name} x {scale} {kw} {k}")
    assert hits > 1000  # the reference answers long rays, too
