"""Caller-supplied rays shared out over the warps of a persistent grid: counts
about a warp, a block, the whole grid and its next share, every ray answered
once and equal to the reference-order walk's answer."""
import pytest

from helpers import assert_bits_equal, random_rays, scene_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["cornell", "interior"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 155_649, 311_295, 311_296, 311_297, 400_003])
def test_rays_about_the_shares(gbdev, name, n):
    (v, t, m), _ = scene_arrays(name)
    s = gbdev.RTScene(v, t, m).build_bvh()
    rays = random_rays(v, n, 40)
    want, got = s.trace_rays(rays, counts=True, eps=1e-4), s.trace_rays(rays, eps=1e-4)
    for k in ("tri", "t", "w", "u", "v"):
        assert_bits_equal(got[k], want[k], f"{name} {n} rays {k}")
