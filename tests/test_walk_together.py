"""Frames whose last paths' walks run eight lanes each, against the same frames
traced one walk a lane in the reference order (which counts its nodes): on
either side of the path count that gives every warp four paths or fewer."""
import pytest

from helpers import assert_bits_equal, scene_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 3, 4])
@pytest.mark.parametrize("size", [(1, 1), (5, 1), (33, 31), (97, 100), (98, 100), (160, 121)])
def test_last_walks_together(gbdev, mode, size):
    (v, t, m), cam = scene_arrays("interior")
    p = gbdev.default_params(eye_depth_max=6, light_depth_max=5, pt_depth_max=7, bilat_radius=2)
    s = gbdev.RTScene(v, t, m).build_bvh()
    images = []
    for counting in (True, False):
        r = gbdev.RTRenderer(*size, mode, p)
        r.set_counting(counting)
        for _ in range(3):
            r.render(s, cam)
        images.append((r.read_buffer(0), r.read_buffer(6)))
    assert_bits_equal(images[1][0], images[0][0], "image")
    assert_bits_equal(images[1][1], images[0][1], "sampleN")
