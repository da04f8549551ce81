"""A scene whose rays often run past the reference's pop bound keeps the
node-by-node walk, others get the ordered one, seen by the three launches a frame
of the ordered walk adds to check its answers.  Images are equal either way."""
import numpy as np
import pytest

from helpers import assert_bits_equal, scene_arrays
from test_ordered import _sticks

pytestmark = pytest.mark.gpu


def _model_in_a_space():
    """The sticks in a space so large that rays from anywhere in it hardly meet them."""
    (v, t, m), cam = _sticks(4000)
    far = np.zeros(6, v.dtype)
    far["pos"] = np.repeat(np.float32([[-600.0], [610.0]]), 3, 0) + np.tile(np.eye(3, dtype=np.float32), (2, 1))
    ft = np.zeros(2, t.dtype)
    for k, corner in enumerate(("v0", "v1", "v2")):
        ft[corner] = len(v) + np.array([k, 3 + k])
    return (np.concatenate([v, far]), np.concatenate([t, ft]), m), cam


@pytest.mark.parametrize("name,ordered", [("interior", True), ("hall_small", True), ("sticks", False), ("model", False)])
def test_walk_of_the_scene(gbdev, name, ordered):
    (v, t, m), cam = {"sticks": lambda: _sticks(4000), "model": _model_in_a_space}.get(name, lambda: scene_arrays(name))()
    s = gbdev.RTScene(v, t, m).build_bvh()
    got = []
    for counting in (True, False):
        r = gbdev.RTRenderer(40, 30, 0, gbdev.default_params(eye_depth_max=5, light_depth_max=4, tail_from=2))
        r.set_counting(counting)
        launches = [r.render(s, cam) is not None and r.last_stats["launches"] for _ in range(3)]
        got.append((launches, r.read_buffer(0)))
    assert got[1][0] == [n + (3 if ordered else 0) for n in got[0][0]]
    assert_bits_equal(got[1][1], got[0][1], name)
