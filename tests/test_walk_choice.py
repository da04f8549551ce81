"""A scene whose rays often run past the reference's pop bound keeps the
node-by-node walk, others get the ordered one, seen by the three launches a frame
of the ordered walk adds to check its answers.  Images are equal either way."""
import pytest

from helpers import assert_bits_equal, scene_arrays
from test_ordered import _sticks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,ordered", [("interior", True), ("hall_small", True), ("sticks", False)])
def test_walk_of_the_scene(gbdev, name, ordered):
    (v, t, m), cam = _sticks(4000) if name == "sticks" else scene_arrays(name)
    s = gbdev.RTScene(v, t, m).build_bvh()
    got = []
    for counting in (True, False):
        r = gbdev.RTRenderer(40, 30, 0, gbdev.default_params(eye_depth_max=5, light_depth_max=4, tail_from=2))
        r.set_counting(counting)
        launches = [r.render(s, cam) is not None and r.last_stats["launches"] for _ in range(3)]
        got.append((launches, r.read_buffer(0)))
    assert got[1][0] == [n + (3 if ordered else 0) for n in got[0][0]]
    assert_bits_equal(got[1][1], got[0][1], name)
