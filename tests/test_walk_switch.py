"""A view most of whose walks pass the reference's pop bound overfills the lists
of such walks; the rest of its sequence then takes the node-by-node walk, with
one band or several and in the modes whose walks wait for their answers.  Seen by
the launches a frame of the ordered walk adds; the images do not change."""
import pytest

from helpers import assert_bits_equal
from test_capped_frames import _params, _scene

pytestmark = pytest.mark.gpu


def _launches(gbdev, size, mode, frames, **options):
    """Launches of the ordered walk's frames beyond those of the counted (node-by-node) walk's."""
    s, _, cam = _scene()
    got = []
    for counting in (True, False):
        r = gbdev.RTRenderer(*size, mode, _params(**options))
        r.set_counting(counting)
        n = []
        for _ in range(frames):
            r.render(s, cam)
            n.append(r.last_stats["launches"])
        got.append((n, r.read_buffer(0)))
    assert_bits_equal(got[1][1], got[0][1], "image")
    return [b - a for a, b in zip(got[0][0], got[1][0])]


@pytest.mark.parametrize("size,bands", [((61, 37), 1), ((61, 37), 3), ((40, 24), 8)], ids=str)
def test_full_lists_of_bands(gbdev, size, bands):
    # a list has 256 records, a band's a share of them: 32 in the last case, whose bands have 120 paths each
    extra = _launches(gbdev, size, 0, 3, bands=bands, tail_from=5)
    assert extra == [3 * bands, 0, 0]


@pytest.mark.parametrize("collect", [False, True])
def test_full_lists_of_walks_that_wait(gbdev, collect):
    # 12,288 paths: a list of 256, and over 1,000 such camera rays
    s, _, cam = _scene()
    got = []
    for counting in (True, False):
        r = gbdev.RTRenderer(128, 96, 1 if collect else 3, _params(tail_from=5, carry_steps=0))
        if collect:
            r.set_mlp(None, collect=True)
        r.set_counting(counting)
        n = []
        for _ in range(3):
            r.render(s, cam)
            n.append(r.last_stats["launches"])
        got.append(n)
    extra = [b - a for a, b in zip(*got)]
    assert extra == [3 + 6, 0, 0]  # three checks, and the answers for each of six launches of walks


def test_lists_with_room(gbdev):
    assert _launches(gbdev, (8, 6), 0, 3, tail_from=2) == [3, 3, 3]


def test_views_after_a_full_list(gbdev):
    """The next sixteen views of the scene keep the node-by-node walk, then the ordered one is tried
    again, and 32 views later; another scene starts anew."""
    s, arrays, cam = _scene()
    other = gbdev.RTScene(*arrays).build_bvh()
    got = []
    for counting in (True, False):
        r = gbdev.RTRenderer(61, 37, 0, _params(tail_from=5))
        r.set_counting(counting)
        n = []
        for k in range(53):
            r.render(s, dict(cam, pos=(5.0, 5.0, 16.0 + 0.01 * k)))
            n.append(r.last_stats["launches"])
        r.render(other, cam)
        n.append(r.last_stats["launches"])
        got.append((n, r.read_buffer(0)))
    extra = [b - a for a, b in zip(got[0][0], got[1][0])]
    assert extra == [3] + 16 * [0] + [3] + 32 * [0] + [3] + 2 * [0] + [3]
    assert_bits_equal(got[1][1], got[0][1], "image")
