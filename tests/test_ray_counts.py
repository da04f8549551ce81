"""gbpt_stats counts the rays of the frame's paths: a path that is run again
because a walk's taken answer was wrong counts once, as in the reference-order
walk (the one that counts its nodes)."""
import pytest

from test_capped_frames import SIZES, _params, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("options", [dict(), dict(tail_from=0), dict(tail_from=5), dict(bands=3)], ids=str)
@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("size", SIZES, ids=str)
def test_rays_of_corrected_paths(gbdev, size, mode, options):
    s, _, cam = _scene()
    got = []
    for counting in (True, False):
        r = gbdev.RTRenderer(*size, mode, _params(**options))
        r.set_counting(counting)
        st = r.render_frames(s, cam, 5)
        got.append({k: st[k] for k in ("rays", "shadow_rays", "paths", "light_vertices", "frame")})
    assert got[1] == got[0]
