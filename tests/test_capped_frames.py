"""Frames with many walks past the reference's 2048 pops, whose taken answers are
checked and run again: several frames side by side, split into bands, with the
tail kernel from the first bounce to none, without carrying, and with the
learned allocator's statistics kept.  The oracle's image, word for word."""
import functools

import numpy as np
import pytest

from helpers import assert_bits_equal, camera_rays
from test_ordered import _sticks

pytestmark = pytest.mark.gpu

SIZES = [(61, 37), (16, 9)]  # more such walks than the lists hold, and fewer


@functools.lru_cache(maxsize=None)
def _scene():
    """The sticks among so many other triangles that few of the scene's rays meet them: it gets the
    ordered walk's tree."""
    import cudapt_gb300 as gb
    (v, t, m), cam = _sticks(6000)
    n = 620  # a far floor of 2 n^2 small triangles
    at = np.linspace(-600, 610, n + 1, dtype=np.float32)
    x, z = np.meshgrid(at, at)
    far = np.zeros((n + 1) ** 2, v.dtype)
    far["pos"] = np.stack([x.ravel(), np.full(x.size, -600, np.float32), z.ravel()], 1)
    far["norm"] = (0.0, 1.0, 0.0)
    i = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).ravel() + len(v)
    ft = np.zeros(2 * n * n, t.dtype)
    for name, corner in (("v0", (0, 0)), ("v1", (n + 2, n + 1)), ("v2", (1, n + 2))):
        ft[name] = np.concatenate([i + corner[0], i + corner[1]])
    v, t = np.concatenate([v, far]), np.concatenate([t, ft])
    s = gb.RTScene(v, t, m).build_bvh()
    assert (s.trace_rays(camera_rays(cam, *SIZES[0], 1), counts=True, eps=1e-4)["nodes"] == 2048).sum() > 100
    launches = []
    for counting in (True, False):  # the ordered walk adds three launches that check its answers
        r = gb.RTRenderer(8, 8, 0, _params(tail_from=2))
        r.set_counting(counting)
        r.render(s, cam)
        launches.append(r.last_stats["launches"])
    assert launches[1] == launches[0] + 3
    return s, (v, t, m), cam


def _params(**kw):
    import cudapt_gb300 as gb
    return gb.default_params(eye_depth_max=5, light_depth_max=4, pt_depth_max=5, warmup_frames=3, filter_radius=2,
                             bilat_radius=2, **kw)


@functools.lru_cache(maxsize=None)
def _oracle_scene():
    import oracle
    return oracle.Scene(*_scene()[1])


@functools.lru_cache(maxsize=None)
def _want(size, mode, light_every):
    import oracle
    cam = _scene()[2]
    ref = oracle.Renderer(*size, mode, _params(light_every=light_every))
    ref.render(_oracle_scene(), cam, 5)
    return ref.get(0), ref.sample_counts()[0]


OPTIONS = [dict(), dict(light_every=1), dict(tail_from=0), dict(tail_from=2), dict(tail_from=5), dict(tail_below=0.5),
           dict(carry_steps=0), dict(carry_steps=1), dict(bands=2), dict(bands=3), dict(bands=8, carry_steps=0),
           dict(bands=2, tail_from=2)]


@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("options", OPTIONS, ids=str)
@pytest.mark.parametrize("size", SIZES, ids=str)
def test_many_corrected_walks(gbdev, orc, size, mode, options):
    s, _, cam = _scene()
    want, counts = _want(size, mode, options.get("light_every", 3))
    for stats in (False, True):  # side by side, and one after another
        r = gbdev.RTRenderer(*size, mode, _params(**options))
        r.render_frames(s, cam, 5, stats=stats)
        assert_bits_equal(r.read_buffer(0), want, f"image, stats {stats}")
        assert_bits_equal(r.read_buffer(6), counts, f"sampleN, stats {stats}")


@pytest.mark.parametrize("tail_from", [-1, 0, 5])
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("size", SIZES, ids=str)
def test_statistics_of_the_learned_allocator(gbdev, size, mode, tail_from):
    """Second moments and path lengths are added to as a path is shaded: walks wait for their answers."""
    s, _, cam = _scene()
    got = []
    for counting in (True, False):
        r = gbdev.RTRenderer(*size, mode, _params(tail_from=tail_from))
        r.set_mlp(None, collect=True)
        r.set_counting(counting)
        r.render_frames(s, cam, 5, stats=False)
        got.append([r.read_buffer(k) for k in (0, 6, 11, 12)])
    for a, b, what in zip(*got, ("image", "sampleN", "second moments", "path lengths")):
        assert_bits_equal(b, a, what)


@pytest.mark.parametrize("size", [(64, 47), (672, 464)], ids=str)  # a thread a ray, and shared out over warps
def test_rays_past_the_bound(gbdev, size):
    s, _, cam = _scene()
    rays = camera_rays(cam, *size, 3)
    for kw in (dict(eps=1e-4), dict(), dict(max_dist=40.0, eps=1e-4)):
        want, got = s.trace_rays(rays, counts=True, **kw), s.trace_rays(rays, **kw)
        assert (want["nodes"] == 2048).mean() > 0.01
        for k in ("tri", "t", "w", "u", "v"):
            assert_bits_equal(got[k], want[k], f"{size} {kw} {k}")
