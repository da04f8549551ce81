"""The ordered walk (the default where nothing is counted) against the
reference-order walk and the oracle, word for word: leaf shapes and tree
depths, rays with zero, tiny, huge, NaN and infinite components, origins
outside its range, distance limits, and walks past the reference's 2048 pops
in every renderer mode."""
import numpy as np
import pytest

from cudapt_gb300 import layouts, scenes
from helpers import assert_bits_equal, camera_rays, random_rays, scene_arrays

pytestmark = pytest.mark.gpu


def _sticks(n=12000, seed=3):
    """Long thin triangles through one room: every ray crosses thousands of boxes."""
    rng = np.random.Generator(np.random.PCG64(seed))
    mb = scenes.MeshBuilder()
    grey = mb.add_material(layouts.material((0.7, 0.6, 0.5), specular=0.5, roughness=0.6))
    lamp = mb.add_material(layouts.material((0.8, 0.8, 0.8), emissive=(6.0, 6.0, 6.0)))
    a = rng.random((n, 3)) * 10
    d = rng.normal(size=(n, 3))
    d *= 6 / np.linalg.norm(d, axis=1, keepdims=True)
    w = rng.normal(size=(n, 3)) * 0.004
    mb.add_tris(np.stack([a, a + d, a + w], 1), grey)
    mb.add_quad((3, 10.5, 3), (7, 10.5, 3), (7, 10.5, 7), (3, 10.5, 7), lamp)
    cam = dict(pos=(5.0, 5.0, 16.0), dir=(0.0, 0.0, -1.0), up=(0.0, 1.0, 0.0), fov=0.9)
    return mb.build(), cam


def _far():
    """A small object far from the origin."""
    (v, t, m), cam = scenes.cornell()
    v = v.copy()
    v["pos"] += np.float32(300.0)
    return (v, t, m), dict(cam, pos=tuple(300.0 + x for x in cam["pos"]))


def _one():
    mb = scenes.MeshBuilder()
    mb.add_tris([[[0, 0, 0], [1, 0, 0], [0, 1, 0]]], mb.add_material(layouts.material()))
    return mb.build(), scenes.cornell()[1]


def _twins():
    """Every triangle four times: leaves of several triangles."""
    (v, t, m), cam = scene_arrays("cornell")
    return (v, np.concatenate([t] * 4), m), cam


SCENES = {
    "cornell": (lambda: scene_arrays("cornell"), 32), "interior": (lambda: scene_arrays("interior"), 32),
    "hall_small": (lambda: scene_arrays("hall_small"), 32), "shallow": (lambda: scene_arrays("interior"), 6),
    "sticks": (_sticks, 32), "far": (_far, 32), "one": (_one, 32), "twins": (_twins, 32),
}


def _rays(v, cam, n):
    rng = np.random.Generator(np.random.PCG64(9))
    r = np.concatenate([random_rays(v, n, 21), camera_rays(cam, 160, 120, 22), random_rays(v, 4096, 23, pad=40.0)])
    odd = random_rays(v, 8192, 24)
    k = rng.integers(0, 12, len(odd))
    for a in range(3):
        odd[(k == a), 3 + a] = 0.0
        odd[(k == 3 + a), 3 + a] *= np.float32(1e-12)
    odd[k == 6, 3:] *= np.float32(1e6)
    odd[k == 7, 3:] = np.nan
    odd[k == 8, 3] = np.nan
    odd[k == 9, 4] = np.inf
    odd[k == 10, 0] = np.inf
    odd[k == 11, :3] *= np.float32(1e4)
    odd[:64, 3:] = 0.0
    return np.concatenate([r, odd]).astype(np.float32)


@pytest.mark.parametrize("name", list(SCENES))
def test_ordered_hits_equal_reference_walk(gbdev, name):
    make, depth = SCENES[name]
    (v, t, m), cam = make()
    s = gbdev.RTScene(v, t, m).build_bvh(max_depth=depth)
    rays = _rays(v, cam, 4096 if name == "sticks" else 40_000)
    for kw in (dict(eps=1e-4), dict(), dict(max_dist=3.0, eps=1e-4), dict(max_dist=0.0), dict(max_dist=3e38),
               dict(max_dist=float("nan"))):
        want = s.trace_rays(rays, counts=True, **kw)
        got = s.trace_rays(rays, **kw)
        for k in ("tri", "t", "w", "u", "v"):
            assert_bits_equal(got[k], want[k], f"{name} {kw} {k}")
        if name == "sticks" and not kw:
            assert (want["nodes"] == 2048).mean() > 0.2  # the reference runs out of pops


@pytest.mark.parametrize("mode,frames", [(0, 4), (1, 4), (2, 4), (3, 3), (4, 4)])
@pytest.mark.parametrize("graphs", [False, True])
def test_frames_with_walks_past_the_pop_limit(gbdev, orc, mode, frames, graphs):
    if graphs and mode not in (0, 4):
        pytest.skip("graphs cover the plain and unidirectional modes")
    (v, t, m), cam = _sticks(6000)
    p = gbdev.default_params(eye_depth_max=5, light_depth_max=4, pt_depth_max=5, warmup_frames=2, filter_radius=2,
                             bilat_radius=2)
    s = gbdev.RTScene(v, t, m).build_bvh()
    r = gbdev.RTRenderer(61, 37, mode, p)
    if graphs:
        r.set_graphs(True)
    for _ in range(frames):
        r.render(s, cam)
    ref = orc.Renderer(61, 37, mode, p)
    ref.render(orc.Scene(v, t, m), cam, frames)
    assert_bits_equal(r.read_buffer(0), ref.get(0), "image")
    assert_bits_equal(r.read_buffer(6), ref.sample_counts()[0], "sampleN")


def test_camera_outside_the_ordered_range(gbdev, orc):
    """A camera farther out than the walk's range takes the reference walk."""
    (v, t, m), cam = scene_arrays("cornell")
    far = dict(cam, pos=(0.5, 0.5, 60.0), fov=0.03)
    p = gbdev.default_params(eye_depth_max=4, light_depth_max=4)
    s = gbdev.RTScene(v, t, m).build_bvh()
    r = gbdev.RTRenderer(40, 40, 0, p)
    ref = orc.Renderer(40, 40, 0, p)
    for _ in range(2):
        r.render(s, far)
    ref.render(orc.Scene(v, t, m), far, 2)
    assert_bits_equal(r.read_buffer(0), ref.get(0), "image")
