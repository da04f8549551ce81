"""Device memory that suffices for a scene but not for the ordered walk's tree:
the scene is uploaded without the tree and answers as before."""
import ctypes

import numpy as np
import pytest

from helpers import assert_bits_equal, random_rays, scene_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("textured", [False, True])
@pytest.mark.parametrize("room", [0, 1, 2, 3])  # of the tree's three allocations
def test_no_memory_for_the_tree(gbdev, textured, room):
    import torch
    (v, t, m), cam = scene_arrays("interior")
    L = gbdev._native.load()
    rays = random_rays(v, 5000, 8)
    n = len(rays)
    s = gbdev.RTScene(v, t, m).build_bvh()
    plain = gbdev.RTScene(v, t, m).build_bvh()
    if textured:
        for q in (s, plain):
            q.set_textures([np.ones((4, 4, 4), np.float32)])
    want = plain.trace_rays(rays, counts=True, eps=1e-4)
    d = torch.from_numpy(rays).cuda()
    out = [torch.empty(n, device="cuda") for _ in range(4)]
    tri = torch.empty(n, dtype=torch.int32, device="cuda")
    needed = 5 + (3 if textured else 0)  # the scene's own arrays
    try:
        L.gbpt_test_fail_allocations(needed + room)
        st = L.gbpt_trace_rays(s.handle, d.data_ptr(), n, ctypes.c_float(1e20), ctypes.c_float(1e-4), 0,
                               out[0].data_ptr(), tri.data_ptr(), *(o.data_ptr() for o in out[1:]), None, None, 1)
    finally:
        L.gbpt_test_fail_allocations(-1)
    assert st == 0, L.gbpt_last_error_string()
    assert_bits_equal(tri.cpu().numpy(), want["tri"], "tri")
    for k, o in zip(("t", "w", "u", "v"), out):
        assert_bits_equal(o.cpu().numpy(), want[k], k)
    extra = []
    for counting in (True, False):
        r = gbdev.RTRenderer(16, 12, 0, gbdev.default_params(tail_from=2))
        r.set_counting(counting)
        r.render(s, cam)
        extra.append(r.last_stats["launches"])
    assert extra[1] - extra[0] == (3 if room == 3 else 0)  # the ordered walk's checks


def test_too_little_for_the_scene_is_reported(gbdev):
    (v, t, m), _ = scene_arrays("interior")
    L = gbdev._native.load()
    for after in range(5):
        s = gbdev.RTScene(v, t, m).build_bvh()
        try:
            L.gbpt_test_fail_allocations(after)
            with pytest.raises(gbdev.GbptError) as e:
                s.trace_rays(random_rays(v, 4, 8))
            assert e.value.status == 2  # GBPT_ERR_OOM
        finally:
            L.gbpt_test_fail_allocations(-1)
        assert len(s.trace_rays(random_rays(v, 4, 8))["tri"]) == 4
