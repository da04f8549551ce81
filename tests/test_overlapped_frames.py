"""Several frames in one call are traced side by side; the image, the sample
counts and the guide planes are those of the same frames one call each."""
import pytest

from helpers import assert_bits_equal, scene_arrays

pytestmark = pytest.mark.gpu


def _compare(gbdev, scene, size, mode, frames, calls=1, setup=None, **params):
    (v, t, m), cam = scene_arrays(scene)
    p = gbdev.default_params(eye_depth_max=5, light_depth_max=4, pt_depth_max=6, warmup_frames=3, filter_radius=2,
                             bilat_radius=2, **params)
    s = gbdev.RTScene(v, t, m).build_bvh()
    one, many = (gbdev.RTRenderer(*size, mode, p) for _ in range(2))
    for r in (one, many):
        if setup:
            setup(r)
    for k in range(calls):
        moved = dict(cam, fov=cam["fov"] * (1.0 + 0.01 * (k // 2)))  # the same camera twice, then another
        for _ in range(frames):
            one.render(s, moved)
        many.render_frames(s, moved, frames, stats=False)
        for what in (0, 1, 2, 3, 6):
            assert_bits_equal(many.read_buffer(what), one.read_buffer(what), f"buffer {what} after call {k}")


@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("frames", [2, 3, 5, 9])
def test_one_call_equals_a_call_a_frame(gbdev, mode, frames):
    _compare(gbdev, "interior", (75, 53), mode, frames, calls=3)


@pytest.mark.parametrize("light_every", [1, 2, 3, 7])
@pytest.mark.parametrize("mode", [0, 3])
def test_light_pass_groups(gbdev, mode, light_every):
    _compare(gbdev, "interior", (40, 31), mode, 8, calls=3, light_every=light_every)


@pytest.mark.parametrize("size", [(1, 1), (512, 255), (512, 257), (1024, 511), (1024, 513)])
def test_sizes_about_the_slot_rule(gbdev, size):
    _compare(gbdev, "cornell", size, 0, 6, calls=2)


@pytest.mark.parametrize("setup", [lambda r: r.set_graphs(True), lambda r: r.set_counting(True), None])
@pytest.mark.parametrize("params", [dict(), dict(bands=2), dict(carry_steps=0), dict(tail_from=0), dict(tail_from=5)])
def test_with_other_scheduling(gbdev, setup, params):
    _compare(gbdev, "interior", (90, 41), 0, 5, setup=setup, **params)


def test_frames_that_only_filter(gbdev):
    _compare(gbdev, "interior", (60, 41), 3, 7, calls=2, render_iterations=4)


def test_on_the_callers_stream(gbdev):
    import torch
    from cudapt_gb300._native import check, load
    st = torch.cuda.Stream()
    _compare(gbdev, "interior", (60, 41), 0, 6, calls=2,
             setup=lambda r: check(load().gbpt_renderer_set_stream(r._h, st.cuda_stream)))


@pytest.mark.parametrize("size", [(256, 227), (256, 228), (342, 341), (342, 342)])
@pytest.mark.parametrize("mode", [0, 3])
def test_sizes_about_the_tail_start(gbdev, mode, size):
    _compare(gbdev, "cornell", size, mode, 4)


@pytest.mark.parametrize("params", [dict(), dict(light_every=1), dict(bands=2, carry_steps=0), dict(bands=3)])
@pytest.mark.parametrize("mode", [0, 1, 3])
def test_light_pass_beside_the_first_walks(gbdev, mode, params):
    """Calls of one frame without statistics start their bounce launches while the light pass runs."""
    (v, t, m), cam = scene_arrays("interior")
    p = gbdev.default_params(eye_depth_max=5, light_depth_max=4, warmup_frames=3, filter_radius=2, bilat_radius=2,
                             tail_from=5, **params)
    s = gbdev.RTScene(v, t, m).build_bvh()
    a, b = (gbdev.RTRenderer(70, 51, mode, p) for _ in range(2))
    for k in range(8):
        moved = dict(cam, fov=cam["fov"] * (1.0 + 0.01 * (k // 4)))
        a.render_frames(s, moved, 1, stats=True)
        b.render_frames(s, moved, 1, stats=False)
        for what in (0, 6):
            assert_bits_equal(b.read_buffer(what), a.read_buffer(what), f"buffer {what} after frame {k}")
