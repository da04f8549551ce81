"""Distributed shared memory may be touched only once every block of the
cluster has started.  A store to a block that has not is undefined and may
fault, so the rule is checked on the kernels' sources: in each kernel that maps
another block's shared memory, a cluster-wide barrier comes before the first
access, outside every loop."""
import glob
import os
import re

import pytest

from helpers import assert_bits_equal, scene_arrays

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
REMOTE = re.compile(r"map_shared_rank|\bmapa\b|ld\.shared::cluster|st\.(async\.)?\S*shared::cluster")
BARRIER = re.compile(r"(this_cluster\(\)|\bcluster)\s*\.\s*sync\(\)|barrier\.cluster\.wait")


def _kernels(src):
    src = re.sub(r"//[^\n]*", "", src)
    for m in re.finditer(r"__global__[^;{]*\{", src):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield m.group(0), src[m.end():i]


def _before_loops(body):
    m = re.search(r"\b(for|while|do)\b", body)
    return body[:m.start()] if m else body


def test_blocks_of_a_cluster_meet_before_they_share_memory():
    found = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "cudapt_gb300", "csrc", "*.cu*"))):
        for head, body in _kernels(open(path).read()):
            first = REMOTE.search(body)
            if not first:
                continue
            found += 1
            early = _before_loops(body[:first.start()])
            assert BARRIER.search(early), f"{os.path.basename(path)}: {head.split('(')[0]} ... has no cluster barrier"
    assert found  # the light pass


@pytest.mark.gpu
@pytest.mark.parametrize("paths", [1, 31, 32, 33, 127, 128, 129])
def test_light_pass_of_one_and_of_eight_blocks(gbdev, orc, paths):
    """Up to 128 light paths run in a cluster of eight blocks, more in one block."""
    (v, t, m), cam = scene_arrays("interior")
    p = gbdev.default_params(light_paths=paths, light_depth_max=5)
    r = gbdev.RTRenderer(20, 16, 0, p)
    r.render(gbdev.RTScene(v, t, m).build_bvh(), cam)
    ref = orc.Renderer(20, 16, 0, p)
    ref.render(orc.Scene(v, t, m), cam, 1)
    want = ref.light_cache()
    assert r.last_stats["light_vertices"] == len(want)
    assert_bits_equal(r.light_cache(len(want)), want, f"{paths} light paths")
