"""The ordered walk's tree made in parts on several threads (from 16384 binary
nodes on) and in one: hits equal the reference walk's on either side."""
import numpy as np
import pytest

from cudapt_gb300 import layouts, scenes
from helpers import assert_bits_equal, random_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 8191, 8192, 8193, 40000])
def test_tree_sizes_about_the_parts_rule(gbdev, n):
    rng = np.random.Generator(np.random.PCG64(n))
    c = rng.uniform(0, 10, (n, 1, 3)) + rng.normal(0, 0.05 + 2.0 / n, (n, 3, 3))
    mb = scenes.MeshBuilder()
    mb.add_tris(c.astype(np.float32), mb.add_material(layouts.material((0.7, 0.6, 0.5), emissive=(1.0, 1.0, 1.0))))
    v, t, m = mb.build()
    s = gbdev.RTScene(v, t, m).build_bvh()
    rays = random_rays(v, 20_000, 5)
    want, got = s.trace_rays(rays, counts=True, eps=1e-4), s.trace_rays(rays, eps=1e-4)
    for k in ("tri", "t", "w", "u", "v"):
        assert_bits_equal(got[k], want[k], f"{n} triangles {k}")
