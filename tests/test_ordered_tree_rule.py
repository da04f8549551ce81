"""Which scenes get the ordered walk's tree.  Its child planes lie outwards by
2^-17 of the scene's largest coordinate, so a scene of small triangles far from
the origin keeps the node-by-node walk: there the moved planes would have a ray
visit several times the leaves."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "gbpt_internal.h"
int main(int argc, char** argv) {  // triangles, their size, the scene's place
  const unsigned n = (unsigned)std::atoi(argv[1]);
  const float size = (float)std::atof(argv[2]), at = (float)std::atof(argv[3]);
  std::vector<gbpt_vertex> v(3 * (size_t)n);
  std::vector<gbpt_triangle> t(n);
  unsigned long long s = 7;
  auto rnd = [&]() { s = s * 6364136223846793005ull + 1442695040888963407ull; return (float)(s >> 40) * 0x1p-24f; };
  for (unsigned i = 0; i < n; i++) {
    float c[3];
    for (float& x : c) x = 10.f * rnd();
    for (int k = 0; k < 3; k++)
      for (int a = 0; a < 3; a++) v[3 * i + k].pos[a] = at + c[a] + size * rnd();
    t[i] = gbpt_triangle{3 * i, 3 * i + 1, 3 * i + 2, 0};
  }
  gbpt::HostBVH bvh;
  if (!gbpt::build_bvh(v.data(), t.data(), n, 32, 4, &bvh)) return 1;
  gbpt::OrderedTree tree;
  const bool ok = gbpt::ordered_tree(bvh, &tree);
  std::printf("%d %u\n", ok ? 1 : 0, tree.leafN);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from cudapt_gb300 import build
    lib = build.build()
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(SRC)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "cudapt_gb300", "csrc"), str(d / "rule.cpp"),
                    "-o", str(d / "rule"), "-L", os.path.dirname(lib), "-lgbpt",
                    "-Wl,-rpath," + os.path.dirname(lib)], check=True)

    def run(*args):
        out = subprocess.run([str(d / "rule"), *map(str, args)], capture_output=True, text=True, timeout=60)
        assert out.returncode == 0, out.stderr
        return tuple(int(x) for x in out.stdout.split())
    return run


@pytest.mark.parametrize("n", [1, 2, 500, 20_000])  # one part, and many parts on several threads
@pytest.mark.parametrize("size", [0.2, 2.0])
def test_scenes_near_the_origin_get_the_tree(program, n, size):
    for at in (0.0, 10.0, 300.0 * size):  # a margin of at most 2.4e-3 * size: leaf boxes grow by a few per cent
        assert program(n, size, at) == (1, n), at


@pytest.mark.parametrize("n", [500, 20_000])
@pytest.mark.parametrize("size", [0.2, 2.0])
def test_small_triangles_far_out_do_not(program, n, size):
    for at in (2.5e5 * size, 2e6 * size):  # a margin of 1.9 sizes and more: boxes of over ten times the area
        assert program(n, size, at)[0] == 0, at


def test_the_line_is_crossed_once(program):
    got = [program(3000, 0.5, at)[0] for at in np.geomspace(100, 1e6, 25)]
    assert got == sorted(got, reverse=True) and got[0] == 1 and got[-1] == 0
