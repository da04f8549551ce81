"""Host memory running out while the ordered walk's tree is made, on any of its
threads and in the starting of a thread too: the tree is given up or the call
throws, the process goes on, and the next call makes the tree."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include "gbpt_internal.h"
std::atomic<long> left{-1};  // allocations until all fail; -1: none does
void* operator new(std::size_t n) {
  if (left.load() >= 0 && left.fetch_sub(1) <= 0) {
    left.store(0);
    throw std::bad_alloc();
  }
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
int main() {
  const unsigned n = 20000;  // 39,999 nodes: parts on eight threads
  std::vector<gbpt_vertex> v(3 * n);
  std::vector<gbpt_triangle> t(n);
  unsigned long long s = 7;
  auto rnd = [&]() { s = s * 6364136223846793005ull + 1442695040888963407ull; return (float)(s >> 40) * 0x1p-24f; };
  for (unsigned i = 0; i < n; i++) {
    float c[3];
    for (float& x : c) x = 10.f * rnd();
    for (int k = 0; k < 3; k++)
      for (int a = 0; a < 3; a++) v[3 * i + k].pos[a] = c[a] + 0.2f * rnd();
    t[i] = gbpt_triangle{3 * i, 3 * i + 1, 3 * i + 2, 0};
  }
  gbpt::HostBVH bvh;
  if (!gbpt::build_bvh(v.data(), t.data(), n, 32, 4, &bvh)) return 1;
  unsigned given_up = 0, made = 0;
  for (long after = 0; after < 4000; after = after < 200 ? after + 1 : after + after / 8) {
    gbpt::OrderedTree tree;
    bool ok = false;
    left.store(after);
    try {
      ok = gbpt::ordered_tree(bvh, &tree);
    } catch (const std::bad_alloc&) {
    }
    left.store(-1);
    (ok ? made : given_up)++;
    if (ok && tree.leafN != n) return 2;
  }
  gbpt::OrderedTree tree;
  if (!gbpt::ordered_tree(bvh, &tree) || tree.leafN != n) return 3;
  std::printf("%u %u\n", given_up, made);
  return given_up > 20 ? 0 : 4;
}
"""


def test_allocations_that_fail(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    csrc = os.path.join(ROOT, "cudapt_gb300", "csrc")
    (tmp_path / "memory.cpp").write_text(SRC)
    exe = str(tmp_path / "memory")
    subprocess.run([gxx, "-std=c++17", "-O1", "-ffp-contract=off", "-I", csrc, str(tmp_path / "memory.cpp"),
                    os.path.join(csrc, "ordered_tree.cpp"), os.path.join(csrc, "bvh_build.cpp"), "-o", exe,
                    "-lpthread"], check=True)
    for _ in range(3):  # which thread meets the failure differs from run to run
        out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
        assert out.returncode == 0, (out.returncode, out.stdout, out.stderr)
