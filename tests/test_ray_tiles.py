"""k_resolve_rays looks through a call's rays 256 at a time, a grid apart.  Its
loop, taken from the kernel's source, is compiled for the CPU: it ends, and
every tile is taken once, up to the largest ray count."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdint>
#include <cstdio>
struct Dim { uint32_t x; };
constexpr uint32_t kCapThreads = 256;
int main() {
  const uint32_t counts[] = {1, 255, 256, 257, 155648, 155649, 311296, 4000000, 0x80000001u, 0xFFFDA000u, 0xFFFFFEFFu,
                             0xFFFFFF00u, 0xFFFFFF01u, 0xFFFFFFFFu};
  const Dim gridDim{608};
  for (uint32_t n : counts) {
    const uint64_t want = ((uint64_t)n + 255) / 256;
    uint64_t tiles = 0, sum = 0;
    for (Dim blockIdx{0}; blockIdx.x < gridDim.x; blockIdx.x++) {
      @LOOP@ {
        if (++tiles > want) { std::printf("%u rays: the loop does not end\n", n); return 1; }
        if (base % 256 != 0 || base >= n) { std::printf("%u rays: tile at %llu\n", n, (unsigned long long)base); return 1; }
        sum += base / 256;
      }
    }
    if (tiles != want || sum != want * (want - 1) / 2) { std::printf("%u rays: tiles missing\n", n); return 1; }
  }
  return 0;
}
"""


def test_every_tile_once(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    src = open(os.path.join(ROOT, "cudapt_gb300", "csrc", "kernels_wave.cu")).read()
    body = src[src.index("k_resolve_rays(DevScene S"):]
    loop = re.search(r"for \([^{]*\)(?= \{)", body).group(0)
    assert "base" in loop and "gridDim" in loop
    f = tmp_path / "tiles.cpp"
    f.write_text(SRC.replace("@LOOP@", loop))
    subprocess.run([gxx, "-std=c++17", "-O2", str(f), "-o", str(tmp_path / "tiles")], check=True)
    out = subprocess.run([str(tmp_path / "tiles")], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
