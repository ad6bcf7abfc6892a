"""Host-side check of the Cartesian near-boundary list (interior_range,
shell_count and shell_decode of csrc/wql3d_device.cuh, compiled here from that
header): with and without PML on each of the six faces, also where the two
slabs of an axis overlap or a slab is wider than the axis, every point belongs
to the strict interior or to exactly one entry of the list, and no entry lies
outside the block.  No GPU is involved."""
import os
import subprocess

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "wql3d_device.cuh"
using namespace wql3d;
int main() {
  int bad = 0, blocks = 0;
  const int axis[3] = {13, 16, 21};
  for (int nx : axis) for (int ny : axis) for (int nz : axis) for (int np : {6, 7, 8, 11, 14, 22})
    for (int pml = 0; pml < 64; ++pml) {
      Blk<double> b;
      memset(&b, 0, sizeof b);
      const int n[3] = {b.nx = nx, b.ny = ny, b.nz = nz};
      for (int a = 0; a < 3; ++a)
        interior_range(n[a], (pml >> (2 * a)) & 1 ? np : 6, (pml >> (2 * a + 1)) & 1 ? np : 6, b.lo[a], b.hi[a]);
      std::vector<int> hit((size_t)nx * ny * nz, 0);
      bool ok = true;
      for (long long i = 0; i < shell_count(b); ++i) {
        int p[3];
        shell_decode(b, (int)i, p[0], p[1], p[2]);
        if (p[0] < 1 || p[0] > nx || p[1] < 1 || p[1] > ny || p[2] < 1 || p[2] > nz) { ok = false; continue; }
        hit[(p[0] - 1) + nx * ((p[1] - 1) + ny * (p[2] - 1))]++;
      }
      for (int z = 1; z <= nz; ++z) for (int y = 1; y <= ny; ++y) for (int x = 1; x <= nx; ++x) {
        const int p[3] = {x, y, z};
        bool in = true;
        for (int a = 0; a < 3; ++a) {
          // strict interior: off every closure and out of every slab
          in = in && p[a] > ((pml >> (2 * a)) & 1 ? np : 6) && p[a] <= n[a] - ((pml >> (2 * a + 1)) & 1 ? np : 6);
          const bool box = p[a] >= b.lo[a] && p[a] <= b.hi[a];
          if (in && !box) ok = false;
        }
        ok = ok && hit[(x - 1) + nx * ((y - 1) + ny * (z - 1))] == (in ? 0 : 1);
      }
      ++blocks;
      if (!ok && bad++ < 5) printf("block %d %d %d slab %d faces %d\n", nx, ny, nz, np, pml);
    }
  printf("%d blocks, %d wrong\n", blocks, bad);
  return bad != 0;
}
"""


def test_every_point_once(tmp_path):
    from waveqlab3d_q_gpu_b200 import build
    src, exe = tmp_path / "cover.cu", tmp_path / "cover"
    src.write_text(PROGRAM)
    subprocess.run([os.environ.get("NVCC", "nvcc")] + build.NVCC_FLAGS +
                   ["-I", os.path.join(build.ROOT, "include"), "-I", build.CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
