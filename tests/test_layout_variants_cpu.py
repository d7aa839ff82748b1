"""Every block layout the kernels use, not only an FP64 batch's: FP32 (entries in
iedge order) and the splits of small single meshes (blocks of 128 and 64
vertices).  A C++ program builds each for annulus grids, expects no violation,
and expects one for each mistake planted in a copy; a second one counts the
layouts that fvm_layout_stats has checked."""
import os
import shutil
import subprocess

import pytest

from fvm2d_gb300 import build as B

GRID = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "fvm_gpu.h"
#include "fvm_layout.h"
using namespace fvm;
static fvm_geom *annulus(int ni, int nr) {
  std::vector<double> c;
  std::vector<int32_t> el, pt;
  for (int j = 0; j < nr; j++)
    for (int i = 0; i < ni; i++) {
      const double r = 1.0 + 0.1 * j, a = 2 * M_PI * (i + 0.3 * (j % 2)) / ni;
      c.push_back(r * std::cos(a));
      c.push_back(r * std::sin(a));
      pt.push_back(j == 0 ? FVM_PT_SOLID : j == nr - 1 ? FVM_PT_FARFIELD : FVM_PT_INTERIOR);
    }
  for (int j = 0; j + 1 < nr; j++)
    for (int i = 0; i < ni; i++) {
      const int a = j * ni + i + 1, b = j * ni + (i + 1) % ni + 1;
      const int32_t t[6] = {a, b, a + ni, b, b + ni, a + ni};
      el.insert(el.end(), t, t + 6);
    }
  static std::vector<std::vector<double>> keep_c;
  static std::vector<std::vector<int32_t>> keep_i;
  keep_c.push_back(c);
  keep_i.push_back(el);
  int32_t *elem = keep_i.back().data();
  const double *coord = keep_c.back().data();
  keep_i.push_back(pt);
  fvm_geom *g = nullptr;
  if (fvm_geom_build(ni * nr, (int)el.size() / 3, coord, elem, keep_i.back().data(), FVM_CELL_MEDIAN, &g))
    return nullptr;
  return g;
}
"""
CHECK = GRID + r"""
static int bad = 0;
static void expect(bool ok, const char *what, int ni, int bv, int fp64) {
  if (!ok) bad++, printf("%s: ni %d blocks of %d fp64 %d\n", what, ni, bv, fp64);
}
int main() {
  const int grids[][2] = {{8, 3}, {16, 16}, {16, 17}, {60, 40}, {97, 31}};
  for (auto &q : grids)
    for (int bv : {256, 128, 64})
      for (int fp64 : {0, 1}) {
        fvm_geom *g = annulus(q[0], q[1]);
        MeshLayout L;
        if (!g || build_layout(g->mesh, bv, fp64, L)) return 2;
        expect(verify_layout(L) == 0 && L.sub == 256 / bv, "valid", q[0], bv, fp64);
        auto wrong = [&](const char *what, auto change) {
          MeshLayout M = L;
          change(M);
          expect(verify_layout(M) > 0, what, q[0], bv, fp64);
        };
        if (L.nblk > 1) {
          wrong("another split's factor", [](MeshLayout &M) { M.sub = M.sub == 1 ? 2 : M.sub / 2; });
          // (eight vertices from a block to its neighbour: the blocks' ranges alone)
          wrong("uneven blocks", [](MeshLayout &M) {
            BlockInfo &b = M.blocks.back();
            b.v0 += 8;
            b.nv -= 8;
          });
        }
        wrong("an edge's local slot", [](MeshLayout &M) { M.be_loc.back() ^= 1u; });
        wrong("an entry of another vertex", [](MeshLayout &M) { M.be_nodes[0].x = M.be_nodes[0].y; });
        wrong("a slot past the block", [](MeshLayout &M) { M.ve_list[0] |= kSlotMask; });
        wrong("a triangle slot", [](MeshLayout &M) { M.vt_list[0] ^= 0x4000; });
        if (fp64) wrong("a flux source", [](MeshLayout &M) { M.ve_src[0] ^= 1; });
        fvm_geom_free(g);
      }
  return bad != 0;
}
"""
# (its own verify_layout takes the library's place)
COUNT = GRID + r"""
#include <set>
#include <utility>
static std::set<std::pair<int, bool>> seen;
namespace fvm {
int64_t verify_layout(const MeshLayout &L) {
  seen.insert({L.sub, !L.ve_src.empty()});
  return 1;
}
}
int main() {
  fvm_geom *g = annulus(60, 40);
  int64_t out[10];
  if (!g || fvm_layout_stats(&g->mesh, out)) return 2;
  printf("%d layouts, %d violations\n", (int)seen.size(), (int)out[9]);
  return seen.size() != 6 || out[9] != 6;
}
"""


@pytest.mark.parametrize("program", [CHECK, COUNT], ids=["invariants", "stats"])
def test_layouts(tmp_path, program):
    cxx = os.environ.get("CXX", "g++")
    if not shutil.which(cxx):
        pytest.skip("no C++ compiler")
    lib = B.build()
    src = tmp_path / "t.cpp"
    src.write_text(program)
    exe = tmp_path / "t"
    subprocess.run([cxx, "-O1", "-std=c++17", "-rdynamic", f"-I{B.SRC}", f"-I{B.INC}",
                    f"-I{B.CUDA_HOME}/include", str(src), lib, f"-Wl,-rpath,{os.path.dirname(lib)}",
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
