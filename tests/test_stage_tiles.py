"""The tile tables of the fused stage kernel (esr_mesh.cpp: build_tiles), built
here on the host from the golden meshes: what the kernel's indexing relies on,
and tiles that stay compact wherever the mesh lies."""
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, load_mesh

MAIN = r'''
#include <cstdio>
#include <cstdlib>
#include <set>
#include "esr_internal.h"
using namespace esr;
static std::vector<double> rd(FILE* f, long n) { std::vector<double> v(n); if (fread(v.data(), 8, n, f) != (size_t)n) exit(9); return v; }
int main(int argc, char** argv) {
  FILE* f = fopen(argv[1], "rb");
  const std::vector<double> h = rd(f, 3);
  const long P = h[0], N = h[1], F = h[2];
  const std::vector<double> pts = rd(f, 2 * P), a = rd(f, 3 * N + 3 * N + 2 * F + F + 3 * N);
  std::vector<int> v(a.begin(), a.end());
  esr_mesh_desc d{};
  d.n_points = P; d.n_cells = N; d.n_faces = F; d.points = pts.data();
  const int* q = v.data();
  d.tris = q; q += 3 * N; d.neighbors = q; q += 3 * N; d.faces = q; q += 2 * F; d.face_markers = q; q += F;
  d.face_connectivity = q; d.force_marker = 2; d.sponge = 1; d.renumber = 1;
  HostMesh hm;
  std::string err;
  if (prepare_mesh(d, hm, err) != 0) { std::printf("prepare: %s\n", err.c_str()); return 2; }
  long bad = 0, ring = 0;
  for (int cells : {32, 64})
    for (bool once : {true, false})
      for (bool owner : {true, false}) {
        const TileSet ts = build_tiles(hm, cells, once, owner);
        std::set<int> owned;
        std::set<std::pair<int, int>> seen;   // interior faces, by their two cells
        long boundary = 0, sides = 0;
        for (const TileHead& t : ts.head) {
          bad += t.n_own < 1 || t.n_own > cells || t.n1 < t.n_own || t.n2 < t.n1 || t.n2 + t.n_ghosts > ts.max_rows;
          ring += cells == 64 && once && owner ? t.n1 - t.n_own : 0;
          const int* list = ts.list.data() + t.list;
          for (int i = 0; i < t.n_own; ++i) bad += !owned.insert(list[i]).second;
          std::set<int> slots;
          for (int i = 0; i < t.n1; ++i) {
            const TileCell& c = ts.cells[t.cells + i];
            bad += c.cell != list[i];
            for (int k = 0; k < 3; ++k) {
              const int j = hm.nbr[4 * (size_t)c.cell + k];
              if (j >= 0) bad += c.nbr[k] >= t.n2 || list[c.nbr[k]] != j;
              else {
                const TileGhost& g = ts.ghosts[t.ghosts + c.nbr[k] - t.n2];
                bad += c.nbr[k] < t.n2 || c.nbr[k] >= t.n2 + t.n_ghosts || g.cell != c.cell || g.edge != k;
              }
              if (i < t.n_own) bad += c.slot[k] != 3 * i + k;
              if (c.slot[k] != kNoSlot) bad += c.slot[k] >= ts.max_slots || !slots.insert(c.slot[k]).second;
            }
          }
          for (int i = 0; i < t.n_faces; ++i) {
            const TileFace& x = ts.faces[t.faces + i];
            bad += !slots.count(x.left);
            const int j = hm.nbr[4 * (size_t)x.cell + x.edge];
            if (x.kind == K_INTERIOR) {
              bad += !slots.count(x.right) || j < 0;
              if (once) bad += owner ? hm.perm[x.cell] > hm.perm[j] : x.cell > j;
              seen.insert({std::min(x.cell, j), std::max(x.cell, j)});
              ++sides;
            } else {
              bad += x.right < t.n2 || x.right >= t.n2 + t.n_ghosts || j >= 0;
              ++boundary;
            }
          }
        }
        bad += (long)owned.size() != N || boundary != hm.n_boundary_slots || (long)seen.size() != (3 * N - boundary) / 2;
        if (!once) bad += sides != 3 * N - boundary;
        bad += ts.max_rows > 10 * cells + 6 * cells || ts.max_slots > 6 * cells;
      }
  std::printf("%ld %.4f\n", bad, (double)ring / N);
  return 0;
}
'''


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    tmp = tmp_path_factory.mktemp("tiles")
    (tmp / "main.cpp").write_text(MAIN)
    csrc = ROOT / "eulersr_b200" / "csrc"
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", str(csrc), "-I", str(ROOT / "include"), str(tmp / "main.cpp"),
                    str(csrc / "esr_mesh.cpp"), "-o", str(tmp / "tiles")], check=True)

    def run(mesh, shift=0.0):
        parts = [[len(mesh.points), len(mesh.tris), len(mesh.faces)], np.asarray(mesh.points) + shift, mesh.tris,
                 mesh.neighbors, mesh.faces, mesh.face_markers, mesh.face_connectivity]
        np.concatenate([np.asarray(p, np.float64).reshape(-1) for p in parts]).tofile(tmp / "mesh.bin")
        r = subprocess.run([str(tmp / "tiles"), str(tmp / "mesh.bin")], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        bad, ring = r.stdout.split()
        return int(bad), float(ring)
    return run


@pytest.mark.parametrize("name", ["diamond_h0.2", "naca0012_h0.2", "diamond_h0.1"])
def test_tiles_cover_the_mesh(program, name):
    """Every cell owned once, every face evaluated, neighbours, ghosts and
    face-state slots by their right local index, within the shared-memory bound."""
    bad, ring = program(load_mesh(name))
    assert bad == 0 and 0 < ring < 1


def test_tiles_are_compact_far_from_the_origin(program):
    """The cells are grouped by their centres in float32; a mesh of size 4 at
    coordinates around 10^7, where float32 steps by 1, still gets the rings that it
    has at the origin."""
    mesh = load_mesh("diamond_h0.1")
    bad, ring = program(mesh)
    bad_far, ring_far = program(mesh, 1.0e7)
    assert bad == bad_far == 0
    assert ring_far <= 1.05 * ring, (ring_far, ring)
