// esr_internal.h -- declarations shared by the host runtime files.
#pragma once
#include <stdint.h>

#include <array>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/eulersr.h"
#include "esr_layout.h"

namespace esr {

struct TileSet;

struct HostMesh {
  int n_cells = 0, n_faces = 0, n_boundary_slots = 0;
  double y_min = 0, y_max = 0;
  std::vector<int> perm;          // new -> old
  std::vector<int> patch_start;   // cells of patch p: [patch_start[p], patch_start[p+1]) in the new order
  std::vector<int> inv;           // old -> new
  std::vector<double> geo;        // n_cells records of G_COUNT values, renumbered
  // The same records formed as the reference forms them on every call, in
  // its operation order, from the points rounded to the run's precision
  // (esr_params.fidelity = ESR_FIDELITY_REFERENCE); float32 adds the
  // per-call least-squares data.
  std::vector<float> geo_ref32;
  std::vector<LsqRef> lsq_ref32;
  std::vector<double> geo_ref64;
  std::vector<float> wall_n_ref32, wall_ds_ref32;
  std::vector<double> wall_n_ref64, wall_ds_ref64;
  std::vector<int> nbr;           // 4 x n_cells (x,y,z neighbours, w packed)
  std::vector<float> centre;      // barycentres (x, y) from the first point, renumbered
  std::vector<int> wall_cell;     // renumbered owner cell of each force face
  std::vector<double> wall_n;     // (nx, ny) per force face
  std::vector<double> wall_ds;    // face length per force face
  double inlet_subsonic[4] = {1.0, 1.0, 0.0, 1.0};
  // tile sets built so far (tiles_of), a few per mesh
  mutable std::mutex tile_mutex;
  mutable std::map<std::array<int, 3>, std::shared_ptr<const TileSet>> tiles;
  // their device tables (StageTables), by device, precision, fidelity and tile size
  mutable std::map<std::array<int, 4>, std::shared_ptr<void>> device_tiles;
};

int prepare_mesh(const esr_mesh_desc& d, HostMesh& hm, std::string& err);
// records `msg` as the calling thread's esr_last_error() and returns `code`
int report_error(int code, const std::string& msg);
std::vector<int> rcm_order(int n, const std::vector<int>& nbr);
std::vector<int> patch_order(int n, const std::vector<int>& nbr, const std::vector<int>& seed,
                             std::vector<int>& patch_start);

// The fused stage kernel's tiles: indices only, the solver adds the geometry
// in its precision (esr_stage.cuh). Local rows: own cells, ring 1, ring 2,
// then one ghost per boundary edge of the own and ring-1 cells.
struct TileCell {           // own or ring-1 cell
  int cell;
  uint16_t nbr[3];          // local row across each edge
  uint16_t slot[3];         // face-state slot of each edge (kNoSlot: no face of the tile)
  uint32_t kinds;           // the mesh's packed slot word
};
struct TileGhost {
  int cell, edge, kind;
};
struct TileFace {
  int cell, edge;           // whose outward normal the face takes
  uint16_t left, right;     // face-state slots of its sides; on a boundary `right` is the ghost's row
  int kind;
};
struct TileSet {
  int n_tiles = 0, max_own = 0, max_rows = 0, max_slots = 0;
  std::vector<int> list;          // cells of the local rows
  std::vector<TileCell> cells;
  std::vector<TileGhost> ghosts;
  std::vector<TileFace> faces;    // each face of the own cells once, or every side of every own cell
  std::vector<TileHead> head;
};
// once: each face once, from its owner; else every side. caller_owner: a
// face's owner is the lower cell of the caller's numbering, else of the kernels'.
TileSet build_tiles(const HostMesh& hm, int cells, bool once, bool caller_owner);
// the same, kept with the mesh for its next solver
std::shared_ptr<const TileSet> tiles_of(const HostMesh& hm, int cells, bool once, bool caller_owner);

}  // namespace esr

// Solvers share the prepared mesh (it does not change once created), so the
// handle may be destroyed while they live.
struct esr_mesh {
  std::shared_ptr<esr::HostMesh> host = std::make_shared<esr::HostMesh>();
  esr::HostMesh& hm = *host;
};
