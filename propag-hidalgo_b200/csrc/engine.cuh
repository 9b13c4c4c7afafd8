// Internal interface between the host code and the propagation kernels.
#pragma once

#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>

#include "dda_columns.cuh"

namespace propag {

// A cell of a global-memory tile.  los is the cell's line of sight to its
// reference, walked once when the cell adopts it (boundaries do not change):
// the cells the walk visits, up to and including the first boundary, and
// kLosBlocked when it met one.
struct alignas(16) CellState {
  float time;
  uint32_t ref;  // packed x | y << 16
  uint32_t los;
  uint32_t pad;
};
constexpr uint32_t kLosBlocked = 0x80000000u;
// The line of sight of a cell that references itself (an ignition): its walk
// visits it twice, or meets a boundary at once.
__host__ __device__ inline uint32_t los_of_self(bool boundary) { return boundary ? kLosBlocked | 1u : 2u; }

// JobDev::max_time of a caller's limit.  A cell that has not burned has the time
// FLT_MAX and no reference, and the kernels follow the reference of every cell
// whose time is below the limit: infinity (no limit) becomes FLT_MAX, below
// which every time of a burned cell lies.
inline float time_limit(float max_time) { return max_time > FLT_MAX ? FLT_MAX : max_time; }

// One scenario as the device sees it.
struct JobDev {
  int32_t W, H;
  float gdx, gdy;
  float max_time;  // time_limit: at most FLT_MAX
  int32_t T;       // tile side in cells (>= max(W, H) means one tile)
  int32_t TX, TY;  // tiles per axis
  int32_t north_up;
  int32_t smem_tile;  // kSmemTile*: where tile launches keep the tile's state
  int32_t refm;       // 1: the reference's arithmetic in time_from, 0: portable
  const float *speed, *az, *ecc;
  float *time;         // the output; shared-memory tiles also keep their state here
  uint32_t *refs;      // state of shared-memory tiles: packed x | y << 16
  uint32_t *los;       // and every cell's line of sight to its reference (CellState::los)
  uint32_t *bnd;       // boundary bits (written by the prep pass)
  // referrer box of every cell (the cells that ever adopted it as their
  // reference): min and max corner, 0xFFFFFFFF in box_x0 = empty
  uint32_t *box_x0, *box_y0, *box_x1, *box_y1;
  const void *ignitions;  // PropagIgnition[n_ignitions]
  uint32_t n_ignitions;
  uint32_t pad;
  uint16_t *out_rx, *out_ry;
  uint32_t *out_bnd;   // caller's boundary output (may alias bnd)
  // Round-down reciprocal of every cell's elliptical speed toward each of its
  // 8 neighbours (plane k: toward the cell whose neighbour k it is), written
  // by the prep pass; null = computed per evaluation instead.  Plane stride
  // tt_plane.
  float *tt;
  int64_t tt_plane;
  // Global-memory tiles keep their state in two copies of packed cell records
  // (sweeps alternate between them) and the fire fields packed beside box_x0;
  // null when every tile is resident in shared memory.
  CellState *st0, *st1;
  float4 *fire4;  // speed, azimuth, eccentricity; w holds box_x0 (as bits)
  int64_t box_x0_step;  // words between the box_x0 of consecutive cells (4 inside fire4, else 1)
  // Grid-wide pending bitmap of global-memory tiles (bit x + y W): cells whose
  // inputs changed since they were last evaluated, outside the tile that
  // changed them; a tile launch's first sweep evaluates only its pending
  // cells.  Null: first sweeps evaluate the whole tile.
  uint32_t *pending;
};

struct Update {
  uint32_t k;     // cell index inside the tile
  float time;
  uint32_t ref;
  uint32_t pad;
};
static_assert(sizeof(Update) == 16, "an update is read back as one 16-byte load");

// An improvement of a global-memory tile's sweep: the cell's new state and its
// index inside the tile (in CellState's spare word).
using TileUpdate = CellState;
// Update entries a CTA keeps in shared memory per sweep parity (the rest go
// to its global update region).
constexpr int kTileUpdSmem = 1024;

// Global-memory scratch of one team slot.  dirty/upd serve tile launches
// whose state stays in global memory: the tile's dirty bitmaps (owner-major:
// each CTA's cells are consecutive bits, see owner_words) and the update
// arrays (one per sweep parity), CTA r of an R-CTA team using entries from
// (parity * R + r) * cap on (cap = global_tile_upd_cap; the first
// kTileUpdSmem of them stay in shared memory); ovf_list/ovf_upd take the
// work-list and update-list entries of shared-memory tiles beyond their
// shared-memory capacity (ovf_cap entries per CTA of the cluster, CTA r at
// offset r * ovf_cap).
struct SlotDev {
  uint32_t *dirty;        // two bitmaps of dirty_words words (alternating by sweep)
  uint32_t dirty_words;
  uint32_t pad0;
  TileUpdate *upd;
  // [0..3] shared-memory tiles' counters, [4] job, [5..7] cluster mode's
  // improving-CTA counts of global-memory tiles (rotating by barrier),
  // [8..11] group mode's two 64-bit barrier arrival words
  uint32_t *ctr;
  uint16_t *ovf_list;
  Update *ovf_upd;
  uint32_t ovf_cap;
  uint32_t pad;
};

// Ownership of a global-memory tile's cells: the tile-linear cells are cut
// into groups of kOwnGroup consecutive cells, and group g belongs to CTA
// g mod R of the team, so that the cells of a front spread over the CTAs
// while a CTA's cells still come in short runs (its neighbour reads share
// sectors).  Groups of 4 cells measured fastest on the 4096^2 scenario with
// 148 CTAs (1 cell and whole 32-cell words were slower).
// The dirty bitmap is owner-major: CTA r's owner_words words start at word
// r * owner_words, and the cells of its l-th group are bits 4 l .. 4 l + 3, so
// that a CTA reads only its own words (23 of them for a 323^2 tile and 148
// CTAs, where a bitmap in tile order has 3 261).
constexpr uint32_t kOwnGroup = 4;
__host__ __device__ inline uint32_t owner_words(uint32_t TN, uint32_t R) {
  return (((TN + kOwnGroup - 1) / kOwnGroup + R - 1) / R + 7) / 8;
}
// Several teams on one job (waves): the tile launches of the reference's
// sequence (rounds of all tiles in row-major order) run as soon as the launches
// they depend on are done.  Words, zeroed before the run:
struct WaveDev {
  uint32_t *done;    // per tile: rounds finished
  uint32_t *claim;   // per tile: rounds taken by a team
  uint32_t *worked;  // per round: a launch of it improved a cell
  uint32_t *sweeps;  // per round: sweeps of its launches
  uint32_t *far;     // [0] a reference lies too far away for `window`; [1] sweeps of all teams, modulo 2^32
  uint32_t tiles;
  int32_t window;    // launches of tiles up to this many tiles apart keep their order
  // A team that waits this long while no team ends a sweep gives the run up (a
  // launch may take longer: a sweep's own waits are bounded by the barrier's).
  unsigned long long stall_ns;
};
constexpr unsigned long long kWaveStallNs = 20000000000ull;
constexpr uint32_t kWaveRounds = 1024;  // rounds the words hold
constexpr uint32_t kWaveTiles = 4096;   // tiles a team's leader looks through

// Update-array entries a CTA of an R-CTA team may need in one sweep of a
// global-memory tile of TN cells: the cells it owns.
__host__ __device__ inline uint32_t global_tile_upd_cap(uint32_t TN, uint32_t R) {
  return owner_words(TN, R) * 32;
}

// Shared memory a CTA needs for a global-memory tile launch: the work list
// of one chunk (tile cell indices, 32 per thread), two sweeps' update entries
// and the crossing times of the line-of-sight walks.
__host__ __device__ inline uint32_t global_tile_list_cap(int threads) { return (uint32_t)threads * 32u; }
__host__ __device__ inline size_t global_tile_list_bytes(int threads) {
  return (size_t)global_tile_list_cap(threads) * 4;
}
__host__ __device__ inline size_t global_tile_cross_off(int threads) {
  return global_tile_list_bytes(threads) + 2 * kTileUpdSmem * sizeof(TileUpdate);
}
__host__ __device__ inline size_t global_tile_smem(int threads) {
  return global_tile_cross_off(threads) + (size_t)kCrossTableLen * 4;
}

// Per-job statistics accumulated on the device (PropagStats order).
struct StatsDev {
  unsigned long long rounds, launches, sweeps, evaluations, improvements, dda_steps,
      refbox_scans, burned, gathers;
  // SM cycles seen by the cluster leader in each phase (barrier wait
  // included): first sweeps of tile launches, evaluate, commit, staging
  unsigned long long cyc_first, cyc_eval, cyc_commit, cyc_stage;
  uint32_t status, max_walk;
  // device clock (%globaltimer, ns) when a cluster took the job and when its
  // propagation finished
  unsigned long long t_start_ns, t_done_ns;
  unsigned long long scan_cells, cyc_wait;
};

constexpr uint32_t kStatusSweepLimit = 1;
// a group barrier wait gave up (group mode); the job's results are invalid
constexpr uint32_t kStatusGroupTimeout = 2;

// Shared-memory tile layout: rows of the tile plus its one-cell halo are
// dealt to the cluster's CTAs round-robin (row hy -> CTA hy % C), so that a
// front of any orientation spreads over all CTAs.  Bytes per cell slot:
// time 4, reference 4, referrer box 4 (halo-local corners, one byte each,
// in units of 1 << box_shift cells), a dirty bit and a box-grown bit.  The work list and
// the update list hold kSmemListCap / kSmemUpdCap entries in shared memory
// and spill beyond that to the slot's global overflow arrays.
// With exact referrer boxes (BoxExact, 8 bytes) a slot takes 16 bytes.
constexpr int kSmemBytesPerCell = 12;
constexpr int kSmemBytesPerCellExact = 16;
constexpr int kSmemListCap = 4096;  // u16 slot indices
constexpr int kSmemUpdCap = 2048;   // u16 slot + f32 time + u32 reference
constexpr int kSmemFixedBytes = 256;
constexpr int kSmemMaxSide = 510;  // halo side whose corners fit a byte at box_shift 1

// JobDev::smem_tile
constexpr int32_t kSmemTileGlobal = 0;  // state in global memory (two copies), bitmaps and update regions in the slot
constexpr int32_t kSmemTileCoarse = 1;  // shared memory, BoxCoarse referrer boxes
constexpr int32_t kSmemTileExact = 2;   // shared memory, BoxExact referrer boxes

__host__ __device__ inline int smem_rows_per_cta(int TH, int C) { return (TH + 2 + C - 1) / C; }
__host__ __device__ inline int smem_cap(int TW, int TH, int C) {
  return smem_rows_per_cta(TH, C) * (TW + 2);
}
__host__ __device__ inline size_t smem_bytes(int TW, int TH, int C, bool exact = false) {
  if (TW + 2 > kSmemMaxSide || TH + 2 > kSmemMaxSide) return ~(size_t)0;  // never fits
  const size_t cap = (size_t)smem_cap(TW, TH, C);
  return cap * (exact ? kSmemBytesPerCellExact : kSmemBytesPerCell) + (cap / 32 + 1) * 8 +
         (size_t)kSmemListCap * 2 +
         (size_t)kSmemUpdCap * 10 + kSmemFixedBytes;
}

}  // namespace propag
