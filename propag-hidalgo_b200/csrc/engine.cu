// Arrival-time propagation on B200: boundary/prep pass, ignition scatter,
// the persistent engine and the post mask.

// Reference semantics (paths relative to the reference project):
//   pre_propagate / find_boundaries   crates/propag/src/propag.cu:345-375,410-421
//   propag / Propagator::run          crates/propag/src/propag.cu:62-109,382-394
//   post_propagate                    crates/propag/src/propag.cu:110-117,396-408
//   host tile loop                    crates/propag/src/propag.rs:482-556
//
// Schedule.  The reference covers the grid with super-grid tiles of
// T x T cells (one cooperative launch each), runs the tiles one after another
// in row-major order, each until a sweep improves nothing, and repeats the
// pass until no tile improved.  Inside a tile every sweep is a Jacobi sweep
// (two grid.sync()s separate the reads from the writes).  This engine keeps
// exactly that schedule, so its results are the reference's for the same T,
// but a sweep only evaluates the cells whose inputs changed:
//   * the 3x3 neighbourhood of every cell that improved in the last sweep;
//   * the 3x3 neighbourhood of every cell whose reference improved in the last
//     sweep (a cell reads the current time of its neighbours' references,
//     propag.cu:221-224).  Each cell keeps the bounding box of the cells that
//     ever adopted it as their reference, so those referrers are found by
//     scanning that box only.
// The first sweep of a tile launch evaluates the whole tile (shared-memory
// tiles) or its pending cells, those whose inputs changed since their last
// evaluation (global-memory tiles).
//
// Mapping.  The engine is one persistent launch whose CTAs form teams; a
// team works on one scenario at a time and pulls scenarios from a queue
// (largest first), so a batch runs concurrently, scenario per team.  Two
// kinds of team:
//   * cluster mode: a thread-block cluster of 1-16 CTAs.  The tile and its
//     halo (time, reference, referrer boxes) are staged into the cluster's
//     distributed shared memory, rows dealt round-robin to the CTAs; a sweep
//     is two phases, evaluate (reads only) and commit (writes the state,
//     marks the next sweep's cells, scans referrer boxes), separated by
//     hardware cluster barriers, and the tile is written back at the end of
//     the launch.  Tiles too large for the cluster's shared memory take the
//     global-memory path below.
//   * group mode: a cooperative launch without clusters whose CTAs form
//     teams of any size (the whole device for one scenario).  The tile state
//     stays in global memory in two copies, so that a sweep is one phase; the
//     team meets at a counter barrier in global memory whose wait is bounded
//     (see Team).  A lone scenario of enough tiles is run by several teams
//     (waves_kernel): tile launches that cannot read each other's cells run at
//     the same time, and a team's wait for the launches it depends on is
//     bounded too.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>
#include <vector>

#include "dda_columns.cuh"
#include "engine.cuh"
#include "propag_device.cuh"
#include "tile_index.cuh"

namespace cg = cooperative_groups;

namespace propag {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kEngineThreads = 512;
constexpr uint32_t kEmptyBox = 0xFFFFFFFFu;

// The GPU's global nanosecond clock (comparable across SMs and launches).
__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Per-scenario constants of the eight neighbour directions, in the
// reference's neighbour order (j outer, i inner, centre skipped): the bearing
// from the neighbour to the cell and their distance, computed with the same
// operations as time_from, so using them is bit-identical to recomputing.
struct DirConst {
  float bearing[8];
  float dist[8];
};

__device__ __forceinline__ void dir_consts(const JobDev &j, DirConst &d) {
  const bool nu = j.north_up != 0, refm = j.refm != 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int kk = k < 4 ? k : k + 1;
    const int di = kk % 3 - 1, dj = kk / 3 - 1;
    d.bearing[k] = bearing(di, dj, 0, 0, nu, refm);
    d.dist[k] = cell_distance(di, dj, j.gdx, j.gdy, refm);
  }
}

// Round-down reciprocal of the elliptical speed of a cell with fire f toward
// the cell it is neighbour k of, so that step_time(ftime, dc.dist[k], inv)
// is bit-identical to time_from(neighbour -> cell).
__device__ __forceinline__ float dir_inv_speed(const DirConst &dc, int k, const Fire &f, bool refm) {
  return inv_speed(dc.bearing[k], f, refm);
}

// ---------------------------------------------------------------- prep ----
// Boundary bits (find_boundaries) packed with a warp ballot, plus the initial
// state: time = FLT_MAX, no reference, empty referrer boxes; and the
// reciprocal direct-spread speeds toward the 8 neighbours (when the job has them).
// only_if: when given and zero, nothing is done (a second start of a job that
// turned out not to need one).
__global__ void __launch_bounds__(256) prep_kernel(const JobDev *__restrict__ jobs,
                                                   const uint32_t *__restrict__ only_if) {
  if (only_if && *only_if == 0u) return;
  const JobDev j = jobs[blockIdx.y];
  __shared__ DirConst dc;
  if (j.tt) {
    if (threadIdx.x == 0) dir_consts(j, dc);
    __syncthreads();
  }
  const bool refm = j.refm != 0;
  const int64_t N = (int64_t)j.W * j.H;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w0 = warp * 32; w0 < N; w0 += nwarps * 32) {
    const int64_t i = w0 + lane;
    bool b = false;
    if (i < N) {
      const int x = (int)(i % j.W), y = (int)(i / j.W);
      const Fire me{__ldg(j.speed + i), __ldg(j.az + i), __ldg(j.ecc + i)};
#pragma unroll
      for (int di = -1; di < 2; ++di) {
#pragma unroll
        for (int dj = -1; dj < 2; ++dj) {
          if (di == 0 && dj == 0) continue;
          const int nx = x + di, ny = y + dj;
          if (nx < 0 || ny < 0 || nx >= j.W || ny >= j.H) continue;
          const int64_t n = nx + (int64_t)ny * j.W;
          const Fire nb{__ldg(j.speed + n), __ldg(j.az + n), __ldg(j.ecc + n)};
          b |= !similar_fires(nb, me) && me.speed_max < nb.speed_max;
        }
      }
      if (j.fire4) {  // packed records of global-memory tiles
        j.fire4[i] = make_float4(me.speed_max, me.azimuth_max, me.eccentricity, __uint_as_float(kEmptyBox));
        const CellState none{FLT_MAX, kNoRef, 0u, 0u};
        j.st0[i] = none;
        j.st1[i] = none;
      } else {
        if (j.tt && me.speed_max != 0.0f) {
#pragma unroll
          for (int k = 0; k < 8; ++k) j.tt[k * j.tt_plane + i] = dir_inv_speed(dc, k, me, refm);
        }
        j.time[i] = FLT_MAX;
        j.refs[i] = kNoRef;
        j.box_x0[i] = kEmptyBox;
      }
      j.box_y0[i] = kEmptyBox;
      j.box_x1[i] = 0u;
      j.box_y1[i] = 0u;
    }
    const unsigned word = __ballot_sync(kFull, b);
    if (lane == 0) {
      j.bnd[w0 >> 5] = word;
      if (j.pending) j.pending[w0 >> 5] = 0u;
    }
  }
}

// ------------------------------------------------------------- ignition ----
// Later ignitions overwrite earlier ones in the same cell (GDAL burn order);
// every cell whose time is not f32::MAX references itself
// (crates/propag/src/propag.rs:441-449).  One block per job, a thread per
// ignition: the last entry of a cell is found with a maximum over the entries'
// positions in the cell's box_x1 (0 so far), which then gets its value.  (One
// thread took 1.3 to 1.6 us per ignition, a chain of dependent global accesses:
// 26 us for 20 and 4.9 ms for 3000; 7 and 57 us now.)
constexpr int kIgniteThreads = 256;
__global__ void __launch_bounds__(kIgniteThreads) ignite_kernel(const JobDev *__restrict__ jobs,
                                                                const uint32_t *__restrict__ only_if) {
  if (only_if && *only_if == 0u) return;
  const JobDev j = jobs[blockIdx.x];
  struct Ign {
    uint32_t x, y;
    float t;
  };
  const Ign *const ign = (const Ign *)j.ignitions;
  const bool packed = j.fire4 != nullptr;
  // every ignition inside the grid: fn(position, ignition, cell)
  auto each = [&](auto fn) {
    for (uint32_t k = threadIdx.x; k < j.n_ignitions; k += kIgniteThreads) {
      const Ign g = ign[k];
      if (g.x < (uint32_t)j.W && g.y < (uint32_t)j.H) fn(k, g, g.x + (int64_t)g.y * j.W);
      if (k + kIgniteThreads < k) break;
    }
  };
  float *const time = packed ? &j.st0[0].time : j.time;
  const int64_t step = packed ? (int64_t)(sizeof(CellState) / 4) : 1;  // words between cells' times
  each([&](uint32_t k, const Ign &, int64_t c) { atomicMax(j.box_x1 + c, k + 1u); });
  __syncthreads();
  each([&](uint32_t k, const Ign &g, int64_t c) {
    if (__ldcg(j.box_x1 + c) == k + 1u) time[c * step] = g.t;
  });
  __syncthreads();
  // entries of the same cell write the same values
  each([&](uint32_t, const Ign &g, int64_t c) {
    const float t = __ldcg(time + c * step);
    if (t == FLT_MAX) {
      j.box_x1[c] = 0u;
      if (packed) j.st1[c].time = t;
      return;
    }
    const uint32_t r = pack_ref((int)g.x, (int)g.y);
    const uint32_t los = los_of_self((j.bnd[c >> 5] >> (c & 31)) & 1u);
    if (packed) {
      const CellState cell{t, r, los, 0u};
      j.st0[c] = cell;
      j.st1[c] = cell;
    } else {
      j.refs[c] = r;
      j.los[c] = los;
    }
    j.box_x0[c * j.box_x0_step] = j.box_x1[c] = g.x;
    j.box_y0[c] = j.box_y1[c] = g.y;
    // the neighbours of the burning cells are the cells that can improve first
    if (!j.pending || !(t < j.max_time && j.speed[c] != 0.0f)) return;
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const int ax = (int)g.x + dx, ay = (int)g.y + dy;
        if ((dx || dy) && ax >= 0 && ay >= 0 && ax < j.W && ay < j.H) {
          const int64_t n = ax + (int64_t)ay * j.W;
          atomicOr(j.pending + (n >> 5), 1u << (n & 31));
        }
      }
  });
}

// ------------------------------------------------------- common pieces ----
// The engine kernel is compiled for batches whose jobs all use one arithmetic
// of time_from (PROPAG_ARITH_*: kArithRef, kArithPortable) and for mixed ones
// (kArithMixed, chosen per job): a sweep is one pass of each warp through
// straight-line code, so code that a batch does not use costs instruction
// fetches.
constexpr int kArithPortable = 0, kArithRef = 1, kArithMixed = 2;
template <int kArith>
__device__ __forceinline__ bool arith_of(const JobDev &j) {
  return kArith == kArithMixed ? j.refm != 0 : kArith == kArithRef;
}

struct Best {
  float time;
  uint32_t ref;
};

struct Counters {
  uint32_t dda = 0, gat = 0, walk_max = 0;
  unsigned long long evals = 0, scans = 0, scan_cells = 0;
};

// find_neighbor_which_reaches_first (propag.cu:124-190) evaluated by the 8
// lanes of a lane group (lanes 8c .. 8c+7), lane k taking neighbour k in the
// reference's order.  Every neighbour offers a time that does not depend on
// the best found so far -- the candidate through its reference, or its own
// direct time when the line of sight is blocked or the candidate is not
// faster -- and the sequential loop keeps the first strictly smaller offer;
// so the result is the first minimum of the offers when it beats the cell's
// own time.  An offer that is NaN (of a neighbour whose fire is) is never the
// smaller one there, and counts as infinite here: in a reduction by comparisons
// it would hide the offers behind it.  The line of sight from the neighbour to
// its reference was walked when it adopted the reference, and is read; only the
// walks the sequential loop performs (candidate also faster than every earlier
// offer) are counted, so the counters match the reference's order exactly.
// Called by all 32 lanes.
template <int kArith, typename Acc>
__device__ __forceinline__ Best evaluate_coop(const JobDev &j, const DirConst &dc, const Acc &acc,
                                              int x, int y, Best own, bool valid, uint32_t lane,
                                              Counters &cnt) {
  const float kInf = __int_as_float(0x7f800000);
  const int k = (int)(lane & 7u);
  const int kk = k < 4 ? k : k + 1;
  const int nx = x + kk % 3 - 1, ny = y + kk / 3 - 1;
  float nt = FLT_MAX, rt = FLT_MAX;
  uint32_t nr = kNoRef;
  bool act = false;
  if (valid && nx >= 0 && ny >= 0 && nx < j.W && ny < j.H) {
    acc.cell(nx, ny, nt, nr);
    act = nt < j.max_time && nr != pack_ref(x, y);
  }
  // far from the fire (most cells of a whole tile's first sweep) nothing else
  // is read
  if (!__any_sync(kFull, act)) return own;
  Fire f{0.0f, 0.0f, 0.0f};
  float tt = 0.0f;
  uint32_t los = 0;
  if (act) {
    // one memory round trip for all of these
    const int64_t n = nx + (int64_t)ny * j.W;
    f.speed_max = __ldg(j.speed + n);
    f.azimuth_max = __ldg(j.az + n);
    f.eccentricity = __ldg(j.ecc + n);
    if (j.tt) tt = __ldg(j.tt + k * j.tt_plane + n);
    los = __ldcg(j.los + n);
    rt = acc.time_of(nr);
    act = f.speed_max != 0.0f;
  }
  cnt.gat += act ? 1u : 0u;
  float offer = kInf, cand = kInf;
  uint32_t oref = 0;
  const uint32_t steps = los & ~kLosBlocked;
  bool walked = false;
  if (act) {
    const bool refm = arith_of<kArith>(j);
    const float ntime =
        step_time(nt, dc.dist[k], j.tt ? tt : dir_inv_speed(dc, k, f, refm), refm);
    cand = time_from(ref_x(nr), ref_y(nr), rt, x, y, f, j.gdx, j.gdy, j.north_up != 0, refm);
    offer = ntime;
    oref = pack_ref(nx, ny);
    if (cand < ntime) {
      walked = cand < own.time;
      if (!(walked && (los & kLosBlocked))) {
        offer = cand;
        oref = nr;
      }
    }
    offer = fminf(offer, kInf);  // NaN: infinite
  }
  // running best of the sequential loop before neighbour k (exclusive min)
  float pm = offer;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const float t = __shfl_up_sync(kFull, pm, o);
    if (k >= o && t < pm) pm = t;
  }
  float before = __shfl_up_sync(kFull, pm, 1);
  if (k == 0) before = kInf;
  if (walked && cand < before) {
    cnt.dda += steps;
    cnt.walk_max = max(cnt.walk_max, steps);
  }
  // first minimum of the offers
  float bv = offer;
  uint32_t br = oref;
  int bi = k;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const float ov = __shfl_xor_sync(kFull, bv, o);
    const uint32_t orf = __shfl_xor_sync(kFull, br, o);
    const int oi = __shfl_xor_sync(kFull, bi, o);
    if (ov < bv || (ov == bv && oi < bi)) {
      bv = ov;
      br = orf;
      bi = oi;
    }
  }
  return bv < own.time ? Best{bv, br} : own;
}

// Warp-aggregated append: every lane of the (fully active) warp passes its
// count; one atomic per warp reserves the space.  Returns this lane's slot.
__device__ __forceinline__ uint32_t warp_append(uint32_t *counter, uint32_t cnt, uint32_t lane) {
  uint32_t x = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  const uint32_t total = __shfl_sync(kFull, x, 31);
  uint32_t base = 0;
  if (lane == 31 && total) base = atomicAdd(counter, total);
  base = __shfl_sync(kFull, base, 31);
  return base + x - cnt;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, uint32_t lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, v, o);
    if (lane >= (uint32_t)o) v += y;
  }
  return v;
}

// Referrer box of a changed cell clipped to the tile grown by one cell
// (referrers further out have no neighbour inside the tile).
struct Box {
  int x0, y0, x1, y1;
  __device__ __forceinline__ uint32_t area() const {
    return x0 > x1 || y0 > y1 ? 0u : (uint32_t)(x1 - x0 + 1) * (uint32_t)(y1 - y0 + 1);
  }
};

__device__ __forceinline__ Box clip_box(int bx0, int by0, int bx1, int by1, int tx0, int ty0,
                                        int TW, int TH, int W, int H) {
  Box b;
  b.x0 = max(max(bx0, tx0 - 1), 0);
  b.y0 = max(max(by0, ty0 - 1), 0);
  b.x1 = min(min(bx1, tx0 + TW), W - 1);
  b.y1 = min(min(by1, ty0 + TH), H - 1);
  return b;
}

// One lane's referrer box in a warp's concatenated scan.
struct ScanBox {
  int x0, y0;
  uint32_t bw, want, incl;  // width, packed reference, inclusive end in the concatenation
};

// Walks the concatenation of the warp's boxes, 32 cells per step, so that a
// step is one independent wave of loads; mark_fn(hit, gx, gy) is called once
// per step by every lane.  ref_fn(gx, gy, t) returns a cell's reference and
// time.
template <typename RefFn, typename MarkFn>
__device__ __forceinline__ void warp_scan_boxes(ScanBox *sb, const Box &box, uint32_t want,
                                                const JobDev &j, uint32_t lane, Counters &cnt,
                                                RefFn ref_fn,
                                                MarkFn mark_fn) {
  const uint32_t area = box.area();
  cnt.scans += area ? 1 : 0;
  cnt.scan_cells += area;
  const uint32_t incl = warp_incl_scan(area, lane);
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  if (total == 0) return;
  sb[lane] = ScanBox{box.x0, box.y0, (uint32_t)max(box.x1 - box.x0 + 1, 1), want, incl};
  __syncwarp();
  for (uint32_t q0 = 0; q0 < total; q0 += 32) {
    const uint32_t q = q0 + lane;
    bool hit = false;
    int xx = 0, yy = 0;
    if (q < total) {
      int lo = 0, hi = 31;  // first lane whose inclusive end exceeds q
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sb[mid].incl > q) hi = mid; else lo = mid + 1;
      }
      const ScanBox o = sb[lo];
      const uint32_t a = q - (lo ? sb[lo - 1].incl : 0u);  // offset in lane lo's box
      xx = o.x0 + (int)(a % o.bw);
      yy = o.y0 + (int)(a / o.bw);
      float t;
      const uint32_t r = ref_fn(xx, yy, t);
      // a referrer that burns (a cell that does not burn is skipped by its
      // neighbours; requiring it makes the marked set independent of the
      // order of this sweep's commits)
      hit = r == o.want && t < j.max_time && __ldg(j.speed + xx + (int64_t)yy * j.W) != 0.0f;
    }
    mark_fn(hit, xx, yy);
  }
  __syncwarp();
}

// Division of any 32-bit value by a small divisor (the team's CTA count, the
// tile's width) with a multiplication: the estimate is at most one short.
struct FastDiv {
  uint32_t d, m;  // m = floor((2^32 - 1) / d)
  __device__ __forceinline__ explicit FastDiv(uint32_t v) : d(v), m(0xFFFFFFFFu / v) {}
  __device__ __forceinline__ uint32_t div(uint32_t v, uint32_t &rem) const {
    uint32_t q = __umulhi(v, m);
    rem = v - q * d;
    if (rem >= d) {
      rem -= d;
      ++q;
    }
    return q;
  }
};

// Referrer boxes too large for a warp's scan, left to the whole CTA at the end
// of the sweep's evaluations (corners and the referenced cell, 16 bits each).
struct ScanItem {
  uint32_t lo, hi, want;
};
constexpr uint32_t kScanQueue = 512;
// Boxes up to this many cells are scanned at once by the warp that found them;
// larger ones by the CTA.  The largest box of a sweep set the sweep's time
// while one warp scanned it (4096^2 scenario: the slowest warp's scans took
// 4.7 us of a 10.7 us sweep on average, 12.6 us in a tenth of the sweeps).
constexpr uint32_t kScanInline = 32;

// Whether cell (xx, yy) references `want` and burns in the state X: a cell
// that does not burn is skipped by its neighbours, and requiring it makes the
// marked set independent of the order of this sweep's commits.
__device__ __forceinline__ bool referrer(const JobDev &j, const CellState *__restrict__ X, int xx, int yy,
                                         uint32_t want) {
  const uint32_t c = (uint32_t)xx + (uint32_t)yy * (uint32_t)j.W;
  const uint2 s = __ldcg(reinterpret_cast<const uint2 *>(X + c));
  return s.y == want && __uint_as_float(s.x) < j.max_time && __ldg(&j.fire4[c].x) != 0.0f;
}

// The referrer boxes of a warp's four cells (a box is common to its cell's
// eight lanes): the large ones go to the CTA's queue, the others are scanned
// as one concatenation, 32 cells per step.  hit_fn is called by the lanes
// whose cell is a referrer.
template <typename HitFn>
__device__ __forceinline__ void warp_scan_boxes4(const Box &box, uint32_t want, const JobDev &j,
                                                 const CellState *__restrict__ X, uint32_t lane,
                                                 Counters &cnt, ScanItem *queue, uint32_t *queue_ctr,
                                                 HitFn hit_fn) {
  uint32_t area = box.area();
  if ((lane & 7u) == 0) {
    cnt.scans += area ? 1 : 0;
    cnt.scan_cells += area;
  }
  if (!__any_sync(kFull, area != 0u)) return;
  if (area > kScanInline) {
    uint32_t at = 0;
    if ((lane & 7u) == 0) {
      at = atomicAdd(queue_ctr, 1u);
      if (at < kScanQueue)
        queue[at] = ScanItem{(uint32_t)box.x0 | ((uint32_t)box.y0 << 16), (uint32_t)box.x1 | ((uint32_t)box.y1 << 16), want};
    }
    at = __shfl_sync(0xFFu << (lane & 24u), at, lane & 24u);
    if (at < kScanQueue) area = 0;  // a full queue: scanned here after all
  }
  __syncwarp();
  uint32_t end[4];  // ends of the four boxes in the concatenation
#pragma unroll
  for (int g = 0; g < 4; ++g) end[g] = __shfl_sync(kFull, area, 8 * g) + (g ? end[g - 1] : 0u);
  for (uint32_t q0 = 0; q0 < end[3]; q0 += 32) {
    const uint32_t q = q0 + lane;
    const int g = (q >= end[0]) + (q >= end[1]) + (q >= end[2]);
    const uint32_t begin = g == 0 ? 0u : g == 1 ? end[0] : g == 2 ? end[1] : end[2];
    const int bx0 = __shfl_sync(kFull, box.x0, 8 * g), by0 = __shfl_sync(kFull, box.y0, 8 * g);
    const int bx1 = __shfl_sync(kFull, box.x1, 8 * g);
    const uint32_t w = __shfl_sync(kFull, want, 8 * g);
    if (q < end[3]) {
      const uint32_t bw = (uint32_t)(bx1 - bx0 + 1), a = q - begin;
      const int xx = bx0 + (int)(a % bw), yy = by0 + (int)(a / bw);
      if (referrer(j, X, xx, yy, w)) hit_fn(xx, yy);
    }
  }
}

// The CTA's queued boxes, kScanRun cells a thread in flight.
constexpr int kScanRun = 4;
template <typename HitFn>
__device__ __forceinline__ void cta_scan_boxes(const ScanItem *queue, uint32_t n, const JobDev &j,
                                               const CellState *__restrict__ X, HitFn hit_fn) {
  for (uint32_t i = 0; i < n; ++i) {
    const ScanItem it = queue[i];
    const int bx0 = (int)(it.lo & 0xFFFFu), by0 = (int)(it.lo >> 16);
    const uint32_t bw = (it.hi & 0xFFFFu) - (it.lo & 0xFFFFu) + 1u;
    const uint32_t area = bw * ((it.hi >> 16) - (it.lo >> 16) + 1u);
    const FastDiv by_w(bw);
    for (uint32_t a0 = threadIdx.x; a0 < area; a0 += kScanRun * blockDim.x) {
      uint2 s[kScanRun];
#pragma unroll
      for (int r = 0; r < kScanRun; ++r) {
        const uint32_t a = a0 + (uint32_t)r * blockDim.x;
        s[r] = make_uint2(0u, ~it.want);
        if (a < area) {
          uint32_t col;
          const uint32_t row = by_w.div(a, col);
          s[r] = __ldcg(reinterpret_cast<const uint2 *>(X + (bx0 + (int)col) + (int64_t)(by0 + (int)row) * j.W));
        }
      }
#pragma unroll
      for (int r = 0; r < kScanRun; ++r) {
        if (s[r].y != it.want) continue;
        uint32_t col;
        const int yy = by0 + (int)by_w.div(a0 + (uint32_t)r * blockDim.x, col), xx = bx0 + (int)col;
        if (__uint_as_float(s[r].x) < j.max_time && __ldg(&j.fire4[xx + (int64_t)yy * j.W].x) != 0.0f) hit_fn(xx, yy);
      }
    }
  }
}

// ---- team synchronisation ----
// The CTAs that work on one job meet at every phase boundary: at the hardware
// cluster barrier, or in group mode (G CTAs of a cooperative launch without
// clusters, tiles in global memory) at an arrival word in global memory.
// Group mode alternates between two 64-bit arrival words (barrier k uses
// word k & 1): a CTA arrives with one release reduction adding 1 to the low
// half and, when it improved a cell in the sweep that ends there, 1 to the
// high half; the barrier is complete when the low half reaches the team's
// running target, and the high half's growth since the word's last use is
// the number of CTAs that improved.  The count is exact: a CTA can add to
// word k & 1 again only at barrier k + 2, which no CTA reaches before every
// CTA has arrived at barrier k + 1, i.e. has finished reading barrier k.
// (The low half carries into the high half after 2^32 arrivals on one word,
// billions of sweeps.)  A group wait is bounded: when the other CTAs have
// not all arrived after kGroupWaitNs, or once any CTA of the launch has
// given up, it sets the launch's error flag and returns false, and the
// caller abandons the launch.
constexpr unsigned long long kGroupWaitNs = 2000000000ull;  // 2 s; a phase takes < 50 ms

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_add_u64(unsigned long long *p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <bool kGroup>
struct Team {
  unsigned long long *bar;  // group mode: the two arrival words
  uint32_t *err;            // group mode: the launch's error flag
  int *ok;                  // shared: [0] this CTA's outcome of the last wait, [1] improving CTAs
  uint32_t G;               // CTAs in the group
  uint32_t phase = 0;       // thread 0: barriers passed
  uint32_t target[2] = {0u, 0u};  // thread 0: arrivals expected on each word (low half, modular)
  uint32_t seen[2] = {0u, 0u};    // thread 0: the high half of each word at its last use
  unsigned long long waited = 0;  // thread 0: cycles from arrival to release
  // Cluster mode's count of improving CTAs: three counters in global memory
  // used in rotation by the barriers that count (barrier k: counter k % 3).
  // The cluster's leader clears counter (k + 2) % 3 after barrier k: it was
  // last read right after barrier k - 1, and no CTA adds to it before it has
  // passed barrier k + 1, which the leader reaches after the clear.
  uint32_t *cnt3 = nullptr;
  bool cnt_leader = false;
  uint32_t dsweep = 0;  // every thread: sweeps of global-memory tiles (which dirty bitmap is read)
  uint32_t cnt_phase = 0;  // thread 0: counting barriers passed, mod 3
  // global_fence = false: cluster mode orders shared-memory accesses only.
  // *improved (shared memory, may be null) is not zero when this CTA improved
  // a cell in the phase that ends here; *improving receives the number of the
  // team's CTAs that did.
  __device__ bool sync(bool global_fence = true, const uint32_t *improved_ctr = nullptr,
                       uint32_t *improving = nullptr) {
    const long long t0 = threadIdx.x == 0 ? clock64() : 0;
    if constexpr (!kGroup) {
      if (improving) {
        __syncthreads();  // the CTA's updates are counted
        if (threadIdx.x == 0 && *improved_ctr) atomicAdd(cnt3 + cnt_phase, 1u);
      }
      if (global_fence || improving) __threadfence();
      cg::this_cluster().sync();
      if (threadIdx.x == 0) {
        if (improving) {
          ok[1] = (int)__ldcg(cnt3 + cnt_phase);
          if (cnt_leader) cnt3[(cnt_phase + 2) % 3] = 0u;
          cnt_phase = (cnt_phase + 1) % 3;
        }
        waited += (unsigned long long)(clock64() - t0);
      }
      if (improving) {
        __syncthreads();
        *improving = (uint32_t)ok[1];
      }
      return true;
    } else {
    __syncthreads();
    if (threadIdx.x == 0) {
      const bool improved = improved_ctr && *improved_ctr != 0u;
      const uint32_t w = phase & 1u;
      ++phase;
      target[w] += G;  // every CTA of the group passes the same barriers
      unsigned long long *word = bar + w;
      // the release orders this CTA's writes (made visible to thread 0 by the
      // CTA barrier above) before the arrival
      red_release_add_u64(word, 1ull | ((unsigned long long)(improved ? 1u : 0u) << 32));
      bool good = true;
      const unsigned long long start_ns = globaltimer_ns();
      unsigned long long v = ld_acquire_u64(word);
      while ((int32_t)((uint32_t)v - target[w]) < 0) {
        if (ld_relaxed_u32(err) != 0u || globaltimer_ns() - start_ns > kGroupWaitNs) {
          good = false;
          break;
        }
        __nanosleep(32);
        v = ld_acquire_u64(word);
      }
      if (!good) atomicOr(err, 1u);
      const uint32_t hi = (uint32_t)(v >> 32);
      ok[0] = good ? 1 : 0;
      ok[1] = (int)(hi - seen[w]);
      seen[w] = hi;
      waited += (unsigned long long)(clock64() - t0);
    }
    __syncthreads();
    if (improving) *improving = (uint32_t)ok[1];
    return ok[0] != 0;
    }
  }
};

// Referrer box update for a cell (x, y) that adopted reference r, in the
// global arrays (fire-and-forget reductions).
__device__ __forceinline__ void box_expand_global(const JobDev &j, uint32_t r, int x, int y) {
  const int64_t rc = ref_x(r) + (int64_t)ref_y(r) * j.W;
  atomicMin(j.box_x0 + rc, (uint32_t)x);
  atomicMin(j.box_y0 + rc, (uint32_t)y);
  atomicMax(j.box_x1 + rc, (uint32_t)x);
  atomicMax(j.box_y1 + rc, (uint32_t)y);
}

struct TileDesc {
  int x0, y0, TW, TH;
};

// ================================================ global-memory tiles ====
// The tile's state stays in global memory (L2), in two copies X0 and X1 of
// packed records (time, reference, line of sight): sweep s reads X[s & 1] and
// writes X[(s + 1) & 1], so that a sweep is a single phase between two team
// barriers.  The cells are dealt to the team's R CTAs in groups of four (see
// owner_words), and only a cell's owner writes it.  In sweep s a CTA
//   1. loads its words of the dirty bitmap D[s & 1] (its pending cells on the
//      first sweep), clears them and turns the bits into a work list in
//      shared memory, a chunk at a time; meanwhile it copies its improvements
//      of sweep s - 1 (already in X[s & 1]) into X[(s + 1) & 1];
//   2. evaluates the listed cells against X[s & 1], eight lanes to a cell, and
//      commits each improvement at once, by the lanes that found it: they
//      walk the line of sight to the new reference, write the record to
//      X[(s + 1) & 1], grow the reference's box, mark the 3x3 neighbourhood of
//      a burning cell in D[(s + 1) & 1] and scan the cell's referrer box
//      (reading X[s & 1]);
//   3. meets the team; the barrier reports how many CTAs improved a cell.
// After a sweep without improvements both copies hold the same state.  Marks
// are bit reductions without a return value.  The referrer scans read the
// references as the sweep started: a referrer whose reference changes in this
// sweep improved, so its neighbourhood is marked anyway, and one that did not
// reads the same reference either way -- the marks are those of scans run
// after the commits.
//
// What bounds it: a sweep of a few thousand cells over 148 CTAs is a chain of
// dependent L2 round trips (0.3-0.4 us each) between two barriers (1.3 us), so
// every step above is there to shorten that chain.  The line of sight is
// walked when a cell adopts its reference, by the eight lanes of the cell at
// once, instead of by every neighbour in every later evaluation.

// Where the cells of a global-memory tile keep their dirty bits.
struct TileBits {
  int TW, TH;
  uint32_t wpo;  // words per owner
  FastDiv by_r, by_tw;
  __device__ __forceinline__ TileBits(int tw, int th, uint32_t R)
      : TW(tw), TH(th), wpo(owner_words((uint32_t)tw * (uint32_t)th, R)), by_r(R), by_tw((uint32_t)tw) {}
  // The (up to) three cells of row dy - 1 of the 3x3 neighbourhood of tile
  // cell (lx, ly), centre excluded: bit i of `run` is tile cell k0 + i, with
  // k0 the first cell of a group (so the run spans one group or two).
  __device__ __forceinline__ uint32_t row_run(int lx, int ly, int dy, uint32_t &g) const {
    const int xa = max(lx - 1, 0), xb = min(lx + 1, TW - 1);  // columns inside the tile
    const int ay = ly + dy - 1;
    if (xa > xb || ay < 0 || ay >= TH) return 0u;
    uint32_t run = (2u << (xb - xa)) - 1u;
    if (dy == 1 && lx >= xa && lx <= xb) run &= ~(1u << (lx - xa));
    const uint32_t k0 = (uint32_t)xa + (uint32_t)ay * (uint32_t)TW;
    g = k0 / kOwnGroup;
    return run << (k0 & (kOwnGroup - 1));
  }
  // half 0 raises the run's first group, half 1 its second
  __device__ __forceinline__ void mark_half(uint32_t *dirty, int lx, int ly, int dy, int half) const {
    uint32_t g = 0, owner;
    const uint32_t run = row_run(lx, ly, dy, g);
    const uint32_t bits = half ? run >> kOwnGroup : run & ((1u << kOwnGroup) - 1u);
    if (!bits) return;
    const uint32_t l = by_r.div(g + (uint32_t)half, owner);
    atomicOr(dirty + owner * wpo + (l >> 3), bits << ((l & 7u) * kOwnGroup));
  }
  __device__ __forceinline__ void mark_row(uint32_t *dirty, int lx, int ly, int dy) const {
    uint32_t g = 0, owner;
    const uint32_t run = row_run(lx, ly, dy, g);
    if (!run) return;
    uint32_t l = by_r.div(g, owner);
    const uint32_t lo = run & ((1u << kOwnGroup) - 1u), hi = run >> kOwnGroup;
    if (lo) atomicOr(dirty + owner * wpo + (l >> 3), lo << ((l & 7u) * kOwnGroup));
    if (hi) {  // the next group: the next CTA's
      if (++owner == by_r.d) {
        owner = 0;
        ++l;
      }
      atomicOr(dirty + owner * wpo + (l >> 3), hi << ((l & 7u) * kOwnGroup));
    }
  }
  __device__ __forceinline__ void mark3x3(uint32_t *dirty, int lx, int ly) const {
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) mark_row(dirty, lx, ly, dy);
  }
};

// Neighbour t (0..8, row-major, 4 the centre) of tile cell (lx, ly) when it
// lies outside the tile but inside the grid: raises its bit in the grid-wide
// pending bitmap.  (lx, ly) may lie anywhere in the grid.
__device__ __forceinline__ void mark_pending(uint32_t *pending, const JobDev &j, int x0, int y0, int lx,
                                             int ly, int TW, int TH, int t) {
  const int ax = lx + t % 3 - 1, ay = ly + t / 3 - 1;
  if (t == 4 || (ax >= 0 && ay >= 0 && ax < TW && ay < TH)) return;
  const int gx = x0 + ax, gy = y0 + ay;
  if (gx < 0 || gy < 0 || gx >= j.W || gy >= j.H) return;
  const int64_t g = gx + (int64_t)gy * j.W;
  atomicOr(pending + (g >> 5), 1u << (g & 31));
}
__device__ __forceinline__ bool tile_border(int lx, int ly, int TW, int TH) {
  return lx <= 0 || ly <= 0 || lx >= TW - 1 || ly >= TH - 1;
}

// Takes (reads and clears) the pending bits of tile cells k0 .. k0 + n - 1
// (n <= 32, tile-linear order) from the grid-wide bitmap; bit i of the result
// is cell k0 + i.  The cells of one tile row are consecutive grid cells, so
// each row segment is a funnel shift of two words.
__device__ __forceinline__ uint32_t take_pending(uint32_t *pending, const JobDev &j, int x0, int y0,
                                                 int TW, uint32_t k0, uint32_t n) {
  uint32_t out = 0, done = 0;
  while (done < n) {
    const uint32_t k = k0 + done;
    const uint32_t lx = k % (uint32_t)TW, ly = k / (uint32_t)TW;
    const uint32_t seg = min(n - done, (uint32_t)TW - lx);  // cells left in this row
    const int64_t g = (x0 + (int64_t)lx) + (int64_t)(y0 + (int64_t)ly) * j.W;
    const int64_t wi = g >> 5;
    const uint32_t sh = (uint32_t)(g & 31);
    const bool two = sh + seg > 32;  // the segment reaches the next word (same row)
    const uint64_t w2 =
        (uint64_t)__ldcg(pending + wi) | (two ? (uint64_t)__ldcg(pending + wi + 1) << 32 : 0ull);
    const uint32_t m = seg >= 32 ? 0xFFFFFFFFu : (1u << seg) - 1u;
    const uint32_t bits = (uint32_t)(w2 >> sh) & m;
    if (bits) {
      const uint64_t cm = (uint64_t)bits << sh;
      if ((uint32_t)cm) atomicAnd(pending + wi, ~(uint32_t)cm);
      if ((uint32_t)(cm >> 32)) atomicAnd(pending + wi + 1, ~(uint32_t)(cm >> 32));
    }
    out |= bits << done;
    done += seg;
  }
  return out;
}

struct SweepCtx {
  bool leader;
  Counters cnt;
  unsigned long long sweeps = 0, improvements = 0, max_sweeps = 0;
  unsigned long long cyc[4] = {0, 0, 0, 0};  // first sweeps, evaluate, commit, staging
  long long t_phase = 0;
  bool abort = false;
  bool failed = false;  // a group wait gave up (implies abort)
  __device__ __forceinline__ void tick(int phase) {
    if (leader) {
      const long long now = clock64();
      cyc[phase] += (unsigned long long)(now - t_phase);
      t_phase = now;
    }
  }
};

__device__ __forceinline__ CellState ld_state(const CellState *p) {
  const uint4 v = __ldcg(reinterpret_cast<const uint4 *>(p));
  return CellState{__uint_as_float(v.x), v.y, v.z, v.w};
}
__device__ __forceinline__ void st_state(CellState *p, const CellState &s) {
  *reinterpret_cast<uint4 *>(p) = make_uint4(__float_as_uint(s.time), s.ref, s.los, s.pad);
}

// A global-memory tile's update entries of one sweep: this CTA's first
// kTileUpdSmem in shared memory, the rest in its global update region.
__device__ __forceinline__ CellState get_update(const TileUpdate *sm_upd, const TileUpdate *g_upd,
                                                uint32_t u) {
  return u < (uint32_t)kTileUpdSmem ? sm_upd[u] : ld_state(g_upd + u);
}

// find_neighbor_which_reaches_first (propag.cu:124-190) by the eight lanes of
// a cell, as evaluate_coop, on packed records: the neighbour's line of sight
// to its reference is read with its state instead of walked.  All arithmetic
// but the last sum of the candidate's time is independent of the reference's
// time, and runs while that load is in flight.  own: the cell's state; the
// result is the lanes' common view (best.time < own.time: improved).
// hot: the job's fields that every evaluation reads, and this lane's
// neighbour, in registers (the job itself lives in shared memory).
struct Hot {
  int W, H, dx, dy;  // grid; offset of the lane's neighbour
  float max_time, gdx, gdy;
  float bearing, dist;  // from the neighbour to the cell
  bool north_up;
  const float4 *fire4;
};

template <int kArith>
__device__ __forceinline__ Best evaluate_packed(const JobDev &j, const Hot &h,
                                                const CellState *__restrict__ X, int x, int y, Best own,
                                                bool valid, uint32_t lane, Counters &cnt) {
  const float kInf = __int_as_float(0x7f800000);
  const int k = (int)(lane & 7u);
  const int nx = x + h.dx, ny = y + h.dy;
  const bool refm = arith_of<kArith>(j);
  CellState n{FLT_MAX, kNoRef, 0u, 0u};
  Fire f{0.0f, 0.0f, 0.0f};
  if (valid && (uint32_t)nx < (uint32_t)h.W && (uint32_t)ny < (uint32_t)h.H) {
    const uint32_t c = (uint32_t)nx + (uint32_t)ny * (uint32_t)h.W;  // grids below 2^32 cells
    n = ld_state(X + c);
    const float4 v = __ldg(h.fire4 + c);
    f = Fire{v.x, v.y, v.z};
  }
  const int rx = ref_x(n.ref), ry = ref_y(n.ref);
  const bool act = n.time < h.max_time && f.speed_max != 0.0f && n.ref != pack_ref(x, y);
  float rt = FLT_MAX;
  if (act) rt = __ldcg(&X[(uint32_t)rx + (uint32_t)ry * (uint32_t)h.W].time);
  cnt.gat += act ? 1u : 0u;
  float offer = kInf, cand = kInf;
  uint32_t oref = 0;
  bool walked = false;
  if (act) {
    offer = step_time(n.time, h.dist, inv_speed(h.bearing, f, refm), refm);
    oref = pack_ref(nx, ny);
    const float inv = inv_speed(bearing(rx, ry, x, y, h.north_up, refm), f, refm);
    const float dist = cell_distance(rx - x, ry - y, h.gdx, h.gdy, refm);
    cand = step_time(rt, dist, inv, refm);
    if (cand < offer) {
      walked = cand < own.time;
      if (!(walked && (n.los & kLosBlocked))) {
        offer = cand;
        oref = n.ref;
      }
    }
    offer = fminf(offer, kInf);  // NaN: infinite
  }
  // running best of the sequential loop before neighbour k (exclusive min),
  // and the first minimum of the offers
  float pm = offer, bv = offer;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const float t = __shfl_up_sync(kFull, pm, o);
    const float ov = __shfl_xor_sync(kFull, bv, o);
    if (k >= o && t < pm) pm = t;
    if (ov < bv) bv = ov;
  }
  float before = __shfl_up_sync(kFull, pm, 1);
  if (k == 0) before = kInf;
  if (walked && cand < before) {
    const uint32_t steps = n.los & ~kLosBlocked;
    cnt.dda += steps;
    cnt.walk_max = max(cnt.walk_max, steps);
  }
  const uint32_t g0 = lane & 24u;
  bv = __shfl_sync(kFull, bv, g0);
  const uint32_t at = (__ballot_sync(kFull, offer == bv) >> g0) & 0xFFu;
  const uint32_t br = __shfl_sync(kFull, oref, g0 + (at ? (uint32_t)__ffs(at) - 1u : 0u));
  return bv < own.time ? Best{bv, br} : own;
}

// The line of sight from cell (fx, fy) to (tx, ty) by the eight lanes of a
// cell; the result is a CellState's los.  The walk (propag.h:91-135) visits the
// cells from one to the other inclusive; its t-max accumulators are the
// reference's float arithmetic: start 1/|d|, step +1/|d|, a diagonal step when
// |tmax.x - tmax.y| < 1e-9 (a double comparison in the reference: for a float v,
// (double)v < 1e-9 exactly when v is at most the largest float below 1e-9).
// Called by all 32 lanes; `on` is uniform in each group of eight.
//
// Step by step, for offsets beyond kColumnsMax: every lane generates the walk,
// lane i of the eight looks up the visited cells i, i + 8, ... of each run of
// kCoopSteps, whose bitmap words are thus loaded together.  In remaining
// counts (ri, rj) the walk's end conditions are signs: the target is the only
// cell with both zero, and every step from it leaves the walk's box.
constexpr int kCoopSteps = 16;
__device__ __noinline__ uint32_t walk_los_steps(const uint32_t *__restrict__ bnd, int W, int fx, int fy,
                                                int tx, int ty, bool on, uint32_t lane) {
  const int sx = (tx > fx) - (tx < fx), sy = (ty > fy) - (ty < fy);
  const int adx = abs(tx - fx), ady = abs(ty - fy);
  int ri = on ? adx : -1, rj = ady;
  // 1 / |d|: the float nearest to the reference's double quotient (a quotient
  // of integers below 2^16 lies too far from a midpoint of floats to round
  // differently in one step or two)
  const float ddx = __frcp_rn((float)adx), ddy = __frcp_rn((float)ady);
  float tmx = ddx, tmy = ddy;
  const float kTie = __int_as_float(0x3089705F);  // the largest float below 1e-9
  uint32_t cur = (uint32_t)fx + (uint32_t)fy * (uint32_t)W;  // grids below 2^32 cells
  const uint32_t stepx = (uint32_t)sx, stepy = (uint32_t)(sy * W);
  const uint32_t k = lane & 7u, g0 = lane & 24u;
  uint32_t steps = 0, los = 0;
  while (__any_sync(kFull, (ri | rj) >= 0)) {
    uint32_t ix[kCoopSteps / 8];
    uint32_t mine = 0, nv = 0;  // my visited cells (bit per eight), cells visited in this run
#pragma unroll
    for (int i = 0; i < kCoopSteps; ++i) {
      const bool live = (ri | rj) >= 0;
      if (live) ++nv;
      if (live && k == (uint32_t)(i & 7)) {
        ix[i >> 3] = cur;
        mine |= 1u << (i >> 3);
      }
      const float t = __fsub_rn(tmx, tmy);
      if (t <= kTie) {  // x first, or a tie (a diagonal step)
        tmx = __fadd_rn(tmx, ddx);
        cur += stepx;
        --ri;
      }
      if (t >= -kTie) {
        tmy = __fadd_rn(tmy, ddy);
        cur += stepy;
        --rj;
      }
    }
    uint32_t w[kCoopSteps / 8];
#pragma unroll
    for (int b = 0; b < kCoopSteps / 8; ++b) w[b] = (mine >> b) & 1u ? __ldg(bnd + (ix[b] >> 5)) : 0u;
#pragma unroll
    for (int b = 0; b < kCoopSteps / 8; ++b) {
      const bool hit = ((mine >> b) & 1u) && ((w[b] >> (ix[b] & 31u)) & 1u);
      const uint32_t m = (__ballot_sync(kFull, hit) >> g0) & 0xFFu;
      if (m && !los) los = kLosBlocked | (steps + (uint32_t)b * 8u + (uint32_t)__ffs(m));
    }
    steps += nv;
    if (los) ri = -1;
    // a walk from a cell to itself visits it twice (no step leaves it)
    if (adx + ady == 0 && ri >= 0) {
      steps = 2;
      ri = -1;
    }
  }
  return los ? los : steps;
}

// Accumulated crossing times for tiles whose CTAs have no shared memory left
// for them (uploaded once per device).
__device__ float d_cross[kCrossTableLen];

// In closed form (dda_columns.cuh), lane i of the eight taking columns i, i +
// 8, ..., kRuns at a time: all bitmap words of a run of 8 kRuns columns are
// loaded together, and no step waits for the one before.
template <int kRuns>
__device__ __forceinline__ uint32_t walk_los_runs(const uint32_t *__restrict__ bnd, const float *cross, int W,
                                                  int fx, int fy, int tx, int ty, bool on, uint32_t lane) {
  const int dx = tx - fx, dy = ty - fy;
  const int adx = abs(dx), ady = abs(dy);
  const int P = max(adx, ady), Q = min(adx, ady);
  const int sx = dx < 0 ? -1 : 1, sy = dy < 0 ? -W : W;
  const int step_p = adx >= ady ? sx : sy, step_q = adx >= ady ? sy : sx;
  const uint32_t start = (uint32_t)fx + (uint32_t)fy * (uint32_t)W;  // grids below 2^32 cells
  const float inv_p = __frcp_rn((float)P);
  const uint32_t k = lane & 7u, g0 = lane & 24u;
  const int last = on ? P : -1;
  uint32_t D = 0, los = 0;  // diagonal steps so far; the result once blocked
  for (int c0 = 0; kRuns == 1 ? c0 == 0 : __any_sync(kFull, c0 <= last && !los); c0 += 8 * kRuns) {
    uint32_t hit_in = 0, hit_out = 0, diags = 0;  // bit b: column c0 + 8 b + k
    uint32_t ia[kRuns], wa[kRuns], wb[kRuns];
    int two[kRuns];
#pragma unroll
    for (int b = 0; b < kRuns; ++b) {
      const int c = c0 + 8 * b + (int)k;
      wa[b] = wb[b] = 0u;
      ia[b] = 0u;
      two[b] = 0;
      if (c <= last) {
        int jin, jout;
        bool diag;
        walk_column(cross, P, Q, c, inv_p, jin, jout, diag);
        ia[b] = start + (uint32_t)(c * step_p) + (uint32_t)(jin * step_q);
        two[b] = jout - jin ? step_q : 0;
        if (diag) diags |= 1u << b;
        wa[b] = __ldg(bnd + (ia[b] >> 5));
        wb[b] = __ldg(bnd + ((ia[b] + (uint32_t)two[b]) >> 5));
      }
    }
    uint32_t dm[kRuns];  // the cell's diagonal steps, a byte per eight columns
#pragma unroll
    for (int b = 0; b < kRuns; ++b) dm[b] = (__ballot_sync(kFull, (diags >> b) & 1u) >> g0) & 0xFFu;
#pragma unroll
    for (int b = 0; b < kRuns; ++b) {
      hit_in |= ((wa[b] >> (ia[b] & 31u)) & 1u) << b;
      hit_out |= ((wb[b] >> ((ia[b] + (uint32_t)two[b]) & 31u)) & 1u) << b;
    }
    const bool hit = (hit_in | hit_out) != 0u;
    if (__any_sync(kFull, hit)) {
      // the first boundary's column in this run, from the lanes' masks
      uint32_t first = 0xFFFFu;
      if (hit) first = 8u * (uint32_t)(__ffs(hit_in | hit_out) - 1) + k;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) first = min(first, __shfl_xor_sync(kFull, first, o));
      uint32_t before = 0;  // diagonal steps up to and including that column
#pragma unroll
      for (int b = 0; b < kRuns; ++b) {
        const int upto = (int)first - 8 * b;  // bits 0 .. upto count
        before += (uint32_t)__popc(upto >= 7 ? dm[b] : upto >= 0 ? dm[b] & ((2u << upto) - 1u) : 0u);
      }
      const uint32_t in_hits = __shfl_sync(kFull, hit_in, g0 + (first & 7u));
      if (first != 0xFFFFu && !los) {
        int jin, jout;
        bool diag;
        walk_column(cross, P, Q, c0 + (int)first, inv_p, jin, jout, diag);
        const int r = (in_hits >> (first >> 3)) & 1u ? jin : jout;
        los = kLosBlocked | (uint32_t)(c0 + (int)first + r + 1 - (int)(D + before));
      }
    }
#pragma unroll
    for (int b = 0; b < kRuns; ++b) D += (uint32_t)__popc(dm[b]);
  }
  return los ? los : (uint32_t)(P + Q + 1) - D;
}

// Walks of up to eight columns (the usual ones on rough ground) take the
// single-run code: a third of the instructions.
__device__ __forceinline__ uint32_t walk_los(const uint32_t *__restrict__ bnd, const float *cross, int W,
                                             int fx, int fy, int tx, int ty, bool on, uint32_t lane) {
  const int P = max(abs(tx - fx), abs(ty - fy));
  if (!__any_sync(kFull, on && (uint32_t)(P - 1) > 6u))
    return walk_los_runs<1>(bnd, cross, W, fx, fy, tx, ty, on, lane);
  if (__any_sync(kFull, on && (uint32_t)(P - 1) >= (uint32_t)kColumnsMax))
    return walk_los_steps(bnd, W, fx, fy, tx, ty, on, lane);
  return walk_los_runs<4>(bnd, cross, W, fx, fy, tx, ty, on, lane);
}

// One tile launch with the state in global memory, by a team of R CTAs
// (this one is `rank`).  `list` is shared memory for blockDim.x * 32 entries,
// `sm_upd` for two sweeps' kTileUpdSmem update entries, `cta_ctr` six shared
// counters, `queue` kScanQueue boxes, `cross` the crossing times of the line-of-sight walks.  Returns
// whether any sweep improved a cell.
//
// The referrer box a commit scans is read while the cell is evaluated (before
// or during other commits of the sweep): it holds every referrer adopted in
// earlier sweeps (their growth happened before the last barrier); referrers
// that adopt the cell in this sweep improved, and mark their neighbourhoods
// themselves.  Concurrent growth can only widen the box (a box created in
// this sweep may show the empty marker in a corner: corners are clamped to
// the grid), which costs scan work, never a mark: a scan hits the cells that
// referenced the cell when the sweep started.  With a pending bitmap the
// scans read referrers outside the launching tile too, from X[p]: a launch
// writes only its tile's cells, and both copies agree everywhere when a
// launch ends, so outside the tile X[0] and X[1] hold the same state.
// kWaves: other teams run launches of other tiles of the job at the same time;
// reach is the largest offset (in cells, per axis) of a reference for which
// their launches and this one are independent, *far is set when a cell
// adopts one further away, and far[1] counts the sweeps of all teams.
template <int kArith, bool kGroup, bool kWaves>
__device__ __forceinline__ bool tile_global(const JobDev &j, const DirConst &dc, const SlotDev &s, const TileDesc &td,
                            uint32_t *list, TileUpdate *sm_upd, uint32_t *cta_ctr, ScanItem *queue, const float *cross,
                            uint32_t rank, uint32_t R, SweepCtx &cx, Team<kGroup> &team, int reach,
                            uint32_t *far) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const uint32_t k8 = lane & 7u, g0 = lane & 24u;
  const int x0 = td.x0, y0 = td.y0, TW = td.TW, TH = td.TH;
  const uint32_t TN = (uint32_t)TW * (uint32_t)TH;
  const TileBits tb(TW, TH, R);
  const uint32_t ngroups = (TN + kOwnGroup - 1) / kOwnGroup;
  const uint32_t cap = global_tile_upd_cap(TN, R);
  // the work list holds a chunk of words at a time: usually all of them
  const uint32_t chunk = global_tile_list_cap(blockDim.x) / 32u;
  const CellState *const X[2] = {j.st0, j.st1};
  Hot h;
  {
    const int kk = k8 < 4 ? (int)k8 : (int)k8 + 1;
    h.W = j.W;
    h.H = j.H;
    h.dx = kk % 3 - 1;
    h.dy = kk / 3 - 1;
    h.max_time = j.max_time;
    h.gdx = j.gdx;
    h.gdy = j.gdy;
    h.bearing = dc.bearing[k8];
    h.dist = dc.dist[k8];
    h.north_up = j.north_up != 0;
    h.fire4 = j.fire4;
  }
  uint32_t *const pending = j.pending;
  const uint32_t *const bnd = j.bnd;
  // the launch's counters in registers (the context may live in local memory)
  Counters cnt = cx.cnt;
  bool first = true, worked = false;
  uint32_t q = 0;  // list counter of this chunk: cta_ctr[q]
  int p = 0;       // sweep parity: read X[p], write X[p ^ 1]
  if (threadIdx.x < 1)
    for (int i = 0; i < 6; ++i) cta_ctr[i] = 0u;
  __syncthreads();
  for (;;) {
    ++cx.sweeps;  // every thread counts, so the abort below is uniform
    const CellState *const rs = X[p];
    CellState *const ws = const_cast<CellState *>(X[p ^ 1]);
    // dirty bitmaps by the team's sweep count d: read and clear D[d & 1], mark
    // D[(d + 1) & 1] (cleared by its readers in sweep d - 1)
    const uint32_t dsw = team.dsweep++;
    uint32_t *const dirty = s.dirty + (size_t)(dsw & 1u) * s.dirty_words + (size_t)rank * tb.wpo;
    uint32_t *const dirty_next = s.dirty + (size_t)((dsw + 1u) & 1u) * s.dirty_words;
    TileUpdate *const upd = s.upd + ((size_t)p * R + rank) * cap;
    TileUpdate *const supd = sm_upd + p * kTileUpdSmem;
    uint32_t *const upd_ctr = cta_ctr + 2 + p;
    const uint32_t prev_upd = cta_ctr[2 + (p ^ 1)];  // this CTA's improvements of the previous sweep
    // the neighbours of a referrer
    auto mark_around = [&](int xx, int yy) {
      tb.mark3x3(dirty_next, xx - x0, yy - y0);
      if (pending && tile_border(xx - x0, yy - y0, TW, TH))
        for (int t = 0; t < 9; ++t) mark_pending(pending, j, x0, y0, xx - x0, yy - y0, TW, TH, t);
    };
    for (uint32_t c0 = 0; c0 < tb.wpo; c0 += chunk) {
      if (c0) __syncthreads();  // the previous chunk's list is consumed
      if (threadIdx.x == 0) cta_ctr[5] = 0u;
      const uint32_t c1 = min(tb.wpo, c0 + chunk);
      // ---- 1: this CTA's marked cells into the list ----
      if (!first) {
        // a thread per group: short runs of bits, over as many lanes as there are
        for (uint32_t l = c0 * 8u + threadIdx.x; l < c1 * 8u; l += blockDim.x) {
          const uint32_t v = __ldcg(dirty + (l >> 3));
          uint32_t bits = (v >> ((l & 7u) * kOwnGroup)) & ((1u << kOwnGroup) - 1u);
          if (bits) {
            uint32_t at = atomicAdd(cta_ctr + q, (uint32_t)__popc(bits));
            const uint32_t k0 = (l * R + rank) * kOwnGroup;
            for (; bits; bits &= bits - 1) list[at++] = k0 + (uint32_t)(__ffs(bits) - 1);
          }
        }
      } else {
        // the tile's pending cells (inputs changed since their last
        // evaluation), or every cell
        for (uint32_t l = c0 * 8u + threadIdx.x; l < c1 * 8u; l += blockDim.x) {
          const uint32_t g = l * R + rank;
          if (g >= ngroups) break;
          const uint32_t n = min(kOwnGroup, TN - g * kOwnGroup);
          uint32_t bits = pending ? take_pending(pending, j, x0, y0, TW, g * kOwnGroup, n) : (1u << n) - 1u;
          if (bits) {
            uint32_t at = atomicAdd(cta_ctr + q, (uint32_t)__popc(bits));
            for (; bits; bits &= bits - 1) list[at++] = g * kOwnGroup + (uint32_t)(__ffs(bits) - 1);
          }
        }
      }
      // the previous sweep's improvements into X[p ^ 1], before this sweep's
      // improvements of the same cells (ordered by the barrier below)
      if (c0 == 0)
        for (uint32_t u = threadIdx.x; u < prev_upd; u += blockDim.x) {
          const CellState e = get_update(sm_upd + (p ^ 1) * kTileUpdSmem, s.upd + ((size_t)(p ^ 1) * R + rank) * cap, u);
          uint32_t col;
          const uint32_t row = tb.by_tw.div(e.pad, col);
          st_state(ws + ((uint32_t)x0 + col + ((uint32_t)y0 + row) * (uint32_t)h.W), e);
        }
      __syncthreads();
      for (uint32_t w = c0 + threadIdx.x; w < c1; w += blockDim.x) dirty[w] = 0u;  // marked again in the next sweep at the earliest
      const uint32_t nlist = cta_ctr[q];
      q ^= 1u;
      if (threadIdx.x == 0) {
        cnt.evals += nlist;
        cta_ctr[q] = 0u;  // the next chunk's or sweep's counter (read before the last barrier)
        if (c0 == 0) cta_ctr[2 + (p ^ 1)] = 0u;
      }
      // ---- 2: evaluate and commit, up to four cells a warp, spread over the
      // CTA's warps (a warp's walks and scans take as long as its longest) ----
      const uint32_t per = min(4u, (nlist + nwarps - 1) / nwarps);
      // Longer lists go on with whichever warp is done first: fours differ by
      // their walks and scans, and the CTA waits for its last warp (teams of a
      // few CTAs: 64 scenarios 132/159/260 -> 129/156/253 ms; 4096 x 4096
      // 160/171/179 -> 155/165/179 ms; short lists are not touched).
      auto next_four = [&]() -> uint32_t {
        if (nlist <= 4u * nwarps) return nlist;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(cta_ctr + 5, 4u);
        return 4u * nwarps + __shfl_sync(kFull, at, 0);
      };
      for (uint32_t base = warp * per; base < nlist; base = next_four()) {
        const uint32_t ci = base + (lane >> 3);
        const bool valid = (lane >> 3) < per && ci < nlist;
        uint32_t k = 0;
        int lx = 0, ly = 0, x = 0, y = 0;
        uint32_t c = 0;
        Best own{FLT_MAX, kNoRef};
        uint32_t corner = 0;  // lanes 0..3 of the cell: x0, y0, x1, y1 of its referrer box
        float own_speed = 0.0f;
        if (valid) {
          k = list[ci];
          uint32_t col;
          ly = (int)tb.by_tw.div(k, col);
          lx = (int)col;
          x = x0 + lx;
          y = y0 + ly;
          c = (uint32_t)x + (uint32_t)y * (uint32_t)h.W;
          const CellState o = ld_state(rs + c);
          own = Best{o.time, o.ref};
          if (k8 < 4) {
            const uint32_t *const b = k8 == 0   ? reinterpret_cast<const uint32_t *>(h.fire4 + c) + 3
                                      : k8 == 1 ? j.box_y0 + c
                                      : k8 == 2 ? j.box_x1 + c
                                                : j.box_y1 + c;
            corner = __ldcg(b);
          }
          own_speed = __ldg(&h.fire4[c].x);
        }
        const Best b = evaluate_packed<kArith>(j, h, rs, x, y, own, valid, lane, cnt);
        const bool improved = valid && b.time < own.time;  // common to the cell's lanes
        if (!__any_sync(kFull, improved)) continue;
        // referrer box (whole with a pending bitmap: referrers anywhere mark
        // pending cells; else clipped to the tile grown by one cell)
        Box box{1, 1, 0, 0};
        if (__any_sync(kFull, improved && k8 == 0 && corner != kEmptyBox)) {
          box.x0 = (int)__shfl_sync(kFull, corner, g0);
          box.y0 = (int)__shfl_sync(kFull, corner, g0 + 1);
          box.x1 = (int)__shfl_sync(kFull, corner, g0 + 2);
          box.y1 = (int)__shfl_sync(kFull, corner, g0 + 3);
          if (!improved || (uint32_t)box.x0 == kEmptyBox)
            box = Box{1, 1, 0, 0};
          else if (pending)
            box = Box{max(box.x0, 0), max(box.y0, 0), min(box.x1, h.W - 1), min(box.y1, h.H - 1)};
          else
            box = clip_box(box.x0, box.y0, box.x1, box.y1, x0, y0, TW, TH, h.W, h.H);
        }
        const uint32_t los = walk_los(bnd, cross, h.W, x, y, ref_x(b.ref), ref_y(b.ref), improved, lane);
        const uint32_t adds = __ballot_sync(kFull, improved && k8 == 0);
        uint32_t ai = 0;
        if (lane == 0) ai = atomicAdd(upd_ctr, (uint32_t)__popc(adds));
        ai = __shfl_sync(kFull, ai, 0) + (uint32_t)__popc(adds & ((1u << lane) - 1u));
        if (improved) {
          if (k8 == 0) {
            st_state(ws + c, CellState{b.time, b.ref, los, 0u});
            const CellState e{b.time, b.ref, los, k};
            if (kWaves && max(abs(ref_x(b.ref) - x), abs(ref_y(b.ref) - y)) > reach) *far = 1u;
            if (ai < (uint32_t)kTileUpdSmem)
              supd[ai] = e;
            else
              st_state(upd + ai, e);
          }
          // the reference's box grows to hold (x, y), a corner a lane
          const uint32_t rc = (uint32_t)ref_x(b.ref) + (uint32_t)ref_y(b.ref) * (uint32_t)h.W;
          const uint32_t at = k8 & 1u ? (uint32_t)y : (uint32_t)x;
          if (k8 < 2)
            atomicMin(k8 == 0 ? j.box_x0 + 4 * (size_t)rc : j.box_y0 + rc, at);
          else if (k8 < 4)
            atomicMax(k8 == 2 ? j.box_x1 + rc : j.box_y1 + rc, at);
          // only a burning cell is read by its neighbours
          if (b.time < h.max_time && own_speed != 0.0f) {
            if (k8 < 6) tb.mark_half(dirty_next, lx, ly, (int)(k8 >> 1), (int)(k8 & 1u));
            if (pending && tile_border(lx, ly, TW, TH))
              mark_pending(pending, j, x0, y0, lx, ly, TW, TH, (int)(k8 < 4 ? k8 : k8 + 1));
          }
        }
        warp_scan_boxes4(box, pack_ref(x, y), j, rs, lane, cnt, queue, cta_ctr + 4, mark_around);
      }
    }
    __syncthreads();  // the queue is complete
    const uint32_t queued = min(cta_ctr[4], kScanQueue);
    if (queued) {
      cta_scan_boxes(queue, queued, j, rs, mark_around);
      __syncthreads();
      if (threadIdx.x == 0) cta_ctr[4] = 0u;
    }
    // ---- 3: meet; the barrier reports how many CTAs improved a cell ----
    uint32_t improving = 0;
    const bool met = team.sync(true, upd_ctr, &improving);
    cx.tick(first ? 0 : 1);
    // a sweep's beat: teams that wait for this launch see that it goes on
    if (kWaves && cx.leader) atomicAdd(far + 1, 1u);
    if (!met) {
      cx.failed = cx.abort = true;
      break;
    }
    if (threadIdx.x == 0) cx.improvements += *upd_ctr;  // summed over the team at the job's end
    if (improving == 0) break;  // X[p ^ 1] got the last improvements: both copies agree
    worked = true;
    p ^= 1;
    first = false;
    if (cx.sweeps > cx.max_sweeps) {
      cx.abort = true;
      break;
    }
  }
  // an abandoned launch leaves marks behind: the slot's next tile starts clean
  if (cx.abort)
    for (uint32_t w = rank * blockDim.x + threadIdx.x; w < 2u * s.dirty_words; w += R * blockDim.x) s.dirty[w] = 0u;
  cx.cnt = cnt;
  return worked;
}

// ================================================ shared-memory tiles ====
// Cell slots of the tile and its halo: halo coordinates hx in [0, TW + 2),
// hy in [0, TH + 2) (grid x = x0 - 1 + hx, y = y0 - 1 + hy); row hy lives in
// CTA hy % C at local row hy / C.
struct SmemTile {
  float *time;
  uint32_t *ref;
  // referrer box of each slot restricted to the staged region, in the job's
  // codec (BoxCoarse or BoxExact); the codec's kEmpty when no referrer lies
  // inside
  void *box;
  uint16_t *list;   // this sweep's cells to evaluate (local slot index); kSmemListCap
  uint16_t *uidx;   // pending updates: local slot, time, reference; kSmemUpdCap
  float *utime;
  uint32_t *uref;
  uint32_t *dirty;  // bit per local slot: evaluate in the next sweep
  uint32_t *grown;  // bit per local slot: a referrer joined its staged box in this launch
  uint32_t *ctr;    // [0] list size, [1] local updates, [2..3] cluster updates (parity)
  uint16_t *ovf_list;  // this CTA's global overflow of list / updates
  Update *ovf_upd;
};

__device__ __forceinline__ SmemTile carve_smem(char *base, int cap, int box_bytes, const SlotDev &s,
                                              int rank) {
  SmemTile t;
  t.box = base;  // first: 8-byte aligned for BoxExact
  base += (size_t)cap * box_bytes;
  t.time = (float *)base;
  base += (size_t)cap * 4;
  t.ref = (uint32_t *)base;
  base += (size_t)cap * 4;
  t.utime = (float *)base;
  base += (size_t)kSmemUpdCap * 4;
  t.uref = (uint32_t *)base;
  base += (size_t)kSmemUpdCap * 4;
  t.list = (uint16_t *)base;
  base += (size_t)kSmemListCap * 2;
  t.uidx = (uint16_t *)base;
  base += (size_t)kSmemUpdCap * 2;
  t.dirty = (uint32_t *)(((uintptr_t)base + 3) & ~(uintptr_t)3);
  base = (char *)(t.dirty + (cap / 32 + 1));
  t.grown = (uint32_t *)base;
  base = (char *)(t.grown + (cap / 32 + 1));
  t.ctr = (uint32_t *)(((uintptr_t)base + 15) & ~(uintptr_t)15);
  t.ovf_list = s.ovf_list + (size_t)rank * s.ovf_cap;
  t.ovf_upd = s.ovf_upd + (size_t)rank * s.ovf_cap;
  return t;
}

// Work-list and update-list entries: shared memory first, then the overflow.
__device__ __forceinline__ void list_put(const SmemTile &t, uint32_t i, uint32_t slot) {
  if (i < (uint32_t)kSmemListCap)
    t.list[i] = (uint16_t)slot;
  else
    t.ovf_list[i - kSmemListCap] = (uint16_t)slot;
}
__device__ __forceinline__ uint32_t list_get(const SmemTile &t, uint32_t i) {
  return i < (uint32_t)kSmemListCap ? t.list[i] : __ldcg(t.ovf_list + (i - kSmemListCap));
}
__device__ __forceinline__ void upd_put(const SmemTile &t, uint32_t i, uint32_t slot, float time,
                                        uint32_t ref) {
  if (i < (uint32_t)kSmemUpdCap) {
    t.uidx[i] = (uint16_t)slot;
    t.utime[i] = time;
    t.uref[i] = ref;
  } else {
    t.ovf_upd[i - kSmemUpdCap] = Update{slot, time, ref, 0u};
  }
}
__device__ __forceinline__ void upd_get(const SmemTile &t, uint32_t i, uint32_t &slot, float &time,
                                        uint32_t &ref) {
  if (i < (uint32_t)kSmemUpdCap) {
    slot = t.uidx[i];
    time = t.utime[i];
    ref = t.uref[i];
  } else {
    const Update u = t.ovf_upd[i - kSmemUpdCap];
    slot = u.k;
    time = u.time;
    ref = u.ref;
  }
}

// Staged referrer-box codecs.  A box is [hx0, hx1] x [hy0, hy1] in halo-local
// cells; grow() adds one cell with a compare-and-swap loop (per-field min of
// the low corner, max of the high corner).
//   BoxCoarse: one u32, a byte per corner in units of 1 << sh cells, decoded
//              rounded outwards (4 bytes per slot; halo sides up to 510);
//   BoxExact:  one u64, 16 bits per corner (8 bytes per slot).
struct BoxCoarse {
  using T = uint32_t;
  static constexpr T kEmpty = 0x0000FFFFu;  // x0 = y0 = 255, x1 = y1 = 0
  static __device__ __forceinline__ T pack(int hx0, int hy0, int hx1, int hy1, int sh) {
    return (T)(hx0 >> sh) | ((T)(hy0 >> sh) << 8) | ((T)(hx1 >> sh) << 16) | ((T)(hy1 >> sh) << 24);
  }
  static __device__ __forceinline__ void grow(T *w, int hx, int hy, int sh) {
    const uint32_t px = (uint32_t)(hx >> sh), py = (uint32_t)(hy >> sh);
    const uint32_t lo = px | (py << 8) | 0xFFFF0000u;
    const uint32_t hi = (px << 16) | (py << 24);
    T o = *w;
    for (;;) {
      const T nw = (__vminu4(o, lo) & 0x0000FFFFu) | (__vmaxu4(o, hi) & 0xFFFF0000u);
      if (nw == o) return;
      const T pr = atomicCAS(w, o, nw);
      if (pr == o) return;
      o = pr;
    }
  }
  static __device__ __forceinline__ void decode(T v, int sh, int &hx0, int &hy0, int &hx1, int &hy1) {
    const int m = (1 << sh) - 1;
    hx0 = (int)(v & 0xFFu) << sh;
    hy0 = (int)((v >> 8) & 0xFFu) << sh;
    hx1 = ((int)((v >> 16) & 0xFFu) << sh) + m;
    hy1 = ((int)(v >> 24) << sh) + m;
  }
};

struct BoxExact {
  using T = unsigned long long;
  static constexpr T kEmpty = 0x00000000FFFFFFFFull;  // low corner 0xFFFF, high corner 0
  static __device__ __forceinline__ T pack(int hx0, int hy0, int hx1, int hy1, int) {
    return (T)((uint32_t)hx0 | ((uint32_t)hy0 << 16)) | ((T)((uint32_t)hx1 | ((uint32_t)hy1 << 16)) << 32);
  }
  static __device__ __forceinline__ void grow(T *w, int hx, int hy, int) {
    const uint32_t p = (uint32_t)hx | ((uint32_t)hy << 16);
    T o = *w;
    for (;;) {
      const T nw = (T)__vminu2((uint32_t)o, p) | ((T)__vmaxu2((uint32_t)(o >> 32), p) << 32);
      if (nw == o) return;
      const T pr = atomicCAS(w, o, nw);
      if (pr == o) return;
      o = pr;
    }
  }
  static __device__ __forceinline__ void decode(T v, int, int &hx0, int &hy0, int &hx1, int &hy1) {
    hx0 = (int)(v & 0xFFFFu);
    hy0 = (int)((v >> 16) & 0xFFFFu);
    hx1 = (int)((v >> 32) & 0xFFFFu);
    hy1 = (int)(v >> 48);
  }
};

struct SmemGeom {
  int x0, y0, TW, TH, P, HR, C, rank, rows_mine;
  int sh;    // box_shift: 0 when the halo side fits a byte, else 1
  int lc;    // log2 C (cluster sizes are powers of two): row hy -> CTA hy & (C-1), local row hy >> lc
  uint32_t pm, tm;  // recip_of(P), recip_of(TW)
  __device__ __forceinline__ int owner(int hy) const { return hy & (C - 1); }
  __device__ __forceinline__ int lrow(int hy) const { return hy >> lc; }
  __device__ __forceinline__ int div_p(int s) const { return (int)div_wide((uint32_t)s, pm); }
};

template <typename T>
__device__ __forceinline__ T *rank_ptr(T *local, int r) {
  return cg::this_cluster().map_shared_rank(local, (unsigned)r);
}

// Marks the tile cells of the 3x3 neighbourhood of halo cell (hx, hy) in
// their owners' dirty bitmaps (fire-and-forget reductions on shared memory).
// A row's (up to) three cells are consecutive slots of one owner: one
// reduction, two where they straddle a word.
__device__ __forceinline__ void mark3x3_smem(const SmemTile &sm, const SmemGeom &g, int hx, int hy) {
  const int xa = max(hx - 1, 1), xb = min(hx + 1, g.TW);  // tile columns (halo coordinates)
  if (xa > xb) return;
#pragma unroll
  for (int dy = -1; dy <= 1; ++dy) {
    const int ay = hy + dy;
    if (ay < 1 || ay > g.TH) continue;
    uint32_t run = (1u << (xb - xa + 1)) - 1u;
    if (dy == 0 && hx >= xa && hx <= xb) run &= ~(1u << (hx - xa));
    if (!run) continue;
    const int owner = g.owner(ay);
    const uint32_t l0 = (uint32_t)(g.lrow(ay) * g.P + xa);
    uint32_t *d = owner == g.rank ? sm.dirty : rank_ptr(sm.dirty, owner);
    const uint32_t w = l0 >> 5, b = l0 & 31;
    const uint32_t lo = run << b;
    if (lo) atomicOr(d + w, lo);
    if (b + (uint32_t)(xb - xa) >= 32) {
      const uint32_t hi = run >> (32 - b);
      if (hi) atomicOr(d + w + 1, hi);
    }
  }
}

__device__ __forceinline__ void smem_cell(const SmemTile &sm, const SmemGeom &g, int hx, int hy,
                                          float &t, uint32_t &r) {
  const int owner = g.owner(hy);
  const int li = g.lrow(hy) * g.P + hx;
  if (owner == g.rank) {
    t = sm.time[li];
    r = sm.ref[li];
  } else {
    t = rank_ptr(sm.time, owner)[li];
    r = rank_ptr(sm.ref, owner)[li];
  }
}

__device__ __forceinline__ float smem_time_of(const JobDev &j, const SmemTile &sm,
                                              const SmemGeom &g, uint32_t r) {
  const int hx = ref_x(r) - (g.x0 - 1), hy = ref_y(r) - (g.y0 - 1);
  if (hx >= 0 && hy >= 0 && hx < g.P && hy < g.HR) {
    const int owner = g.owner(hy);
    const int li = g.lrow(hy) * g.P + hx;
    return owner == g.rank ? sm.time[li] : rank_ptr(sm.time, owner)[li];
  }
  return __ldcg(j.time + ref_x(r) + (int64_t)ref_y(r) * j.W);  // outside: static this launch
}

struct SmemAcc {
  const JobDev &j;
  const SmemTile &sm;
  const SmemGeom &g;
  __device__ __forceinline__ void cell(int x, int y, float &t, uint32_t &r) const {
    smem_cell(sm, g, x - (g.x0 - 1), y - (g.y0 - 1), t, r);
  }
  __device__ __forceinline__ float time_of(uint32_t r) const { return smem_time_of(j, sm, g, r); }
};

// One tile launch resident in the cluster's shared memory; B is the staged
// referrer-box codec.
template <class B, int kArith>
__device__ bool tile_smem(const JobDev &j, const DirConst &dc, char *smem, const float *cross, const SlotDev &slot,
                          const TileDesc &td, ScanBox *scan_boxes, SweepCtx &cx, Team<false> &team) {
  using BoxT = typename B::T;
  cg::cluster_group cluster = cg::this_cluster();
  SmemGeom g;
  g.x0 = td.x0;
  g.y0 = td.y0;
  g.TW = td.TW;
  g.TH = td.TH;
  g.P = td.TW + 2;
  g.HR = td.TH + 2;
  g.C = (int)cluster.num_blocks();
  g.lc = __ffs(g.C) - 1;
  g.pm = recip_of((uint32_t)g.P);
  g.tm = recip_of((uint32_t)g.TW);
  g.rank = (int)cluster.block_rank();
  g.rows_mine = g.HR > g.rank ? (g.HR - g.rank + g.C - 1) / g.C : 0;
  g.sh = (sizeof(BoxT) == 4 && (g.P > 256 || g.HR > 256)) ? 1 : 0;
  const SmemTile sm = carve_smem(smem, smem_cap(td.TW, td.TH, g.C), (int)sizeof(BoxT), slot, g.rank);
  BoxT *const sbox = (BoxT *)sm.box;
  const uint32_t lane = threadIdx.x & 31;
  const int nslots = g.rows_mine * g.P;
  const int nwords = (nslots + 31) / 32;

  // ---- stage the tile and its halo (state; referrer boxes restricted to
  // the staged region, where this launch's scans look) ----
  for (int s = threadIdx.x; s < nslots; s += blockDim.x) {
    const int lr = g.div_p(s), hx = s - lr * g.P;
    const int hy = g.rank + lr * g.C;
    const int gx = g.x0 - 1 + hx, gy = g.y0 - 1 + hy;
    float t = FLT_MAX;
    uint32_t r = kNoRef;
    BoxT box = B::kEmpty;
    if (gx >= 0 && gy >= 0 && gx < j.W && gy < j.H) {
      const int64_t c = gx + (int64_t)gy * j.W;
      t = __ldcg(j.time + c);
      r = __ldcg(j.refs + c);
      const uint32_t bx0 = __ldcg(j.box_x0 + c);
      if (bx0 != kEmptyBox) {
        const Box b = clip_box((int)bx0, (int)__ldcg(j.box_y0 + c), (int)__ldcg(j.box_x1 + c),
                               (int)__ldcg(j.box_y1 + c), g.x0, g.y0, g.TW, g.TH, j.W, j.H);
        if (b.x0 <= b.x1 && b.y0 <= b.y1)
          box = B::pack(b.x0 - (g.x0 - 1), b.y0 - (g.y0 - 1), b.x1 - (g.x0 - 1), b.y1 - (g.y0 - 1),
                        g.sh);
      }
    }
    sm.time[s] = t;
    sm.ref[s] = r;
    sbox[s] = box;
  }
  for (int w = threadIdx.x; w < nwords; w += blockDim.x) {
    sm.dirty[w] = 0u;
    sm.grown[w] = 0u;
  }
  if (threadIdx.x == 0) sm.ctr[0] = sm.ctr[1] = sm.ctr[2] = sm.ctr[3] = 0u;
  team.sync(false);
  cx.tick(3);

  // the launch's counters in registers (the context may live in local memory)
  Counters cnt = cx.cnt;
  bool first = true, worked = false;
  int par = 0;
  for (;;) {
    ++cx.sweeps;
    // ---- evaluate: this CTA's list (all its tile cells, or its marks) ----
    // The first sweep's list is implicit: the in-tile rows of this CTA, TW
    // cells each.
    if (!first) {
      for (int w0 = (int)(threadIdx.x & ~31u); w0 < nwords; w0 += blockDim.x) {
        const int w = w0 + (int)lane;
        uint32_t bits = 0;
        if (w < nwords) {
          bits = sm.dirty[w];
          if (bits) sm.dirty[w] = 0u;
        }
        uint32_t at = warp_append(sm.ctr + 0, __popc(bits), lane);
        for (; bits; bits &= bits - 1) list_put(sm, at++, (uint32_t)(w * 32 + __ffs(bits) - 1));
      }
    }
    __syncthreads();
    const uint32_t nlist = first ? (uint32_t)(own_rows(g.TH, g.rank, g.C) * g.TW) : sm.ctr[0];
    if (threadIdx.x == 0) cnt.evals += nlist;
    // four cells per warp, eight lanes per cell
    for (uint32_t base = (threadIdx.x >> 5) * 4; base < nlist; base += (blockDim.x >> 5) * 4) {
      const uint32_t ci = base + (lane >> 3);
      const bool valid = ci < nlist;
      uint32_t s = 0;
      int x = 0, y = 0;
      Best own{FLT_MAX, kNoRef};
      if (valid) {
        s = first ? (uint32_t)own_slot((int)ci, g.rank, g.P, g.tm) : list_get(sm, ci);
        const int lr = g.div_p((int)s), hx = (int)s - lr * g.P, hy = g.rank + lr * g.C;
        x = g.x0 - 1 + hx;
        y = g.y0 - 1 + hy;
        own = Best{sm.time[s], sm.ref[s]};
      }
      const Best b = evaluate_coop<kArith>(j, dc, SmemAcc{j, sm, g}, x, y, own, valid, lane, cnt);
      const bool improved = valid && (lane & 7) == 0 && b.time < own.time;
      const uint32_t at = warp_append(sm.ctr + 1, improved ? 1u : 0u, lane);
      if (improved) upd_put(sm, at, s, b.time, b.ref);
    }
    __syncthreads();
    if (threadIdx.x == 0 && sm.ctr[1]) atomicAdd(rank_ptr(sm.ctr, 0) + 2 + par, sm.ctr[1]);
    team.sync(false);
    cx.tick(first ? 0 : 1);
    const uint32_t total = rank_ptr(sm.ctr, 0)[2 + par];
    if (total == 0) break;
    worked = true;
    // ---- commit, mark, referrer scans (scans may run concurrently with
    // the commits of the same sweep: see tile_global) ----
    if (cx.leader) {
      sm.ctr[2 + (par ^ 1)] = 0u;  // the next sweep's cluster counter
      cx.improvements += total;
    }
    const uint32_t nupd = sm.ctr[1];
    // Some of the warps commit, the others walk the lines of sight to the
    // adopted references (read by other CTAs after the barrier below): both are
    // chains of latencies, a few dozen updates a CTA, and need nothing of each
    // other.  Six and ten of 16: a warp commits up to 32 updates at once, but
    // walks four.  512 x 512 on 16 CTAs, three seeds: 13.1 / 18.3 / 8.9 ms with
    // every warp doing both in turn, 12.1 / 16.6 / 7.8 so (12.2 / 17.0 / 7.8 with
    // eight and eight, 12.2 / 16.3 / 7.8 with four and twelve).
    const uint32_t nwarps = blockDim.x >> 5, warp = threadIdx.x >> 5;
    const uint32_t committers = max(nwarps * 3 / 8, 1u), walkers = max(nwarps - committers, 1u);
    const uint32_t walker = nwarps == 1 ? 0u : warp - committers;  // past `walkers` for the others
    if (walker < walkers) {
      const uint32_t four = min(4u, (nupd + walkers - 1) / walkers);
      for (uint32_t base = walker * four; base < nupd; base += walkers * four) {
        const uint32_t u = base + (lane >> 3);
        const bool on = (lane >> 3) < four && u < nupd;
        uint32_t s = 0, r = 0;
        float t;
        if (on) upd_get(sm, u, s, t, r);
        const int lr = g.div_p((int)s), x = g.x0 - 1 + (int)s - lr * g.P, y = g.y0 - 1 + g.rank + lr * g.C;
        const uint32_t los = walk_los(j.bnd, cross, j.W, x, y, ref_x(r), ref_y(r), on, lane);
        if (on && (lane & 7u) == 0) __stcg(j.los + (uint32_t)x + (uint32_t)y * (uint32_t)j.W, los);
      }
    }
    const uint32_t per = min(32u, (nupd + committers - 1) / committers);
    for (uint32_t base = warp * per; warp < committers && base < nupd; base += committers * per) {
      const uint32_t u = base + lane;
      const bool valid = lane < per && u < nupd;
      uint32_t want = 0;
      Box box{1, 1, 0, 0};
      if (valid) {
        uint32_t s, r;
        float t;
        upd_get(sm, u, s, t, r);
        const int lr = g.div_p((int)s), hx = (int)s - lr * g.P, hy = g.rank + lr * g.C;
        const int x = g.x0 - 1 + hx, y = g.y0 - 1 + hy;
        const float own_speed = __ldg(j.speed + x + (int64_t)y * j.W);  // on its way during the rest
        sm.time[s] = t;
        sm.ref[s] = r;
        // referrer box of r: the staged box inside the staged region (merged
        // into the grid-wide box at the end of the launch), else the
        // grid-wide box in global memory
        const int rhx = ref_x(r) - (g.x0 - 1), rhy = ref_y(r) - (g.y0 - 1);
        if (rhx >= 0 && rhy >= 0 && rhx < g.P && rhy < g.HR) {
          const int owner = g.owner(rhy);
          const int li = g.lrow(rhy) * g.P + rhx;
          // the staged box is rounded outwards, so it may hold (x, y) already
          // while the grid-wide box does not: mark the slot for the merge
          // either way
          B::grow((owner == g.rank ? sbox : rank_ptr(sbox, owner)) + li, hx, hy, g.sh);
          atomicOr((owner == g.rank ? sm.grown : rank_ptr(sm.grown, owner)) + (li >> 5),
                   1u << (li & 31));
        } else {
          box_expand_global(j, r, x, y);
        }
        // only a burning cell is read by its neighbours
        if (t < j.max_time && own_speed != 0.0f) mark3x3_smem(sm, g, hx, hy);
        want = pack_ref(x, y);
        const BoxT pb = sbox[s];
        if (pb != B::kEmpty) {
          // halo-local corners back to grid cells, then clipped to the
          // staged region and the grid
          int bx0, by0, bx1, by1;
          B::decode(pb, g.sh, bx0, by0, bx1, by1);
          box = clip_box(g.x0 - 1 + bx0, g.y0 - 1 + by0, g.x0 - 1 + bx1, g.y0 - 1 + by1, g.x0, g.y0,
                         g.TW, g.TH, j.W, j.H);
        }
      }
      warp_scan_boxes(
          scan_boxes + (threadIdx.x & ~31u), box, want, j, lane, cnt,
          [&](int xx, int yy, float &t) {
            uint32_t r;
            smem_cell(sm, g, xx - (g.x0 - 1), yy - (g.y0 - 1), t, r);
            return r;
          },
          [&](bool hit, int xx, int yy) {
            if (hit) mark3x3_smem(sm, g, xx - (g.x0 - 1), yy - (g.y0 - 1));
          });
    }
    __syncthreads();
    if (threadIdx.x == 0) sm.ctr[0] = sm.ctr[1] = 0u;
    team.sync(false);
    cx.tick(2);
    par ^= 1;
    first = false;
    if (cx.sweeps > cx.max_sweeps) {
      cx.abort = true;
      break;
    }
  }
  // ---- write the tile's state back (halo times and references are
  // unchanged) and merge the staged boxes that grew into the grid-wide boxes
  // (rounded outwards: a box may cover a cell more than its referrers, which
  // costs scan work, never a missed referrer) ----
  for (int s = threadIdx.x; s < nslots; s += blockDim.x) {
    const int lr = g.div_p(s), hx = s - lr * g.P;
    const int hy = g.rank + lr * g.C;
    const int gx = g.x0 - 1 + hx, gy = g.y0 - 1 + hy;
    if (gx < 0 || gy < 0 || gx >= j.W || gy >= j.H) continue;
    const int64_t c = gx + (int64_t)gy * j.W;
    if (hx >= 1 && hx <= g.TW && hy >= 1 && hy <= g.TH) {
      j.time[c] = sm.time[s];
      j.refs[c] = sm.ref[s];
    }
    if (sm.grown[s >> 5] & (1u << (s & 31))) {
      int bx0, by0, bx1, by1;
      B::decode(sbox[s], g.sh, bx0, by0, bx1, by1);
      atomicMin(j.box_x0 + c, (uint32_t)max(g.x0 - 1 + bx0, 0));
      atomicMin(j.box_y0 + c, (uint32_t)max(g.y0 - 1 + by0, 0));
      atomicMax(j.box_x1 + c, (uint32_t)min(g.x0 - 1 + bx1, j.W - 1));
      atomicMax(j.box_y1 + c, (uint32_t)min(g.y0 - 1 + by1, j.H - 1));
    }
  }
  if (threadIdx.x == 0) sm.ctr[0] = sm.ctr[1] = 0u;
  team.sync();
  cx.tick(3);
  cx.cnt = cnt;
  return worked;
}

// ================================================================ engine ====
// Accumulated crossing times of the line-of-sight walks (dda_columns.cuh).
__device__ __forceinline__ void fill_cross(float *cross) {
  for (int n = 1 + (int)threadIdx.x; n <= kColumnsMax; n += blockDim.x) {
    const float step = __frcp_rn((float)n);
    float t = step;
    for (int i = 1; i <= n; ++i, t = __fadd_rn(t, step)) cross[cross_at(n, i)] = t;
  }
}

// A warp's counters into the job's statistics.  Called by all 32 lanes.
__device__ __forceinline__ void add_counters(Counters &cnt, StatsDev *st, uint32_t lane) {
  unsigned long long evals = cnt.evals, scans = cnt.scans, scan_cells = cnt.scan_cells;
  for (int o = 16; o > 0; o >>= 1) {
    cnt.dda += __shfl_xor_sync(kFull, cnt.dda, o);
    cnt.gat += __shfl_xor_sync(kFull, cnt.gat, o);
    cnt.walk_max = max(cnt.walk_max, __shfl_xor_sync(kFull, cnt.walk_max, o));
    scans += __shfl_xor_sync(kFull, scans, o);
    scan_cells += __shfl_xor_sync(kFull, scan_cells, o);
    evals += __shfl_xor_sync(kFull, evals, o);
  }
  if (lane == 0) {
    if (cnt.dda) atomicAdd(&st->dda_steps, (unsigned long long)cnt.dda);
    if (cnt.gat) atomicAdd(&st->gathers, (unsigned long long)cnt.gat);
    if (scans) atomicAdd(&st->refbox_scans, scans);
    if (scan_cells) atomicAdd(&st->scan_cells, scan_cells);
    if (evals) atomicAdd(&st->evaluations, evals);
    if (cnt.walk_max) atomicMax(&st->max_walk, cnt.walk_max);
  }
}

// Cluster mode (group == 0): every cluster is one team.  Group mode
// (group = G > 1, launched cooperatively without clusters): CTAs
// [g * G, (g + 1) * G) form team g, which keeps its tiles in global memory
// and meets at the bounded counter barrier of its slot.
template <int kArith, bool kGroup>
__global__ void __launch_bounds__(kEngineThreads, 1)
    engine_kernel(const JobDev *__restrict__ jobs, uint32_t n_jobs, const SlotDev *__restrict__ slots,
                  uint32_t *__restrict__ queue, StatsDev *__restrict__ stats,
                  unsigned long long max_sweeps, const uint32_t *__restrict__ order, uint32_t group) {
  extern __shared__ __align__(16) char dyn_smem[];
  const uint32_t csize = kGroup ? group : cg::this_cluster().num_blocks();
  const uint32_t slot_id = blockIdx.x / csize;
  const SlotDev s = slots[slot_id];
  const uint32_t rank = kGroup ? blockIdx.x % csize : cg::this_cluster().block_rank();
  const uint32_t tid = rank * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31;
  __shared__ DirConst dc;
  __shared__ JobDev js;
  __shared__ ScanBox scan_boxes[kEngineThreads];  // or the scan queue of global-memory tiles
  static_assert(sizeof(ScanItem) * kScanQueue <= sizeof(ScanBox) * kEngineThreads, "the scan queue fits");
  __shared__ int team_ok[2];
  __shared__ uint32_t cta_ctr[6];  // global-memory tiles: work-list and update counts (two each), scan queue, cells taken
  Team<kGroup> team{reinterpret_cast<unsigned long long *>(s.ctr + 8), queue + 1, team_ok, csize};
  team.cnt3 = s.ctr + 5;  // cluster mode: slot counters 5..7
  team.cnt_leader = rank == 0;
  float *const cross = reinterpret_cast<float *>(dyn_smem + global_tile_cross_off(blockDim.x));
  uint32_t taken = 0xFFFFFFFFu;  // tid 0: the queue position it took last

  for (;;) {
    if (tid == 0) {
      taken = atomicAdd(queue, 1u);
      s.ctr[4] = taken;
      s.ctr[0] = s.ctr[1] = s.ctr[2] = s.ctr[3] = 0;
    }
    if (!team.sync()) break;
    // teams take the jobs in queue order; `order` (when given) maps queue
    // positions to jobs, e.g. largest first so that the longest jobs start early
    const uint32_t q = __ldcg(s.ctr + 4);
    if (q >= n_jobs) return;
    const uint32_t jid = order ? __ldg(order + q) : q;
    if (threadIdx.x == 0) {
      js = jobs[jid];
      dir_consts(js, dc);
    }
    __syncthreads();
    const JobDev &j = js;  // shared-memory copy: frees registers
    // accumulated crossing times of the line-of-sight walks (a shared-memory
    // tile of another job may have used the space since the last time)
    if (j.smem_tile == kSmemTileGlobal) fill_cross(cross);
    StatsDev *st = stats + jid;
    if (tid == 0) st->t_start_ns = globaltimer_ns();
    SweepCtx cx;
    cx.leader = tid == 0;
    cx.max_sweeps = max_sweeps;
    cx.t_phase = clock64();
    unsigned long long rounds = 0, launches = 0;
    for (;;) {  // rounds
      ++rounds;
      bool round_worked = false;
      for (int t = 0; t < j.TX * j.TY && !cx.abort; ++t) {  // tiles, row-major
        ++launches;
        TileDesc td;
        td.x0 = (t % j.TX) * j.T;
        td.y0 = (t / j.TX) * j.T;
        td.TW = min(j.T, j.W - td.x0);
        td.TH = min(j.T, j.H - td.y0);
        bool w = false;
        if constexpr (!kGroup) {
          if (j.smem_tile == kSmemTileExact)
            w = tile_smem<BoxExact, kArith>(j, dc, dyn_smem, d_cross, s, td, scan_boxes, cx, team);
          else if (j.smem_tile == kSmemTileCoarse)
            w = tile_smem<BoxCoarse, kArith>(j, dc, dyn_smem, d_cross, s, td, scan_boxes, cx, team);
        }
        if (kGroup || j.smem_tile == kSmemTileGlobal)
          w = tile_global<kArith, kGroup, false>(
              j, dc, s, td, reinterpret_cast<uint32_t *>(dyn_smem),
              reinterpret_cast<TileUpdate *>(dyn_smem + global_tile_list_bytes(blockDim.x)), cta_ctr,
              reinterpret_cast<ScanItem *>(scan_boxes), cross, rank, csize, cx, team, 0, nullptr);
        round_worked |= w;
      }
      if (!round_worked || cx.abort) break;
    }
    // per-job statistics
    add_counters(cx.cnt, st, lane);
    // every CTA's own improvements (global-memory tiles), or the cluster's
    // total counted by its leader (shared-memory tiles)
    if (threadIdx.x == 0 && cx.improvements) atomicAdd(&st->improvements, cx.improvements);
    if (cx.leader) {
      st->rounds = rounds;
      st->launches = launches;
      st->sweeps = cx.sweeps;
      st->cyc_first = cx.cyc[0];
      st->cyc_eval = cx.cyc[1];
      st->cyc_commit = cx.cyc[2];
      st->cyc_stage = cx.cyc[3];
      if (cx.abort) st->status = cx.failed ? kStatusGroupTimeout : kStatusSweepLimit;
      st->t_done_ns = globaltimer_ns();
      st->cyc_wait = team.waited;
    }
    if (cx.failed || !team.sync()) break;
  }
  // A group wait gave up: this team's job and every job no team has taken
  // yet are reported failed (the other teams stop at their next wait).
  if (tid == 0) {
    for (uint32_t q = taken; q < n_jobs; q = atomicAdd(queue, 1u))
      stats[order ? __ldg(order + q) : q].status = kStatusGroupTimeout;
  }
}

// ================================================================= waves ====
// One job by several teams.  The reference runs the launches one after
// another: rounds of all tiles in row-major order.  Launches of tiles more than
// `window` tiles apart are independent as long as no reference lies more than
// window * T - 1 cells from its cell (per axis): a launch reads and marks cells
// within that many cells of its own tile's border, plus one, and the tiles in
// between are window * T cells wide.  So a launch (round r, tile t) may run as
// soon as, within the window, the tiles ahead of t have finished round r and
// those behind it round r - 1, and round r is known to take place (a launch of
// round r - 1 improved a cell).  Every launch then reads what it reads in
// sequence: times, references and all work counts are the same.  A cell that
// adopts a reference further away than that sets *far: the teams stop, and the
// job is started again, its launches in sequence (wave_end_kernel).
//
// Why: a sweep is a chain of latencies whose length hardly depends on the CTAs
// that share it, and one tile's front is too small for 148 of them.  4096^2, 20
// ignitions: 443 ms in sequence, 201 ms with four teams of 37 CTAs; 2048^2 with 20:
// 184 and 98.
constexpr uint32_t kWaveStop = 0xFFFFFFFFu, kWaveIdle = 0xFFFFFFFEu;
constexpr unsigned long long kWavePickNs = 1000000ull;  // 1 ms: a team's members wait that long at their barrier

// The first launch in sequence that may run and no team has taken: round << 12
// | tile; kWaveStop when the job is finished (or cannot go on), kWaveIdle when
// nothing was to be had for kWavePickNs.  By one warp; `done` is shared memory
// for w.tiles words.
__device__ __noinline__ uint32_t wave_pick(const WaveDev &w, int TX, int TY, const uint32_t *err,
                                           uint32_t *done, uint32_t lane) {
  const unsigned long long start = globaltimer_ns();
  for (;;) {
    if (ld_relaxed_u32(err) != 0u || ld_relaxed_u32(w.far) != 0u) return kWaveStop;
    uint32_t low = 0xFFFFFFFFu;
    for (uint32_t t = lane; t < w.tiles; t += 32) {
      const uint32_t d = ld_relaxed_u32(w.done + t);
      done[t] = d;
      low = min(low, d);
    }
    low = __reduce_min_sync(kFull, low);
    __threadfence();  // what those launches wrote is read after their `done`
    __syncwarp();
    // all tiles have finished round `low`, and it improved nothing
    if (low >= 1 && ld_relaxed_u32(w.worked + low) == 0u) return kWaveStop;
    uint32_t best = 0xFFFFFFFFu;
    for (uint32_t t = lane; t < w.tiles; t += 32) {
      const uint32_t d = done[t], r = d + 1;
      if (ld_relaxed_u32(w.claim + t) != d) continue;
      if (r >= kWaveRounds) {
        *w.far = 1u;
        continue;
      }
      if (r > 1 && ld_relaxed_u32(w.worked + d) == 0u) continue;
      const int x = (int)t % TX, y = (int)t / TX;
      bool ready = true;
      for (int v = max(y - w.window, 0); v <= min(y + w.window, TY - 1) && ready; ++v)
        for (int u = max(x - w.window, 0); u <= min(x + w.window, TX - 1); ++u) {
          const uint32_t o = (uint32_t)(u + v * TX);
          ready = ready && done[o] >= (o < t ? r : d);
        }
      if (ready) best = min(best, r << 12 | t);
    }
    best = __reduce_min_sync(kFull, best);
    if (best != 0xFFFFFFFFu) {
      uint32_t got = 0;
      if (lane == 0) {
        const uint32_t r = best >> 12;
        got = atomicCAS(w.claim + (best & 0xFFFu), r - 1, r) == r - 1;
      }
      if (__shfl_sync(kFull, got, 0)) {
        __threadfence();
        return best;
      }
    } else {
      if (globaltimer_ns() - start > kWavePickNs) return kWaveIdle;
      __nanosleep(200);
    }
    __syncwarp();
  }
}

template <int kArith>
__global__ void __launch_bounds__(kEngineThreads, 1)
    waves_kernel(const JobDev *__restrict__ jobs, const SlotDev *__restrict__ slots, uint32_t *__restrict__ err,
                 StatsDev *__restrict__ st, WaveDev w, uint32_t group) {
  extern __shared__ __align__(16) char dyn_smem[];
  const SlotDev s = slots[blockIdx.x / group];
  const uint32_t rank = blockIdx.x % group;
  const uint32_t tid = rank * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  __shared__ DirConst dc;
  __shared__ JobDev js;
  __shared__ ScanItem queue[kScanQueue];
  __shared__ int team_ok[2];
  __shared__ uint32_t cta_ctr[6];
  Team<true> team{reinterpret_cast<unsigned long long *>(s.ctr + 8), err, team_ok, group};
  float *const cross = reinterpret_cast<float *>(dyn_smem + global_tile_cross_off(blockDim.x));
  uint32_t *const list = reinterpret_cast<uint32_t *>(dyn_smem);  // between launches: the leader's copy of w.done
  if (threadIdx.x == 0) {
    js = jobs[0];
    dir_consts(js, dc);
  }
  __syncthreads();
  const JobDev &j = js;
  fill_cross(cross);
  if (blockIdx.x == 0 && threadIdx.x == 0) st->t_start_ns = globaltimer_ns();
  SweepCtx cx;
  cx.leader = tid == 0;
  cx.max_sweeps = ~0ull;
  cx.t_phase = clock64();
  uint32_t turn = 0, seen = 0;  // leader: the beats (sweeps of all teams) at the last look
  unsigned long long idle_since = 0;
  for (;;) {
    // the leader's warp picks; its word alternates, so that it is not
    // overwritten before every CTA has read it
    if (rank == 0 && threadIdx.x < 32) {
      uint32_t pick = wave_pick(w, j.TX, j.TY, err, list, lane);
      if (lane == 0) {
        const uint32_t beats = ld_relaxed_u32(w.far + 1);
        if (pick != kWaveIdle || beats != seen || idle_since == 0) {
          seen = beats;
          idle_since = globaltimer_ns();
        } else if (globaltimer_ns() - idle_since > w.stall_ns) {
          atomicOr(err, 1u);
          pick = kWaveStop;
        }
        s.ctr[turn & 1u] = pick;
      }
    }
    if (!team.sync()) {
      cx.failed = true;
      break;
    }
    const uint32_t pick = __ldcg(s.ctr + (turn & 1u));
    ++turn;
    if (pick == kWaveIdle) continue;
    if (pick == kWaveStop) break;
    const uint32_t r = pick >> 12, t = pick & 0xFFFu;
    TileDesc td;
    td.x0 = ((int)t % j.TX) * j.T;
    td.y0 = ((int)t / j.TX) * j.T;
    td.TW = min(j.T, j.W - td.x0);
    td.TH = min(j.T, j.H - td.y0);
    const unsigned long long before = cx.sweeps;
    const bool worked = tile_global<kArith, true, true>(
        j, dc, s, td, list, reinterpret_cast<TileUpdate *>(dyn_smem + global_tile_list_bytes(blockDim.x)), cta_ctr,
        queue, cross, rank, group, cx, team, w.window * j.T - 1, w.far);
    if (cx.abort) break;
    if (tid == 0) {
      atomicAdd(w.sweeps + r, (uint32_t)(cx.sweeps - before));
      if (worked) atomicOr(w.worked + r, 1u);
      __threadfence();  // the team's writes (its last barrier made them visible here), then `done`
      atomicExch(w.done + t, r);
    }
  }
  add_counters(cx.cnt, st, lane);
  if (threadIdx.x == 0 && cx.improvements) atomicAdd(&st->improvements, cx.improvements);
  if (tid == 0) {
    atomicAdd(&st->cyc_first, cx.cyc[0]);
    atomicAdd(&st->cyc_eval, cx.cyc[1]);
    atomicAdd(&st->cyc_wait, team.waited);
    atomicMax(&st->t_done_ns, globaltimer_ns());
    if (cx.failed || ld_relaxed_u32(err) != 0u) atomicMax(&st->status, kStatusGroupTimeout);
  }
}

// After the waves: the schedule's counts, or a second start.  redo: the queue
// (position, error flag) of the engine launch that follows, which takes the job
// only when *w.far is set.
__global__ void wave_end_kernel(WaveDev w, StatsDev *__restrict__ st, uint32_t *__restrict__ redo) {
  if (threadIdx.x != 0) return;
  redo[1] = 0u;
  if (st->status != 0u) *w.far = 0u;  // a wait gave up: reported, not repeated
  if (*w.far != 0u) {
    *st = StatsDev{};
    redo[0] = 0u;
    return;
  }
  redo[0] = 1u;  // past the last job
  unsigned long long sweeps = 0;
  uint32_t r = 1;
  for (; r < kWaveRounds; ++r) {
    sweeps += w.sweeps[r];
    if (w.worked[r] == 0u) break;
  }
  st->rounds = r;
  st->launches = (unsigned long long)r * w.tiles;
  st->sweeps = sweeps;
}

// ---------------------------------------------------------------- post ----
// post_propagate (propag.cu:110-117): time = FLT_MAX where the cell's own fire
// is null or the time is past max_time; references unpacked into the x/y
// outputs; burned cells counted.
__global__ void __launch_bounds__(256) post_kernel(const JobDev *__restrict__ jobs,
                                                   StatsDev *__restrict__ stats) {
  const JobDev j = jobs[blockIdx.y];
  const int64_t N = (int64_t)j.W * j.H;
  unsigned long long burned = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (int64_t)gridDim.x * blockDim.x) {
    float t;
    uint32_t r;
    if (j.st0) {
      const uint2 v = *reinterpret_cast<const uint2 *>(j.st0 + i);
      t = __uint_as_float(v.x);
      r = v.y;
    } else {
      t = j.time[i];
      r = j.refs[i];
    }
    if (__ldg(j.speed + i) == 0.0f || t > j.max_time) t = FLT_MAX;
    j.time[i] = t;
    burned += t < FLT_MAX;
    if (j.out_rx) j.out_rx[i] = (uint16_t)(r & 0xFFFFu);
    if (j.out_ry) j.out_ry[i] = (uint16_t)(r >> 16);
  }
  for (int o = 16; o > 0; o >>= 1) burned += __shfl_xor_sync(kFull, burned, o);
  if ((threadIdx.x & 31) == 0 && burned) atomicAdd(&stats[blockIdx.y].burned, burned);
}

// ------------------------------------------------------------ launchers ----
static unsigned grid_for(uint64_t cells, int sms) {
  uint64_t blocks = (cells + 255) / 256;
  const uint64_t cap = (uint64_t)sms * 8;
  if (blocks > cap) blocks = cap;
  return blocks ? (unsigned)blocks : 1u;
}

cudaError_t launch_prep(const JobDev *jobs, uint32_t n_jobs, uint64_t max_cells, int sms,
                        const uint32_t *only_if, cudaStream_t stream) {
  dim3 grid(grid_for(max_cells, sms), n_jobs);
  prep_kernel<<<grid, 256, 0, stream>>>(jobs, only_if);
  return cudaGetLastError();
}

cudaError_t launch_ignite(const JobDev *jobs, uint32_t n_jobs, const uint32_t *only_if,
                          cudaStream_t stream) {
  ignite_kernel<<<n_jobs, kIgniteThreads, 0, stream>>>(jobs, only_if);
  return cudaGetLastError();
}

static cudaLaunchConfig_t engine_config(int csize, int threads, unsigned blocks, size_t smem,
                                        cudaLaunchAttribute *attr, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

using EngineKernel = void (*)(const JobDev *, uint32_t, const SlotDev *, uint32_t *, StatsDev *, unsigned long long,
                              const uint32_t *, uint32_t);
static EngineKernel engine_for(int arith, bool group) {
  if (arith == kArithRef) return group ? engine_kernel<kArithRef, true> : engine_kernel<kArithRef, false>;
  if (arith == kArithPortable)
    return group ? engine_kernel<kArithPortable, true> : engine_kernel<kArithPortable, false>;
  return group ? engine_kernel<kArithMixed, true> : engine_kernel<kArithMixed, false>;
}

template <typename K>
static cudaError_t engine_attrs(K kernel, size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

int engine_threads() { return kEngineThreads; }

// The walks' crossing times on the current device.
cudaError_t upload_cross_table() {
  std::vector<float> t(kCrossTableLen);
  for (int n = 1; n <= kColumnsMax; ++n) {
    const float step = 1.0f / (float)n;
    float v = step;
    for (int i = 1; i <= n; ++i, v += step) t[(size_t)cross_at(n, i)] = v;
  }
  return cudaMemcpyToSymbol(d_cross, t.data(), t.size() * sizeof(float));
}

// Clusters of csize CTAs resident at once, of the kernel that launch_engine
// runs for this arithmetic and kind of team.
cudaError_t engine_max_clusters(int csize, int threads, size_t smem, int arith, bool group, int *n) {
  const EngineKernel kernel = engine_for(arith, group);
  cudaError_t e = engine_attrs(kernel, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = engine_config(csize, threads, (unsigned)csize, smem, attr, 0);
  return cudaOccupancyMaxActiveClusters(n, kernel, &cfg);
}

// arith: the jobs' common arithmetic (their JobDev::refm), or kArithMixed (2).
// group == 0: n_slots clusters of csize CTAs.  group > 1: n_slots teams of
// `group` CTAs in one cooperative launch (all CTAs co-resident, which the
// teams' barriers need; the launch fails rather than run otherwise).
// phantom > 0 (self-test of the bounded wait, one slot only): the team counts
// `phantom` CTAs more than the launch holds, so its barriers never complete.
cudaError_t launch_engine(const JobDev *jobs, uint32_t n_jobs, const SlotDev *slots,
                          uint32_t n_slots, int csize, int threads, size_t smem, uint32_t *queue,
                          StatsDev *stats, unsigned long long max_sweeps, const uint32_t *order,
                          uint32_t group, uint32_t phantom, int arith, cudaStream_t stream) {
  const EngineKernel kernel = engine_for(arith, group > 1);
  cudaError_t e = engine_attrs(kernel, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr[1];
  if (group > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_slots * group, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (phantom && n_slots != 1) return cudaErrorInvalidValue;
    return cudaLaunchKernelEx(&cfg, kernel, jobs, n_jobs, slots, queue, stats, max_sweeps,
                              order, group + phantom);
  }
  cudaLaunchConfig_t cfg = engine_config(csize, threads, n_slots * (unsigned)csize, smem, attr, stream);
  return cudaLaunchKernelEx(&cfg, kernel, jobs, n_jobs, slots, queue, stats, max_sweeps, order,
                            0u);
}

using WavesKernel = void (*)(const JobDev *, const SlotDev *, uint32_t *, StatsDev *, WaveDev, uint32_t);
static WavesKernel waves_for(int arith) {
  return arith == kArithRef ? waves_kernel<kArithRef> : waves_kernel<kArithPortable>;
}

// CTAs of the waves kernel resident at once.
cudaError_t waves_max_ctas(int threads, size_t smem, int arith, int *n) {
  cudaError_t e = engine_attrs(waves_for(arith), smem);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = engine_config(1, threads, 1, smem, attr, 0);
  return cudaOccupancyMaxActiveClusters(n, waves_for(arith), &cfg);
}

// One job by `teams` teams of `group` CTAs (a cooperative launch), then the
// counts or the order to start again; err: the launch's error flag.
cudaError_t launch_waves(const JobDev *job, const SlotDev *slots, uint32_t teams, uint32_t group, int threads,
                         size_t smem, uint32_t *err, StatsDev *stats, const WaveDev &w, uint32_t *redo, int arith,
                         cudaStream_t stream) {
  const WavesKernel kernel = waves_for(arith);
  cudaError_t e = engine_attrs(kernel, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(teams * group, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kernel, job, slots, err, stats, w, group);
  if (e != cudaSuccess) return e;
  wave_end_kernel<<<1, 32, 0, stream>>>(w, stats, redo);
  return cudaGetLastError();
}

cudaError_t launch_post(const JobDev *jobs, uint32_t n_jobs, uint64_t max_cells, int sms,
                        StatsDev *stats, cudaStream_t stream) {
  dim3 grid(grid_for(max_cells, sms), n_jobs);
  post_kernel<<<grid, 256, 0, stream>>>(jobs, stats);
  return cudaGetLastError();
}

}  // namespace propag
