// The rasterisation kernels (see raster.cu for the passes and the host
// side).  Kept in a header of their own so that the CPU tests can compile
// the same source for the host, with the CUDA built-ins replaced by a
// thread-level emulation (tests/emul/).
#pragma once

#include <cfloat>
#include <cstdint>

#include "propag_b200.h"
#include "raster.hpp"

namespace propag {
namespace raster_dev {

constexpr int kRasterThreads = 256;  // every kernel below assumes 8 warps
constexpr int kRowWords = 2048;      // row mask words of the widest grid: 65536 columns
constexpr int kMaskWords = 4096;     // a CTA's row masks
constexpr int kRasterWarps = kRasterThreads / 32;

__global__ void __launch_bounds__(kRasterThreads) fill_winner_kernel(int32_t *win, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    win[i] = -1;
}

// The index of the last part whose `before` is <= i (`before` strictly
// increasing from 0).
template <typename T>
__device__ __forceinline__ uint64_t find_part(const T *parts, uint64_t n, uint64_t i) {
  uint64_t lo = 0, hi = n - 1;
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo + 1) / 2;
    if (parts[mid].before <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(kRasterThreads)
    segment_kernel(const RasterSeg *__restrict__ segs, uint64_t nseg, uint64_t samples, int64_t W,
                   int64_t H, int32_t *__restrict__ win) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < samples;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const RasterSeg &g = segs[find_part(segs, nseg, i)];
    const int64_t s = g.s0 + (int64_t)(i - g.before);
    int64_t c, r;
    if (seg_sample(g, s, W, H, c, r)) atomicMax(win + r * W + c, g.feature);
  }
}

// Threads that share a polygon row: eight while a row's mask fits their share
// of the CTA's shared memory (grids up to 4096 columns), a warp (16384) or the
// CTA.  Most polygons of a fuel map are narrow and of a few dozen edges: the
// search for the polygon, the crossings and the prefix leave the lanes of a
// wider group idle, and the kernel is bound by its instructions.  1200
// polygons of 20 to 480 cells on a 3001 x 2003 grid: 1005 us with a CTA and
// every column of the grid per row, 141 us with a warp and the polygon's own
// columns, 63 us with eight threads and four mask words a step.  Looking at a
// winner before raising it costs more than the atomics it saves (92 us).
__host__ __device__ __forceinline__ int polygon_row_threads(int64_t W) {
  return W <= 32 * (kMaskWords / (kRasterThreads / 8)) ? 8 : W <= 32 * (kMaskWords / kRasterWarps) ? 32 : kRasterThreads;
}

// A barrier of the threads that share a row.  (The CPU emulation has block
// barriers only; its blocks meet all of them together.)
#if defined(__CUDACC__)
#define PG_ROW_SYNC(in_warp) \
  do {                       \
    if (in_warp)             \
      __syncwarp();          \
    else                     \
      __syncthreads();       \
  } while (0)
#else
#define PG_ROW_SYNC(in_warp) __syncthreads()
#endif

// W <= 32 * kRowWords.
__global__ void __launch_bounds__(kRasterThreads, 8)
    polygon_kernel(const RasterPoly *__restrict__ polys, uint64_t npoly, uint64_t rows,
                   const RasterEdge *__restrict__ edges, int64_t W, int32_t *__restrict__ win) {
  struct Row {
    int32_t *first;  // the winner of the first column looked at
    int32_t quads, feature;
  };
  struct alignas(16) Quad {
    uint32_t w[4];
  };
  __shared__ Quad quad_masks[kMaskWords / 4];
  __shared__ Row row_of[kRasterThreads / 8];
  __shared__ uint32_t warp_parity[kRasterWarps];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int gn = polygon_row_threads(W);  // threads of a row
  const int at_once = kRasterThreads / gn, row_words = kMaskWords / at_once;
  const bool in_warp = gn <= 32;
  const int gt = tid & (gn - 1), slot = tid / gn;
  uint32_t *const mask = &quad_masks[0].w[0] + slot * row_words;
  // lanes of this row ahead of this one
  const uint32_t lower = ((1u << lane) - 1u) & ~((1u << (lane & ~(gn - 1))) - 1u);
  for (uint64_t base = (uint64_t)blockIdx.x * at_once; base < rows; base += (uint64_t)gridDim.x * at_once) {
    const uint64_t item = base + (uint64_t)slot;
    RasterPoly p{};
    int64_t r = 0;
    int c0 = 0, c1 = -1;  // the columns looked at: c0 a multiple of 32
    if (item < rows) {
      p = polys[find_part(polys, npoly, item)];
      r = (int64_t)p.row0 + (int64_t)(item - p.before);
      c0 = p.col0 > 0 ? p.col0 / 32 * 32 : 0;
      c1 = (int)min((int64_t)p.col1, W - 1);
    }
    const int n = c1 >= c0 ? c1 - c0 + 1 : 0, nw = (n + 31) / 32;  // columns and mask words in use
    const int quads = (nw + 3) / 4;
    for (int w = gt; w < 4 * quads; w += gn) mask[w] = 0u;
    if (gt == 0) row_of[slot] = Row{win + r * W + c0, quads, p.feature};
    PG_ROW_SYNC(in_warp);
    // a crossing toggles the first column whose centre is at or right of it
    const double yc = (double)r + 0.5;
    for (uint32_t k = gt; nw > 0 && k < p.count; k += gn) {
      double x;
      if (!edge_crossing(edges[p.first + k], yc, x)) continue;
      int64_t c = crossing_cell(x, W);
      if (c > c1) continue;
      c = c > c0 ? c - c0 : 0;
      atomicXor(&mask[c >> 5], 1u << (c & 31));
    }
    PG_ROW_SYNC(in_warp);
    // inside = odd number of toggles at or left of the column: an inclusive
    // prefix XOR along the row (within a word by shifts, across words and
    // threads by the parity of everything ahead)
    const int per = (nw + gn - 1) / gn;  // words per thread
    const int w0 = min(nw, gt * per), w1 = min(nw, w0 + per);
    uint32_t par = 0;
    for (int w = w0; w < w1; ++w) par ^= (uint32_t)__popc(mask[w]) & 1u;
    const uint32_t vote = __ballot_sync(0xFFFFFFFFu, par != 0u);
    uint32_t carry = (uint32_t)__popc(vote & lower) & 1u;
    if (!in_warp) {
      if (lane == 0) warp_parity[wid] = (uint32_t)__popc(vote) & 1u;
      __syncthreads();
      for (int k = 0; k < wid; ++k) carry ^= warp_parity[k];
    }
    for (int w = w0; w < w1; ++w) {
      const uint32_t b = mask[w];
      uint32_t m = b;
      m ^= m << 1;
      m ^= m << 2;
      m ^= m << 4;
      m ^= m << 8;
      m ^= m << 16;
      if (carry) m = ~m;
      if (w == nw - 1 && (n & 31)) m &= (1u << (n & 31)) - 1u;  // columns past the last one
      mask[w] = m;
      carry ^= (uint32_t)__popc(b) & 1u;
    }
    PG_ROW_SYNC(in_warp);
    // a warp to a mask word, 32 winners side by side, four words a step
    const int first_row = in_warp ? wid * (32 / gn) : 0, rows_here = in_warp ? 32 / gn : 1;
    const uint32_t bit = 1u << lane;
    for (int i = first_row; i < first_row + rows_here; ++i) {
      const Row o = row_of[i];
      const Quad *const quad = quad_masks + i * (row_words / 4);
      const int q0 = in_warp ? 0 : wid, dq = in_warp ? 1 : kRasterWarps;
      int32_t *at = o.first + 128 * q0 + lane;
      for (int q = q0; q < o.quads; q += dq, at += 128 * dq) {
        const Quad m = quad[q];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (m.w[k] & bit) atomicMax(at + 32 * k, o.feature);
      }
    }
    PG_ROW_SYNC(in_warp);  // the mask is reused by the next row
  }
}

// In place: the winner raster (int32 in the float buffer) becomes times.
__global__ void __launch_bounds__(kRasterThreads)
    finish_times_kernel(float *times, const float *__restrict__ value, int64_t n) {
  int32_t *win = reinterpret_cast<int32_t *>(times);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t w = win[i];
    times[i] = w >= 0 ? value[w] : FLT_MAX;
  }
}

__global__ void __launch_bounds__(kRasterThreads)
    finish_codes_kernel(const int32_t *__restrict__ win, const uint8_t *__restrict__ value,
                        uint8_t *__restrict__ out, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t w = win[i];
    out[i] = w >= 0 ? value[w] : (uint8_t)255;
  }
}

// ---- ignition list of a time raster ------------------------------------------
constexpr int kChunk = 4096;  // cells per CTA iteration of the count and write passes
constexpr int kChunkSteps = kChunk / kRasterThreads;

__global__ void __launch_bounds__(kRasterThreads)
    count_burning_kernel(const float *__restrict__ t, int64_t n, uint64_t chunks,
                         uint32_t *__restrict__ counts) {
  __shared__ uint32_t part[kRasterThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (uint64_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
    const int64_t base = (int64_t)ch * kChunk;
    uint32_t k = 0;
    for (int j = threadIdx.x; j < kChunk; j += kRasterThreads) {
      const int64_t i = base + j;
      if (i < n && t[i] != FLT_MAX) ++k;
    }
    for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(0xFFFFFFFFu, k, o);
    if (lane == 0) part[wid] = k;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t s = 0;
      for (int w = 0; w < kRasterThreads / 32; ++w) s += part[w];
      counts[ch] = s;
    }
    __syncthreads();
  }
}

// One CTA: offsets[k] = sum of counts[0 .. k), offsets[chunks] = the total.
__global__ void __launch_bounds__(1024)
    scan_counts_kernel(const uint32_t *__restrict__ counts, uint64_t chunks,
                       uint64_t *__restrict__ offsets) {
  __shared__ uint64_t part[1024];
  const uint64_t per = (chunks + blockDim.x - 1) / blockDim.x;
  const uint64_t a = min(chunks, (uint64_t)threadIdx.x * per), b = min(chunks, a + per);
  uint64_t s = 0;
  for (uint64_t k = a; k < b; ++k) s += counts[k];
  part[threadIdx.x] = s;
  __syncthreads();
  for (unsigned d = 1; d < blockDim.x; d <<= 1) {
    const uint64_t v = threadIdx.x >= d ? part[threadIdx.x - d] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  uint64_t run = part[threadIdx.x] - s;
  for (uint64_t k = a; k < b; ++k) {
    offsets[k] = run;
    run += counts[k];
  }
  if (threadIdx.x == blockDim.x - 1) offsets[chunks] = part[threadIdx.x];
}

// Burning cells (time != FLT_MAX, NaN included) in row-major order.  Chunks
// without one are passed over, the others loaded whole before the one barrier
// that their counts need: 24 us with a barrier pair per 256 cells, 12 us now
// (40 ignitions on a 3001 x 2003 grid).
__global__ void __launch_bounds__(kRasterThreads)
    write_burning_kernel(const float *__restrict__ t, int64_t n, int64_t W, uint64_t chunks,
                         const uint64_t *__restrict__ offsets, PropagIgnition *__restrict__ out,
                         uint64_t max_out) {
  __shared__ uint32_t warp_count[kChunk / 32];  // burning cells of each run of 32
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (uint64_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
    const uint64_t first = offsets[ch];
    if (offsets[ch + 1] == first) continue;  // most chunks: nothing burns
    const int64_t base = (int64_t)ch * kChunk;
    float v[kChunkSteps];
#pragma unroll
    for (int j = 0; j < kChunkSteps; ++j) {
      const int64_t i = base + j * kRasterThreads + threadIdx.x;
      v[j] = i < n ? t[i] : FLT_MAX;
    }
#pragma unroll
    for (int j = 0; j < kChunkSteps; ++j) {
      const uint32_t vote = __ballot_sync(0xFFFFFFFFu, v[j] != FLT_MAX);
      if (lane == 0) warp_count[j * kRasterWarps + wid] = (uint32_t)__popc(vote);
    }
    __syncthreads();
    uint64_t at = first;
#pragma unroll
    for (int j = 0; j < kChunkSteps; ++j) {
      const uint32_t vote = __ballot_sync(0xFFFFFFFFu, v[j] != FLT_MAX);
      uint32_t ahead = (uint32_t)__popc(vote & ((1u << lane) - 1u)), total = 0;
      for (int w = 0; w < kRasterWarps; ++w) {
        const uint32_t k = warp_count[j * kRasterWarps + w];
        if (w < wid) ahead += k;
        total += k;
      }
      if (v[j] != FLT_MAX && at + ahead < max_out) {
        const int64_t i = base + j * kRasterThreads + threadIdx.x;
        PropagIgnition g;
        g.x = (uint32_t)(i % W);
        g.y = (uint32_t)(i / W);
        g.time = v[j];
        out[at + ahead] = g;
      }
      at += total;
    }
    __syncthreads();  // warp_count is rewritten by the next chunk
  }
}

}  // namespace raster_dev
}  // namespace propag
