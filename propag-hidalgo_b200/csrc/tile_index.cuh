// Index arithmetic of shared-memory tiles.  A tile's rows and its halo's (hy in
// [0, TH + 2), hx in [0, P), P = TW + 2) are dealt to the C CTAs of a cluster
// round-robin: row hy lives in CTA hy % C at local row hy / C, and a cell's
// slot is local row * P + hx.  A test enumerates the slots on the host.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define PG_TILE_INDEX __host__ __device__ __forceinline__
#else
#define PG_TILE_INDEX inline
#endif

namespace propag {

// s / d as the high word of s * recip_of(d): ceil(2^32 / d), exact for s < 2^16
// and 2 <= d < 2^12.  2^32 / 1 does not fit the word: recip_of(1) is 0, which
// div_any takes for a division by one and div_wide does not expect.
PG_TILE_INDEX uint32_t recip_of(uint32_t d) { return d > 1u ? 0xFFFFFFFFu / d + 1u : 0u; }
PG_TILE_INDEX uint32_t div_wide(uint32_t s, uint32_t recip) {
#if defined(__CUDA_ARCH__)
  return __umulhi(s, recip);
#else
  return (uint32_t)((uint64_t)s * recip >> 32);
#endif
}
PG_TILE_INDEX uint32_t div_any(uint32_t s, uint32_t recip) { return recip ? div_wide(s, recip) : s; }

// The tile's own rows (hy = 1 .. TH) of CTA `rank` of C: the first one's local
// row and their number.
PG_TILE_INDEX int own_rows_first(int rank) { return rank == 0 ? 1 : 0; }
PG_TILE_INDEX int own_rows(int TH, int rank, int C) {
  const int n = TH >= rank ? (TH - rank) / C - own_rows_first(rank) + 1 : 0;
  return n > 0 ? n : 0;
}
// Slot of the k-th of their cells (rows in order, TW cells each); recip_tw =
// recip_of(TW).
PG_TILE_INDEX int own_slot(int k, int rank, int P, uint32_t recip_tw) {
  const int row = (int)div_any((uint32_t)k, recip_tw);
  return (own_rows_first(rank) + row) * P + 1 + (k - row * (P - 2));
}

}  // namespace propag
