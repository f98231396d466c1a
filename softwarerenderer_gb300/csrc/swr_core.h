// Host launchers of the generic device primitives (swr_core.cu) and of the pipeline
// stages (swr_stages.cuh, instantiated per shader program).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "swr_device.cuh"

namespace swr {

// Blocks used by the fixed-grid scan / sort kernels (each owns a contiguous chunk).
constexpr int kScanBlocks = 304;  // 2 x 152 SMs

// Exclusive prefix sum of in[0..n) into out, where n = min(*n_dev, n_max) when n_dev is
// given (device-resident length) else n_max.  total (device) receives the sum, or
// SWR_COUNT_MAX when it is that or more: the prefixes are then of no use.
// scratch needs scan_scratch_words(n_max) words.  Two kernels: block partial sums, then
// each block prefixes the partials before it and scans its chunk.
size_t scan_scratch_words(uint32_t n_max);
void scan_exclusive(const uint32_t* in, uint32_t* out, const uint32_t* n_dev, uint32_t n_max,
                    uint32_t* total, uint32_t* scratch, cudaStream_t s);

// Places the (tile, segment) cells of a binned draw: every non-empty tile gets a range of
// *total (advanced by the entries), its cells in segment order.  Ranges are handed out as
// blocks of 32 tiles come, not in tile order: nothing needs one tile's range to follow
// another's, and the exclusive scan that put them in order was two launches (10 us of a small
// draw's chain; on 256 meshes' 491,520 mostly empty tiles 79 us).  The same kernel makes the
// lists of t, so that empty tiles cost the later kernels nothing.  SWR_COUNT_MAX entries or more
// set SWR_F_PAIR_OVERFLOW (*total is then of no use).
//   count       per cell (layout `cells`)
//   fill_start  the starts in that layout (segment-major only; tile-major it is t.start itself)
//   heavy_min   tiles of more entries go to t.heavy, up to t.heavy_cap, and not to t.list
//   sort_min    tiles of more entries go to t.sort
//   front_min   tiles of more entries go to t.list's front (rasterized first), others to its back
struct CellsArgs {
  uint32_t* status;
  const uint32_t* count;
  SwrCells cells;
  uint32_t* fill_start;
  uint32_t* total;
  SwrTiles t;
  uint32_t heavy_min, sort_min, front_min;
  const uint32_t* target_tile_base;  // per target, for the tile -> target lookup
  int ntargets;
};
void place_cells(const CellsArgs& a, cudaStream_t s);

// Stable LSD radix sort of (key, value) pairs by the low `bits` bits of key; three kernels
// per 8-bit pass (block histograms, per-digit offsets, stable scatter).
// n = min(*n_dev, n_max).  Ping-pongs between (k0,v0) and (k1,v1); returns 0 when the
// result ends in (k0, v0), 1 when it ends in (k1, v1).  scratch: sort_scratch_words(n_max).
size_t sort_scratch_words(uint32_t n_max);
int radix_sort_pairs(uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1,
                     const uint32_t* n_dev, uint32_t n_max, int bits, uint32_t* scratch,
                     cudaStream_t s);

// start[t] = first index i of sorted keys[0..n) with keys[i] >= t, for t in [0, ntiles].
void segment_starts(const uint32_t* keys, const uint32_t* n_dev, uint32_t n_max,
                    uint32_t ntiles, uint32_t* start, cudaStream_t s);

}  // namespace swr
