// Raster-stage kernels of the built-in pixel shaders: the launch wrappers and the PsOps table
// entry of one shader, instantiated per shader in the swr_ps_*.cu translation units (split
// so that the build compiles them in parallel).
#pragma once
#include "swr_ops.h"

namespace swr {
namespace {

constexpr int kGrid = 152 * 8;

template <class PS>
void run_direct(const DirectArgs& a, cudaStream_t s) {
  const uint32_t nb = (a.nprims + SWR_BATCH_PRIMS - 1) / SWR_BATCH_PRIMS, nv = (a.nverts + 255) / 256;
  const uint32_t want = nb > nv ? nb : nv;
  const uint32_t grid = want < (uint32_t)kGrid ? want : (uint32_t)kGrid;
  if (grid) swr::launch(k_direct_vertices<PS::AVarCount, PS::PVarCount>, grid, 256, 0, s, a);
}

template <class PS>
void run_setup(const SetupArgs& a, cudaStream_t s) {
  swr::launch(k_setup<PS>, a.grid ? a.grid : (uint32_t)kGrid, kSetupThreads, 0, s, a);
}

template <class PS>
void run_pairs(const uint32_t* status, uint32_t cap_prims, const float* recs, const uint32_t* tile_count,
               const uint32_t* pair_off, const uint32_t* npairs, uint32_t cap_pairs,
               const SwrDrawDesc* draws, const SwrTargetDesc* targets, int tile, uint32_t* keys,
               uint32_t* vals, uint32_t* status_w, cudaStream_t s) {
  swr::launch(k_emit_pairs<PS>, kGrid, 256, 0, s, status, cap_prims, recs, tile_count, pair_off, npairs, cap_pairs,
                                         draws, targets, tile, keys, vals, status_w);
}

template <class PS>
void run_fill(const uint32_t* status, uint32_t cap_prims, const float* recs,
              uint32_t* cell_count, const uint32_t* fill_start, const uint32_t* pairs, uint32_t ncells, SwrCells cells, int seg_shift,
              uint32_t cap_pairs,
              const SwrDrawDesc* draws, const SwrTargetDesc* targets, int tile, uint32_t* bin, uint32_t* status_w,
              cudaStream_t s) {
  swr::launch(k_fill_bins<PS>, kGrid, 256, 0, s, status, cap_prims, recs, cell_count, fill_start, pairs, ncells, cells,
                                        seg_shift, cap_pairs, draws, targets, tile, bin, status_w);
}

template <class PS>
void run_raster(const RasterArgs& a, uint32_t ntiles, int tile, cudaStream_t s) {
  constexpr int kChunk = SwrRasterChunk<PS>::value;  // primitives staged in shared memory per bin chunk
  if (!ntiles) return;
  if constexpr (SwrOverwrite<PS>::value) {
    if (a.boxes) {
      swr::launch(k_overwrite<PS, 16, true, false>, ntiles, 256, 0, s, a);
    } else {
      const uint32_t grid = a.slices > 1 ? ntiles * (uint32_t)a.slices : ntiles;
      if (tile == 32 && a.has_block) swr::launch(k_overwrite<PS, 32, false, true>, grid, 256, 0, s, a);
      else if (tile == 32) swr::launch(k_overwrite<PS, 32, false, false>, grid, 256, 0, s, a);
      else if (a.has_block) swr::launch(k_overwrite<PS, 16, false, true>, grid, 256, 0, s, a);
      else swr::launch(k_overwrite<PS, 16, false, false>, grid, 256, 0, s, a);
    }
  } else {
    if (a.boxes) {  // a small draw: 16-px tiles, one CTA each
      if (a.has_span) swr::launch(k_raster<PS, 16, kChunk, true, true>, ntiles, 256, 0, s, a);
      else swr::launch(k_raster<PS, 16, kChunk, false, true>, ntiles, 256, 0, s, a);
      return;
    }
    // one CTA per tile; Block-only submissions run the instantiation without the Span-mode passes
    uint32_t grid = ntiles;
    if (a.quad_all) grid = 4 * ntiles;
    else if (a.dslice || a.quad) grid = 4 * a.tiles.heavy_cap + ntiles;  // the heavy tiles' runs or quadrants first
    if (tile == 32) {
      if (a.has_span) swr::launch(k_raster<PS, 32, kChunk, true>, grid, 256, 0, s, a);
      else swr::launch(k_raster<PS, 32, kChunk, false>, grid, 256, 0, s, a);
    } else {
      constexpr int kBlockThreads = SwrRasterThreadsBlock<PS>::value;
      if (grid == ntiles && ntiles > SWR_RASTER_LOOP) {
        const uint32_t half = (ntiles + 1) / 2;
        if (a.has_span) swr::launch(k_raster_two<PS, kChunk, true, 256>, half, 256, 0, s, a);
        else swr::launch(k_raster_two<PS, kChunk, false, kBlockThreads>, half, kBlockThreads, 0, s, a);
      } else if (a.has_span) swr::launch(k_raster<PS, 16, kChunk, true>, grid, 256, 0, s, a);
      else swr::launch(k_raster<PS, 16, kChunk, false, false, kBlockThreads>, grid, kBlockThreads, 0, s, a);
    }
  }
}

template <class PS>
void run_lp_setup(const SetupArgs& a, cudaStream_t s) {
  swr::launch(k_lp_setup<PS>, kGrid, kLpSetupThreads, 0, s, a);
}

template <class PS>
void run_lp_frags(const LpFragArgs& a, cudaStream_t s) {
  swr::launch(k_lp_frags<PS>, kGrid, 256, 0, s, a);
}

template <class PS>
void run_lp_raster(const LpRasterArgs& a, cudaStream_t s) {
  if (a.tiles.ntiles) swr::launch(k_lp_raster<PS>, SWR_LP_PARTS * a.tiles.heavy_cap + a.tiles.ntiles, 256, 0, s, a);
}

template <class PS>
PsOps make_ps() {
  PsOps o;
  o.A = PS::AVarCount;
  o.P = PS::PVarCount;
  o.R = Rec<PS>::R;
  o.S = VLayout<PS::AVarCount, PS::PVarCount>::S;
  o.direct_vertices = &run_direct<PS>;
  o.setup = &run_setup<PS>;
  o.emit_pairs = &run_pairs<PS>;
  o.raster = &run_raster<PS>;
  o.fill_bins = &run_fill<PS>;
  o.lp_R = LpRec<PS>::R;
  o.lp_setup = &run_lp_setup<PS>;
  o.lp_frags = &run_lp_frags<PS>;
  o.lp_raster = &run_lp_raster<PS>;
  o.needs_eq = SwrNeedsEquations<PS>::value;
  o.overwrite = SwrOverwrite<PS>::value;
  o.state_bytes = (int)sizeof(typename PS::State);
  o.depth_min = SwrDepthMin<PS>::value;
  o.slice_chunks = SwrRasterSlices<PS>::value;
  o.chunk = SwrRasterChunk<PS>::value;
  return o;
}

}  // namespace
}  // namespace swr
