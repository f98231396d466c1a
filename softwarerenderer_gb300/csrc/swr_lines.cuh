// Points and lines: VertexProcessor::clipPoints / clipLines (VertexProcessor.cpp:152-215,
// LineClipper.cpp:30-56) and Rasterizer::drawPointTemplate / drawLineTemplate
// (Rasterizer.h:150-222).
//
//   k_assemble_lp_count / _emit  one CTA per batch: outcodes, parametric line clipping
//                                (endpoints replaced by lerps at t0 / t1), point rejection;
//                                survivors keep submission order
//   k_lp_setup                   per primitive: DDA step count and per-step increments
//   k_lp_frags                   one fragment per DDA step, numbered in primitive order, then
//                                step order: the stepped position by exact fold, the
//                                per-step scissor test, the pixel; counts (tile, segment) cells
//   k_lp_fill                    fragment numbers into their tile's bin (the triangles' cells:
//                                a tile's fragments in SWR_SEGS runs of fragment numbers);
//                                k_sort_tiles orders cells above SWR_LP_CHUNK entries and all
//                                cells of heavy tiles, the tile's CTA the others
//   k_lp_raster                  one CTA per 16 x 16 tile, four per heavy one: each thread owns a
//                                pixel and applies its fragments in order (a line may hit a
//                                pixel twice)
//
// Binning by tile took the place of a stable radix sort of all fragments by pixel (three
// 8-bit passes of three kernels, then one thread per covered pixel searching each fragment's
// primitive).  Sizes below: 1M points and 122,880 lines (0.5M fragments) at 1920x1080.
#pragma once
#include "swr_stages.cuh"

namespace swr {

// Line / point record for pixel shader PS: steps, draw id, start vertex, per-step increment;
// each vertex is x, y, z, w, avar[NA], pvar[NP].
template <class PS>
struct LpRec {
  enum { NA = PS::AVarCount, NP = PS::PVarCount, NV = 4 + NA + NP, R = 2 + 2 * NV };
};

template <int A, int P>
__device__ uint32_t assemble_lp_one(const AssembleArgs& g, const SwrDrawDesc& D, uint32_t p) {
  typedef VLayout<A, P> L;
  const uint32_t gp = D.pbase + p;
  const int per = D.draw_mode == 0 ? 1 : 2;
  uint32_t idx[2] = {0, 0};
  for (int k = 0; k < per; ++k) {
    idx[k] = D.indices[(size_t)per * p + k];
    if (idx[k] >= D.nverts) {
      atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_BAD_INDEX);
      g.tri_flags[gp] = 0;
      return 0;
    }
  }
  const uint32_t r0 = D.vbase + idx[0], r1 = D.vbase + idx[per - 1];
  const float* v0 = g.ptv + (size_t)r0 * L::S;
  const float* v1 = g.ptv + (size_t)r1 * L::S;
  const int m0 = __float_as_int(v0[7]), m1 = __float_as_int(v1[7]);
  uint2 ref = make_uint2(r0, r1);
  uint32_t kept = 0;
  if (per == 1) {  // clipPoints: any outcode bit rejects
    kept = m0 == 0;
  } else if ((m0 | m1) == 0) {
    kept = 1;
  } else {
    // LineClipper against every plane whose bit is set in either outcode; each test uses
    // the original endpoints, t0 only grows and t1 only shrinks.
    const int m = m0 | m1;
    const float pl[6][4] = {{-1, 0, 0, 1}, {1, 0, 0, 1}, {0, -1, 0, 1}, {0, 1, 0, 1}, {0, 0, -1, 1}, {0, 0, 1, 1}};
    float t0 = 0.0f, t1 = 1.0f;
    bool gone = false;
    for (int k = 0; k < 6 && !gone; ++k) {
      if (!(m & (1 << k))) continue;
      const float d0 = Clipper<A, P>::dist(v0, pl[k][0], pl[k][1], pl[k][2], pl[k][3]);
      const float d1 = Clipper<A, P>::dist(v1, pl[k][0], pl[k][1], pl[k][2], pl[k][3]);
      const bool n0 = d0 < 0.0f, n1 = d1 < 0.0f;
      if (n0 && n1) {
        gone = true;
      } else if (n0) {
        const float t = swr_div(-d0, swr_sub(d1, d0));
        t0 = (t0 < t) ? t : t0;
      } else {
        const float t = swr_div(d0, swr_sub(d0, d1));
        t1 = (t < t1) ? t : t1;
      }
    }
    if (!gone) {
      // endpoints with a non-zero outcode are replaced (VertexProcessor.cpp:201-213)
      const int nnew = (m0 ? 1 : 0) + (m1 ? 1 : 0);
      const uint32_t vb = atomicAdd(&g.status[SWR_ST_CLIP_VERTS], (uint32_t)nnew);
      if (vb + nnew > g.cap_clip_verts) {
        atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_CLIP_OVERFLOW);
        g.tri_flags[gp] = 0;
        return 0;
      }
      uint32_t next = vb;
      for (int e = 0; e < 2; ++e) {
        if (!(e ? m1 : m0)) continue;
        const float t = e ? t1 : t0;  // Helper::interpolateVertex(v0, v1, t)
        const float s = swr_sub(1.0f, t);
        float* o = g.clipv + (size_t)next * L::S;
        for (int c = 0; c < 4; ++c) o[c] = swr_add(swr_mul(v0[c], s), swr_mul(v1[c], t));
        for (int i = 0; i < A; ++i)
          o[L::OFF_A + i] = swr_add(swr_mul(v0[L::OFF_A + i], s), swr_mul(v1[L::OFF_A + i], t));
        for (int i = 0; i < P; ++i)
          o[L::OFF_P + i] = swr_add(swr_mul(v0[L::OFF_P + i], s), swr_mul(v1[L::OFF_P + i], t));
        to_screen(D, o[0], o[1], o[2], o[3], o[4], o[5], o[6]);
        o[7] = __int_as_float(0);
        if (e) ref.y = SWR_CLIP_REF | next; else ref.x = SWR_CLIP_REF | next;
        next++;
      }
      kept = 1;
    }
  }
  g.tri_flags[gp] = (uint8_t)kept;
  g.lp_refs[gp] = ref;
  return kept;
}

template <int A, int P>
__global__ void __launch_bounds__(256) k_assemble_lp_count(AssembleArgs g) {
  swr_pdl_entry();
  __shared__ uint32_t tmp[32];
  const uint32_t b = blockIdx.x;
  const int d = g.ndraws > 1 ? swr_find_le(g.draw_bbase, g.ndraws, b) : 0;
  const SwrDrawDesc& D = g.draws[d];
  const uint32_t p0 = (b - D.bbase) * SWR_BATCH_PRIMS;
  uint32_t sum = 0;
  for (int j = 0; j < 4; ++j) {
    const uint32_t p = p0 + j * 256 + threadIdx.x;  // consecutive threads, consecutive primitives
    if (p < D.nprims) sum += assemble_lp_one<A, P>(g, D, p);
  }
  uint32_t tot;
  swr_block_exscan(sum, tmp, &tot);
  if (threadIdx.x == 0) g.batch_base[b] = tot;
  uint32_t total;
  if (swr_last_block_scan(g.batch_base, gridDim.x, g.done, &total) && threadIdx.x == 0) {
    g.status[SWR_ST_PRIMS] = total;
    if (total > g.cap_prims) atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_PRIM_OVERFLOW);
  }
}

static __global__ void __launch_bounds__(256) k_assemble_lp_emit(AssembleArgs g) {
  swr_pdl_entry();
  __shared__ uint32_t tmp[32];
  if (g.status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  const uint32_t b = blockIdx.x;
  const int d = g.ndraws > 1 ? swr_find_le(g.draw_bbase, g.ndraws, b) : 0;
  const SwrDrawDesc& D = g.draws[d];
  const uint32_t p0 = (b - D.bbase) * SWR_BATCH_PRIMS;
  uint32_t keep[4], sum = 0;
  for (int j = 0; j < 4; ++j) {
    const uint32_t p = p0 + threadIdx.x * 4 + j;
    keep[j] = (p < D.nprims && p < p0 + SWR_BATCH_PRIMS) ? g.tri_flags[D.pbase + p] & 1u : 0u;
    sum += keep[j];
  }
  uint32_t tot;
  uint32_t rank = swr_block_exscan(sum, tmp, &tot);
  const uint32_t base = g.batch_base[b];
  for (int j = 0; j < 4; ++j) {
    if (!keep[j]) continue;
    const uint2 r = g.lp_refs[D.pbase + p0 + threadIdx.x * 4 + j];
    g.tris[base + rank] = make_uint4(r.x, r.y, 0u, (uint32_t)d);
    rank++;
  }
}

// Words between the records of consecutive primitives: points have no step, so their records
// end after the start vertex.
template <class PS>
__device__ __forceinline__ int lp_stride(int draw_mode) {
  return draw_mode == 0 ? 2 + LpRec<PS>::NV : LpRec<PS>::R;
}

constexpr int kLpSetupThreads = 128;

// Per primitive: start vertex and per-step increment (computeVertexStep, Rasterizer.h:210-222).
// Bound by memory: one or two gathered vertex records in, one record out.  Records are staged
// in shared memory (odd stride: no bank conflicts) and written as contiguous words; one
// thread storing its own 64-byte record word by word took 74 us for 1M points.
template <class PS>
__global__ void __launch_bounds__(kLpSetupThreads) k_lp_setup(SetupArgs g) {
  swr_pdl_entry();
  typedef LpRec<PS> RL;
  constexpr int RS = RL::R | 1;
  __shared__ float stage[kLpSetupThreads * RS];
  if (g.status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  uint32_t np = g.status[SWR_ST_PRIMS];
  if (np > g.cap_prims) np = g.cap_prims;
  const int mode = g.draws[0].draw_mode;  // points and lines are drawn one draw at a time
  const uint32_t W = (uint32_t)lp_stride<PS>(mode);
  // 16-byte aligned vertex records: words 0-3 clip position, 4-6 screen x, y, z, then avars and pvars
  auto vertex = [&](uint32_t ref, float* o) {
    const float* vp = (ref & SWR_CLIP_REF) ? g.clipv + (size_t)(ref & ~SWR_CLIP_REF) * g.S : g.ptv + (size_t)ref * g.S;
    const float4 q = __ldg((const float4*)vp + 1);
    o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = __ldg(vp + 3);
    for (int i = 0; i < RL::NA; ++i) o[4 + i] = i < g.vs_a ? __ldg(vp + g.off_a + i) : 0.0f;
    for (int i = 0; i < RL::NP; ++i) o[4 + RL::NA + i] = i < g.vs_p ? __ldg(vp + g.off_p + i) : 0.0f;
  };
  for (uint32_t p0 = blockIdx.x * kLpSetupThreads; p0 < np; p0 += gridDim.x * kLpSetupThreads) {
    const uint32_t p = p0 + threadIdx.x;
    if (p < np) {
      const uint4 t = g.tris[p];
      float a[RL::NV];
      vertex(t.x, a);
      float* rec = stage + threadIdx.x * RS;
      int steps = 1;
      if (mode == 1) {
        float b[RL::NV];
        vertex(t.y, b);
        const int adx = abs(swr_trunc_int(b[0]) - swr_trunc_int(a[0]));
        const int ady = abs(swr_trunc_int(b[1]) - swr_trunc_int(a[1]));
        steps = adx > ady ? adx : ady;
        const float fs = (float)steps;
        for (int i = 0; i < RL::NV; ++i) rec[2 + RL::NV + i] = swr_div(swr_sub(b[i], a[i]), fs);
      }
      rec[0] = __int_as_float(steps);
      rec[1] = __int_as_float((int)t.w);
      for (int i = 0; i < RL::NV; ++i) rec[2 + i] = a[i];
      g.tile_count[p] = (uint32_t)(steps > 0 ? steps : 0);
    }
    __syncthreads();
    const uint32_t words = min((uint32_t)kLpSetupThreads, np - p0) * W;
    float* dst = g.recs + (size_t)p0 * W;
    for (uint32_t i = threadIdx.x; i < words; i += kLpSetupThreads) {
      const uint32_t k = i / W;
      dst[i] = stage[k * RS + (i - k * W)];
    }
    __syncthreads();
  }
}

// Stepped vertex component i after j steps.  stepVertex (Rasterizer.h:196-207) advances z
// only with InterpolateZ and w only with InterpolateW; x, y and the variables always.
template <class PS>
__device__ __forceinline__ float lp_value(const float* rec, int i, int j) {
  typedef LpRec<PS> RL;
  if (j == 0 || (i == 2 && !PS::InterpolateZ) || (i == 3 && !PS::InterpolateW)) return rec[2 + i];
  return swr_fold(rec[2 + i], rec[2 + RL::NV + i], j);
}

#define SWR_LP_TILE 16                // tile edge of the point / line bins (one pixel per thread)
#define SWR_LP_CHUNK 256              // fragments per raster chunk (one per thread)
#define SWR_LP_INVALID 0xffffffffu    // key of a fragment that reaches no target pixel
#define SWR_LP_HEAVY 4096             // tiles of more fragments are rasterized by SWR_LP_PARTS CTAs,
#define SWR_LP_PARTS 4                // each for its quarter of the tile's rows,
#define SWR_LP_SLOTS 64               // this many tiles at most

struct LpFragArgs {
  const uint32_t* status;
  uint32_t cap_prims;
  const float* recs;
  const uint32_t* steps;      // per primitive: its fragments
  const uint32_t* frag_off;   // their exclusive scan
  const uint32_t* nfrags;     // device total (SWR_COUNT_MAX: that or more)
  uint32_t cap_frags;
  const SwrDrawDesc* draws;
  const SwrTargetDesc* targets;
  uint32_t* keys;             // per fragment: tile * 256 + pixel in the tile, or SWR_LP_INVALID
  uint32_t* prims;            // per fragment: its primitive
  uint32_t* cell_count;       // per (tile, segment): fragments
  SwrCells cells;
  int seg_shift;              // segment = fragment number >> seg_shift
  uint32_t* status_w;
};

// Fragments of the primitives, one warp per 32 consecutive primitives whose fragments are
// spread over its lanes 32 at a time, so a long line does not hold up the warp and no
// fragment has to search for its primitive.  Fewer primitives a warp where they have many
// fragments each, about SWR_LP_FRAGS in all: 2,500 lines of 20 steps are 78 warps of 32, too few
// to hide each step's latency (the binning stage 57 us, 27 this way).
#ifndef SWR_LP_FRAGS
#define SWR_LP_FRAGS 128
#endif
template <class PS>
__global__ void __launch_bounds__(256) k_lp_frags(LpFragArgs g) {
  swr_pdl_entry();
  typedef LpRec<PS> RL;
  if (g.status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  // The sum of the steps, never wrapped: screen-space lines are not clipped, and one may take
  // 2^31 - 1 steps.  Past the queue nothing is written; past SWR_COUNT_MAX no queue would do.
  const uint32_t nf = *g.nfrags;
  if (nf > g.cap_frags || nf == SWR_COUNT_MAX) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      atomicOr(&g.status_w[SWR_ST_FLAGS], SWR_F_PAIR_OVERFLOW);
      g.status_w[SWR_ST_PAIRS] = nf;
    }
    return;
  }
  uint32_t np = g.status[SWR_ST_PRIMS];
  if (np > g.cap_prims) np = g.cap_prims;
  const SwrDrawDesc& D = g.draws[0];
  const SwrTargetDesc& T = g.targets[D.target];
  const uint32_t W = (uint32_t)lp_stride<PS>(D.draw_mode);
  const float sx0 = (float)D.sc_minx, sx1 = (float)D.sc_maxx, sy0 = (float)D.sc_miny, sy1 = (float)D.sc_maxy;
  const int width = T.width, height = T.height, tiles_x = T.tiles_x;
  const int lane = threadIdx.x & 31;
  // one fragment per lane (every lane of the warp calls it)
  auto put = [&](bool on, uint32_t f, uint32_t prim, float x, float y) {
    uint32_t key = SWR_LP_INVALID;
    if (on && f < g.cap_frags) {
      // Rasterizer::scissorTest on the stepped float position (Rasterizer.h:144-147)
      if (x >= sx0 && x < sx1 && y >= sy0 && y < sy1) {
        const int ix = swr_trunc_int(x), iy = swr_trunc_int(y);
        if (ix >= 0 && iy >= 0 && ix < width && iy < height)
          key = ((uint32_t)((iy / SWR_LP_TILE) * tiles_x + ix / SWR_LP_TILE) << 8) |
                (uint32_t)((iy % SWR_LP_TILE) * SWR_LP_TILE + ix % SWR_LP_TILE);
      }
      g.keys[f] = key;
      g.prims[f] = prim;
    }
    const uint32_t cell = key != SWR_LP_INVALID ? g.cells.at(key >> 8, f >> g.seg_shift) : SWR_LP_INVALID;
    const uint32_t peers = __match_any_sync(0xffffffffu, cell);  // neighbours share cells
    if (cell != SWR_LP_INVALID && lane == __ffs(peers) - 1) atomicAdd(&g.cell_count[cell], (uint32_t)__popc(peers));
  };
  uint32_t per = 32;  // primitives a warp: 32, or as many as SWR_LP_FRAGS fragments belong to
  while (per > 1 && (uint64_t)nf * per > (uint64_t)np * SWR_LP_FRAGS) per >>= 1;
  const uint32_t stride = gridDim.x * (blockDim.x >> 5) * per;
  for (uint32_t p0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per; p0 < np; p0 += stride) {
    const uint32_t p = p0 + (uint32_t)lane;
    uint32_t cnt = 0, off = 0;
    float x = 0.0f, y = 0.0f, dx = 0.0f, dy = 0.0f;
    if ((uint32_t)lane < per && p < np) {
      cnt = g.steps[p];
      off = g.frag_off[p];
      const float* rec = g.recs + (size_t)p * W;
      x = rec[2];
      y = rec[3];
      if (cnt > 1) {
        dx = rec[2 + RL::NV];
        dy = rec[3 + RL::NV];
      }
    }
    if (__reduce_max_sync(0xffffffffu, cnt) <= 1u) {  // points, lines of one step
      put(cnt != 0, off, p, x, y);
      continue;
    }
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    for (uint32_t base = 0; base < total; base += 32) {
      const uint32_t j = base + (uint32_t)lane;
      int src = 0;  // owner: the number of lanes whose inclusive count is <= j
#pragma unroll
      for (int step = 16; step; step >>= 1) {
        const uint32_t v = __shfl_sync(0xffffffffu, inc, src + step - 1);
        if (v <= j) src += step;
      }
      src = src < 31 ? src : 31;
      const uint32_t first = __shfl_sync(0xffffffffu, inc - cnt, src);
      const uint32_t ooff = __shfl_sync(0xffffffffu, off, src);
      const float ox = __shfl_sync(0xffffffffu, x, src), oy = __shfl_sync(0xffffffffu, y, src);
      const float odx = __shfl_sync(0xffffffffu, dx, src), ody = __shfl_sync(0xffffffffu, dy, src);
      const bool on = j < total;
      const int k = on ? (int)(j - first) : 0;
      put(on, ooff + (uint32_t)k, p0 + (uint32_t)src, swr_fold(ox, odx, k), swr_fold(oy, ody, k));
    }
  }
}

// Fragment numbers into their cells (arbitrary order inside a cell); takes every count of
// k_lp_frags back, so the counters are zero again after the draw.
static __global__ void __launch_bounds__(256) k_lp_fill(const uint32_t* status, const uint32_t* nfrags,
                                                        uint32_t cap_frags, const uint32_t* keys,
                                                        uint32_t* cell_count, const uint32_t* fill_start,
                                                        SwrCells cells, int seg_shift, uint32_t* bin) {
  swr_pdl_entry();
  if (status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;  // (k_lp_frags counted nothing then)
  const uint32_t nf = min(*nfrags, cap_frags);
  const int lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t f0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; f0 < nf; f0 += stride) {
    const uint32_t f = f0 + (uint32_t)lane;
    const uint32_t key = f < nf ? keys[f] : SWR_LP_INVALID;
    const uint32_t cell = key != SWR_LP_INVALID ? cells.at(key >> 8, f >> seg_shift) : SWR_LP_INVALID;
    const uint32_t peers = __match_any_sync(0xffffffffu, cell);
    const int leader = __ffs(peers) - 1;
    uint32_t pos = 0;
    if (cell != SWR_LP_INVALID && lane == leader) {
      const uint32_t n = (uint32_t)__popc(peers);
      pos = fill_start[cell] + atomicSub(&cell_count[cell], n) - n;
    }
    pos = __shfl_sync(0xffffffffu, pos, leader);
    if (cell != SWR_LP_INVALID) bin[pos + (uint32_t)__popc(peers & ((1u << lane) - 1u))] = f;
  }
}

struct LpRasterArgs {
  const uint32_t* status;
  const float* recs;
  const uint32_t* frag_off;
  const uint32_t* keys;        // per fragment (LpFragArgs)
  const uint32_t* prims;
  SwrTiles tiles;              // the tiles with fragments, their bins and cells
  const uint32_t* bin_raw;     // fragment numbers, unordered inside a cell
  const uint32_t* bin;         // ordered by k_sort_tiles, for cells of more than SWR_LP_CHUNK entries
                               // and all cells of tiles of more than SWR_LP_HEAVY
  const SwrDrawDesc* draws;
  const SwrTargetDesc* targets;
  uint32_t* status_w;
};

// The words of an interpolated fragment: f(i, word) for each.
template <class PS>
struct LpPixelWords {
  enum { W = PS::InterpolateW ? 2 : 0, value = 1 + W + PS::AVarCount + PS::PVarCount };
};
template <class PS, class F>
__device__ __forceinline__ void lp_words(GpuPixel<PS>& pd, F f) {
  typedef LpPixelWords<PS> PW;
  f(0, pd.z);
  if (PS::InterpolateW) {
    f(1, pd.w);
    f(2, pd.invw);
  }
#pragma unroll
  for (int a = 0; a < PS::AVarCount; ++a) f(1 + PW::W + a, pd.avar[a]);
#pragma unroll
  for (int a = 0; a < PS::PVarCount; ++a) f(1 + PW::W + PS::AVarCount + a, pd.pvar[a]);
}

// Rasterizer::pixelDataFromVertex (Rasterizer.h:161-173) of step j of a primitive's record.
template <class PS>
__device__ __forceinline__ void lp_pixel(const float* rec, int j, int fx, int fy, GpuPixel<PS>& pd) {
  typedef LpRec<PS> RL;
  pd.x = fx;
  pd.y = fy;
  pd.eq = nullptr;  // points and lines carry no triangle equations
  pd.z = 0.0f;
  if (PS::InterpolateZ) pd.z = lp_value<PS>(rec, 2, j);
  if (PS::InterpolateW) {
    pd.w = lp_value<PS>(rec, 3, j);
    pd.invw = swr_div(1.0f, pd.w);
  }
  for (int a = 0; a < RL::NA; ++a) pd.avar[a] = lp_value<PS>(rec, 4 + a, j);
  for (int a = 0; a < RL::NP; ++a) pd.pvar[a] = lp_value<PS>(rec, 4 + RL::NA + a, j);
}

// A quarter of the rows of a heavy tile, whose cells are all ordered: the CTA looks through the
// tile's fragments 512 at a time, keeps those of its rows, in order, and rasterizes them in chunks
// as k_lp_raster does, its first 64 threads owning the pixels.  A chunk is a chain of a few
// microseconds however few pixels it is for, and one CTA had all of a tile's: 10,000 lines inside
// one tile, 80,000 fragments, took 1811 us in the raster, four CTAs 870; 100,000 points 959 and 432.
// Tiles of fewer fragments have most cells within a chunk, and ordering those ahead costs more
// than this gains (1M points on a sphere 213 us a draw, 278 with the line at 2,048).
// The lists lie where the other tiles' masks do: more shared memory is less cache for all.
struct LpHeavy {
  enum { FIND = 512, CH = SWR_LP_CHUNK, PART = 256 / SWR_LP_PARTS };
  uint32_t mask[CH / 32][PART];  // per pixel: the chunk's fragments that hit it
  uint32_t f[FIND];              // the finds: fragment number
  uint8_t pix[FIND];             // and pixel, from the first row's first
  uint32_t count[FIND / 32];
};

template <class PS, class Shared>
__device__ __forceinline__ uint2 lp_heavy_rows(const LpRasterArgs& g, uint4 entry, int first, Shared& sh) {
  typedef LpHeavy H;
  static_assert(sizeof(H) <= sizeof(sh.mask), "the lists fit the masks' place");
  H& h = *(H*)sh.mask;
  const uint32_t tile = entry.x, b = entry.y, total = entry.z - entry.y;
  const SwrDrawDesc& D = g.draws[0];
  const SwrTargetDesc& T = g.targets[D.target];
  const SwrUniforms& U = D.u;
  const uint32_t W = (uint32_t)lp_stride<PS>(D.draw_mode);
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ox = (int)(tile % (uint32_t)T.tiles_x) * SWR_LP_TILE;
  const int oy = (int)(tile / (uint32_t)T.tiles_x) * SWR_LP_TILE + first / SWR_LP_TILE;
  const int x = ox + tid % SWR_LP_TILE, y = oy + tid / SWR_LP_TILE;
  const bool in = tid < H::PART && x < T.width && y < T.height;
  uint32_t frags = 0;
  typename PS::State st;
  if (in) PS::load(st, x, y, U);
  for (uint32_t base = 0; base < total; base += H::FIND) {
    constexpr int R = H::FIND / H::CH;
    uint32_t f[R], key[R], bal[R];
    __syncthreads();  // the previous finds are no longer read
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t i = base + (uint32_t)(r * H::CH + tid);
      f[r] = i < total ? g.bin[b + i] : 0u;
      key[r] = i < total ? (g.keys[f[r]] & 255u) - (uint32_t)first : 256u;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      bal[r] = __ballot_sync(0xffffffffu, key[r] < (uint32_t)H::PART);
      if (lane == 0) h.count[r * (H::CH / 32) + warp] = (uint32_t)__popc(bal[r]);
    }
    __syncthreads();
    static_assert(R * (H::CH / 32) <= 32, "one count per lane");
    const uint32_t cnt = lane < R * (H::CH / 32) ? h.count[lane] : 0u;
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const int m = (int)__shfl_sync(0xffffffffu, inc, 31);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t at = __shfl_sync(0xffffffffu, inc - cnt, r * (H::CH / 32) + warp) +
                          (uint32_t)__popc(bal[r] & ((1u << lane) - 1u));
      if (key[r] < (uint32_t)H::PART) {
        h.f[at] = f[r];
        h.pix[at] = (uint8_t)key[r];
      }
    }
    for (int c0 = 0; c0 < m; c0 += H::CH) {
      const int n = min((int)H::CH, m - c0), words = (n + 31) / 32;
      if (tid < H::PART)
        for (int w = 0; w < words; ++w) h.mask[w][tid] = 0u;
      __syncthreads();
      if (tid < n) {
        const uint32_t fr = h.f[c0 + tid], prim = g.prims[fr];
        const int pix = h.pix[c0 + tid], j = D.draw_mode == 0 ? 0 : (int)(fr - g.frag_off[prim]);
        sh.put(tid, g.recs + (size_t)prim * W, prim, j, ox + pix % SWR_LP_TILE, oy + pix / SWR_LP_TILE, U);
        atomicOr(&h.mask[tid >> 5][pix], 1u << (tid & 31));
      }
      __syncthreads();
      if (in)
        for (int w = 0; w < words; ++w)
          for (uint32_t s = h.mask[w][tid]; s; s &= s - 1u) {
            frags++;
            sh.take(w * 32 + __ffs(s) - 1, x, y, st, U);
          }
      __syncthreads();  // the chunk is no longer read
    }
  }
  if (!in || !frags) return make_uint2(0u, 0u);
  PS::store(st, x, y, U);
  return make_uint2(frags, st.writes);  // (fragments and writes)
}

// A chunk's fragments in shared memory.
template <class PS>
struct LpChunk {
  enum { CH = SWR_LP_CHUNK, CW = CH / 32, COMPACT = !SwrNoCompact<PS>::value };
  uint32_t mask[CW][256];  // per pixel: the chunk's fragments that hit it
  uint32_t prim[CH];
  float z[COMPACT ? CH : 1];
  typename PS::Color color[COMPACT ? CH : 1];
  float words[COMPACT ? 1 : LpPixelWords<PS>::value * CH];  // shaders with side effects: interpolated, not shaded
  // Interpolates (and shades) step j of a primitive as the k-th fragment ...
  __device__ __forceinline__ void put(int k, const float* rec, uint32_t p, int j, int fx, int fy, const SwrUniforms& U) {
    prim[k] = p;
    GpuPixel<PS> pd;
    if constexpr (COMPACT) {
      lp_pixel<PS>(rec, j, fx, fy, pd);
      z[k] = pd.z;
      color[k] = PS::shade(pd, U);
    } else {
      lp_pixel<PS>(rec, j, 0, 0, pd);
      lp_words<PS>(pd, [&](int i, float& v) { words[i * CH + k] = v; });
    }
  }
  // ... and applies it to the pixel (x, y) it hits.
  __device__ __forceinline__ void take(int k, int x, int y, typename PS::State& st, const SwrUniforms& U) {
    if constexpr (COMPACT) {
      PS::apply(st, z[k], color[k], (int)prim[k]);
    } else {
      GpuPixel<PS> pd;
      pd.x = x;
      pd.y = y;
      pd.eq = nullptr;  // points and lines carry no triangle equations
      lp_words<PS>(pd, [&](int i, float& v) { v = words[i * CH + k]; });
      PS::drawPixel(pd, (int)prim[k], st, U);
    }
  }
};

// One CTA per listed 16 x 16 tile, one pixel per thread (the first SWR_LP_PARTS * heavy_cap CTAs take
// the heavy tiles' rows: lp_heavy_rows).  A chunk is as many whole cells of the
// tile's bin as hold at most 256 fragments (a larger cell, ordered by k_sort_tiles, is a run of
// chunks by itself): one fragment per thread is ranked inside its cell, interpolated, shaded
// and marked under its rank in its pixel's set; then each thread applies its pixel's
// fragments in increasing order (shaders with side effects of their own are not shaded ahead:
// each gets its interpolated fragments' words there, one drawPixel at a time.  Interpolated
// there as well, in lanes that few of a tile's pixels keep busy, 200,000 lines of 40 steps of a
// user shader took 3435 us a draw; this way 1394).  Bound by the latency of the dependent gathers bin ->
// primitive -> record.  Ordering the cells here instead of ahead (a warp ranking each cell of
// 17 to 64 entries, a bitmap above) took the two sorts from 184 to 4 us on the points and
// from 64 to 4 us on the lines.
template <class PS>
__global__ void __launch_bounds__(256) k_lp_raster(const __grid_constant__ LpRasterArgs g) {
  swr_pdl_entry();
  constexpr int CH = SWR_LP_CHUNK;
  static_assert(CH == 256 && SWR_SEGS == 32, "one fragment per thread, one cell per lane");
  __shared__ uint32_t sraw[CH];
  __shared__ uint32_t scs[SWR_SEGS + 1];
  __shared__ LpChunk<PS> sh;
  __shared__ uint32_t sfr[64];
  if (blockIdx.x == 0 && threadIdx.x == 0) swr_close_status(g.status_w);
  if (g.status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  uint4 entry;
  auto report = [&](uint32_t frags, uint32_t passes) {
    uint32_t tot, ptot;
    swr_block_sum2(frags, passes, sfr, tot, ptot);
    if (threadIdx.x == 0 && tot) {
      atomicAdd((unsigned long long*)&g.status_w[SWR_ST_SHADED_LO], (unsigned long long)tot);
      atomicAdd((unsigned long long*)&g.status_w[SWR_ST_PASSES_LO], (unsigned long long)ptot);
    }
  };
  const uint32_t nheavy = SWR_LP_PARTS * g.tiles.heavy_cap;
  if (blockIdx.x < nheavy) {
    if (blockIdx.x / SWR_LP_PARTS >= min(g.tiles.counts[0], g.tiles.heavy_cap)) return;
    const uint2 done = lp_heavy_rows<PS>(g, __ldg(g.tiles.heavy + blockIdx.x / SWR_LP_PARTS),
                                         (int)(blockIdx.x % SWR_LP_PARTS) * LpHeavy::PART, sh);
    report(done.x, done.y);
    return;
  }
  if (!swr_listed_tile(g.tiles, blockIdx.x - nheavy, entry)) return;
  const uint32_t tile = entry.x, b = entry.y, e = entry.z;
  const uint32_t* cells = g.tiles.start + (size_t)tile * SWR_SEGS;
  const SwrDrawDesc& D = g.draws[0];
  const SwrTargetDesc& T = g.targets[D.target];
  const SwrUniforms& U = D.u;
  const int mode = D.draw_mode;
  const uint32_t W = (uint32_t)lp_stride<PS>(mode);
  const int tid = (int)threadIdx.x, lane = tid & 31;
  const int x = (int)(tile % (uint32_t)T.tiles_x) * SWR_LP_TILE + tid % SWR_LP_TILE;
  const int y = (int)(tile / (uint32_t)T.tiles_x) * SWR_LP_TILE + tid / SWR_LP_TILE;
  const bool in = x < T.width && y < T.height;
  typename PS::State st;
  if (in) PS::load(st, x, y, U);
  if (tid <= SWR_SEGS) scs[tid] = (tid < SWR_SEGS ? cells[tid] : e) - b;
  uint32_t frags = 0, passes = 0;
  const uint32_t total = e - b;
  __syncthreads();
  uint32_t c0 = 0;  // first entry of the chunk, relative to b
  int cell = 0;     // the cell it lies in
  while (c0 < total) {
    // the chunk: cells [cell, last), or a run of an ordered cell that is larger than a chunk
    const int last = __popc(__ballot_sync(0xffffffffu, scs[lane + 1] <= c0 + CH));
    const bool whole = last > cell && scs[cell] == c0;
    const uint32_t c1 = whole ? scs[last] : min(c0 + CH, scs[cell + 1]);
    const int n = (int)(c1 - c0);
    const int words = (n + 31) / 32;
    __syncthreads();  // the previous chunk's shared state is no longer read
    uint32_t f = 0;
    if (tid < n) {
      f = whole ? g.bin_raw[b + c0 + tid] : g.bin[b + c0 + tid];
      sraw[tid] = f;
    }
    for (int w = 0; w < words; ++w) sh.mask[w][tid] = 0u;
    __syncthreads();
    if (tid < n) {
      const uint32_t prim = g.prims[f];
      const int pix = (int)(g.keys[f] & 255u);
      const int j = mode == 0 ? 0 : (int)(f - g.frag_off[prim]);
      int k = tid;  // the fragment's place in the chunk
      if (whole) {
        const uint32_t at = c0 + (uint32_t)tid;
        int lo = cell, hi = last - 1;  // its cell: the last one starting at or before it
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (scs[mid] <= at) lo = mid; else hi = mid - 1;
        }
        const int r0 = (int)(scs[lo] - c0), r1 = (int)(scs[lo + 1] - c0);
        k = r0;
        for (int i = r0; i < r1; ++i) k += sraw[i] < f;  // numbers are unique
      }
      sh.put(k, g.recs + (size_t)prim * W, prim, j, x - tid % SWR_LP_TILE + pix % SWR_LP_TILE,
             y - tid / SWR_LP_TILE + pix / SWR_LP_TILE, U);
      atomicOr(&sh.mask[k >> 5][pix], 1u << (k & 31));
    }
    __syncthreads();
    c0 = c1;
    while (cell < SWR_SEGS && scs[cell + 1] <= c0) ++cell;
    if (!in) continue;
    for (int w = 0; w < words; ++w) {
      uint32_t m = sh.mask[w][tid];
      while (m) {
        const int k = w * 32 + __ffs(m) - 1;
        m &= m - 1u;
        frags++;
        sh.take(k, x, y, st, U);
      }
    }
  }
  if (in && frags) {
    PS::store(st, x, y, U);
    passes = st.writes;
  }
  report(frags, passes);
}

}  // namespace swr
