// Pipeline stages of the GB300 rasterizer, templated on the shader programs.
//
//   k_vertex          VertexShader::processVertex once per vertex + outcodes + divide and
//                     viewport (VertexProcessor.cpp:122-150, :347-377)
//   k_assemble_count  one CTA per 1024-primitive batch: outcode OR, polygon clipping
//                     (PolyClipper.cpp:45-81), fan split and culling (VertexProcessor.cpp:
//                     217-263, :319-345); counts survivors per batch
//   k_assemble_emit   writes the surviving triangles in the reference's effective order:
//                     per batch, the input slots in order, then every extra fan triangle
//                     in parent order (VertexProcessor.cpp:254-260)
//   k_setup           TriangleEquations (TriangleEquations.h:47-71) and the raster-mode
//                     decision, bounding boxes and tile counts per primitive
//   k_front           small draws: the stages up to k_assemble_emit in one launch
//   k_fill_bins       primitive ids into (tile, primitive segment) cells; k_emit_pairs:
//                     (tile, primitive) pairs in primitive order for a stable radix sort
//   k_raster          one CTA per listed screen tile (k_raster_two: per two); each thread owns
//                     pixels and walks the tile's bin in primitive order, reproducing Span
//                     (Rasterizer.h:309-411) and Block (Rasterizer.h:225-306,
//                     PixelShaderBase.h:55-112) coverage and incrementally stepped
//                     interpolants exactly, with the effects of calling the pixel shader in
//                     the same per-pixel order as the reference
//   k_overwrite       the same for shaders without depth test that only overwrite
//
// All arithmetic on the parity path uses the _rn intrinsics (no FMA contraction).
#pragma once
#include "swr_device.cuh"
#include "swr_math.h"

namespace swr {

// ---------------------------------------------------------------------------------
// Post-transform vertex record (floats): 0-3 clip x,y,z,w | 4-6 screen x,y,z | 7 outcode
// | 8.. avar[A] | pvar[P].  Stride rounded to 16 bytes.
template <int A, int P>
struct VLayout {
  enum { NA = A, NP = P, OFF_A = 8, OFF_P = 8 + A, S = ((8 + A + P + 3) / 4) * 4 };
};

template <int A, int P>
struct VsOut {
  float x, y, z, w;
  float avar[A > 0 ? A : 1];
  float pvar[P > 0 ? P : 1];
};

__device__ __forceinline__ int outcode(float x, float y, float z, float w) {
  // VertexProcessor::clipMask (VertexProcessor.cpp:122-132)
  int m = 0;
  if (swr_sub(w, x) < 0.0f) m |= 0x01;
  if (swr_add(x, w) < 0.0f) m |= 0x02;
  if (swr_sub(w, y) < 0.0f) m |= 0x04;
  if (swr_add(y, w) < 0.0f) m |= 0x08;
  if (swr_sub(w, z) < 0.0f) m |= 0x10;
  if (swr_add(z, w) < 0.0f) m |= 0x20;
  return m;
}

// Perspective divide, viewport and depth range (VertexProcessor.cpp:364-373).
__device__ __forceinline__ void to_screen(const SwrDrawDesc& D, float x, float y, float z, float w,
                                          float& sx, float& sy, float& sz) {
  const float iw = swr_div(1.0f, w);
  const float nx = swr_mul(x, iw), ny = swr_mul(y, iw), nz = swr_mul(z, iw);
  sx = swr_add(swr_mul(D.vp_px, nx), D.vp_ox);
  sy = swr_add(swr_mul(D.vp_py, -ny), D.vp_oy);
  sz = swr_add(swr_mul(swr_mul(0.5f, swr_sub(D.df, D.dn)), nz), swr_mul(0.5f, swr_add(D.dn, D.df)));
}

// Vertex shading of every vertex, grid-stride over the launch's threads.
template <class VS>
__device__ __forceinline__ void vertex_stage(const SwrDrawDesc* __restrict__ draws, int ndraws,
                                             const uint32_t* __restrict__ draw_vbase, uint32_t nverts,
                                             float* __restrict__ ptv) {
  typedef VLayout<VS::AVarCount, VS::PVarCount> L;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nverts; v += gridDim.x * blockDim.x) {
    const int d = ndraws > 1 ? swr_find_le(draw_vbase, ndraws, v) : 0;
    const SwrDrawDesc& D = draws[d];
    const uint32_t local = v - D.vbase;
    SwrVertexInput in;
#pragma unroll
    for (int a = 0; a < VS::AttribCount; ++a)
      in.p[a] = (const char*)D.attrib[a] + (size_t)D.attrib_stride[a] * (size_t)local;
    VsOut<VS::AVarCount, VS::PVarCount> o;
    VS::processVertex(in, &o, D.u);
    float rec[L::S];
    rec[0] = o.x; rec[1] = o.y; rec[2] = o.z; rec[3] = o.w;
    to_screen(D, o.x, o.y, o.z, o.w, rec[4], rec[5], rec[6]);
    rec[7] = __int_as_float(outcode(o.x, o.y, o.z, o.w));
#pragma unroll
    for (int i = 0; i < VS::AVarCount; ++i) rec[L::OFF_A + i] = o.avar[i];
#pragma unroll
    for (int i = 0; i < VS::PVarCount; ++i) rec[L::OFF_P + i] = o.pvar[i];
#pragma unroll
    for (int i = 8 + VS::AVarCount + VS::PVarCount; i < L::S; ++i) rec[i] = 0.0f;
    float4* dst = (float4*)(ptv + (size_t)v * L::S);
#pragma unroll
    for (int i = 0; i < L::S / 4; ++i) dst[i] = make_float4(rec[4 * i], rec[4 * i + 1], rec[4 * i + 2], rec[4 * i + 3]);
  }
}

template <class VS>
__global__ void __launch_bounds__(256) k_vertex(const SwrDrawDesc* __restrict__ draws, int ndraws,
                                                const uint32_t* __restrict__ draw_vbase,
                                                uint32_t nverts, float* __restrict__ ptv) {
  swr_pdl_entry();
  vertex_stage<VS>(draws, ndraws, draw_vbase, nverts, ptv);
}

// Direct Rasterizer path: RasterizerVertex (x, y, z, w, avar[16], pvar[16]) records are
// already in screen space; convert them to the post-transform layout of the pixel shader.
// Primitives whose first index is -1 are skipped (Rasterizer::drawTriangleList,
// Rasterizer.h:134-141); others keep their order: the same launch counts the kept ones of
// every SWR_BATCH_PRIMS submitted, and its last block turns the counts into bases (a flag
// per primitive and a scan of them were three more launches, 10 us of a list draw's chain).
struct DirectArgs {
  const float* rv;
  uint32_t nverts;
  float* ptv;
  const int32_t* idx;
  uint32_t nprims;
  int per;             // indices per primitive
  uint32_t* base;      // per SWR_BATCH_PRIMS primitives: kept ones before them
  uint32_t* done;      // zero between draws
  uint32_t* status;
  uint32_t cap_prims;
};

template <int A, int P>
__global__ void __launch_bounds__(256) k_direct_vertices(DirectArgs g) {
  swr_pdl_entry();
  __shared__ uint32_t tmp[32];
  typedef VLayout<A, P> L;
  const uint32_t nb = (g.nprims + SWR_BATCH_PRIMS - 1) / SWR_BATCH_PRIMS;
  for (uint32_t b = blockIdx.x; b < nb; b += gridDim.x) {
    uint32_t c = 0, tot;
    for (uint32_t p = b * SWR_BATCH_PRIMS + threadIdx.x; p < min(g.nprims, (b + 1) * SWR_BATCH_PRIMS); p += 256)
      c += g.idx[(size_t)g.per * p] != -1;
    swr_block_exscan(c, tmp, &tot);
    if (threadIdx.x == 0) g.base[b] = tot;
  }
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < g.nverts; v += gridDim.x * blockDim.x) {
    const float* s = g.rv + (size_t)v * 36;
    float* o = g.ptv + (size_t)v * L::S;
    o[0] = s[0]; o[1] = s[1]; o[2] = s[2]; o[3] = s[3];
    o[4] = s[0]; o[5] = s[1]; o[6] = s[2]; o[7] = __int_as_float(0);
    for (int i = 0; i < A; ++i) o[L::OFF_A + i] = s[4 + i];
    for (int i = 0; i < P; ++i) o[L::OFF_P + i] = s[20 + i];
  }
  uint32_t total;
  if (swr_last_block_scan(g.base, nb, g.done, &total) && threadIdx.x == 0) {
    g.status[SWR_ST_PRIMS] = total;
    if (total > g.cap_prims) atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_PRIM_OVERFLOW);
  }
}

// One block per SWR_BATCH_PRIMS primitives, four consecutive ones per thread.
static __global__ void __launch_bounds__(256) k_direct_emit(DirectArgs g, uint4* __restrict__ tris) {
  swr_pdl_entry();
  __shared__ uint32_t tmp[32];
  if (g.status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  const uint32_t p0 = blockIdx.x * SWR_BATCH_PRIMS + threadIdx.x * 4;
  int32_t first[4];
  uint32_t c = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    first[k] = p0 + k < g.nprims ? g.idx[(size_t)g.per * (p0 + k)] : -1;
    c += first[k] != -1;
  }
  uint32_t at = g.base[blockIdx.x] + swr_block_exscan(c, tmp);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (first[k] == -1) continue;
    uint32_t r[3] = {0, 0, 0};
    for (int j = 0; j < g.per; ++j) {
      const int32_t i = j ? g.idx[(size_t)g.per * (p0 + k) + j] : first[k];
      if (i < 0 || (uint32_t)i >= g.nverts)
        atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_BAD_INDEX);
      else
        r[j] = (uint32_t)i;
    }
    tris[at++] = make_uint4(r[0], r[1], r[2], 0u);
  }
}

// ---------------------------------------------------------------------------------
// Triangle assembly, clipping and culling.

// Polygon clipper over a per-thread vertex pool (clip-space x,y,z,w + A + P values).
// A convex cut adds one vertex per plane (at most 9 in total); exact zeros in the plane
// distances can add more, so both the polygon and the pool are bounds-checked and a
// polygon that would exceed them is reported (SWR_F_CLIP_COMPLEX) and dropped.
template <int A, int P>
struct Clipper {
  enum { NV = 4 + A + P, POOL = 24, MAXPOLY = 16 };
  float pool[POOL][NV];
  int npool;
  int poly[MAXPOLY + 1];
  int npoly;
  bool bad;

  __device__ void lerp(int i0, int i1, float t) {  // Helper::interpolateVertex (PolyClipper.h:34-48)
    const float s = swr_sub(1.0f, t);
    float* r = pool[npool];
#pragma unroll
    for (int k = 0; k < NV; ++k) r[k] = swr_add(swr_mul(pool[i0][k], s), swr_mul(pool[i1][k], t));
    npool++;
  }

  __device__ static float dist(const float* v, float a, float b, float c, float d) {
    return swr_add(swr_add(swr_add(swr_mul(a, v[0]), swr_mul(b, v[1])), swr_mul(c, v[2])), swr_mul(d, v[3]));
  }

  __device__ static int sgn(float v) { return (0.0f < v) - (v < 0.0f); }

  // PolyClipper::clipToPlane (PolyClipper.cpp:45-81).
  __device__ void clip(float a, float b, float c, float d) {
    if (npoly < 3 || bad) return;
    int out[MAXPOLY + 1];
    int nout = 0;
    int iprev = poly[0];
    poly[npoly] = iprev;
    float dprev = dist(pool[iprev], a, b, c, d);
    for (int i = 1; i <= npoly; ++i) {
      const int icur = poly[i];
      const float dcur = dist(pool[icur], a, b, c, d);
      if (dprev >= 0.0f) {
        if (nout >= MAXPOLY) { bad = true; return; }
        out[nout++] = iprev;
      }
      if (sgn(dcur) != sgn(dprev)) {
        if (nout >= MAXPOLY || npool >= POOL) { bad = true; return; }
        const float t = dcur < 0.0f ? swr_div(dprev, swr_sub(dprev, dcur))
                                    : swr_div(-dprev, swr_sub(dcur, dprev));
        lerp(iprev, icur, t);
        out[nout++] = npool - 1;
      }
      iprev = icur;
      dprev = dcur;
    }
    for (int i = 0; i < nout; ++i) poly[i] = out[i];
    npoly = nout;
  }
};

// facing test of VertexProcessor::cullTriangles (VertexProcessor.cpp:330-343):
// returns 0 = drop, 1 = keep, 3 = keep and swap v0 <-> v2.
__device__ __forceinline__ int cull_decision(int cull, float x0, float y0, float x1, float y1,
                                             float x2, float y2) {
  const float facing = swr_sub(swr_mul(swr_sub(x0, x1), swr_sub(y2, y1)),
                               swr_mul(swr_sub(x2, x1), swr_sub(y0, y1)));
  if (facing < 0.0f) return cull == 2 ? 0 : 1;
  return cull == 1 ? 0 : 3;
}

struct AssembleArgs {
  const SwrDrawDesc* draws;
  int ndraws;
  const uint32_t* draw_bbase;
  const float* ptv;
  float* clipv;             // clip-generated vertices (post-transform layout)
  SwrClipEntry* clip_table;
  uint32_t* clip_slot;      // per submitted primitive (valid when clipped)
  uint8_t* tri_flags;       // per submitted primitive: bit0 keep, bit1 swap, bit2 clipped
  uint2* batch_counts;      // per batch: (kept input slots, kept extra fan triangles)
  uint32_t* batch_base;     // per batch, survivors before it (points, lines; triangles: scan)
  uint4* tris;              // output primitives: v0, v1, v2 references + draw id
  uint2* lp_refs;           // per submitted point / line: endpoint references after clipping
  uint32_t* done;           // counting blocks finished (zero between launches)
  uint32_t scan;            // triangles: k_assemble_count writes batch_base (SWR_SCAN_BATCHES)
  uint32_t* draw_prim_base; // per draw: index of its first emitted primitive (optional)
  uint32_t* status;
  uint32_t cap_clip_slots, cap_clip_verts, cap_prims;
};

// SAME: the vertex records were written by this launch (k_geometry, k_front), so they are read
// with plain loads; k_assemble_count reads them through the read-only path.
template <int A, int P, bool SAME>
__device__ void assemble_one(const AssembleArgs& g, const SwrDrawDesc& D, uint32_t p, uint32_t i0,
                             uint32_t i1, uint32_t i2, uint32_t& in_kept, uint32_t& ex_kept) {
  typedef VLayout<A, P> L;
  in_kept = ex_kept = 0;
  const uint32_t gp = D.pbase + p;
  if (i0 >= D.nverts || i1 >= D.nverts || i2 >= D.nverts) {
    atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_BAD_INDEX);
    g.tri_flags[gp] = 0;
    return;
  }
  const uint32_t r[3] = {D.vbase + i0, D.vbase + i1, D.vbase + i2};
  const float* v[3] = {g.ptv + (size_t)r[0] * L::S, g.ptv + (size_t)r[1] * L::S, g.ptv + (size_t)r[2] * L::S};
  // words 4-7 of a record (16-byte aligned: S is a multiple of 4): screen x, y, z, outcode
  float4 q[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) q[k] = SAME ? *(const float4*)(v[k] + 4) : __ldg((const float4*)(v[k] + 4));
  const int m = __float_as_int(q[0].w) | __float_as_int(q[1].w) | __float_as_int(q[2].w);
  if (m == 0) {
    const int c = cull_decision(D.cull, q[0].x, q[0].y, q[1].x, q[1].y, q[2].x, q[2].y);
    g.tri_flags[gp] = (uint8_t)c;
    in_kept = c & 1;
    return;
  }
  // Clip in the reference's plane order +X, -X, +Y, -Y, +Z, -Z (VertexProcessor.cpp:237-242).
  Clipper<A, P> cp;
  for (int k = 0; k < 3; ++k) {
    cp.pool[k][0] = v[k][0]; cp.pool[k][1] = v[k][1]; cp.pool[k][2] = v[k][2]; cp.pool[k][3] = v[k][3];
    for (int i = 0; i < A; ++i) cp.pool[k][4 + i] = v[k][L::OFF_A + i];
    for (int i = 0; i < P; ++i) cp.pool[k][4 + A + i] = v[k][L::OFF_P + i];
    cp.poly[k] = k;
  }
  cp.npool = 3;
  cp.npoly = 3;
  cp.bad = false;
  if (m & 0x01) cp.clip(-1.0f, 0.0f, 0.0f, 1.0f);
  if (m & 0x02) cp.clip(1.0f, 0.0f, 0.0f, 1.0f);
  if (m & 0x04) cp.clip(0.0f, -1.0f, 0.0f, 1.0f);
  if (m & 0x08) cp.clip(0.0f, 1.0f, 0.0f, 1.0f);
  if (m & 0x10) cp.clip(0.0f, 0.0f, -1.0f, 1.0f);
  if (m & 0x20) cp.clip(0.0f, 0.0f, 1.0f, 1.0f);
  if (cp.bad) atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_CLIP_COMPLEX);
  if (cp.npoly < 3 || cp.bad) {
    g.tri_flags[gp] = 4;  // clipped away entirely
    g.clip_slot[gp] = 0xffffffffu;
    return;
  }
  // Screen positions of the polygon (generated vertices are transformed here).
  float sx[Clipper<A, P>::MAXPOLY], sy[Clipper<A, P>::MAXPOLY], sz[Clipper<A, P>::MAXPOLY];
  int nnew = 0;
  for (int k = 0; k < cp.npoly; ++k) {
    const int pi = cp.poly[k];
    if (pi < 3) {
      sx[k] = v[pi][4]; sy[k] = v[pi][5]; sz[k] = v[pi][6];
    } else {
      to_screen(D, cp.pool[pi][0], cp.pool[pi][1], cp.pool[pi][2], cp.pool[pi][3], sx[k], sy[k], sz[k]);
      nnew++;
    }
  }
  uint32_t keep = 0, swap = 0;  // bit k: fan triangle (p0, p[k+1], p[k+2])
  for (int k = 0; k + 2 < cp.npoly; ++k) {
    const int c = cull_decision(D.cull, sx[0], sy[0], sx[k + 1], sy[k + 1], sx[k + 2], sy[k + 2]);
    if (c & 1) keep |= 1u << k;
    if (c & 2) swap |= 1u << k;
  }
  // Queue places of the warp's polygons that got here together, with one atomic per word: added
  // by every polygon for itself the two words bound the kernel (1M-triangle soup, a third of it
  // clipped: 385 us, per warp 250).  nnew <= 16: its prefix over the lanes from five ballots.
  const uint32_t act = __activemask(), lt = (1u << (threadIdx.x & 31)) - 1u;
  uint32_t vpre = 0, vsum = 0;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const uint32_t m2 = __ballot_sync(act, (nnew >> k) & 1);
    vpre += (uint32_t)__popc(m2 & lt) << k;
    vsum += (uint32_t)__popc(m2) << k;
  }
  const int lead = __ffs(act) - 1;
  uint32_t slot = 0, vb = 0;
  if (!(act & lt)) {
    slot = atomicAdd(&g.status[SWR_ST_CLIP_SLOTS], (uint32_t)__popc(act));
    vb = atomicAdd(&g.status[SWR_ST_CLIP_VERTS], vsum);
  }
  slot = __shfl_sync(act, slot, lead) + (uint32_t)__popc(act & lt);
  vb = __shfl_sync(act, vb, lead) + vpre;
  if (slot >= g.cap_clip_slots || vb + nnew > g.cap_clip_verts) {
    atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_CLIP_OVERFLOW);
    g.tri_flags[gp] = 4;
    g.clip_slot[gp] = 0xffffffffu;
    return;
  }
  SwrClipEntry ent;
  int nv = 0;
  for (int k = 0; k < cp.npoly; ++k) {
    const int pi = cp.poly[k];
    if (pi < 3) {
      ent.ref[k] = r[pi];
    } else {
      const uint32_t id = vb + nv++;
      float* o = g.clipv + (size_t)id * L::S;
      o[0] = cp.pool[pi][0]; o[1] = cp.pool[pi][1]; o[2] = cp.pool[pi][2]; o[3] = cp.pool[pi][3];
      o[4] = sx[k]; o[5] = sy[k]; o[6] = sz[k]; o[7] = __int_as_float(0);
      for (int i = 0; i < A; ++i) o[L::OFF_A + i] = cp.pool[pi][4 + i];
      for (int i = 0; i < P; ++i) o[L::OFF_P + i] = cp.pool[pi][4 + A + i];
      ent.ref[k] = SWR_CLIP_REF | id;
    }
  }
  ent.n = (uint16_t)cp.npoly;
  ent.keep = (uint16_t)keep;
  ent.swap = (uint16_t)swap;
  g.clip_table[slot] = ent;
  g.clip_slot[gp] = slot;
  g.tri_flags[gp] = 4;
  in_kept = keep & 1u;
  ex_kept = __popc(keep >> 1);
}

// Triangles [p0, p0 + count) of a draw, clamped to the draw: their count.
__device__ __forceinline__ uint32_t batch_count(const SwrDrawDesc& D, uint32_t p0, uint32_t count) {
  return p0 < D.nprims ? min(count, D.nprims - p0) : 0u;
}

#define SWR_HALF (SWR_BATCH_PRIMS / 2)  // triangles per assembly CTA (half a batch)

// One CTA per half batch (512 triangles, one per thread): clip / cull and count the
// survivors: batch_counts[h] = (kept input slots, kept extra fan triangles).
template <int A, int P, bool SAME>
__device__ __forceinline__ void assemble_count_block(const AssembleArgs& g, uint32_t hb) {
  __shared__ uint32_t tmp[64];
  const uint32_t b = hb >> 1;
  const int d = g.ndraws > 1 ? swr_find_le(g.draw_bbase, g.ndraws, b) : 0;
  const SwrDrawDesc& D = g.draws[d];
  const uint32_t p0 = (b - D.bbase) * SWR_BATCH_PRIMS + (hb & 1) * SWR_HALF;
  const uint32_t n = batch_count(D, p0, SWR_HALF);
  uint32_t ik = 0, ek = 0;
  const uint32_t q = threadIdx.x;
  if (q < n) {
    const uint32_t* ix = D.indices + (size_t)3 * (p0 + q);
    assemble_one<A, P, SAME>(g, D, p0 + q, __ldg(ix), __ldg(ix + 1), __ldg(ix + 2), ik, ek);
  }
  uint32_t tin, tex;
  swr_block_sum2(ik, ek, tmp, tin, tex);
  if (threadIdx.x == 0) g.batch_counts[hb] = make_uint2(tin, tex);
}

template <int A, int P>
__global__ void __launch_bounds__(SWR_HALF) k_assemble_count(AssembleArgs g) {
  swr_pdl_entry();
  assemble_count_block<A, P, false>(g, blockIdx.x);
  if (!g.scan) return;
  uint32_t total;
  const uint32_t nb = gridDim.x / 2;
  const bool last = swr_last_block_scan(
      [&](uint32_t b) {
        const uint4 c = __ldcg((const uint4*)g.batch_counts + b);
        return c.x + c.y + c.z + c.w;
      },
      g.batch_base, nb, g.done, &total);
  if (last && threadIdx.x == 0) g.batch_base[nb] = total;
}

// Batches above which the counting launch's last block turns the counts into bases.  Up to it
// every emitting block sums the counts before it: those sums grow with the square of the
// batches, the scan costs every counting block an atomic and the launch a serial tail.  256
// meshes, 6,810 batches: emit 115 us summed, 71 scanned, for 30 us more in the counting launch
// (2861 -> 2838 us in all); 1,024 batches of a soup take the same time either way, and 320
// batches of one mesh are slower scanned (95.7 -> 97.6 us in all).
#ifndef SWR_SCAN_BATCHES
#define SWR_SCAN_BATCHES 2048
#endif

// Writes the surviving triangles of one batch at their effective-order positions.  The
// batch base is the sum of the totals of the batches before it, from the counting launch's scan
// (SCAN) or summed here; the last batch publishes the primitive count (and flags an undersized
// primitive queue).
template <int A, int P, bool SCAN>
__device__ __forceinline__ void assemble_emit_block(const AssembleArgs& g, uint32_t hb, uint32_t nhb) {
  __shared__ uint32_t tmp[64];
  __shared__ uint32_t tmps[32];
  // An overflow of the count stage (flags set by atomics, of this launch in k_geometry and
  // k_front).  One that another block of this stage found does not count: the last block
  // still has to publish the primitive count the queue must grow to.
  if (__ldcg(&g.status[SWR_ST_FLAGS]) & (SWR_F_ANY_OVERFLOW & ~SWR_F_PRIM_OVERFLOW)) return;
  const uint32_t b = hb >> 1, half = hb & 1;
  const int d = g.ndraws > 1 ? swr_find_le(g.draw_bbase, g.ndraws, b) : 0;
  const SwrDrawDesc& D = g.draws[d];
  const uint32_t p0 = (b - D.bbase) * SWR_BATCH_PRIMS + half * SWR_HALF;
  const uint32_t n = batch_count(D, p0, SWR_HALF);
  // base: the batch's first emitted primitive; dbase: the draw's (primitive-source output)
  uint32_t base, dbase;
  if (SCAN) {
    base = g.batch_base[b];
    dbase = g.batch_base[D.bbase];
  } else {
    uint32_t before = 0, dbefore = 0;
    for (uint32_t i = threadIdx.x; i < 2 * b; i += blockDim.x) {
      const uint32_t c = g.batch_counts[i].x + g.batch_counts[i].y;
      before += c;
      if (i < 2 * D.bbase) dbefore += c;
    }
    swr_block_sum2(before, dbefore, tmp, base, dbase);
  }
  const uint2 c0 = g.batch_counts[2 * b], c1 = g.batch_counts[2 * b + 1];
  const uint32_t batch_in = c0.x + c1.x, batch_total = batch_in + c0.y + c1.y;
  // primitive ids seen by the pixel shader are per draw, as with one drawElements call each
  if (g.draw_prim_base && b == D.bbase && half == 0 && threadIdx.x == 0) g.draw_prim_base[d] = base;
  // effective order within the batch: every kept input slot (first half, then second),
  // then every extra fan triangle (first half's, then second's)
  const uint32_t in_base = base + (half ? c0.x : 0u);
  const uint32_t ex_base = base + batch_in + (half ? c0.y : 0u);
  const uint32_t q = threadIdx.x;
  uint32_t fl = 0, slot = 0xffffffffu, keep = 0, i0 = 0, i1 = 0, i2 = 0;
  if (q < n) {
    const uint32_t* ix = D.indices + (size_t)3 * (p0 + q);  // read early: used after the scan
    i0 = __ldg(ix);
    i1 = __ldg(ix + 1);
    i2 = __ldg(ix + 2);
    fl = g.tri_flags[D.pbase + p0 + q];
    if (fl & 4) {
      slot = g.clip_slot[D.pbase + p0 + q];
      if (slot != 0xffffffffu) keep = g.clip_table[slot].keep;
    } else {
      keep = fl & 1;
    }
  }
  // one scan of (kept input slot, extra fan triangles) packed in 16-bit halves: at most 512
  // and 512 * 13 per half batch, so the low half never carries
  uint32_t tot;
  const uint32_t ex = swr_block_exscan((keep & 1u) | ((uint32_t)__popc(keep >> 1) << 16), tmps, &tot);
  uint32_t rin = (ex & 0xffffu) + in_base;
  uint32_t rex = (ex >> 16) + ex_base;
  if (hb == nhb - 1 && threadIdx.x == 0) {
    g.status[SWR_ST_PRIMS] = base + batch_total;
    if (base + batch_total > g.cap_prims) atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_PRIM_OVERFLOW);
  }
  if (base + batch_total > g.cap_prims) {
    if (threadIdx.x == 0) atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_PRIM_OVERFLOW);
    return;
  }
  // source triangle (draw-relative) of the primitive emitted at global position `at`
  auto record_src = [&](uint32_t at, uint32_t src) {
    if (!D.prim_src) return;
    const uint32_t k = at - dbase;
    if (k < D.prim_src_cap) D.prim_src[k] = (int32_t)src;
    else atomicOr(&g.status[SWR_ST_FLAGS], SWR_F_SRC_OVERFLOW);
  };
  if (keep) {
    if (!(fl & 4)) {
      uint32_t r0 = D.vbase + i0, r1 = D.vbase + i1, r2 = D.vbase + i2;
      if (fl & 2) { const uint32_t t = r0; r0 = r2; r2 = t; }
      record_src(rin, p0 + q);
      g.tris[rin++] = make_uint4(r0, r1, r2, (uint32_t)d);
    } else {
      // first fan triangle in the input slot, the others after all of the batch's slots
      const SwrClipEntry e = g.clip_table[slot];
      for (int k = 0; k + 2 < e.n; ++k) {
        if (!((e.keep >> k) & 1)) continue;
        uint32_t r0 = e.ref[0], r1 = e.ref[k + 1], r2 = e.ref[k + 2];
        if ((e.swap >> k) & 1) { const uint32_t t = r0; r0 = r2; r2 = t; }
        if (k == 0) {
          record_src(rin, p0 + q);
          g.tris[rin++] = make_uint4(r0, r1, r2, (uint32_t)d);
        } else {
          record_src(rex, p0 + q);
          g.tris[rex++] = make_uint4(r0, r1, r2, (uint32_t)d);
        }
      }
    }
  }
}

template <int A, int P>
__global__ void __launch_bounds__(SWR_HALF) k_assemble_emit(AssembleArgs g) {
  swr_pdl_entry();
  if (g.scan) assemble_emit_block<A, P, true>(g, blockIdx.x, gridDim.x);
  else assemble_emit_block<A, P, false>(g, blockIdx.x, gridDim.x);
}

// Grid barrier of a cooperative launch: bar[0] counts arrivals, bar[1] is the generation.
// The wait is bounded: past its limit the barrier sets SWR_F_BARRIER_TIMEOUT and returns
// false, and the caller skips the rest of its work (every CTA ends; none waits forever).
__device__ __forceinline__ bool swr_grid_sync(uint32_t* bar, uint32_t* status) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile uint32_t* gen = bar + 1;
    const uint32_t g0 = *gen;
    __threadfence();
    ok = 1;
    if (atomicAdd(bar, 1u) == gridDim.x - 1) {
      atomicExch(bar, 0u);  // reset before the release: the next barrier counts from zero
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      uint32_t spins = 0;
      while (*gen == g0) {
        if (++spins > (1u << 24)) {  // seconds of waiting: give up
          atomicOr(&status[SWR_ST_FLAGS], SWR_F_BARRIER_TIMEOUT);
          ok = 0;
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// The geometry front end of a draw or batch in one persistent cooperative launch: vertex
// shading, then assembly's count and emit over every half batch, the CTAs staying resident
// and meeting at grid barriers between the stages (512 threads, the assembly's CTA size).
template <class VS>
__global__ void __launch_bounds__(SWR_HALF) k_geometry(const SwrDrawDesc* draws, int ndraws, const uint32_t* draw_vbase,
                                                       uint32_t nverts, float* ptv, AssembleArgs g, uint32_t nhb,
                                                       uint32_t* bar) {
  swr_pdl_entry();
  vertex_stage<VS>(draws, ndraws, draw_vbase, nverts, ptv);
  if (!swr_grid_sync(bar, g.status)) return;
  for (uint32_t hb = blockIdx.x; hb < nhb; hb += gridDim.x) {
    assemble_count_block<VS::AVarCount, VS::PVarCount, true>(g, hb);
    __syncthreads();  // the block's shared scratch is reused by its next half batch
  }
  if (!swr_grid_sync(bar, g.status)) return;
  for (uint32_t hb = blockIdx.x; hb < nhb; hb += gridDim.x) {
    assemble_emit_block<VS::AVarCount, VS::PVarCount, false>(g, hb, nhb);
    __syncthreads();
  }
}

// The geometry front end of a small draw: descriptor upload, vertex shading and assembly in
// one CTA.  Such a draw is bound by its chain of dependent launches (4 us each, whatever they
// do); see small_draw in swr_capi.cu for the sizes.
struct FrontArgs {
  SwrDrawDesc draw;      // the draw's descriptors, by value; with `staged` they are in place already
  SwrTargetDesc target;
  int staged;
  SwrDrawDesc* draws;
  SwrTargetDesc* targets;
  uint32_t nverts, nhb;  // vertices, half batches
  float* ptv;
  AssembleArgs aa;
};

template <class VS>
__global__ void __launch_bounds__(SWR_HALF) k_front(const __grid_constant__ FrontArgs a) {
  swr_pdl_entry();
  AssembleArgs g = a.aa;
  if (!a.staged) {
    g.draws = &a.draw;
    const uint32_t* s = (const uint32_t*)&a.draw;
    uint32_t* d = (uint32_t*)a.draws;
    for (uint32_t i = threadIdx.x; i < sizeof(SwrDrawDesc) / 4; i += SWR_HALF) d[i] = s[i];
    s = (const uint32_t*)&a.target;
    d = (uint32_t*)a.targets;
    for (uint32_t i = threadIdx.x; i < sizeof(SwrTargetDesc) / 4; i += SWR_HALF) d[i] = s[i];
    if (threadIdx.x < 5) g.status[SWR_ST_CLIP_SLOTS + threadIdx.x] = 0u;  // the draw's working counters
    __threadfence();  // the counters are zero before this CTA's atomics reach them
  }
  vertex_stage<VS>(g.draws, 1, nullptr, a.nverts, a.ptv);
  __syncthreads();
  for (uint32_t hb = 0; hb < a.nhb; ++hb) {
    assemble_count_block<VS::AVarCount, VS::PVarCount, true>(g, hb);
    __syncthreads();  // the block's shared scratch is reused by its next half batch
  }
  for (uint32_t hb = 0; hb < a.nhb; ++hb) {
    assemble_emit_block<VS::AVarCount, VS::PVarCount, false>(g, hb, a.nhb);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------
// Triangle setup.

// Setup record layout for pixel shader PS (32-bit words).
template <class PS>
struct Rec {
  enum {
    NA = PS::AVarCount,
    NP = PS::PVarCount,
    IZ = PS::InterpolateZ ? 1 : 0,
    IW = (PS::InterpolateW || PS::PVarCount > 0) ? 1 : 0,
    NEQ = IZ + IW + NA + NP,
    EQ0 = 18,
    R = ((EQ0 + 3 * NEQ + 3) / 4) * 4,
    EQ_Z = 0,
    EQ_W = IZ,
    EQ_A = IZ + IW,
    EQ_P = IZ + IW + NA
  };
  // word 0 flags: bit0 drawable, bit1 block mode, bits2-4 tie of e0..e2, bit5 bottom half,
  //               bit6 top half
  // word 1 draw id; words 2-5 pixel bbox x0, y0, x1, y1 (inclusive, clamped to target)
  // block: words 6-14 e0.a e0.b e0.c e1.a e1.b e1.c e2.a e2.b e2.c
  // span:  words 6-11 bottom half yb0 yb1 t.x t.y is1 is2; 12-17 top half yt_hi yt_lo b.x b.y is1 is2
  // words 18.. (a, b, c) per interpolated equation: z, invw, avar[NA], pvar[NP]
};

struct Edge {
  float a, b, c;
  bool tie;
};

__device__ __forceinline__ Edge make_edge(float x0, float y0, float x1, float y1) {
  // EdgeEquation::init (EdgeEquation.h:37-43)
  Edge e;
  e.a = swr_sub(y0, y1);
  e.b = swr_sub(x1, x0);
  e.c = swr_div(-swr_add(swr_mul(e.a, swr_add(x0, x1)), swr_mul(e.b, swr_add(y0, y1))), 2.0f);
  e.tie = e.a != 0.0f ? e.a > 0.0f : e.b > 0.0f;
  return e;
}

// EdgeEquation::test (EdgeEquation.h): v > 0, or v == 0 on a tie edge.  Written as one
// comparison against a per-edge threshold: with denormals kept (no flush to zero) no float
// lies strictly between 0 and 2^-149, so v > 0 is v >= 2^-149; v == 0 (either zero) with
// the tie is v >= 0; NaN fails both, as it fails the reference's two comparisons.
__device__ __forceinline__ bool edge_test(float v, bool tie) { return v >= (tie ? 0.0f : 0x1p-149f); }

__device__ __forceinline__ void param_eq(float p0, float p1, float p2, const Edge& e0, const Edge& e1,
                                         const Edge& e2, float f, float* o) {
  // ParameterEquation::init (ParameterEquation.h:36-48)
  o[0] = swr_mul(f, swr_add(swr_add(swr_mul(p0, e0.a), swr_mul(p1, e1.a)), swr_mul(p2, e2.a)));
  o[1] = swr_mul(f, swr_add(swr_add(swr_mul(p0, e0.b), swr_mul(p1, e1.b)), swr_mul(p2, e2.b)));
  o[2] = swr_mul(f, swr_add(swr_add(swr_mul(p0, e0.c), swr_mul(p1, e1.c)), swr_mul(p2, e2.c)));
}

struct SetupArgs {
  const uint4* tris;
  const uint32_t* status;  // SWR_ST_PRIMS = primitive count
  uint32_t cap_prims;
  const float* ptv;
  const float* clipv;
  int S, off_a, off_p, vs_a, vs_p;
  const SwrDrawDesc* draws;
  const SwrTargetDesc* targets;
  float* recs;
  uint32_t* tile_count;
  int tile;  // tile edge in pixels
  uint32_t* cell_count;  // per (tile, primitive segment): bin entries (counted with atomics)
  SwrCells cells;
  int seg_shift;         // primitive segment = primitive index >> seg_shift (< SWR_SEGS)
  uint32_t* boxes;       // small draws (null otherwise): per primitive its packed tile box instead of
                         // cell counts (SWR_NO_BOX: no tile); bin entries are summed in the status
  uint32_t* status_w;    // small draws: the status words
  uint32_t grid;         // CTAs to launch (0: the default)
};

// A tile box packed in a word, 8 bits each: x0 | y0 << 8 | x1 << 16 | y1 << 24 (inclusive).
#define SWR_NO_BOX 0x000000ffu  // x0 = 255 > x1 = 0: hits no tile
__device__ __forceinline__ bool swr_box_hit(uint32_t box, uint32_t tx, uint32_t ty) {
  return tx >= (box & 255u) && tx <= ((box >> 16) & 255u) && ty >= ((box >> 8) & 255u) && ty <= (box >> 24);
}

// Whether any of a small draw's n boxes hits a tile (whole CTA): asked first, at the cost of one
// barrier, by k_overwrite and where the boxes are several windows of k_raster's.  On a large
// target nearly every tile's answer is no.  1,024 triangles of 8 px, us a draw with the windows
// gone through in every tile / this way / general route: 1920x1080 55 / 48 / 48, 3840x2160
// 125 / 79 / 74, 4080x4080 218 / 118 / 110.
__device__ __forceinline__ bool direct_any(const uint32_t* boxes, uint32_t n, uint32_t tile, uint32_t tiles_x) {
  const uint32_t tx = tile % tiles_x, ty = tile / tiles_x;
  bool hit = false;
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) hit |= swr_box_hit(boxes[i], tx, ty);
  return __syncthreads_or(hit);
}

// A warp's (primitive, tile) pairs, spread over its lanes 32 at a time and handed to
// put(owner lane, tile) in groups of four per lane, so that one large primitive does not
// serialise the warp and the pairs' memory operations are in flight together.  Every lane
// brings the tile box of its primitive: `cnt` tiles (0: none), nx a row, from (tx0, ty0), in
// a target of tiles_x tiles a row starting at tile tbase.  `put` returns nothing; it is called
// by whole warps with on = false for lanes without a pair.  Counting by serial walks
// per lane, k_setup took 104 us on the Benchmark program and 192 us on the 1M-triangle soup;
// this way 85 and 98, and with the counters segment-major (SwrCells) 37 and 81.
template <class F>
__device__ __forceinline__ void warp_tiles(int cnt, int nx, int tx0, int ty0, uint32_t tbase, int tiles_x, F put) {
  constexpr int G = 4;
  const int lane = threadIdx.x & 31;
  int inc = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  const int total = __shfl_sync(0xffffffffu, inc, 31);
  for (int base = 0; base < total; base += 32 * G) {
    int owner[G];
    uint32_t tile[G];
    bool on[G];
#pragma unroll
    for (int u = 0; u < G; ++u) {
      on[u] = false;
      if (base + u * 32 >= total) continue;  // (uniform)
      const int j = base + u * 32 + lane;
      int src = 0;  // owner: the number of lanes whose inclusive count is <= j
#pragma unroll
      for (int step = 16; step; step >>= 1) {
        const int v = __shfl_sync(0xffffffffu, inc, src + step - 1);
        if (v <= j) src += step;
      }
      src = src < 31 ? src : 31;
      const int first = __shfl_sync(0xffffffffu, inc - cnt, src);
      const int onx = __shfl_sync(0xffffffffu, nx, src);
      const int otx0 = __shfl_sync(0xffffffffu, tx0, src);
      const int oty0 = __shfl_sync(0xffffffffu, ty0, src);
      const uint32_t otb = __shfl_sync(0xffffffffu, tbase, src);
      const int otw = __shfl_sync(0xffffffffu, tiles_x, src);
      const int local = j - first;
      const int ry = local / onx;
      owner[u] = src;
      tile[u] = otb + (uint32_t)((oty0 + ry) * otw + otx0 + (local - ry * onx));
      on[u] = j < total;
    }
    put(owner, tile, on);
  }
}

struct SpanHalf {
  float ox, oy, is1, is2;
  int y0, y1;  // bottom: rows [y0, y1); top: rows (y1, y0]
};

// x extent (xl of the first pixel, xr exclusive) of row y of a span half.
__device__ __forceinline__ void span_row(const SpanHalf& h, int y, int minx, int maxx, int& xl, int& xr) {
  const float dy = swr_add(swr_sub((float)y, h.oy), 0.5f);
  const float c1 = swr_add(swr_add(h.ox, swr_mul(h.is1, dy)), 0.5f);
  const float c2 = swr_add(swr_add(h.ox, swr_mul(h.is2, dy)), 0.5f);
  xl = swr_maxi(minx, swr_trunc_int(c1));
  xr = swr_mini(maxx, swr_trunc_int(c2));
}

// Records are assembled in shared memory and written out as contiguous float4 runs
// (one record per thread would be a 4-byte store per 160-byte stride).
constexpr int kSetupThreads = 128;

template <class PS>
__global__ void __launch_bounds__(kSetupThreads) k_setup(SetupArgs g) {
  swr_pdl_entry();
  typedef Rec<PS> RL;
  // records staged with an odd stride, so the threads' scalar stores of one field fall in
  // 32 different banks (a stride of R = 40 words put 32 threads in 4 banks)
  constexpr int RS = RL::R + 1;
  __shared__ float stage[kSetupThreads * RS];
  // a small draw's queue requests are final here (bin entries are no queue of it)
  if (g.boxes && blockIdx.x == 0 && threadIdx.x == 0) swr_close_status(g.status_w);
  if (g.status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  uint32_t np = g.status[SWR_ST_PRIMS];
  if (np > g.cap_prims) np = g.cap_prims;
  for (uint32_t p0 = blockIdx.x * kSetupThreads; p0 < np; p0 += gridDim.x * kSetupThreads) {
  const uint32_t p = p0 + threadIdx.x;
  int cnt = 0, tnx = 1, tx0 = 0, ty0 = 0, tiles_x = 0;  // the primitive's tiles
  uint32_t tbase = 0;
  if (p < np) {
    const uint4 t = g.tris[p];
    const SwrDrawDesc& D = g.draws[t.w];
    const SwrTargetDesc& T = g.targets[D.target];
    const uint32_t rr[3] = {t.x, t.y, t.z};
    float x[3], y[3], z[3], w[3];
    float av[3][RL::NA > 0 ? RL::NA : 1], pv[3][RL::NP > 0 ? RL::NP : 1];
    // Post-transform records (16-byte aligned): words 0-3 clip position, 4-6 screen x, y, z,
    // then the vertex shader's avars and pvars.  Records of at most 16 words with the avars
    // at word 8 and 0 or 3 of them (every built-in vertex shader) are read as float4s;
    // scattered scalar reads of 9 words per vertex made the stage L1-wavefront bound.
    const bool vec = g.S <= 16 && g.off_a == 8 && g.off_p == 8 + g.vs_a && (g.vs_a == 0 || g.vs_a == 3);
    for (int k = 0; k < 3; ++k) {
      const float* vp = (rr[k] & SWR_CLIP_REF) ? g.clipv + (size_t)(rr[k] & ~SWR_CLIP_REF) * g.S
                                               : g.ptv + (size_t)rr[k] * g.S;
      if (vec) {
        const float4 q0 = __ldg((const float4*)vp), q1 = __ldg((const float4*)vp + 1);
        const float4 q2 = g.S > 8 ? __ldg((const float4*)vp + 2) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float4 q3 = g.S > 12 ? __ldg((const float4*)vp + 3) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float at[8] = {q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z, q3.w};
        w[k] = q0.w;
        x[k] = q1.x; y[k] = q1.y; z[k] = q1.z;
#pragma unroll
        for (int i = 0; i < RL::NA; ++i) av[k][i] = i < g.vs_a ? at[i] : 0.0f;
#pragma unroll
        for (int i = 0; i < RL::NP; ++i) pv[k][i] = i < g.vs_p ? (g.vs_a ? at[(3 + i) & 7] : at[i]) : 0.0f;
      } else {
        x[k] = vp[4]; y[k] = vp[5]; z[k] = vp[6]; w[k] = vp[3];
        for (int i = 0; i < RL::NA; ++i) av[k][i] = i < g.vs_a ? vp[g.off_a + i] : 0.0f;
        for (int i = 0; i < RL::NP; ++i) pv[k][i] = i < g.vs_p ? vp[g.off_p + i] : 0.0f;
      }
    }
    float* rec = stage + threadIdx.x * RS;
    uint32_t tiles = 0, box = SWR_NO_BOX;
    // TriangleEquations: e0 = (v1, v2), e1 = (v2, v0), e2 = (v0, v1)
    const Edge e0 = make_edge(x[1], y[1], x[2], y[2]);
    const Edge e1 = make_edge(x[2], y[2], x[0], y[0]);
    const Edge e2 = make_edge(x[0], y[0], x[1], y[1]);
    const float area2 = swr_add(swr_add(e0.c, e1.c), e2.c);
    int flags = 0;
    int bx0 = 0, by0 = 0, bx1 = -1, by1 = -1;
    if (!(area2 <= 0.0f)) {
      flags = 1 | (e0.tie ? 4 : 0) | (e1.tie ? 8 : 0) | (e2.tie ? 16 : 0);
      const float factor = swr_div(1.0f, area2);
      float* eq = rec + RL::EQ0;
      if (RL::IZ) param_eq(z[0], z[1], z[2], e0, e1, e2, factor, eq + 3 * RL::EQ_Z);
      const float iw0 = swr_div(1.0f, w[0]), iw1 = swr_div(1.0f, w[1]), iw2 = swr_div(1.0f, w[2]);
      if (RL::IW) param_eq(iw0, iw1, iw2, e0, e1, e2, factor, eq + 3 * RL::EQ_W);
      for (int i = 0; i < RL::NA; ++i) param_eq(av[0][i], av[1][i], av[2][i], e0, e1, e2, factor, eq + 3 * (RL::EQ_A + i));
      for (int i = 0; i < RL::NP; ++i)
        param_eq(swr_mul(pv[0][i], iw0), swr_mul(pv[1][i], iw1), swr_mul(pv[2][i], iw2), e0, e1, e2, factor,
                 eq + 3 * (RL::EQ_P + i));
      // Raster mode (Rasterizer.h:414-446); Adaptive compares the float ratio as double.
      bool block = D.raster_mode == 1;
      if (D.raster_mode == 2) {
        const float fx0 = swr_minf(swr_minf(x[0], x[1]), x[2]), fx1 = swr_maxf(swr_maxf(x[0], x[1]), x[2]);
        const float fy0 = swr_minf(swr_minf(y[0], y[1]), y[2]), fy1 = swr_maxf(swr_maxf(y[0], y[1]), y[2]);
        const float orient = swr_div(swr_sub(fx1, fx0), swr_sub(fy1, fy0));
        block = (double)orient > 0.4 && (double)orient < 1.6;
      }
      if (block) {
        flags |= 2;
        // Rasterizer.h:235-255
        int mnx = swr_trunc_int(swr_minf(swr_minf(x[0], x[1]), x[2]));
        int mxx = swr_trunc_int(swr_maxf(swr_maxf(x[0], x[1]), x[2]));
        int mny = swr_trunc_int(swr_minf(swr_minf(y[0], y[1]), y[2]));
        int mxy = swr_trunc_int(swr_maxf(swr_maxf(y[0], y[1]), y[2]));
        mnx = swr_maxi(mnx, D.sc_minx);
        mxx = swr_mini(mxx, D.sc_maxx);
        mny = swr_maxi(mny, D.sc_miny);
        mxy = swr_mini(mxy, D.sc_maxy);
        mnx &= ~(SWR_BLOCK - 1);
        mxx &= ~(SWR_BLOCK - 1);
        mny &= ~(SWR_BLOCK - 1);
        mxy &= ~(SWR_BLOCK - 1);
        const int sx = (mxx - mnx) / SWR_BLOCK + 1, sy = (mxy - mny) / SWR_BLOCK + 1;
        // Blocks visited by i in [0, sx*sy): (mnx + (i % sx) * 8, mny + (i / sx) * 8).
        if (sx > 0 && sy > 0) {
          bx0 = mnx; bx1 = mnx + SWR_BLOCK * (sx - 1) + SWR_BLOCK - 1;
          by0 = mny; by1 = mny + SWR_BLOCK * (sy - 1) + SWR_BLOCK - 1;
        } else if (sx < 0 && sy < 0) {
          bx0 = mnx; bx1 = mnx + SWR_BLOCK * (-sx - 1) + SWR_BLOCK - 1;
          by0 = mny - SWR_BLOCK * (-sy - 1); by1 = mny + SWR_BLOCK - 1;
        }
        rec[6] = e0.a; rec[7] = e0.b; rec[8] = e0.c;
        rec[9] = e1.a; rec[10] = e1.b; rec[11] = e1.c;
        rec[12] = e2.a; rec[13] = e2.b; rec[14] = e2.c;
      } else {
        // Rasterizer.h:318-357
        int it = 0, im = 1, ib = 2;
        if (y[it] > y[im]) { const int q = it; it = im; im = q; }
        if (y[im] > y[ib]) { const int q = im; im = ib; ib = q; }
        if (y[it] > y[im]) { const int q = it; it = im; im = q; }
        const float dy = swr_sub(y[ib], y[it]);
        const float iy = swr_sub(y[im], y[it]);
        SpanHalf bot, top;
        bool has_bot = false, has_top = false;
        float lx, ly, rx, ry;
        if (y[im] == y[it]) {
          lx = x[im]; ly = y[im]; rx = x[it]; ry = y[it];
          if (lx > rx) { float q = lx; lx = rx; rx = q; q = ly; ly = ry; ry = q; }
          has_top = true;
        } else if (y[im] == y[ib]) {
          lx = x[im]; ly = y[im]; rx = x[ib]; ry = y[ib];
          if (lx > rx) { float q = lx; lx = rx; rx = q; q = ly; ly = ry; ry = q; }
          has_bot = true;
        } else {
          const float v4x = swr_add(x[it], swr_mul(swr_div(swr_sub(x[ib], x[it]), dy), iy));
          lx = x[im]; ly = y[im]; rx = v4x; ry = y[im];
          if (lx > rx) { float q = lx; lx = rx; rx = q; q = ly; ly = ry; ry = q; }
          has_bot = has_top = true;
        }
        if (has_bot) {  // drawBottomFlatTriangle(t, l, r) (Rasterizer.h:361-385)
          bot.ox = x[it]; bot.oy = y[it];
          bot.is1 = swr_div(swr_sub(lx, x[it]), swr_sub(ly, y[it]));
          bot.is2 = swr_div(swr_sub(rx, x[it]), swr_sub(ry, y[it]));
          bot.y0 = swr_trunc_int(swr_add(y[it], 0.5f));
          bot.y1 = swr_trunc_int(swr_add(ly, 0.5f));
        } else {
          bot.ox = bot.oy = bot.is1 = bot.is2 = 0.0f;
          bot.y0 = bot.y1 = 0;
        }
        if (has_top) {  // drawTopFlatTriangle(l, r, b) (Rasterizer.h:388-411)
          top.ox = x[ib]; top.oy = y[ib];
          top.is1 = swr_div(swr_sub(x[ib], lx), swr_sub(y[ib], ly));
          top.is2 = swr_div(swr_sub(x[ib], rx), swr_sub(y[ib], ry));
          top.y0 = swr_trunc_int(swr_sub(y[ib], 0.5f));
          top.y1 = swr_trunc_int(swr_sub(ly, 0.5f));
        } else {
          top.ox = top.oy = top.is1 = top.is2 = 0.0f;
          top.y0 = top.y1 = 0;
        }
        if (has_bot) flags |= 32;
        if (has_top) flags |= 64;
        rec[6] = __int_as_float(bot.y0); rec[7] = __int_as_float(bot.y1);
        rec[8] = bot.ox; rec[9] = bot.oy; rec[10] = bot.is1; rec[11] = bot.is2;
        rec[12] = __int_as_float(top.y0); rec[13] = __int_as_float(top.y1);
        rec[14] = top.ox; rec[15] = top.oy; rec[16] = top.is1; rec[17] = top.is2;
        // Conservative pixel box: rows inside the target, x from the end rows of each
        // half (the span edges are linear in y up to rounding, hence the 2 px margin).
        int rx0 = 0x7fffffff, rx1 = -0x7fffffff, ry0 = 0x7fffffff, ry1 = -0x7fffffff;
        for (int hh = 0; hh < 2; ++hh) {
          const SpanHalf& h = hh ? top : bot;
          if (!(hh ? has_top : has_bot)) continue;
          int lo = hh ? h.y1 + 1 : h.y0, hi = hh ? h.y0 : h.y1 - 1;
          lo = swr_maxi(lo, 0);
          hi = swr_mini(hi, T.height - 1);
          if (lo > hi) continue;
          ry0 = swr_mini(ry0, lo);
          ry1 = swr_maxi(ry1, hi);
          for (int e = 0; e < 2; ++e) {
            int xl, xr;
            span_row(h, e ? hi : lo, D.sc_minx, D.sc_maxx, xl, xr);
            rx0 = swr_mini(rx0, xl);
            rx1 = swr_maxi(rx1, xr - 1);
          }
        }
        if (ry0 <= ry1) {
          bx0 = swr_maxi(rx0 - 2, D.sc_minx);
          bx1 = swr_mini(rx1 + 2, D.sc_maxx - 1);
          by0 = ry0;
          by1 = ry1;
        }
      }
      bx0 = swr_maxi(bx0, 0);
      by0 = swr_maxi(by0, 0);
      bx1 = swr_mini(bx1, T.width - 1);
      by1 = swr_mini(by1, T.height - 1);
      if (bx0 <= bx1 && by0 <= by1) {
        const int tshift = __ffs(g.tile) - 1;  // tiles are 16 or 32 pixels; the box is >= 0
        tx0 = bx0 >> tshift;
        ty0 = by0 >> tshift;
        const int tx1 = bx1 >> tshift, ty1 = by1 >> tshift;
        tnx = tx1 - tx0 + 1;
        cnt = tnx * (ty1 - ty0 + 1);
        tiles = (uint32_t)cnt;
        box = (uint32_t)tx0 | (uint32_t)ty0 << 8 | (uint32_t)tx1 << 16 | (uint32_t)ty1 << 24;
        tbase = T.tile_base;
        tiles_x = T.tiles_x;
      } else {
        flags = 0;
      }
    }
    rec[0] = __int_as_float(flags);
    rec[1] = __int_as_float((int)t.w);
    rec[2] = __int_as_float(bx0); rec[3] = __int_as_float(by0);
    rec[4] = __int_as_float(bx1); rec[5] = __int_as_float(by1);
    if (g.boxes) {
      g.boxes[p] = box;
      if (tiles) atomicAdd(&g.status_w[SWR_ST_PAIRS], tiles);
    } else {
      g.tile_count[p] = flags ? tiles : 0u;
    }
  }
  if (g.cell_count) {
    if (__reduce_max_sync(0xffffffffu, (uint32_t)cnt) <= 2u) {  // small primitives: every lane its own tiles
      const uint32_t seg = p >> g.seg_shift;
      for (int i = 0; i < cnt; ++i) {
        const int tx = tx0 + (i < tnx ? i : i - tnx), ty = ty0 + (i < tnx ? 0 : 1);
        atomicAdd(&g.cell_count[g.cells.at(tbase + (uint32_t)(ty * tiles_x + tx), seg)], 1u);
      }
    } else {
      const uint32_t pw = p0 + (threadIdx.x & ~31u);
      warp_tiles(cnt, tnx, tx0, ty0, tbase, tiles_x, [&](const int (&owner)[4], const uint32_t (&tile)[4], const bool (&on)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (on[u]) atomicAdd(&g.cell_count[g.cells.at(tile[u], (pw + (uint32_t)owner[u]) >> g.seg_shift)], 1u);
      });
    }
  }
  __syncthreads();
  const uint32_t nrec = min((uint32_t)kSetupThreads, np - p0);
  float4* dst = (float4*)(g.recs + (size_t)p0 * RL::R);
  for (uint32_t i = threadIdx.x; i < nrec * (RL::R / 4); i += kSetupThreads) {
    const uint32_t t = i / (RL::R / 4);
    const float* src = stage + t * RS + (i - t * (RL::R / 4)) * 4;
    dst[i] = make_float4(src[0], src[1], src[2], src[3]);
  }
  __syncthreads();
  }
}

// (tile, primitive) pairs in primitive order.
template <class PS>
__global__ void __launch_bounds__(256) k_emit_pairs(const uint32_t* status, uint32_t cap_prims, const float* recs,
                                                    const uint32_t* tile_count, const uint32_t* pair_off,
                                                    const uint32_t* npairs, uint32_t cap_pairs,
                                                    const SwrDrawDesc* draws, const SwrTargetDesc* targets,
                                                    int tile, uint32_t* keys, uint32_t* vals,
                                                    uint32_t* status_w) {
  swr_pdl_entry();
  typedef Rec<PS> RL;
  if (status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  if (*npairs > cap_pairs) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      atomicOr(&status_w[SWR_ST_FLAGS], SWR_F_PAIR_OVERFLOW);
      status_w[SWR_ST_PAIRS] = *npairs;
    }
    return;
  }
  uint32_t np = status[SWR_ST_PRIMS];
  if (np > cap_prims) np = cap_prims;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
    if (!tile_count[p]) continue;
    const float* rec = recs + (size_t)p * RL::R;
    const int d = __float_as_int(rec[1]);
    const SwrTargetDesc& T = targets[draws[d].target];
    const int tx0 = __float_as_int(rec[2]) / tile, ty0 = __float_as_int(rec[3]) / tile;
    const int tx1 = __float_as_int(rec[4]) / tile, ty1 = __float_as_int(rec[5]) / tile;
    uint32_t o = pair_off[p];
    for (int ty = ty0; ty <= ty1; ++ty)
      for (int tx = tx0; tx <= tx1; ++tx) {
        keys[o] = T.tile_base + (uint32_t)(ty * T.tiles_x + tx);
        vals[o] = p;
        o++;
      }
  }
}

// Segmented binning.  The primitive list is cut into SWR_SEGS contiguous segments; a
// (tile, segment) cell holds the segment's primitives that touch the tile.  Cells are laid
// out tile-major, so a tile's bin is one contiguous range ordered by segment; inside a cell
// the fill order is arbitrary; k_raster (or k_sort_tiles ahead of it, for tiles it cannot
// order itself) restores increasing primitive order.
#ifndef SWR_FILL_TILES
#define SWR_FILL_TILES 512
#endif
template <class PS>
__global__ void __launch_bounds__(256) k_fill_bins(const uint32_t* status, uint32_t cap_prims, const float* recs,
                                                   uint32_t* cell_count, const uint32_t* fill_start,
                                                   const uint32_t* pairs, uint32_t ncells, SwrCells cells, int seg_shift,
                                                   uint32_t cap_pairs, const SwrDrawDesc* draws,
                                                   const SwrTargetDesc* targets, int tile, uint32_t* bin,
                                                   uint32_t* status_w) {
  swr_pdl_entry();
  typedef Rec<PS> RL;
  // cell_count is all zero between draws: every entry counted by k_setup is taken back
  // here, and a draw that stops early zeroes the counts instead
  const uint32_t total = *pairs;
  const bool overflow = status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW;
  if (overflow || total > cap_pairs) {
    if (!overflow && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&status_w[SWR_ST_FLAGS], SWR_F_PAIR_OVERFLOW);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ncells; i += gridDim.x * blockDim.x) cell_count[i] = 0u;
    return;
  }
  uint32_t np = status[SWR_ST_PRIMS];
  if (np > cap_prims) np = cap_prims;
  // draw 0's target, read up front: every primitive of a single-draw submission uses it
  const SwrTargetDesc& T0 = targets[draws[0].target];
  const uint32_t tb0 = T0.tile_base;
  const int tw0 = T0.tiles_x;
  const int tshift = __ffs(tile) - 1;  // tiles are 16 or 32 pixels; pixel boxes are >= 0
  const int lane = threadIdx.x & 31;
  // One warp per `per` consecutive primitives (the loop is uniform per warp): 32, or as many as
  // SWR_FILL_TILES entries belong to.  A warp works through its entries 128 at a time, each a
  // chain of an atomic and a store, so few primitives of many tiles have to spread over warps:
  // 40,960 triangles of 94 tiles took 87 us as 1,280 warps of 32, and take 45 as 10,240 of 4
  // (256 or 1,024 entries a warp: 1 % of the draw slower).
  uint32_t per = 32;
  while (per > 1 && (uint64_t)total * per > (uint64_t)np * SWR_FILL_TILES) per >>= 1;
  const uint32_t stride = gridDim.x * (blockDim.x >> 5) * per;
  for (uint32_t p0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per; p0 < np; p0 += stride) {
    const uint32_t p = (uint32_t)lane < per ? p0 + (uint32_t)lane : 0xffffffffu;
    // record words 0-5: flags (0: no tile, as tile_count), draw, pixel box (two float4
    // reads of the 16-byte aligned record)
    int tx0 = 0, ty0 = 0, nx = 1, cnt = 0;
    uint32_t tbase = tb0;
    int tiles_x = tw0;
    if (p < np) {
      const float4 q0 = __ldg((const float4*)(recs + (size_t)p * RL::R));
      const float4 q1 = __ldg((const float4*)(recs + (size_t)p * RL::R) + 1);
      if (__float_as_int(q0.x)) {
        const int d = __float_as_int(q0.y);
        if (d != 0) {
          const SwrTargetDesc& T = targets[draws[d].target];
          tbase = T.tile_base;
          tiles_x = T.tiles_x;
        }
        tx0 = __float_as_int(q0.z) >> tshift;
        ty0 = __float_as_int(q0.w) >> tshift;
        nx = (__float_as_int(q1.x) >> tshift) - tx0 + 1;
        cnt = nx * ((__float_as_int(q1.y) >> tshift) - ty0 + 1);
      }
    }
    const uint32_t seg = p >> seg_shift;
    auto put = [&](uint32_t prim, uint32_t pseg, uint32_t tb, int tw, int tx, int ty) {
      const uint32_t cell = cells.at(tb + (uint32_t)(ty * tw + tx), pseg);
      const uint32_t pos = atomicSub(&cell_count[cell], 1u) - 1u;
      bin[fill_start[cell] + pos] = prim;
    };
    if (__reduce_max_sync(0xffffffffu, (uint32_t)cnt) <= 2u) {
      // small primitives (the common case): every lane its own tiles
      for (int i = 0; i < cnt; ++i) put(p, seg, tbase, tiles_x, tx0 + (i < nx ? i : i - nx), ty0 + (i < nx ? 0 : 1));
      continue;
    }
    warp_tiles(cnt, nx, tx0, ty0, tbase, tiles_x, [&](const int (&owner)[4], const uint32_t (&tile)[4], const bool (&on)[4]) {
      uint32_t at[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t cell = cells.at(tile[u], (p0 + (uint32_t)owner[u]) >> seg_shift);
        if (on[u]) at[u] = fill_start[cell] + atomicSub(&cell_count[cell], 1u) - 1u;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (on[u]) bin[at[u]] = p0 + (uint32_t)owner[u];
    });
  }
}

// Orders the cells of the listed tiles (ids in `in`, increasing within a cell in `out`): one
// CTA per tile, its cells dealt to the CTA's warps.  Cells of up to 32 ids are ranked by
// shuffles; larger ones through a bitmap of the segment's id range [seg << shift, (seg + 1) <<
// shift) in the warp's slice of shared memory (bm_words words; only those between the cell's
// smallest and largest id are touched): set one bit per id, prefix-count the words across the
// lanes, write the set bits out in order.  A range that does not fit the bitmap (queues of more
// than 32M ids) is gone through in windows of what does, unless ranking 32 ids at a time takes
// less (the windows' words cost their number, ranks the square of the ids): 100,000 lines of 300
// steps over each other, 30M fragments, took 28 s a draw with every such cell ranked, 75 ms so.  Cells of
// at most cell_min ids in tiles of at most all_min are left alone.
static __global__ void __launch_bounds__(256) k_sort_tiles(const uint32_t* status, const SwrTiles tiles, int seg_shift,
                                                           uint32_t bm_words, uint32_t cell_min, uint32_t all_min,
                                                           const uint32_t* in, uint32_t* out) {
  swr_pdl_entry();
  extern __shared__ uint32_t smem_bm[];
  if (status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  uint32_t* bm = smem_bm + (size_t)wib * bm_words;
  const uint32_t R = 1u << seg_shift;
  const uint32_t nsort = min(tiles.counts[3], tiles.ntiles);
  for (uint32_t i = blockIdx.x; i < nsort; i += gridDim.x) {
    const uint4 entry = tiles.sort[i];
    const uint32_t* cells = tiles.start + (size_t)entry.x * SWR_SEGS;
    for (uint32_t c = wib; c < SWR_SEGS; c += nwarps) {  // (uniform per warp, like all below)
      const uint32_t s = cells[c], e = c + 1 < SWR_SEGS ? cells[c + 1] : entry.z;
      const uint32_t m = e > s ? e - s : 0u;
      if (m == 0 || (m <= cell_min && entry.z - entry.y <= all_min)) continue;
      auto rank = [&]() {
        for (uint32_t i0 = 0; i0 < m; i0 += 32) {
          const uint32_t val = i0 + lane < m ? in[s + i0 + lane] : 0xffffffffu;
          uint32_t rank = 0;
          for (uint32_t j0 = 0; j0 < m; j0 += 32) {
            const uint32_t w = j0 + lane < m ? in[s + j0 + lane] : 0xffffffffu;
#pragma unroll 8
            for (int l = 0; l < 32; ++l) rank += __shfl_sync(0xffffffffu, w, l) < val;
          }
          if (i0 + lane < m) out[s + rank] = val;
        }
      };
      if (m <= 32) {
        rank();
        continue;
      }
      const uint32_t lo_id = c << seg_shift;
      uint32_t lo = 0xffffffffu, hi = 0u;
      for (uint32_t j = lane; j < m; j += 32) {
        const uint32_t v = in[s + j] - lo_id;
        if (v < R) {
          lo = min(lo, v);
          hi = max(hi, v);
        }
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      if (lo > hi) continue;
      const uint32_t last = hi >> 5;
      if (R / 32 > bm_words && (uint64_t)m * m <= 4ull * (last - (lo >> 5) + 1)) {
        rank();
        continue;
      }
      uint32_t base = 0;  // ids written by the windows before
      for (uint32_t w0 = lo >> 5; w0 <= last; w0 += bm_words) {  // (once, where the range fits)
        const uint32_t nw = min(bm_words, last - w0 + 1);
        for (uint32_t w = lane; w < nw; w += 32) bm[w] = 0u;
        __syncwarp();
#pragma unroll 4
        for (uint32_t j = lane; j < m; j += 32) {
          const uint32_t v = in[s + j] - lo_id, w = (v >> 5) - w0;
          if (v < R && w < nw) atomicOr(&bm[w], 1u << (v & 31));
        }
        __syncwarp();
        const uint32_t per = (nw + 31) / 32;  // lane l owns words [l * per, (l + 1) * per) of the window
        const uint32_t a = min(nw, (uint32_t)lane * per), b = min(nw, a + per);
        uint32_t cnt = 0;
        for (uint32_t w = a; w < b; ++w) cnt += __popc(bm[w]);
        uint32_t inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += y;
        }
        uint32_t pos = base + inc - cnt;
        base += __shfl_sync(0xffffffffu, inc, 31);
        for (uint32_t w = a; w < b; ++w) {
          uint32_t bits = bm[w];
          while (bits) {
            const int bit = __ffs(bits) - 1;
            bits &= bits - 1u;
            if (pos < m) out[s + pos] = lo_id + ((w0 + w) << 5) + (uint32_t)bit;
            ++pos;
          }
        }
        __syncwarp();
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// Tile rasterization.

template <class PS>
struct GpuPixel {  // PixelData (PixelData.h:35-146) as seen by drawPixel
  int x, y;
  float z, w, invw;
  float avar[PS::AVarCount > 0 ? PS::AVarCount : 1];
  float pvar[PS::PVarCount > 0 ? PS::PVarCount : 1];
  const float* eq;  // the triangle's parameter equations (PixelData::equations); null for points and lines
};

// PixelData::computePerspectiveDerivatives(*equations, i, ddx, ddy) for the pixel shaders
// (found by argument-dependent lookup from swr_programs.h).
template <class PS>
__device__ __forceinline__ void swr_persp_deriv(const GpuPixel<PS>& p, int i, float& ddx, float& ddy) {
  if (!p.eq) {
    ddx = ddy = 0.0f;
    return;
  }
  typedef Rec<PS> RL;
  swr_persp_deriv_eq(p.eq + 3 * (RL::EQ_P + i), p.eq + 3 * RL::EQ_W, p.x, p.y, ddx, ddy);
}

struct RasterArgs {
  const uint32_t* status;
  SwrTiles tiles;              // the tiles to rasterize, their bins and cells (k_cells); or, with
                               // tiles.list null, all of them:
  const uint32_t* tile_start;  // bin start of tile t at tile_start[t] (plus the end)
  const uint32_t* bin;         // primitive ids, each tile's range in increasing order
  const uint32_t* bin_raw;     // optional: the unsorted ids (cells); tiles of <= SWR_RASTER_SORT
                               // entries order them in the kernel, and have no range in `bin`
  const float* recs;
  const SwrDrawDesc* draws;
  const SwrTargetDesc* targets;
  const uint32_t* draw_prim_base;    // per draw first primitive (null: a single draw from 0)
  uint32_t* status_w;
  uint32_t ntiles;
  int slices;                        // k_overwrite: CTAs per tile of more than SWR_RASTER_SORT entries
                                     // (1: no slicing), each over a slice of its bin
  uint32_t* best;                    // their pixels' winners, primitive id + 1, [tile][TILE * TILE]
  uint32_t* best_done;               // per tile: the slices finished (both zero between draws)
  int has_span;                      // some draw rasterizes in Span or Adaptive mode (selects k_raster<..., true>)
  int has_block;                     // some draw rasterizes in Block or Adaptive mode
  // Quadrant CTAs (quad; 16-px tiles): a heavy tile -- more than three chunks of bin entries;
  // k_cells lists up to tiles.heavy_cap of them -- is rasterized by four CTAs, one per 8 x 8
  // quadrant, each walking the whole bin for its own pixels, so the slowest tiles no longer
  // set the kernel's length.  CTAs [0, 4 heavy_cap) take the listed tiles' quadrants; CTA
  // 4 heavy_cap + i takes entry i of the list of the others.  With quad_all every tile is split
  // (CTA 4 i + q: quadrant q of entry i): an 8-px raster tile over 16-px bins.
  int quad;
  int quad_all;
  // Sliced heavy tiles (depth-min shaders, SwrDepthMin): with dslice set, each tile of
  // tiles.heavy is rasterized by SWR_DSLICES CTAs instead, each over a run of whole chunks of
  // its ordered bin and from the draw's starting State; each writes its States to
  // dslice_state, and the last of the tile's CTAs to finish merges them in bin order
  // (swr_depth_merge) and stores.  CTAs [0, SWR_DSLICES heavy_cap) take the listed tiles'
  // slices; CTA SWR_DSLICES heavy_cap + i takes entry i of the list of the others.
  int dslice;
  // Small draws (k_raster<..., true>): no bins; every CTA picks its tile's primitives, in order,
  // from the packed tile boxes of all `status[SWR_ST_PRIMS]` primitives.
  const uint32_t* boxes;
  uint32_t cap_prims;
  void* dslice_state;      // [slot][slice][TILE * TILE] PS::State
  uint32_t* dslice_done;   // per slot: the slices finished (zero between draws)
};

// v <- fl(v + a) repeated k times for 0 <= k <= 7 (steps inside one 8x8 block), as
// predicated adds so the lanes of a warp never diverge.
__device__ __forceinline__ float fold7(float v, float a, int k) {
#pragma unroll
  for (int i = 0; i < 7; ++i) v = i < k ? swr_add(v, a) : v;
  return v;
}

// Block classification of Rasterizer.h:263-304 for the block at (bx, by): 0 = skipped,
// 1 = drawBlock<false> (every pixel), 2 = drawBlock<true> (per-pixel edge tests).
__device__ __forceinline__ int block_class(const float* r, int flags, int bx, int by) {
  const float fx = swr_add((float)bx, 0.5f), fy = swr_add((float)by, 0.5f);
  const float s = (float)(SWR_BLOCK - 1);
  bool t00[3], t01[3], t10[3], t11[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const float ea = r[6 + 3 * j], eb = r[7 + 3 * j], ec = r[8 + 3 * j];
    const bool tie = (flags >> (2 + j)) & 1;
    const float ev = swr_eval(ea, eb, ec, fx, fy);
    const float v01 = swr_add(ev, swr_mul(eb, s));
    const float v10 = swr_add(ev, swr_mul(ea, s));
    const float v11 = swr_add(v01, swr_mul(ea, s));
    t00[j] = edge_test(ev, tie);
    t01[j] = edge_test(v01, tie);
    t10[j] = edge_test(v10, tie);
    t11[j] = edge_test(v11, tie);
  }
  const int inside = (t00[0] && t00[1] && t00[2]) + (t01[0] && t01[1] && t01[2]) +
                     (t10[0] && t10[1] && t10[2]) + (t11[0] && t11[1] && t11[2]);
  if (inside == 4) return 1;
  if (inside == 0) {
    const bool s00 = (t00[0] == t00[1]) == t00[2], s01 = (t01[0] == t01[1]) == t01[2];
    const bool s10 = (t10[0] == t10[1]) == t10[2], s11 = (t11[0] == t11[1]) == t11[2];
    if (s00 && s01 && s10 && s11) return 0;
  }
  return 2;
}

// Four rows, 4 * half to 4 * half + 3, of drawBlock<true> (PixelShaderBase.h:64-93): the row
// start is the block corner's edge value stepped row by row by b (eo.stepY), pixels step by a
// (ei.stepX).  Returns the rows' coverage bits, 8 per row.  Four rows a lane: their starts
// follow from each other (a row of its own costs a lane 21 predicated steps to reach it),
// and a chunk's partial blocks still fill the CTA.
__device__ __forceinline__ uint32_t block_rows_bits(const float* r, int flags, int bx, int by, int half) {
  const float fx = swr_add((float)bx, 0.5f), fy = swr_add((float)by, 0.5f);
  const float t0 = (flags & 4) ? 0.0f : 0x1p-149f, t1 = (flags & 8) ? 0.0f : 0x1p-149f;
  const float t2 = (flags & 16) ? 0.0f : 0x1p-149f;  // thresholds of edge_test
  const float a0 = r[6], b0 = r[7], a1 = r[9], b1 = r[10], a2 = r[12], b2 = r[13];
  float i0 = swr_eval(a0, b0, r[8], fx, fy), i1 = swr_eval(a1, b1, r[11], fx, fy), i2 = swr_eval(a2, b2, r[14], fx, fy);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    i0 = half ? swr_add(i0, b0) : i0;
    i1 = half ? swr_add(i1, b1) : i1;
    i2 = half ? swr_add(i2, b2) : i2;
  }
  uint32_t m = 0;
#pragma unroll
  for (int row = 0; row < 4; ++row) {
    float c0 = i0, c1 = i1, c2 = i2;
#pragma unroll
    for (int col = 0; col < SWR_BLOCK; ++col) {
      if (c0 >= t0 && c1 >= t1 && c2 >= t2) m |= 1u << (row * 8 + col);
      c0 = swr_add(c0, a0);
      c1 = swr_add(c1, a1);
      c2 = swr_add(c2, a2);
    }
    i0 = swr_add(i0, b0);
    i1 = swr_add(i1, b1);
    i2 = swr_add(i2, b2);
  }
  return m;
}

// Runs of pixels a Span-mode primitive covers inside the pixel rectangle [x0, x1) x [y0, y1)
// (x0 a multiple of 8, the rectangle inside the target), by one thread straight from words 0-19
// of its setup record: run(y, xa, xb, xs) for pixels [xa, xb) of row y, xs the row's span
// start.  The coverage of k_raster's masks: each row's span inside the box's 8-px blocks.
template <class Run>
__device__ __forceinline__ void span_runs(const float4& q0, const float4& q1, const float4& q2, const float4& q3,
                                          const float4& q4, int sc_minx, int sc_maxx, int x0, int x1, int y0, int y1,
                                          Run run) {
  const int flags = __float_as_int(q0.x);
  const int ylo = max(__float_as_int(q0.w), y0), yhi = min(__float_as_int(q1.y) + 1, y1);
  const int cx0 = max(__float_as_int(q0.z) & ~(SWR_BLOCK - 1), x0);
  const int cx1 = min((__float_as_int(q1.x) | (SWR_BLOCK - 1)) + 1, x1);
  SpanHalf bot, top;
  bot.y0 = __float_as_int(q1.z); bot.y1 = __float_as_int(q1.w);
  bot.ox = q2.x; bot.oy = q2.y; bot.is1 = q2.z; bot.is2 = q2.w;
  top.y0 = __float_as_int(q3.x); top.y1 = __float_as_int(q3.y);
  top.ox = q3.z; top.oy = q3.w; top.is1 = q4.x; top.is2 = q4.y;
  for (int y = ylo; y < yhi; ++y) {
    const bool in_bot = (flags & 32) && y >= bot.y0 && y < bot.y1;
    const bool in_top = (flags & 64) && y > top.y1 && y <= top.y0;
    if (!in_bot && !in_top) continue;
    int xl, xr;
    span_row(in_bot ? bot : top, y, sc_minx, sc_maxx, xl, xr);
    const int xa = max(xl, cx0), xb = min(xr, cx1);
    if (xb > xa) run(y, xa, xb, xl);
  }
}

// The same of rows [ylo, yhi) of one Block-mode block at (bx, by), wx pixels of it wide, of
// class cls (block_class; 1 whole, 2 by the stepped edge tests, as block_rows_bits):
// run(y, xa, xb).
template <class Run>
__device__ __forceinline__ void block_runs(const float* r, int flags, int cls, int bx, int by, int wx, int ylo,
                                           int yhi, Run run) {
  const float t0 = (flags & 4) ? 0.0f : 0x1p-149f, t1 = (flags & 8) ? 0.0f : 0x1p-149f;
  const float t2 = (flags & 16) ? 0.0f : 0x1p-149f;  // thresholds of edge_test
  const float fx = swr_add((float)bx, 0.5f), fy = swr_add((float)by, 0.5f);
  float i0 = swr_eval(r[6], r[7], r[8], fx, fy), i1 = swr_eval(r[9], r[10], r[11], fx, fy);
  float i2 = swr_eval(r[12], r[13], r[14], fx, fy);
  for (int y = by; y < yhi; ++y) {
    uint32_t m = (1u << wx) - 1u;
    if (cls == 2) {
      if (y >= ylo) {
        float c0 = i0, c1 = i1, c2 = i2;
#pragma unroll
        for (int col = 0; col < SWR_BLOCK; ++col) {
          if (!(c0 >= t0 && c1 >= t1 && c2 >= t2)) m &= ~(1u << col);
          c0 = swr_add(c0, r[6]);
          c1 = swr_add(c1, r[9]);
          c2 = swr_add(c2, r[12]);
        }
      }
      i0 = swr_add(i0, r[7]);
      i1 = swr_add(i1, r[10]);
      i2 = swr_add(i2, r[13]);
    }
    if (y < ylo) continue;
    while (m) {  // the row's runs (one, up to rounding)
      const int a = __ffs(m) - 1, b = a + __ffs(~(m >> a)) - 1;
      m &= ~0u << b;
      run(y, bx + a, bx + b);
    }
  }
}

// Primitive id handed to the pixel shader: the index within its own draw.
__device__ __forceinline__ int prim_id(const RasterArgs& g, const float* rec, uint32_t p) {
  return (int)(p - (g.draw_prim_base ? g.draw_prim_base[__float_as_int(rec[1])] : 0u));
}

// 32 x 32 bits turned across a warp: lane l brings row l, lane p leaves with column p (bit l =
// bit p of lane l's row).
__device__ __forceinline__ uint32_t warp_transpose(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j; j >>= 1, m ^= m << j) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & ~m) | ((y & ~m) >> j)) : ((x & m) | ((y & m) << j));
  }
  return x;
}

// A 64-bit word or'ed over the warp.
__device__ __forceinline__ uint64_t warp_or(uint64_t x) {
  const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)x), hi = __reduce_or_sync(0xffffffffu, (uint32_t)(x >> 32));
  return lo | (uint64_t)hi << 32;
}

// Rebuilds the reference's incrementally stepped PixelData for pixel (x, y): the value
// at the evaluation point (block corner or span start) stepped kb times along y and ka
// times along x (PixelData::init/stepY/stepX, PixelData.h:61-125).
template <class PS>
__device__ __forceinline__ void build_pixel(const float* eq, bool blockmode, float fx, float fy, int ka, int kb,
                                            GpuPixel<PS>& pd) {
  typedef Rec<PS> RL;
  // Block pixels step kb rows then ka columns from the block corner; Span pixels ka columns
  // from their span start (kb == 0).  The mode is uniform per primitive (and per warp).
  auto stepped = [&](const float* q3) {
    const float e = swr_eval(q3[0], q3[1], q3[2], fx, fy);
    return blockmode ? fold7(fold7(e, q3[1], kb), q3[0], ka) : swr_fold(e, q3[0], ka);
  };
  if (RL::IW) {
    pd.invw = stepped(eq + 3 * RL::EQ_W);
    pd.w = swr_div(1.0f, pd.invw);
  }
#pragma unroll
  for (int i = 0; i < RL::NA; ++i) pd.avar[i] = stepped(eq + 3 * (RL::EQ_A + i));
#pragma unroll
  for (int i = 0; i < RL::NP; ++i) pd.pvar[i] = swr_mul(stepped(eq + 3 * (RL::EQ_P + i)), pd.w);
}

// Depth a depth-tested shader's State holds (the value its depth test compares against).
template <class State>
__device__ __forceinline__ float swr_state_depth(const State& s) {
  return s.depth;
}

// Conservative depth cull of one primitive in one tile.  A covered pixel's z is the z
// equation (a, b, c) evaluated ((a fx) + (b fy)) + c at the walk's start and then stepped k
// times by b or a (build_z).  With u = 2^-24 and every walk coordinate |x| <= X, 0 <= y <= Y,
// the exact plane values along the walk and the evaluation's terms are bounded by
// Q = |a| X + |b| Y + |c|; the evaluation errs by at most 3.0001 u Q (a three-term naive
// dot product) and each step adds at most u (Q + error so far), so for k u <= 1e-3 the
// stepped z is within u Q (3.01 + 1.001 k) + (k + 3) 2^-149 (underflow) of the exact plane
// value, which 2^-23 (k + 4) Q + 2^-126 bounds.  The exact plane minimum over the covered
// pixel centres [x0, x1] x [y0, y1] is bounded from below with downward-rounded arithmetic.
// Returns true when every covered pixel's z is >= dmax.
__device__ __forceinline__ bool z_not_below(float a, float b, float c, float x0, float x1, float y0, float y1,
                                            float X, float Y, int k, float dmax) {
  if (k > 16384) return false;
  const float q = __fadd_ru(__fadd_ru(__fmul_ru(fabsf(a), X), __fmul_ru(fabsf(b), Y)), fabsf(c));
  if (!(q <= 0x1p100f)) return false;  // no overflow anywhere on the walk (and no NaN)
  const float zlo = __fadd_rd(__fadd_rd(__fmul_rd(a, a >= 0.0f ? x0 : x1), __fmul_rd(b, b >= 0.0f ? y0 : y1)), c);
  const float margin = __fadd_ru(__fmul_ru(q, __fmul_ru((float)(k + 4), 0x1p-23f)), 0x1p-126f);
  return __fsub_rd(zlo, margin) >= dmax;
}

// A State written by another CTA of the same launch (after its fence): loaded through L2,
// never from a possibly stale L1 line.
template <class State>
__device__ __forceinline__ void swr_ld_state(State& d, const State* p) {
  static_assert(sizeof(State) % 4 == 0, "States are whole words");
  uint32_t* o = (uint32_t*)&d;
  const uint32_t* i = (const uint32_t*)p;
#pragma unroll
  for (int k = 0; k < (int)(sizeof(State) / 4); ++k) o[k] = __ldcg(i + k);
}

template <class PS>
__device__ __forceinline__ float build_z(const float* eq, bool blockmode, float fx, float fy, int ka, int kb) {
  typedef Rec<PS> RL;
  if (!RL::IZ) return 0.0f;
  const float* q3 = eq + 3 * RL::EQ_Z;
  const float e = swr_eval(q3[0], q3[1], q3[2], fx, fy);
  // Span pixels start from their own row (kb == 0); the mode is uniform per primitive
  return blockmode ? fold7(fold7(e, q3[1], kb), q3[0], ka) : swr_fold(e, q3[0], ka);
}

// PixelData of pixel (x, y) of the primitive with setup record r (in global memory); pd.z is
// the caller's.
template <class PS, bool SPAN>
__device__ __forceinline__ void pixel_of_record(const float* r, const SwrDrawDesc* draws, int x, int y, GpuPixel<PS>& pd) {
  typedef Rec<PS> RL;
  const int flags = __float_as_int(r[0]);
  const bool blockmode = !SPAN || (flags & 2);
  float fx, fy;
  int ka, kb;
  if (blockmode) {
    fx = swr_add((float)(x & ~7), 0.5f);
    fy = swr_add((float)(y & ~7), 0.5f);
    ka = x & 7;
    kb = y & 7;
  } else {  // from its row's span start
    const SwrDrawDesc& D = draws[__float_as_int(r[1])];
    const bool in_bot = (flags & 32) && y >= __float_as_int(r[6]) && y < __float_as_int(r[7]);
    SpanHalf h;
    h.ox = in_bot ? r[8] : r[14]; h.oy = in_bot ? r[9] : r[15];
    h.is1 = in_bot ? r[10] : r[16]; h.is2 = in_bot ? r[11] : r[17];
    int xl, xr;
    span_row(h, y, D.sc_minx, D.sc_maxx, xl, xr);
    fx = swr_add((float)xl, 0.5f);
    fy = swr_add((float)y, 0.5f);
    ka = x - xl;
    kb = 0;
  }
  pd.x = x;
  pd.y = y;
  pd.eq = r + RL::EQ0;
  build_pixel<PS>(pd.eq, blockmode, fx, fy, ka, kb, pd);
}

// One CTA per screen tile, 256 threads.  Per chunk of CH primitives of the tile's bin:
//   A. stage in shared memory what coverage and depth need of the setup records.  Shaders with
//      the depth cull, behind depths already written: only of primitives that may show; a
//      thread per bin entry decides (verdict), and the others are only counted;
//   B. exact coverage masks per (primitive, 8 x 8 block): one thread per pair classifies
//      Block-mode blocks (the reference's corner test); one thread per four rows builds
//      Span-mode rows from [xl, xr) (kept as each row's interpolation start) and finishes
//      partially covered blocks with the reference's stepped edge tests;
//   C0. depth cull: per 8 x 4 pixel region, primitives whose z cannot pass any depth test of
//      the chunk there (z_not_below against the region's largest depth) are only counted;
//   C2. each thread visits, in primitive order, the primitives covering the pixels it owns:
//      the stepped z and the depth test against the pixel's register-resident State.  Shaders
//      with side effects of their own run drawPixel() there instead.
// At the end of the tile every pixel is shaded once, from the record of the last primitive
// that passed its depth test.  Bound by SM issue and by the latency of the short stages
// between barriers.
//   Against shading fragments ahead of their depth tests, small primitives' compacted one
// fragment per thread (whole draws): 4K soup 5212 -> 4217 us, 60k-triangle list 283 -> 207,
// 256 meshes 3202 -> 3172, 16 differentiable views 637 -> 596, dense 1080p mesh 117 -> 113.
// DIRECT: the raster of a small draw, which has no bins (RasterArgs.boxes).
// A heavy tile of a depth-min shader (RasterArgs.dslice) is run by up to SWR_DSLICES CTAs,
// each over its own run of whole chunks from the draw's starting State; the last run to
// finish merges the runs' States in bin order (swr_depth_merge) and stores.
//
// raster_tile: the work of CTA `bid` of a launch that gives every tile its own; false when it
// has none.
template <class PS, int TILE, int CH, bool SPAN, bool DIRECT, int NT>
__device__ __forceinline__ bool raster_tile(const RasterArgs& g, uint32_t bid) {
  typedef Rec<PS> RL;
  constexpr int PPT = TILE * TILE / NT;  // pixels per thread
  constexpr int NWARP = NT / 32;
  constexpr int NBX = TILE / SWR_BLOCK;   // blocks per tile row
  constexpr int NB = NBX * NBX;
  constexpr bool kCull = SWR_DEPTH_CULL && SwrDepthCull<PS>::value;
  // Shaders without side effects are shaded once per pixel, after the tile's depth tests: a
  // fragment that passes only records its primitive, and the last one that did is shaded from
  // its record.
  constexpr bool kDefer = !SwrNoCompact<PS>::value;
  // Shaders with side effects interpolate every fragment in the walk.  In Span mode its steps
  // from the row's span start are a loop whose course depends on the primitive (swr_fold), and
  // lanes that visit different ones wait for each other: the warp's lanes then visit the same
  // primitives, unless that is many more steps than the pixel with most of them takes.  A
  // depth-tested user shader at 1920x1080, us a draw with every pixel on its own / together /
  // by that rule: 20,000 triangles of 300 px 27700 / 21800 / 21700, 200,000 of 40 px
  // 8560 / 6790 / 6890, 200,000 of 6 px 396 / 544 / 422.  Block mode's are at most 14 predicated
  // steps, the same for every primitive: there each pixel goes on its own.
  constexpr bool kTogether = !kDefer && SPAN;
  static_assert(!kDefer || (PS::HasDepth && RL::IZ), "a deferred fragment is one that passes the depth test");
  // Staged records: words 0-23 where only coverage and z are read (header, edges or span
  // halves, the z equation), 28 words apart so that the lanes' different records spread over
  // the banks; else whole.
  constexpr int RW4 = kDefer ? 6 : RL::R / 4, SR4 = kDefer ? 7 : RL::R / 4, SR = SR4 * 4;
  static_assert(RL::EQ0 + 3 * RL::EQ_Z + 3 <= 24, "the z equation lies in the first 24 words");
  __shared__ float4 srec4[CH * SR4];
  float* srec = (float*)srec4;
  __shared__ uint64_t smask[CH * NB];
  __shared__ int2 sspan[SPAN ? CH * TILE : 1];  // Span mode: each tile row's [xl, xr)
  __shared__ uint32_t sids[CH];
  __shared__ uint32_t sfr[64];
  __shared__ uint32_t slast;  // sliced heavy tile: this run is the last to finish
  __shared__ uint16_t spart[CH * NB];  // partially covered (primitive, block) pairs
  __shared__ uint32_t snpart;
  __shared__ uint32_t ssorted[SWR_RASTER_SORT];  // the tile's ordered bin (self-sorted tiles)
  __shared__ uint32_t scs[SWR_SEGS + 1];          // its cell starts relative to the bin start
  static_assert(sizeof(srec4) >= SWR_RASTER_SORT * 4, "raw bin staging fits the record area");
  // Regions of 8 x 4 pixels (half blocks), eight to a 16 x 16 sub-tile: a warp's q-th is region
  // q * NWARP + warp.
  constexpr int NREG = TILE * TILE / 32;
  __shared__ uint32_t swd[NREG];  // per region: order key of the largest depth it holds
  // Depth cull: the next primitives to rasterize, in order (up to CH - 1 left over plus a batch
  // of NT), and per pixel row the coverage of primitives that were only counted (+1 at a run's
  // first pixel, -1 past its last; used where the target records counts)
  __shared__ uint32_t ssurv[kCull ? CH + NT : 1];
  // a batch's primitives to count: Span ones from the front, Block ones from the back; their
  // partially covered blocks (entry * NB + block)
  __shared__ uint32_t scul[kCull ? NT : 1];
  constexpr int SCP = 1024;
  __shared__ uint16_t scp[kCull ? SCP : 1];
  __shared__ int scnt[kCull ? TILE * (TILE + 1) : 1];
  constexpr int NW = CH / 32;      // 32-primitive words of a chunk
  static_assert(CH % 32 == 0 && CH <= 128 && CH <= NT, "chunks of 32, 64, 96 or 128 primitives");
  __shared__ uint32_t sculr[kCull ? NREG * NW : 1];  // per region: primitives only counted there
  __shared__ int sminx[kCull && SPAN ? CH : 1];  // Span mode: leftmost start of a span reaching the tile
  constexpr int HW = (CH + 63) / 64;  // 64-primitive words of a chunk
  // the draw's queue requests are final (nothing after this stage counts)
  if (!DIRECT && bid == 0 && threadIdx.x == 0) swr_close_status(g.status_w);
  if (g.status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return false;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t frags = 0, passes = 0;
  // One CTA per tile (a persistent grid pulling tiles from a counter measured no faster on
  // the dense mesh and slower where few tiles carry the work: they gather on fewer SMs).
  uint32_t tile = bid, slice = 0;
  int quad = -1;  // the 8 x 8 quadrant (block) this CTA rasterizes alone, -1: the whole tile
  int dslot = -1;  // sliced heavy tile: its list slot (slice = its run)
  uint32_t b = 0, e = 0;
  int ti = 0;  // its target
  if constexpr (!DIRECT) {
    if (g.tiles.list) {
      uint4 entry;
      constexpr uint32_t kRuns = SWR_DSLICES > 4 ? SWR_DSLICES : 4;
      static_assert(kRuns == 4 && SWR_DSLICES == 4, "four CTAs per heavy tile, as runs or as quadrants");
      const bool heavy = (SwrDepthMin<PS>::value && g.dslice) || (TILE == 16 && g.quad);
      const uint32_t nq = heavy ? 4u * g.tiles.heavy_cap : 0u;
      if (bid < nq) {
        const uint32_t slot = bid >> 2;
        if (slot >= min(g.tiles.counts[0], g.tiles.heavy_cap)) return false;
        entry = __ldg(g.tiles.heavy + slot);
        if (SwrDepthMin<PS>::value && g.dslice) {
          slice = bid & 3u;
          dslot = (int)slot;
        } else {
          quad = (int)(bid & 3u);
        }
      } else {
        uint32_t i = bid - nq;
        if (TILE == 16 && g.quad_all) {
          quad = (int)(i & 3u);
          i >>= 2;
        }
        if (!swr_listed_tile(g.tiles, i, entry)) return false;
      }
      tile = entry.x;
      b = entry.y;
      e = entry.z;
      ti = (int)entry.w;
    } else {
      if (tile >= g.ntiles) return false;
      b = g.tile_start[tile];
      e = g.tile_start[tile + 1];
    }
  } else {
    if (tile >= g.ntiles) return false;
  }
  // Small draws: the tile's primitives out of the next windows of NT boxes, in order, until
  // ssorted (SWR_RASTER_SORT) may not hold another window's, or none is left (e: their count).
  uint32_t scan_pos = 0, scan_np = 0;
  auto gather = [&]() {
    const uint32_t tx = tile % (uint32_t)g.targets[0].tiles_x, ty = tile / (uint32_t)g.targets[0].tiles_x;
    e = 0;
    while (scan_pos < scan_np && e <= SWR_RASTER_SORT - NT) {
      const uint32_t i = scan_pos + threadIdx.x;
      const bool hit = i < scan_np && swr_box_hit(g.boxes[i], tx, ty);
      const uint32_t bal = __ballot_sync(0xffffffffu, hit);
      __syncthreads();  // the previous window's counts (or the last chunk's ids) are no longer read
      if (lane == 0) scs[warp] = (uint32_t)__popc(bal);
      __syncthreads();
      uint32_t at = e, all = 0;
#pragma unroll
      for (int w = 0; w < NWARP; ++w) {
        const uint32_t c = scs[w];
        if (w < warp) at += c;
        all += c;
      }
      if (hit) ssorted[at + (uint32_t)__popc(bal & ((1u << lane) - 1u))] = i;
      e += all;
      scan_pos += NT;
    }
  };
  if constexpr (DIRECT) {
    scan_np = min(g.status[SWR_ST_PRIMS], g.cap_prims);
    if (scan_np > NT && !direct_any(g.boxes, scan_np, tile, (uint32_t)g.targets[0].tiles_x)) return true;
    gather();
  }
  if (b == e) return true;  // uniform per CTA
  // the chunks this CTA rasterizes: the whole bin, or a sliced heavy tile's run
  uint32_t cb = b, ce = e;
  int nsl = 1;
  if (dslot >= 0) {
    const uint32_t nch = (e - b + CH - 1) / CH;
    nsl = (int)min(nch, (uint32_t)SWR_DSLICES);
    if ((int)slice >= nsl) return false;  // (uniform per tile: these CTAs take no part)
    cb = b + (uint32_t)((uint64_t)nch * slice / (uint32_t)nsl) * CH;
    ce = min(e, b + (uint32_t)((uint64_t)nch * (slice + 1) / (uint32_t)nsl) * CH);
  }
  const SwrTargetDesc& T = g.targets[ti];
  const SwrUniforms& U = g.draws[T.first_draw].u;
  const uint32_t lt = tile - T.tile_base;
  const int ox = (int)(lt % (uint32_t)T.tiles_x) * TILE, oy = (int)(lt / (uint32_t)T.tiles_x) * TILE;
  // Thread -> pixels: each warp covers 8 x 4 half blocks.
  int px[PPT], py[PPT], blk[PPT];
  bool in[PPT];
  typename PS::State st[PPT];
#pragma unroll
  for (int q = 0; q < PPT; ++q) {
    const int reg = q * NWARP + warp, sub = reg >> 3, hb = (reg & 7) >> 1;
    const int lx = (sub % (TILE / 16)) * 16 + (hb & 1) * 8 + (lane & 7);
    const int ly = (sub / (TILE / 16)) * 16 + (hb >> 1) * 8 + (reg & 1) * 4 + (lane >> 3);
    px[q] = ox + lx;
    py[q] = oy + ly;
    blk[q] = (ly >> 3) * NBX + (lx >> 3);
    in[q] = px[q] < T.width && py[q] < T.height && (quad < 0 || blk[q] == quad);
    if (in[q]) PS::load(st[q], px[q], py[q], U);
  }
  // A tile of at most SWR_RASTER_SORT entries orders its own bin: the cells (increasing id
  // segments) are contiguous, so an id's position is its cell's start plus the number of
  // smaller ids in that cell.  The raw ids are staged in the record area (used only later).
  const bool self_sort = DIRECT || (g.bin_raw && e - b <= (uint32_t)SWR_RASTER_SORT);
  if (!DIRECT && self_sort) {
    uint32_t* sraw = (uint32_t*)srec4;
    const uint32_t ntot = e - b;
    if (threadIdx.x <= SWR_SEGS)
      scs[threadIdx.x] = (threadIdx.x < SWR_SEGS ? g.tiles.start[(size_t)tile * SWR_SEGS + threadIdx.x] : e) - b;
    for (uint32_t j = threadIdx.x; j < ntot; j += NT) sraw[j] = g.bin_raw[b + j];
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < ntot; j += NT) {
      int lo = 0, hi = SWR_SEGS - 1;  // the cell holding j: last c with scs[c] <= j
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (scs[mid] <= j) lo = mid; else hi = mid - 1;
      }
      const uint32_t v = sraw[j], c_end = scs[lo + 1];
      uint32_t pos = scs[lo];
      for (uint32_t k = scs[lo]; k < c_end; ++k) pos += sraw[k] < v;
      ssorted[pos < ntot ? pos : 0] = v;
    }
  }
  // the CTA's pixels: the tile or its quadrant, inside the target
  const int rx0 = ox + (quad < 0 ? 0 : (quad % NBX) * SWR_BLOCK), ry0 = oy + (quad < 0 ? 0 : (quad / NBX) * SWR_BLOCK);
  const int rx1 = min(rx0 + (quad < 0 ? TILE : SWR_BLOCK), T.width), ry1 = min(ry0 + (quad < 0 ? TILE : SWR_BLOCK), T.height);
  const bool counts = U.frag_count != nullptr;  // per-pixel drawPixel counts are recorded
  bool cull_on = false;  // some region holds no +inf depth (else nothing can be culled)
  uint32_t stands[PPT];  // kDefer: the last primitive to pass the pixel's depth test (none: ~0)
#pragma unroll
  for (int q = 0; q < PPT; ++q) stands[q] = 0xffffffffu;
  auto bin_id = [&](uint32_t i) { return self_sort ? ssorted[i - b] : __ldg(g.bin + i); };
  // Whether a primitive's fragments here all fail their depth tests for certain -- its z is
  // provably not below the largest depth of any region its box meets (z_not_below, as C0, over
  // the box instead of the covered pixels): 1 a Span, 2 a Block primitive that need only be
  // counted, 0 one to rasterize, 3 one that covers nothing here.
  auto verdict = [&](uint32_t p) -> int {
    const float4* rc = (const float4*)(g.recs + (size_t)p * RL::R);
    const float4 q0 = __ldg(rc), q1 = __ldg(rc + 1), q4 = __ldg(rc + 4);
    const float zc = __ldg(&rc[5].x);
    const int flags = __float_as_int(q0.x);
    const int x0 = max(__float_as_int(q0.z), rx0), x1 = min(__float_as_int(q1.x), rx1 - 1);
    const int y0 = max(__float_as_int(q0.w), ry0), y1 = min(__float_as_int(q1.y), ry1 - 1);
    if (!(flags & 1) || x0 > x1 || y0 > y1) return 3;
    // Span pixels are stepped from their row's start.  Within a half a row's start is a
    // monotone function of the row (every operation of span_row is, for finite slopes), so none
    // lies left of the box, which spans the end rows' -- or of the scissor, where the box is
    // cut off at 0.
    int smin = 0;
    if (SPAN && !(flags & 2)) {
      const float4 q2 = __ldg(rc + 2);
      if (!(fabsf(q2.z) < 0x1p100f && fabsf(q4.x) < 0x1p100f)) return 0;
      smin = __float_as_int(q0.z);
      if (smin <= 0) smin = min(0, g.draws[__float_as_int(q0.y)].sc_minx);
    }
    for (int cy = (y0 - oy) >> 2; cy <= (y1 - oy) >> 2; ++cy)
      for (int cx = (x0 - ox) >> 3; cx <= (x1 - ox) >> 3; ++cx) {
        // region of the 8 x 4 cell (cx, cy): sub-tile, then the warp that owns it
        const int reg = ((cy >> 2) * (TILE / 16) + (cx >> 1)) * 8 + ((cx & 1) + ((cy >> 1) & 1) * 2) * 2 + (cy & 1);
        const uint32_t key = swd[reg];
        if (key == 0u || key >= 0xff800000u) return 0;
        const float dmax = __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
        const int xa = max(x0, ox + cx * 8), xb = min(x1, ox + cx * 8 + 7);
        const int ya = max(y0, oy + cy * 4), yb = min(y1, oy + cy * 4 + 3);
        int steps = 2 * (SWR_BLOCK - 1);
        float X = (float)xb + 0.5f;
        if (SPAN && !(flags & 2)) {
          steps = max(0, xb - smin);
          if (smin < 0) X = fmaxf(X, (float)(-smin) + 0.5f);
        }
        const float fyb = (float)yb + 0.5f;
        if (!z_not_below(q4.z, q4.w, zc, (float)xa + 0.5f, (float)xb + 0.5f, (float)ya + 0.5f, fyb, X, fyb, steps, dmax))
          return 0;
      }
    return SPAN && !(flags & 2) ? 1 : 2;
  };
  auto add_run = [&](int y, int xa, int xb) {  // pixels [xa, xb) of row y: covered once more, failing
    frags += (uint32_t)(xb - xa);
    if (counts) {
      atomicAdd(&scnt[(y - oy) * (TILE + 1) + xa - ox], 1);
      atomicAdd(&scnt[(y - oy) * (TILE + 1) + xb - ox], -1);
    }
  };
  // Counts the listed primitives: ns Span ones a thread each, nb Block ones a thread per 8 x 8
  // block, then a thread per partially covered block.
  auto count_listed = [&](int ns, int nb) {
    if constexpr (SPAN) {
      for (int i = threadIdx.x; i < ns; i += NT) {
        const float4* rc = (const float4*)(g.recs + (size_t)scul[i] * RL::R);
        const float4 q0 = __ldg(rc);
        const SwrDrawDesc& D = g.draws[__float_as_int(q0.y)];
        span_runs(q0, __ldg(rc + 1), __ldg(rc + 2), __ldg(rc + 3), __ldg(rc + 4), D.sc_minx, D.sc_maxx, rx0, rx1, ry0,
                  ry1, [&](int y, int xa, int xb, int) { add_run(y, xa, xb); });
      }
    }
    auto count_block = [&](int i, bool classify) -> int {
      const int j = i % NB;
      const int bx = ox + (j % NBX) * SWR_BLOCK, by = oy + (j / NBX) * SWR_BLOCK;
      const float4* rc = (const float4*)(g.recs + (size_t)scul[NT - 1 - i / NB] * RL::R);
      const float4 q0 = __ldg(rc), q1 = __ldg(rc + 1), q2 = __ldg(rc + 2), q3 = __ldg(rc + 3);
      const float r[15] = {0, 0, 0, 0, 0, 0, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z};
      int cls = 2;
      if (classify) {
        if (bx < rx0 || bx >= rx1 || by < ry0 || by >= ry1 || bx > __float_as_int(q1.x) || by > __float_as_int(q1.y) ||
            bx + SWR_BLOCK - 1 < __float_as_int(q0.z) || by + SWR_BLOCK - 1 < __float_as_int(q0.w))
          return 0;
        cls = block_class(r, __float_as_int(q0.x), bx, by);
        if (cls == 0 || cls == 2) return cls;
      }
      block_runs(r, __float_as_int(q0.x), cls, bx, by, min(SWR_BLOCK, rx1 - bx), by, min(by + SWR_BLOCK, ry1), add_run);
      return 1;
    };
    for (int i = threadIdx.x; i < nb * NB; i += NT)
      if (count_block(i, true) == 2) {
        const uint32_t at = atomicAdd(&snpart, 1u);
        if (at < SCP) scp[at] = (uint16_t)i; else count_block(i, false);
      }
    __syncthreads();
    const int m = min((int)snpart, SCP);
    for (int t = threadIdx.x; t < m; t += NT) count_block(scp[t], false);
  };
  if (kCull && counts)
    for (int i = threadIdx.x; i < TILE * (TILE + 1); i += NT) scnt[i] = 0;  // (first used past the next barrier)
  while (true) {  // once; small draws: per gathered run of the tile's primitives
  uint32_t c0 = cb;        // next bin entry
  uint32_t nsurv = 0;      // depth cull: primitives waiting in ssurv
  while (c0 < ce || nsurv) {
    __syncthreads();  // the previous chunk's shared state is no longer read; ssorted is complete
    int n;
    if constexpr (kCull) {
      // Region depth bounds (tiles of more than one chunk): per region an order-preserving key
      // of the largest depth its pixels hold (NaN depths, which every fragment fails, and
      // pixels outside the target are ignored; key 0: none usable).  A region holding +inf can
      // cull nothing (z is finite); the barrier's OR tells whether any region can.
      if (ce - cb > (uint32_t)CH) {
        bool my_ok = false;
#pragma unroll
        for (int q = 0; q < PPT; ++q) {
          const float dq = swr_state_depth(st[q]);
          const uint32_t u = __float_as_uint(dq);
          const uint32_t kq = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
          const uint32_t key = __reduce_max_sync(0xffffffffu, in[q] && !swr_isnan(dq) ? kq : 0u);
          if (lane == 0) swd[q * NWARP + warp] = key;
          my_ok |= key != 0u && key < 0xff800000u;  // uniform per warp
        }
        cull_on = __syncthreads_or(my_ok);
      }
      // The next chunk's primitives.  Behind depths already written, one thread per entry
      // counts the primitives that cannot show, and only the others are kept (in order).
      while (nsurv < (uint32_t)CH && c0 < ce) {
        if (!cull_on) {
          const uint32_t take = min((uint32_t)CH - nsurv, ce - c0);
          if (threadIdx.x < take) ssurv[nsurv + threadIdx.x] = bin_id(c0 + threadIdx.x);
          nsurv += take;
          c0 += take;
          continue;
        }
        const uint32_t take = min((uint32_t)NT, ce - c0);
        uint32_t p = 0;
        int v = 3;
        if (threadIdx.x < take) {
          p = bin_id(c0 + threadIdx.x);
          v = verdict(p);
        }
        const uint32_t lt_mask = (1u << lane) - 1u;
        const uint32_t bk = __ballot_sync(0xffffffffu, v == 0), bs = __ballot_sync(0xffffffffu, v == 1);
        const uint32_t bb = __ballot_sync(0xffffffffu, v == 2);
        __syncthreads();  // the previous batch's lists are no longer read
        if (lane == 0) scs[warp] = (uint32_t)(__popc(bk) | __popc(bs) << 8 | __popc(bb) << 16);
        if (threadIdx.x == 0) snpart = 0;
        __syncthreads();
        uint32_t at_k = nsurv;
        int ns = 0, nb = 0, at_s = 0, at_b = 0;
#pragma unroll
        for (int w = 0; w < NWARP; ++w) {
          const uint32_t c = scs[w];
          if (w < warp) {
            at_k += c & 255u;
            at_s += (int)((c >> 8) & 255u);
            at_b += (int)(c >> 16);
          }
          nsurv += c & 255u;
          ns += (int)((c >> 8) & 255u);
          nb += (int)(c >> 16);
        }
        if (v == 0) ssurv[at_k + (uint32_t)__popc(bk & lt_mask)] = p;
        if (v == 1) scul[at_s + __popc(bs & lt_mask)] = p;
        if (v == 2) scul[NT - 1 - at_b - __popc(bb & lt_mask)] = p;
        __syncthreads();
        count_listed(ns, nb);
        c0 += take;
      }
      __syncthreads();
      if (nsurv == 0) break;
      n = (int)min((uint32_t)CH, nsurv);
      if (threadIdx.x < n) sids[threadIdx.x] = ssurv[threadIdx.x];
    } else {
      n = (int)min((uint32_t)CH, ce - c0);
      if (threadIdx.x < n) sids[threadIdx.x] = bin_id(c0 + threadIdx.x);
    }
    if (threadIdx.x == 0) snpart = 0;
    if (kCull && SPAN && threadIdx.x < CH) sminx[threadIdx.x] = 0x7fffffff;
    // A: the chunk's setup records (ids read from their source: sids is published by the
    // barrier below)
    {
      const float4* recs4 = (const float4*)g.recs;
#pragma unroll 4
      for (int i = threadIdx.x; i < n * RW4; i += NT) {
        const int k = i / RW4, w = i - k * RW4;
        const uint32_t id = kCull ? ssurv[k] : bin_id(c0 + k);
        srec4[k * SR4 + w] = recs4[(size_t)id * (RL::R / 4) + w];
      }
    }
    __syncthreads();
    uint32_t left = 0;  // depth cull: this thread's share of the primitives waiting after this chunk
    if constexpr (kCull) {
      if (threadIdx.x + n < nsurv) left = ssurv[threadIdx.x + n];
    } else {
      c0 += n;
    }
    // B1: coverage per (primitive, block).  Fully covered / skipped blocks and Span rows are
    // finished here; partially covered Block-mode blocks are queued for B2.
    for (int i = threadIdx.x; i < n * NB; i += NT) {
      const int k = i / NB, j = i - k * NB;
      const float* r = srec + k * SR;
      const int flags = __float_as_int(r[0]);
      if (SPAN && (flags & 3) == 1) continue;  // Span mode: rows below, masks after the barrier
      if (quad >= 0 && j != quad) {  // another CTA's quadrant
        smask[i] = 0;
        continue;
      }
      const int bx = ox + (j % NBX) * SWR_BLOCK, by = oy + (j / NBX) * SWR_BLOCK;
      uint64_t m = 0;
      const bool hit = (flags & 1) && bx <= __float_as_int(r[4]) && bx + SWR_BLOCK - 1 >= __float_as_int(r[2]) &&
                       by <= __float_as_int(r[5]) && by + SWR_BLOCK - 1 >= __float_as_int(r[3]);
      if (hit) {  // Block mode (every valid primitive of a k_raster<..., false> launch)
        const int cls = block_class(r, flags, bx, by);
        if (cls == 1) m = ~0ull;
        if (cls == 2) spart[atomicAdd(&snpart, 1u)] = (uint16_t)i;
      }
      smask[i] = m;
    }
    if constexpr (SPAN) {
      // B1 (Span mode): four rows of a primitive per thread: each row's span [xl, xr), kept as the
      // row's interpolation start, and its half of the masks of the blocks it crosses
      constexpr int NR = TILE / 4;
      for (int i = threadIdx.x; i < n * NR; i += NT) {
        const int k = i / NR, br = i - k * NR;
        const float* r = srec + k * SR;
        const int flags = __float_as_int(r[0]);
        if ((flags & 3) != 1) continue;
        const int rows0 = __float_as_int(r[3]), rows1 = __float_as_int(r[5]);
        const SwrDrawDesc& D = g.draws[__float_as_int(r[1])];
        const int minx = D.sc_minx, maxx = D.sc_maxx;
        const int ya = oy + br * 4;
        uint32_t m[NBX];
#pragma unroll
        for (int j = 0; j < NBX; ++j) m[j] = 0u;
        int lmin = 0x7fffffff;  // leftmost start of a span reaching the tile
#pragma unroll
        for (int rr = 0; rr < 4; ++rr) {
          const int y = ya + rr;
          int2 sp = make_int2(1, 0);
          if (y >= rows0 && y <= rows1) {
            const bool in_bot = (flags & 32) && y >= __float_as_int(r[6]) && y < __float_as_int(r[7]);
            const bool in_top = (flags & 64) && y > __float_as_int(r[13]) && y <= __float_as_int(r[12]);
            if (in_bot || in_top) {
              SpanHalf h;
              h.ox = in_bot ? r[8] : r[14]; h.oy = in_bot ? r[9] : r[15];
              h.is1 = in_bot ? r[10] : r[16]; h.is2 = in_bot ? r[11] : r[17];
              span_row(h, y, minx, maxx, sp.x, sp.y);
            }
          }
          sspan[k * TILE + br * 4 + rr] = sp;
          if (sp.x < sp.y && sp.y > ox) lmin = min(lmin, sp.x);
#pragma unroll
          for (int j = 0; j < NBX; ++j) {
            const int bx = ox + j * SWR_BLOCK;
            const int c0b = min(max(sp.x, bx), bx + SWR_BLOCK) - bx, c1b = min(max(sp.y, bx), bx + SWR_BLOCK) - bx;
            // columns [c0b, c1b): none where c1b <= c0b
            m[j] |= ((0xffu << c0b) & ~(0xffffffffu << c1b) & 0xffu) << (rr * 8);
          }
        }
#pragma unroll
        for (int j = 0; j < NBX; ++j) {
          const int bx = ox + j * SWR_BLOCK, jj = (br >> 1) * NBX + j;
          const bool hit = bx <= __float_as_int(r[4]) && bx + SWR_BLOCK - 1 >= __float_as_int(r[2]) && (quad < 0 || jj == quad);
          ((uint32_t*)&smask[k * NB + jj])[br & 1] = hit ? m[j] : 0u;
        }
        if (kCull && lmin != 0x7fffffff) atomicMin(&sminx[k], lmin);
      }
    }
    __syncthreads();
    if constexpr (kCull) {  // the waiting primitives move up
      if (threadIdx.x + n < nsurv) ssurv[threadIdx.x] = left;
      nsurv -= n;
    }
    // B2: partially covered blocks, four rows per lane: one half of the block's mask
    {
      const int np2 = (int)snpart * 2;
      for (int t = threadIdx.x; t < np2; t += NT) {
        const int i = spart[t >> 1];
        const int k = i / NB, j = i - k * NB;
        const float* r = srec + k * SR;
        ((uint32_t*)&smask[i])[t & 1] = block_rows_bits(r, __float_as_int(r[0]), ox + (j % NBX) * SWR_BLOCK,
                                                        oy + (j / NBX) * SWR_BLOCK, t & 1);
      }
    }
    __syncthreads();
    // C0 (depth-tested shaders): per (region, primitive) whether every covered pixel's z is
    // provably not below the region's largest depth at the chunk's start (z_not_below over
    // the covered pixels' box in the region).  Depths only decrease, so such fragments fail
    // their depth tests: the primitive is only counted there.
    if (kCull && cull_on) {
      for (int t = threadIdx.x; t < NREG * CH; t += NT) {
        const int reg = t / CH, k = t - reg * CH;  // reg uniform per warp (CH is a multiple of 32)
        bool culled = false;
        if (k < n && (__float_as_int(srec[k * SR]) & 1)) {
          const int q = reg >> 3, w = reg & 7, hb = w >> 1;
          const int lx0 = (q % (TILE / 16)) * 16 + (hb & 1) * 8;
          const int ly0 = (q / (TILE / 16)) * 16 + (hb >> 1) * 8 + (w & 1) * 4;
          const uint32_t mh = (uint32_t)(smask[k * NB + (ly0 >> 3) * NBX + (lx0 >> 3)] >> ((w & 1) * 32));
          const uint32_t key = swd[reg];
          if (mh && key != 0u && key < 0xff800000u) {
            const float dmax = __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
            uint32_t c = mh | (mh >> 16);
            c |= c >> 8;
            c &= 0xffu;
            const int x0 = ox + lx0 + __ffs(c) - 1, x1 = ox + lx0 + 31 - __clz(c);
            const int y0 = oy + ly0 + ((__ffs(mh) - 1) >> 3), y1 = oy + ly0 + ((31 - __clz(mh)) >> 3);
            const float* r = srec + k * SR;
            // walk bounds: Block mode steps <= 7 rows then <= 7 columns inside the block;
            // Span mode steps from the row's span start (every covered pixel lies in a row
            // whose span reaches the tile) to the pixel
            int steps = 2 * (SWR_BLOCK - 1);
            float X = (float)x1 + 0.5f;
            if (SPAN && !(__float_as_int(r[0]) & 2)) {
              const int smin = sminx[k];
              steps = max(0, x1 - smin);
              if (smin < 0) X = fmaxf(X, (float)(-smin) + 0.5f);
            }
            const float* zq = r + RL::EQ0 + 3 * RL::EQ_Z;
            const float fy1 = (float)y1 + 0.5f;
            culled = z_not_below(zq[0], zq[1], zq[2], (float)x0 + 0.5f, (float)x1 + 0.5f, (float)y0 + 0.5f, fy1, X,
                                 fy1, steps, dmax);
          }
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, culled);
        if (lane == 0) sculr[reg * NW + (k >> 5)] = bal;
      }
      __syncthreads();
    }
    // C2: fragments in primitive order.  Each warp owns one 8 x 4 half block per sub-tile q;
    // the chunk's masks of that half block, one primitive per lane, are turned across the warp
    // into each pixel's set of covering primitives, which its lane visits in increasing order.
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
      const int half = (py[q] >> 2) & 1;
      uint64_t mine[HW];
#pragma unroll
      for (int w = 0; w < HW; ++w) mine[w] = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        if (w && w * 32 >= n) break;  // (uniform)
        const int k = w * 32 + lane;
        const uint32_t cov = warp_transpose(k < n ? (uint32_t)(smask[k * NB + blk[q]] >> (half * 32)) : 0u, lane);
        mine[w >> 1] |= (uint64_t)(in[q] ? cov : 0u) << ((w & 1) * 32);
      }
      if constexpr (kDefer) {  // (other shaders count a fragment when they draw it)
        uint32_t cnt = 0;
#pragma unroll
        for (int w = 0; w < HW; ++w) cnt += (uint32_t)__popcll(mine[w]);
        frags += cnt;
        st[q].frags += cnt;
      }
      if (kCull && cull_on) {
        // primitives culled in this warp's region fail the depth test: counted only
        const uint32_t* cr = sculr + (q * NWARP + warp) * NW;
#pragma unroll
        for (int w = 0; w < HW; ++w)
          mine[w] &= ~((uint64_t)cr[2 * w] | (2 * w + 1 < NW ? (uint64_t)cr[2 * w + 1] << 32 : 0ull));
      }
      int won = -1;  // kDefer: the chunk's last primitive to pass the pixel's depth test
      // kTogether: the primitives of any of the warp's pixels where they are not many more than
      // one pixel's, else the pixel's own
      auto visits = [&](uint64_t own) -> uint64_t {
        if (!kTogether) return own;
        const uint64_t any = warp_or(own);
        return 4 * __popcll(any) <= 7 * (int)__reduce_max_sync(0xffffffffu, (uint32_t)__popcll(own)) ? any : own;
      };
      uint64_t hits = visits(mine[0]);
      uint64_t later = HW > 1 ? visits(mine[HW - 1]) : 0ull;
      int kbase = 0;
      while (true) {  // (one copy of the loop body for both words)
        if (!hits) {
          if (HW == 1 || !later) break;
          hits = later;
          later = 0;
          kbase = 64;
        }
        const int k = kbase + __ffsll((long long)hits) - 1;
        hits &= hits - 1ull;
        if (kTogether && !((mine[HW > 1 ? k >> 6 : 0] >> (k & 63)) & 1ull)) continue;
        const float* r = srec + k * SR;
        const bool blockmode = !SPAN || (__float_as_int(r[0]) & 2);
        float fx, fy;
        int ka, kb;
        if (blockmode) {
          fx = swr_add((float)(px[q] & ~7), 0.5f);
          fy = swr_add((float)(py[q] & ~7), 0.5f);
          ka = px[q] & 7;
          kb = py[q] & 7;
        } else {
          const int xs = sspan[k * TILE + (py[q] - oy)].x;
          fx = swr_add((float)xs, 0.5f);
          fy = swr_add((float)py[q], 0.5f);
          ka = px[q] - xs;
          kb = 0;
        }
        const float* eq = r + RL::EQ0;
        const float z = build_z<PS>(eq, blockmode, fx, fy, ka, kb);
        if constexpr (kDefer) {
          if (z < st[q].depth) {
            st[q].depth = z;
            st[q].writes++;
            won = k;
          }
        } else {
          frags++;
          GpuPixel<PS> pd;
          pd.x = px[q];
          pd.y = py[q];
          pd.eq = eq;
          pd.z = z;
          build_pixel<PS>(eq, blockmode, fx, fy, ka, kb, pd);
          PS::drawPixel(pd, prim_id(g, r, sids[k]), st[q], g.draws[__float_as_int(r[1])].u);
        }
      }
      if (kDefer && won >= 0) stands[q] = sids[won];
    }
  }
  if constexpr (!DIRECT) break;
  gather();
  if (e == 0) break;
  ce = e;
  }
  if constexpr (kDefer) {  // shade the fragments that stand
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
      if (stands[q] == 0xffffffffu) continue;
      const float* r = g.recs + (size_t)stands[q] * RL::R;
      GpuPixel<PS> pd;
      pd.z = st[q].depth;
      pixel_of_record<PS, SPAN>(r, g.draws, px[q], py[q], pd);
      // its write, against a depth that lets it pass; its test was counted in the walk
      st[q].depth = __int_as_float(0x7f800000);
      PS::apply(st[q], pd.z, PS::shade(pd, g.draws[__float_as_int(r[1])].u), prim_id(g, r, stands[q]));
      st[q].frags--;
      st[q].writes--;
    }
  }
  if (kCull && counts) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
      int c = 0;
      for (int k = 0; k <= px[q] - ox; ++k) c += scnt[(py[q] - oy) * (TILE + 1) + k];
      if (in[q]) st[q].frags += (uint32_t)c;
    }
  }
  if constexpr (SwrDepthMin<PS>::value && !DIRECT) {
    if (dslot >= 0) {
      // this run's States, then the last run to finish merges the tile's runs in bin order
      // (each thread owns the same pixels in every run's CTA)
      typename PS::State* ss = (typename PS::State*)g.dslice_state + (size_t)dslot * SWR_DSLICES * (TILE * TILE);
#pragma unroll
      for (int q = 0; q < PPT; ++q)
        if (in[q]) {
          ss[(size_t)slice * (TILE * TILE) + (py[q] - oy) * TILE + (px[q] - ox)] = st[q];
          passes += st[q].writes;
        }
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) slast = atomicAdd(&g.dslice_done[dslot], 1u) == (uint32_t)(nsl - 1);
      __syncthreads();
      if (slast) {
        __threadfence();
#pragma unroll
        for (int q = 0; q < PPT; ++q)
          if (in[q]) {
            const int pi = (py[q] - oy) * TILE + (px[q] - ox);
            typename PS::State m;
            swr_ld_state(m, ss + pi);
            for (int sl = 1; sl < nsl; ++sl) {
              typename PS::State o;
              swr_ld_state(o, ss + (size_t)sl * (TILE * TILE) + pi);
              swr_depth_merge(m, o);
            }
            PS::store(m, px[q], py[q], U);
          }
        if (threadIdx.x == 0) g.dslice_done[dslot] = 0u;  // ready for the next draw
      }
      uint32_t tot, ptot;
      swr_block_sum2(frags, passes, sfr, tot, ptot);
      if (threadIdx.x == 0 && tot) {
        atomicAdd((unsigned long long*)&g.status_w[SWR_ST_SHADED_LO], (unsigned long long)tot);
        atomicAdd((unsigned long long*)&g.status_w[SWR_ST_PASSES_LO], (unsigned long long)ptot);
      }
      return true;
    }
  }
#pragma unroll
  for (int q = 0; q < PPT; ++q)
    if (in[q]) {
      PS::store(st[q], px[q], py[q], U);
      passes += st[q].writes;
    }
  // fragment statistics: drawPixel calls and colour writes
  uint32_t tot, ptot;
  swr_block_sum2(frags, passes, sfr, tot, ptot);
  if (threadIdx.x == 0 && tot) {
    atomicAdd((unsigned long long*)&g.status_w[SWR_ST_SHADED_LO], (unsigned long long)tot);
    atomicAdd((unsigned long long*)&g.status_w[SWR_ST_PASSES_LO], (unsigned long long)ptot);
  }
  return true;
}

// (32-px tiles: four pixels a thread want the registers of four CTAs per SM, whatever the shader.
// Planned for as many as 16-px tiles, the Lambert, Lambert-textured and differentiable shaders
// spilled: 2,000 triangles of 300 px at 640x480 in Adaptive mode, Lambert-textured, 1042 us a draw
// with six CTAs, 773 with four.)
template <class PS, int TILE, int CH, bool SPAN, bool DIRECT = false, int NT = 256>
__global__ void __launch_bounds__(NT, SWR_RASTER_MINB ? SWR_RASTER_MINB
                                       : TILE == 32      ? 4
                                       : SPAN            ? SwrRasterOccupancy<PS>::value
                                                         : SwrRasterOccupancy<PS>::block * (256 / NT))
    k_raster(RasterArgs g) {
  swr_pdl_entry();
  raster_tile<PS, TILE, CH, SPAN, DIRECT, NT>(g, blockIdx.x);
}

// Draws of more than SWR_RASTER_LOOP tiles: a CTA for every two, which rasterizes its entry of
// the list and the one a grid further on.  Meshes leave most of a batch's tiles empty, and a CTA
// that finds none costs 1 ns of launching: 256 meshes of 491,520 tiles took 2741 us, this way
// 2540 (one for every four tiles or eight: 1 % slower).  Up to the line two tiles a CTA lose (32,400
// tiles of a soup 4134 -> 4185 us).  Above it they lose only where no tile is empty and the CTAs
// are of 128 threads; how many are empty the host does not know.  One target, us a draw with one
// tile a CTA / two: 129,600 tiles, 1M-triangle soup in Block mode 3913 / 3852, in Span mode
// 3409 / 3436; Lambert-textured in Block mode, 262,144 small triangles 683 / 721, 16,384 of them
// 273 / 227; 262,144 tiles 1133 / 1189 and 426 / 313.
#ifndef SWR_RASTER_LOOP
#define SWR_RASTER_LOOP 65536
#endif
template <class PS, int CH, bool SPAN, int NT>
__global__ void __launch_bounds__(NT, SWR_RASTER_MINB ? SWR_RASTER_MINB
                                       : SPAN            ? SwrRasterOccupancy<PS>::value
                                                         : SwrRasterOccupancy<PS>::block * (256 / NT))
    k_raster_two(RasterArgs g) {
  swr_pdl_entry();
  for (uint32_t bid = blockIdx.x; bid < g.ntiles && raster_tile<PS, 16, CH, SPAN, false, NT>(g, bid); bid += gridDim.x)
    __syncthreads();  // the tile's shared state is no longer read
}

// ---------------------------------------------------------------------------------
// Overwrite shaders (SwrOverwrite): a pixel ends with the colour of its last covering
// primitive -- the one with the largest id -- and with the number of primitives covering it.
// Neither needs the bin in order, and only one fragment per pixel needs shading.
//
// One CTA per tile, or g.slices CTAs over parts of a tile's bin of more than SWR_RASTER_SORT
// entries.  Entries are taken from the bin's end (the largest ids up to the order inside a
// cell); an entry adds up the lengths of its rows' runs here and writes its id over smaller
// ones in the tile's winners, and once every pixel has a winner, entries below all of them only
// count.  The last CTA of a tile shades its winners.
//
// Of 128 entries and more, a thread first classifies one each: a Span primitive whose two end
// rows per half show that it misses the tile's columns or covers all of them, and that can win
// no pixel, is counted there.  The others are listed and walked four rows a work item; walked
// by one thread each, a warp waited for the tallest of its 32 (17 lanes active; the 40,960
// large triangles below: 257 us, 210 this way).  Fewer entries are split into rows at once, down
// to single ones (a small draw's large triangles would leave one thread walking 256 pixels).
// Nothing is staged: a record is read from the cache by the threads that need it.
//
// Bound by latency: the record reads and the barriers around the lists, at five CTAs per SM
// (four, with all the registers wanted: 354 us a draw, five 333).  The 40,960 triangles of the
// reference's Benchmark program (640x480, 240M fragments): bins ordered and walked in
// 64-primitive chunks pixel by pixel, 1888 us a draw; this way 333.
//
// MASKS: some draw is in Block or Adaptive mode.
template <class PS, int TILE, bool DIRECT, bool MASKS>
__global__ void __launch_bounds__(256, 5) k_overwrite(RasterArgs g) {
  swr_pdl_entry();
  typedef Rec<PS> RL;
  constexpr int PPT = TILE * TILE / 256;
  static_assert(RL::R >= 20, "words 0-19 of a record are read as five float4s");
  static_assert(PPT == 1 || TILE * TILE <= 1024, "a tile's pixels are listed in swalk");
  __shared__ uint32_t sbest[TILE * TILE];      // per pixel: winner's id + 1
  __shared__ int scnt[TILE * (TILE + 1)];      // per row: +1 at a run's first pixel, -1 past its last
  __shared__ uint32_t sred[8];
  __shared__ uint32_t sfr[32];
  __shared__ uint32_t slast;
  constexpr uint32_t OVB = 1024;  // entries classified at a time
  __shared__ uint32_t swalk[OVB], snwalk;
  // Block primitives' coverage masks, as k_raster's, LIGHT primitives at a time
  constexpr int NBX = TILE / SWR_BLOCK, NB = NBX * NBX;
  constexpr uint32_t LIGHT = 32;
  __shared__ uint64_t smask[MASKS ? LIGHT * NB : 1];
  // the draw's queue requests are final (nothing after this stage counts)
  if (blockIdx.x == 0 && threadIdx.x == 0 && !DIRECT) swr_close_status(g.status_w);
  if (g.status[SWR_ST_FLAGS] & SWR_F_ANY_OVERFLOW) return;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t tile = blockIdx.x, slice = 0, n = 0, hi = 0;
  int nsl = 1, ti = 0;
  if constexpr (DIRECT) {
    n = min(g.status[SWR_ST_PRIMS], g.cap_prims);
    if (!direct_any(g.boxes, n, tile, (uint32_t)g.targets[0].tiles_x)) return;
  } else {
    if (g.slices > 1) {
      tile = blockIdx.x / (uint32_t)g.slices;
      slice = blockIdx.x - tile * (uint32_t)g.slices;
    }
    uint32_t b, e;
    if (g.tiles.list) {
      uint4 entry;
      if (!swr_listed_tile(g.tiles, tile, entry)) return;
      tile = entry.x;
      b = entry.y;
      e = entry.z;
      ti = (int)entry.w;
    } else {
      if (tile >= g.ntiles) return;
      b = g.tile_start[tile];
      e = g.tile_start[tile + 1];
    }
    hi = e;
    n = e - b;
    if (n > (uint32_t)SWR_RASTER_SORT && g.slices > 1) {
      nsl = g.slices;
      const uint32_t lo = b + (uint32_t)((uint64_t)n * slice / (uint32_t)nsl);
      hi = b + (uint32_t)((uint64_t)n * (slice + 1) / (uint32_t)nsl);
      n = hi - lo;
    } else if (slice) {
      return;
    }
  }
  if (tile >= g.ntiles || n == 0) return;  // (a slice of more than SWR_RASTER_SORT entries is never empty)
  const SwrTargetDesc& T = g.targets[ti];
  const SwrUniforms& U = g.draws[T.first_draw].u;
  const uint32_t lt = tile - T.tile_base;
  const uint32_t tx = lt % (uint32_t)T.tiles_x, ty = lt / (uint32_t)T.tiles_x;
  const int ox = (int)tx * TILE, oy = (int)ty * TILE;
  const int xend = min(ox + TILE, T.width), yend = min(oy + TILE, T.height);
  const bool counts = U.frag_count != nullptr;
#pragma unroll
  for (int q = 0; q < PPT; ++q) sbest[q * 256 + tid] = 0u;
  for (int i = tid; i < TILE * (TILE + 1); i += 256) scnt[i] = 0;
  __syncthreads();
  uint32_t smin = 0;  // no pixel's winner is below it
  uint32_t frags = 0;
  // Part `part` of 2^lp of primitive p in the tile: a share of the rows, in Block mode block after
  // block.
  auto cover = [&](uint32_t p, int part, int lp, bool span_only = false) {
    const float4* rc = (const float4*)(g.recs + (size_t)p * RL::R);
    const float4 q0 = __ldg(rc), q1 = __ldg(rc + 1), q2 = __ldg(rc + 2), q3 = __ldg(rc + 3), q4 = __ldg(rc + 4);
    const int flags = __float_as_int(q0.x);
    if (!(flags & 1)) return;
    const uint32_t key = p + 1u;
    auto run = [&](int y, int xa, int xb) {
      const int row = y - oy;
      frags += (uint32_t)(xb - xa);
      if (key > smin)
        for (int i = row * TILE + xa - ox; i < row * TILE + xb - ox; ++i)
          if (*(volatile uint32_t*)&sbest[i] < key) atomicMax(&sbest[i], key);
      if (counts) {
        atomicAdd(&scnt[row * (TILE + 1) + xa - ox], 1);
        atomicAdd(&scnt[row * (TILE + 1) + xb - ox], -1);
      }
    };
    if (!(flags & 2)) {
      const int rows = TILE >> lp, y0 = oy + part * rows, y1 = min(y0 + rows, yend);
      const SwrDrawDesc& D = g.draws[__float_as_int(q0.y)];
      span_runs(q0, q1, q2, q3, q4, D.sc_minx, D.sc_maxx, ox, xend, y0, y1,
                [&](int y, int xa, int xb, int) { run(y, xa, xb); });
      return;
    }
    if (span_only || (!MASKS && !DIRECT)) return;  // (without MASKS a binned draw has no Block primitives)
    const float r[15] = {0, 0, 0, 0, 0, 0, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z};
    constexpr int ROWS = SWR_BLOCK * NB;  // the blocks' rows, block by block
    for (int h = part * (ROWS >> lp), he = h + (ROWS >> lp); h < he;) {
      const int j = h / SWR_BLOCK, r0 = h % SWR_BLOCK, r1 = min(r0 + he - h, SWR_BLOCK);
      h += r1 - r0;
      const int bx = ox + (j % NBX) * SWR_BLOCK, by = oy + (j / NBX) * SWR_BLOCK;
      const int ylo = max(by + r0, __float_as_int(q0.w)), yhi = min(min(by + r1, __float_as_int(q1.y) + 1), yend);
      if (ylo >= yhi || bx >= xend || bx > __float_as_int(q1.x) || bx + SWR_BLOCK - 1 < __float_as_int(q0.z)) continue;
      const int cls = block_class(r, flags, bx, by);
      if (cls) block_runs(r, flags, cls, bx, by, min(SWR_BLOCK, xend - bx), ylo, yhi, run);
    }
  };
  int round = 0;
  auto raise_smin = [&]() {  // (uniform)
    __syncthreads();
    uint32_t m = 0xffffffffu;
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
      const int i = q * 256 + tid;
      if (ox + i % TILE < xend && oy + i / TILE < yend) m = min(m, sbest[i]);
    }
    m = __reduce_min_sync(0xffffffffu, m);
    if (lane == 0) sred[warp] = m;
    __syncthreads();
    smin = sred[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) smin = min(smin, sred[w]);
  };
  // Whether primitive p has to be walked row by row.  A Span primitive whose halves each miss
  // the tile's columns or cover all of theirs, in all the rows they have here, only adds its
  // fragments: an extent's ends are monotone functions of the row within a half (every
  // operation of span_row is, for finite slopes), so the end rows tell.
  auto classify = [&](uint32_t p) -> bool {
    const float4* rc = (const float4*)(g.recs + (size_t)p * RL::R);
    const float4 q0 = __ldg(rc), q1 = __ldg(rc + 1), q2 = __ldg(rc + 2), q3 = __ldg(rc + 3), q4 = __ldg(rc + 4);
    const int flags = __float_as_int(q0.x);
    if (!(flags & 1)) return false;
    if (flags & 2) return true;
    const SwrDrawDesc& D = g.draws[__float_as_int(q0.y)];
    const int ylo = max(__float_as_int(q0.w), oy), yhi = min(__float_as_int(q1.y) + 1, yend);
    const int cx0 = max(__float_as_int(q0.z) & ~(SWR_BLOCK - 1), ox);
    const int cx1 = min((__float_as_int(q1.x) | (SWR_BLOCK - 1)) + 1, xend);
    if (cx0 >= cx1) return false;
    bool walk = false;
    int area = 0, fy0[2], fy1[2];  // covered rows of each half
    int pb1 = INT_MIN, pb0 = INT_MAX;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      SpanHalf hf;
      hf.ox = t ? q3.z : q2.x; hf.oy = t ? q3.w : q2.y; hf.is1 = t ? q4.x : q2.z; hf.is2 = t ? q4.y : q2.w;
      int y0 = t ? __float_as_int(q3.y) : __float_as_int(q1.z), y1 = t ? __float_as_int(q3.x) : __float_as_int(q1.w);
      if (t) { y0 = y0 < INT_MAX ? y0 + 1 : y0; y1 = y1 < INT_MAX ? y1 + 1 : y1; }  // (y1, y0] as [y1 + 1, y0 + 1)
      y0 = max(y0, ylo);
      y1 = min(y1, yhi);
      fy0[t] = fy1[t] = 0;
      if (!(flags & (t ? 64 : 32)) || y0 >= y1) continue;
      if (t && y0 < pb1 && y1 > pb0) walk = true;  // rows of both halves
      pb0 = y0;
      pb1 = y1;
      int a0, b0, a1, b1;
      span_row(hf, y0, D.sc_minx, D.sc_maxx, a0, b0);
      span_row(hf, y1 - 1, D.sc_minx, D.sc_maxx, a1, b1);
      if (!(fabsf(hf.is1) < 0x1p100f && fabsf(hf.is2) < 0x1p100f)) {
        walk = true;
      } else if (max(a0, a1) <= cx0 && min(b0, b1) >= cx1) {
        area += (y1 - y0) * (cx1 - cx0);
        fy0[t] = y0;
        fy1[t] = y1;
      } else if (!(max(b0, b1) <= cx0 || min(a0, a1) >= cx1)) {
        walk = true;
      }
    }
    if (walk || (area && p + 1u > smin)) return true;
    frags += (uint32_t)area;
    if (counts && area)
#pragma unroll
      for (int t = 0; t < 2; ++t)
        for (int y = fy0[t]; y < fy1[t]; ++y) {
          atomicAdd(&scnt[(y - oy) * (TILE + 1) + cx0 - ox], 1);
          atomicAdd(&scnt[(y - oy) * (TILE + 1) + cx1 - ox], -1);
        }
    return false;
  };
  // parts of a primitive: see above (n << shift items in all)
  const int shift = n >= 128u ? 0 : (n >= 32u ? 2 : n >= 16u ? (TILE == 16 ? 3 : 4) : (TILE == 16 ? 4 : 5));
  const uint32_t* bin = g.bin_raw ? g.bin_raw : g.bin;
  const uint64_t items = (uint64_t)n << shift;
  if (MASKS && (!g.has_span || n < 400u)) {
    // Block primitives by masks, LIGHT at a time: one thread per (primitive, block) classifies it,
    // one per half of a partially covered block steps its rows, and each pixel takes the largest of
    // the ids covering it.  Scattered by their rows like Span primitives, lanes at skipped, whole
    // and partial blocks waited for each other: 40,960 triangles of 60 px, us a draw so / this
    // way: 640x480 510 / 225, 1920x1080 468 / 229, 3840x2160 1222 / 343, 4080x4080 1756 / 516.
    // Tiles of more entries in a draw that has Span primitives too scatter both, since those only
    // count once every pixel's winner is known (40,960 triangles of 300 px in Adaptive mode at
    // 640x480: 1760, all by masks 2490).
    if (g.has_span)
      for (uint32_t t = (uint32_t)tid; t < n << shift; t += 256)
        cover(bin[hi - 1u - (t >> shift)], (int)(t & ((1u << shift) - 1u)), shift, true);
    for (uint32_t base = 0; base < n; base += LIGHT) {
      const uint32_t m = min(LIGHT, n - base);
      __syncthreads();  // the previous masks and ids are no longer read; Span's winners are written
      if (tid == 0) snwalk = 0u;
      if ((uint32_t)tid < m) swalk[tid] = bin[hi - 1u - (base + (uint32_t)tid)];
      __syncthreads();
      auto block_of = [&](uint32_t t, int& bx, int& by) -> const float* {
        const int j = (int)(t % NB);
        bx = ox + (j % NBX) * SWR_BLOCK;
        by = oy + (j / NBX) * SWR_BLOCK;
        return g.recs + (size_t)swalk[t / NB] * RL::R;
      };
      for (uint32_t t = (uint32_t)tid; t < m * NB; t += 256) {
        int bx, by;
        const float* r = block_of(t, bx, by);
        const float4 q0 = __ldg((const float4*)r), q1 = __ldg((const float4*)r + 1);
        const int flags = __float_as_int(q0.x);
        int cls = 0;
        if ((flags & 3) == 3 && bx <= __float_as_int(q1.x) && bx + SWR_BLOCK - 1 >= __float_as_int(q0.z) &&
            by <= __float_as_int(q1.y) && by + SWR_BLOCK - 1 >= __float_as_int(q0.w))
          cls = block_class(r, flags, bx, by);
        smask[t] = cls == 1 ? ~0ull : 0ull;
        if (cls == 2) swalk[LIGHT + atomicAdd(&snwalk, 1u)] = t;
      }
      __syncthreads();
      const uint32_t halves = 2u * snwalk;
      for (uint32_t h = (uint32_t)tid; h < halves; h += 256) {
        int bx, by;
        const uint32_t t = swalk[LIGHT + (h >> 1)];
        const float* r = block_of(t, bx, by);
        ((uint32_t*)&smask[t])[h & 1u] = block_rows_bits(r, __float_as_int(r[0]), bx, by, (int)(h & 1u));
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < PPT; ++q) {
        const int reg = q * 8 + warp, sub = reg >> 3, hb = (reg & 7) >> 1;  // the warp's half block (raster_tile)
        const int lx = (sub % (TILE / 16)) * 16 + (hb & 1) * 8 + (lane & 7);
        const int ly = (sub / (TILE / 16)) * 16 + (hb >> 1) * 8 + (reg & 1) * 4 + (lane >> 3);
        const int blk = (ly >> 3) * NBX + (lx >> 3);
        uint32_t cov = warp_transpose((uint32_t)lane < m ? (uint32_t)(smask[lane * NB + blk] >> ((reg & 1) * 32)) : 0u, lane);
        if (ox + lx >= xend || oy + ly >= yend || !cov) continue;
        const uint32_t c = (uint32_t)__popc(cov);
        frags += c;
        uint32_t b = sbest[ly * TILE + lx];
        for (; cov; cov &= cov - 1u) b = max(b, swalk[__ffs(cov) - 1] + 1u);
        sbest[ly * TILE + lx] = b;
        if (counts) {
          uint32_t* fc = U.frag_count + (size_t)(oy + ly) * (size_t)U.width + (size_t)(ox + lx);
          if (nsl > 1) atomicAdd(fc, c); else *fc += c;
        }
      }
    }
  } else if (shift == 0) {
    for (uint32_t base = 0; base < n; ++round) {
      const uint32_t m = min(n - base, round < 3 ? 256u : OVB);
      __syncthreads();  // the previous list is no longer read
      if (tid == 0) snwalk = 0u;
      __syncthreads();
      for (uint32_t k0 = 0; k0 < m; k0 += 256) {
        const uint32_t k = k0 + (uint32_t)tid;
        const uint32_t p = k >= m ? 0u : DIRECT ? n - 1u - (base + k) : bin[hi - 1u - (base + k)];
        const bool walk = k < m && (!DIRECT || swr_box_hit(g.boxes[p], tx, ty)) && classify(p);
        const uint32_t bal = __ballot_sync(0xffffffffu, walk);
        uint32_t at = 0;
        if (lane == 0 && bal) at = atomicAdd(&snwalk, (uint32_t)__popc(bal));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (walk) swalk[at + (uint32_t)__popc(bal & ((1u << lane) - 1u))] = p;
      }
      __syncthreads();
      // four rows an item; few primitives of a small draw's window: one
      constexpr int LT = TILE == 16 ? 4 : 5;
      const int lp = DIRECT && snwalk < 32u ? LT : LT - 2;
      const uint32_t work = snwalk << lp;
      for (uint32_t t = (uint32_t)tid; t < work; t += 256) cover(swalk[t >> lp], (int)(t & ((1u << lp) - 1u)), lp);
      base += m;
      // (a later, larger bound would save little; nothing was walked: there is no larger one)
      if (round < 3 && base < n && snwalk) raise_smin();
    }
  } else
  for (uint64_t base = 0; base < items; base += 256, ++round) {
    const uint64_t it = base + (uint64_t)tid;
    if (it < items) {
      const uint32_t k = (uint32_t)(it >> shift);
      const int part = (int)((uint32_t)it & ((1u << shift) - 1u));
      if constexpr (DIRECT) {
        const uint32_t p = n - 1u - k;
        if (swr_box_hit(g.boxes[p], tx, ty)) cover(p, part, shift);
      } else {
        cover(bin[hi - 1u - k], part, shift);
      }
    }
    if (round < 3 && base + 256 < items) raise_smin();
  }
  __syncthreads();
  uint32_t tot;
  swr_block_exscan(frags, sfr, &tot);
  if (tid == 0 && tot) {  // every fragment writes
    atomicAdd((unsigned long long*)&g.status_w[SWR_ST_SHADED_LO], (unsigned long long)tot);
    atomicAdd((unsigned long long*)&g.status_w[SWR_ST_PASSES_LO], (unsigned long long)tot);
  }
  uint32_t best[PPT];
#pragma unroll
  for (int q = 0; q < PPT; ++q) {
    const int i = q * 256 + tid;
    const int x = ox + i % TILE, y = oy + i / TILE;
    best[q] = sbest[i];
    if (!counts || x >= xend || y >= yend) continue;
    int c = 0;
    for (int k = 0; k <= i % TILE; ++k) c += scnt[(i / TILE) * (TILE + 1) + k];
    if (!c) continue;
    uint32_t* fc = U.frag_count + (size_t)y * (size_t)U.width + (size_t)x;
    if (nsl > 1) atomicAdd(fc, (uint32_t)c); else *fc += (uint32_t)c;
  }
  if (nsl > 1) {
    uint32_t* gb = g.best + (size_t)tile * (TILE * TILE);
#pragma unroll
    for (int q = 0; q < PPT; ++q)
      if (best[q]) atomicMax(&gb[q * 256 + tid], best[q]);
    __threadfence();
    __syncthreads();
    if (tid == 0) slast = atomicAdd(&g.best_done[tile], 1u) == (uint32_t)(nsl - 1);
    __syncthreads();
    if (!slast) return;
    __threadfence();
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
      best[q] = __ldcg(&gb[q * 256 + tid]);
      if (best[q]) gb[q * 256 + tid] = 0u;  // ready for the next draw
    }
    if (tid == 0) g.best_done[tile] = 0u;
  }
  // A thread's pixels are shaded one after the other: where it has several, the tile's winners are
  // first dealt out over the CTA (few of a tile's pixels may have one).
  uint32_t shade = PPT;
  if constexpr (PPT > 1) {
    __syncthreads();  // swalk and sbest are no longer read
    if (tid == 0) snwalk = 0u;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < PPT; ++q) {
      const int i = q * 256 + tid;
      const bool on = best[q] && ox + i % TILE < xend && oy + i / TILE < yend;
      const uint32_t bal = __ballot_sync(0xffffffffu, on);
      uint32_t at = 0;
      if (lane == 0 && bal) at = atomicAdd(&snwalk, (uint32_t)__popc(bal));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (on) swalk[at + (uint32_t)__popc(bal & ((1u << lane) - 1u))] = (uint32_t)i;
      sbest[i] = best[q];
    }
    __syncthreads();
    shade = (snwalk + 255u) / 256u;
  }
  for (uint32_t q = 0; q < shade; ++q) {
    int i = tid;
    uint32_t b = best[0];
    if constexpr (PPT > 1) {
      const uint32_t t = q * 256u + (uint32_t)tid;
      if (t >= snwalk) break;
      i = (int)swalk[t];
      b = sbest[i];
    }
    const int x = ox + i % TILE, y = oy + i / TILE;
    if (!b || x >= xend || y >= yend) continue;
    const uint32_t p = b - 1u;
    const float* r = g.recs + (size_t)p * RL::R;
    GpuPixel<PS> pd;
    pd.z = 0.0f;  // (no depth: SwrOverwrite)
    pixel_of_record<PS, true>(r, g.draws, x, y, pd);
    typename PS::State st;
    PS::load(st, x, y, U);
    PS::apply(st, pd.z, PS::shade(pd, g.draws[__float_as_int(r[1])].u), prim_id(g, r, p));
    st.frags = 0;  // counted above
    PS::store(st, x, y, U);
  }
}

}  // namespace swr
