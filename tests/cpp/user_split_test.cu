// A caller's own shaders drawn in one call and in many calls of a few primitives each: their
// framebuffers must be the same bytes, since primitives reach drawPixel in submission order either
// way.  (Triangles outside the frustum in part are left out: the fans they are clipped to are drawn
// at the end of their batch of 1,024, VertexProcessor.cpp:227-262, which a call of a few ends.)  Covers what only large draws reach: pixels of a warp visiting shared and own primitives
// (Span mode, large and small triangles), 32-px tiles, and tiles of thousands of points' and lines'
// fragments.
#include <swr/Renderer.h>

#include <cstdio>
#include <limits>
#include <vector>

#include "user_scene.h"
#include "user_shaders.h"

namespace {

constexpr int W = 200, H = 120;

void cuda_ok(cudaError_t e) {
  if (e != cudaSuccess) {
    fprintf(stderr, "%s\n", cudaGetErrorString(e));
    exit(2);
  }
}

void abi_ok(int rc) {
  if (rc != SWR_OK) {
    fprintf(stderr, "%s\n", swr_status_string(rc));
    exit(3);
  }
}

template <class T>
T* to_device(const std::vector<T>& v) {
  T* p = nullptr;
  cuda_ok(cudaMalloc(&p, v.size() * sizeof(T)));
  cuda_ok(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
  return p;
}

struct Case {
  int mode, raster, tile, n;
  float size;        // extent of a primitive in pixels
  float x0, x1, y0, y1;  // where they lie
};

// Buffers after drawing the case in calls of `piece` primitives.
template <class PS>
std::vector<uint32_t> draw(const Case& k, int piece, UserTarget t) {
  const int per = k.mode + 1;
  UserLcg g(77);
  std::vector<float> pos;
  std::vector<uint32_t> attr;
  std::vector<int> idx;
  for (int i = 0; i < k.n; ++i) {
    const float cx = k.x0 + g.unit() * (k.x1 - k.x0), cy = k.y0 + g.unit() * (k.y1 - k.y0);
    bool inside = true;
    for (int j = 0; j < per; ++j) {
      const float x = cx + (g.unit() - 0.5f) * k.size, y = cy + (g.unit() - 0.5f) * k.size;
      pos.insert(pos.end(), {x / (W * 0.5f) - 1.0f, 1.0f - y / (H * 0.5f), (float)(g.next() % 8) / 8.0f - 0.5f, g.unit()});
      attr.insert(attr.end(), {g.next() | 0xff000000u, user_float_bits(g.unit()), user_float_bits(g.unit())});
      inside = inside && x > 0.5f && x < W - 0.5f && y > 0.5f && y < H - 0.5f;
    }
    for (int j = 0; j < per && (inside || k.mode != SWR_DRAW_TRIANGLE); ++j) idx.push_back(per * i + j);
  }
  const int prims = (int)idx.size() / per;
  cuda_ok(cudaMemset(t.color, 0, W * H * 4));
  cuda_ok(cudaMemset(t.count, 0, W * H * 4));
  std::vector<float> inf(W * H, std::numeric_limits<float>::infinity());
  cuda_ok(cudaMemcpy(t.depth, inf.data(), W * H * 4, cudaMemcpyHostToDevice));
  swr_context* c = nullptr;
  abi_ok(swr_create(&c));
  abi_ok(swr_set_vertex_program(c, swr::vertex_program<FogVS>()));
  abi_ok(swr_set_pixel_program(c, swr::pixel_program<PS>()));
  abi_ok(swr_set_tile_size(c, k.tile));
  abi_ok(swr_set_raster_mode(c, k.raster));
  abi_ok(swr_set_scissor_rect(c, 0, 0, W, H));
  abi_ok(swr_set_viewport(c, 0, 0, W, H));
  abi_ok(swr_set_cull_mode(c, SWR_CULL_NONE));
  SwrUniforms u;
  memset(&u, 0, sizeof(u));
  u.width = W;
  u.height = H;
  u.color = (void*)&u;  // a target key only
  abi_ok(swr_set_uniforms(c, &u));
  float* p0 = to_device(pos);
  uint32_t* p1 = to_device(attr);
  int* di = to_device(idx);
  abi_ok(swr_set_vertex_attrib_pointer(c, 0, 16, p0, pos.size() * 4));
  abi_ok(swr_set_vertex_attrib_pointer(c, 1, 12, p1, attr.size() * 4));
  for (int at = 0; at < prims; at += piece) {
    const int m = piece < prims - at ? piece : prims - at;
    for (int attempt = 0;; ++attempt) {
      abi_ok(swr_draw_elements(c, k.mode, (uint64_t)m * per, (const uint32_t*)di + (size_t)at * per, nullptr));
      const int rc = swr_finish(c, nullptr, nullptr);
      if (rc == SWR_EOVERFLOW && attempt < 3) continue;
      abi_ok(rc);
      break;
    }
  }
  std::vector<uint32_t> out(3 * W * H);
  cuda_ok(cudaMemcpy(out.data(), t.color, W * H * 4, cudaMemcpyDeviceToHost));
  cuda_ok(cudaMemcpy(out.data() + W * H, t.depth, W * H * 4, cudaMemcpyDeviceToHost));
  cuda_ok(cudaMemcpy(out.data() + 2 * W * H, t.count, W * H * 4, cudaMemcpyDeviceToHost));
  cudaFree(p0);
  cudaFree(p1);
  cudaFree(di);
  abi_ok(swr_destroy(c));
  return out;
}

template <class PS>
int check(const Case& k, int piece, UserTarget t, const char* name) {
  const std::vector<uint32_t> whole = draw<PS>(k, k.n, t), parts = draw<PS>(k, piece, t);
  size_t bad = 0, hit = 0;
  for (size_t i = 0; i < whole.size(); ++i) {
    bad += whole[i] != parts[i];
    hit += i >= 2 * W * H && whole[i] != 0;
  }
  if (bad || !hit)
    printf("%s mode %d raster %d tile %d n %d size %g: %zu words differ, %zu pixels hit\n", name, k.mode, k.raster,
           k.tile, k.n, k.size, bad, hit);
  return bad || !hit;
}

}  // namespace

int main() {
  UserTarget t = {nullptr, nullptr, nullptr, W, H};
  cuda_ok(cudaMalloc(&t.color, W * H * 4));
  cuda_ok(cudaMalloc(&t.depth, W * H * 4));
  cuda_ok(cudaMalloc(&t.count, W * H * 4));
  cuda_ok(cudaMemcpyToSymbol(g_target, &t, sizeof(t)));
  const float mvp[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1};
  cuda_ok(cudaMemcpyToSymbol(g_mvp, mvp, sizeof(mvp)));
  int bad = 0;
  for (int raster = 0; raster < 3; ++raster)
    for (int tile : {16, 32})
      for (float size : {7.0f, 30.0f, 250.0f}) {
        const Case k = {SWR_DRAW_TRIANGLE, raster, tile, 1500, size, -10, W + 10, -10, H + 10};
        bad += check<StripePS>(k, 37, t, "stripe");
        bad += check<LastWriterPS>(k, 101, t, "last writer");
      }
  // points and lines: over the target, and thousands of fragments in one tile and in a few
  for (int mode : {SWR_DRAW_POINT, SWR_DRAW_LINE}) {
    const Case ks[3] = {{mode, 0, 16, 5000, 40.0f, 0, W, 0, H},
                        {mode, 0, 16, 12000, 4.0f, 20, 28, 20, 28},
                        {mode, 0, 16, 12000, 6.0f, 180, W, 110, H}};
    for (const Case& k : ks) {
      bad += check<StripePS>(k, 300, t, "stripe");
      bad += check<LastWriterPS>(k, 300, t, "last writer");
    }
  }
  printf(bad ? "%d cases differ\n" : "ok\n", bad);
  return bad != 0;
}
