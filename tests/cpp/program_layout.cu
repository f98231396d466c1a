// Prints swr_program_layout() and the size of every argument structure that the launchers of a
// caller's shader program exchange with the library (tests/test_program_layout.py).
#include "../../softwarerenderer_gb300/csrc/swr_ops.h"

#include <cstdio>

int main() {
  const int n = (int)(sizeof(swr_program().sizes) / 4);
  uint32_t s[64] = {};
  swr_program_layout(s);
  printf("layout");
  for (int i = 0; i < n; ++i) printf(" %u", s[i]);
#define SIZE(t) printf("\n%s %zu", #t, sizeof(t))
  SIZE(swr::VsOps);
  SIZE(swr::PsOps);
  SIZE(SwrDrawDesc);
  SIZE(SwrTargetDesc);
  SIZE(SwrUniforms);
  SIZE(SwrCells);
  SIZE(swr::AssembleArgs);
  SIZE(swr::FrontArgs);
  SIZE(swr::DirectArgs);
  SIZE(swr::SetupArgs);
  SIZE(swr::RasterArgs);
  SIZE(swr::LpFragArgs);
  SIZE(swr::LpRasterArgs);
  printf("\n");
  return 0;
}
