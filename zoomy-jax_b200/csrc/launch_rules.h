// Launch shapes chosen on the host from sizes alone: plain C++ without CUDA, so that
// they can be checked on any machine over the whole range of sizes.
#pragma once

#include <algorithm>

namespace zb {

// A multigrid level on strips (csrc/poisson.cu, mg_down_strip / mg_up_strip): strips of
// `cols` columns over items of `rows` rows, four items a CTA.
struct MgStrips {
  int strips, rows, ctas;
  bool dot;   // the way up leaves its partial sums of z.q, one per CTA
};

// The rows of an item spread the level over two warps per scheduler (1184), four rows at
// least, 64 at most; even, because the pipeline restricts pairs of rows.  With `dot` the
// CTAs' partial sums have to fit `parts` slots: items grow until they do, at most to the
// level's height.  A level of more than 4 x parts strips does not fit even then (8 rows
// and 900,000 columns): it keeps its shape and a pass of its own forms z.q.
inline MgStrips mg_strips(int nx, int ny, int cols, bool dot, int parts) {
  MgStrips s;
  s.strips = (ny + cols - 1) / cols;
  const int want = (int)((long long)s.strips * nx / 1184 + 1) & ~1;
  auto ctas = [&](int rows) {
    return (int)(((long long)s.strips * (((long long)nx + rows - 1) / rows) + 3) / 4);
  };
  s.rows = std::min(std::max(4, want), 64);
  s.dot = dot;
  if (dot) {
    int r = s.rows;
    while (ctas(r) > parts && r < nx) r *= 2;   // r < 2 nx, nx < 2^30
    s.dot = ctas(r) <= parts;
    if (s.dot) s.rows = r;
  }
  s.ctas = ctas(s.rows);
  return s;
}

// Channels that one launch of an elementwise kernel with a 32-bit index takes of
// [channels][pixels] planes: at most 2^31 elements, so that the index plus a grid's stride
// stays below 2^32.  (16, 16) networks train on batches of up to 2.8e8 pixels in 180 GB,
// more than 2^32 elements of 16 channels; every usual batch is one launch.
inline int plane_slice(int channels, long long pixels) {
  return (int)std::max(1LL, std::min<long long>(channels, (1LL << 31) / pixels));
}

}  // namespace zb
