// Launch shapes chosen on the host from sizes alone: plain C++ without CUDA, so that
// they can be checked on any machine over the whole range of sizes.
#pragma once

#include <algorithm>
#include <cmath>

#ifdef __CUDACC__
#define ZB_HOST_DEVICE __host__ __device__
#else
#define ZB_HOST_DEVICE
#endif

namespace zb {

// ── order-2 stages of a Cartesian grid (csrc/swe2d.cu) ──────────────────────
constexpr int SW = 28;          // output columns per strip

// The strips of a full-coverage grid whose lanes 28 s - 2 .. 28 s + 29 all lie
// inside it (strips 1 .. the count).
ZB_HOST_DEVICE inline int full_mid_strips(int ny) {
  const int ns = (ny + SW - 1) / SW, mh = ny >= 30 ? (ny - 30) / SW : 0;
  return mh > ns - 1 ? ns - 1 : mh;
}

// Row-chunk heights of a single grid's items.  An item of S rows marches S + 4
// (two halo rows each side): long chunks save halo rows, short ones spread a
// small grid over more warps.  A row of a CTA (four items) takes about a + b k,
// k the CTAs on its SM -- a lone warp is bound by its own dependent
// instructions, so the first CTA costs most (float32 1 + 0.3 k us for the two
// stages, k <= 4; float64 2.6 + 0.7 k, k <= 2; fitted to 250 timings of 15 grid
// sizes, mean error 5 %).  The height is the least modelled time over the
// candidates: whole waves of interior CTAs, the last wave with the boundary
// CTAs beside it, and a tail where those do not fit.  Measured on a B200 (us per
// step, minmod eta / HLL-HR; 64 rows everywhere after it): float32 512^2 25 / 94,
// 1024^2 59 / 97, 1448^2 93 / 137, 2048^2 174 / 174; float64 512^2 62 / 230,
// 1024^2 177 / 245, 2048^2 571 / 571; over the 15 sizes within 0.5 % (float64
// 2 %) of the best of ten fixed heights on average.
// A grid of fewer than 6 x 592 strip rows (about 300^2) takes the general body
// everywhere in one uniform list: its two-row boundary items and four-row
// boundary chunks would outlast the rest (256^2 float32 17.6 against 20.5,
// 64^2 14 against 20; 400^2 24 against 22.6).  So does a grid without a middle
// strip (fewer than 58 columns), where every item is a boundary item, in chunks of
// four rows or more: in four-row chunks it marched twice its rows (20000 x 56 float32
// 104 us, now 81, float64 275, now 212; 100000 x 40 508 and 357, 1369 and 983), and
// shorter ones lose there (2000 x 50 float32, three rows 22.0, four 20.0).
struct StripRows {
  int sx, sxc;   // output rows of an interior and of a boundary-strip item
  bool single;   // one uniform list of items of sx rows, every item in the general body
};

inline StripRows strip_rows(int nx, int ny, bool f32) {
  constexpr int SXC = 4;
  const double A = f32 ? 1.0 : 2.6, B = f32 ? 0.3 : 0.7, CPS = f32 ? 4 : 2;
  const double EDGE_ROWS = 8.0 * (f32 ? 1.3 : 1.1);   // a boundary item, in interior rows
  const double SLOTS = 148.0 * CPS, FULL = A + B * CPS;
  const int ns = (ny + SW - 1) / SW, nmid = full_mid_strips(ny);
  StripRows p;
  const bool small = (double)ns * nx < 6.0 * 592.0;
  p.single = small || nmid == 0;
  p.sxc = SXC;
  p.sx = 1;
  const int strips = p.single ? ns : nmid, rows = p.single ? nx : std::max(nx - 4, 1);
  const double ne =
      p.single ? 0.0 : ((ns - nmid) * ((nx + SXC - 1) / SXC) + 2.0 * nmid) / 4.0;
  double best = 1e300;
  for (int s : {2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32, 40, 48, 64}) {
    const int n = (rows + s - 1) / s, h = (rows + n - 1) / n;   // chunks of equal height
    const double L = h + 4, ctas = strips * (double)n / 4.0;
    const double q = std::floor(ctas / SLOTS), r = ctas - q * SLOTS, last = r + ne;
    const double own = r > 0.0 ? L : 0.0;
    double cost = L * q * FULL;
    if (last <= SLOTS)
      cost += std::max(own, ne > 0.0 ? EDGE_ROWS : 0.0) *
              (A + B * (f32 ? std::max(1.0, last / 148.0) : std::ceil(last / 148.0)));
    else
      cost += (own + EDGE_ROWS * std::max(0.5, (last - SLOTS) / SLOTS)) * FULL;
    if (cost < best) {
      best = cost;
      p.sx = h;
    }
  }
  if (p.single && !small) p.sx = std::max(p.sx, SXC);
  return p;
}

// ── multigrid and training kernels ──────────────────────────────────────────

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
