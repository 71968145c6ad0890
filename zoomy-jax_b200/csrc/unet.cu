// Learned multigrid smoother: a small convolutional U-Net with bf16 weights
// and float32 accumulation, its training kernels (forward, backward, Adam) and
// its use as the level-0 smoother of the pressure V-cycle.
//
// The reference's learned V-cycle (zoomy_jax/gnn_blueprint/
// vcycle_structured_gnn.py:74-122, 145-200; graph_mp_multibranch.py:9-16;
// trained by train_vcycle_structured_poisson.py:168-306) smooths each level
// with tanh message-passing layers over the residual.  On a Cartesian grid the
// same local learned operator is a convolution; here it is a two-level U-Net:
//
//   in  = [r / s, c / cmax]                  (2 channels; s = RMS of r)
//   e1  = tanh(conv3x3(in,  2  -> C1))        level 0
//   e2  = tanh(conv3x3(e1,  C1 -> C1))
//   m1  = tanh(conv3x3(pool2(e2), C1 -> C2))  level 1 (2x2 average pool)
//   m2  = tanh(conv3x3(m1,  C2 -> C2))
//   o1  = tanh(conv3x3([up2(m2), e2], C2+C1 -> C1))   (nearest upsample)
//   out = conv3x3(o1, C1 -> 1)
//   correction = s * dx^2 / c * out           (1-homogeneous in r)
//
// with c the cell mean of the four face coefficients.  Activations are
// channel planes [C][B][H][W] in float32; weights [Cout][Cin][3][3] in bf16
// (the training keeps a float32 master copy and rounds it to bf16 for every
// forward, so the gradients are those of the bf16 network).  Convolutions run on
// the tensor cores (conv_tc.cuh): inference through chunked bf16 activations
// (conv3x3_cb8), training and its data gradients through the planes (conv3x3_tc);
// conv3x3_fwd, direct in float32 on the FMA pipe, is the exactness reference
// (zb_unet_conv_impl 0).  Weight gradients run on the FMA pipe (conv3x3_wgrad,
// conv3x3_wgrad_up).  Zero padding at image borders.
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <cstring>
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "conv_tc.cuh"
#include "launch_rules.h"

namespace zb {
namespace unet {

constexpr int TS = 16;          // pixel tile side
constexpr int NTT = TS * TS;    // threads per conv CTA
constexpr int CCH = 8;          // input channels per shared-memory chunk
constexpr int NT = 256;

enum { ACT_NONE = 0, ACT_TANH = 1, ACT_TANH_SFU = 2 };   // see conv_tc.cuh


// out[co][b][y][x] = act(bias[co] + sum_ci sum_tap w[co][ci][tap] in[ci][b][y+dy][x+dx])
// by a 16 x 16 pixel tile with a 1-pixel halo per 8-channel input chunk in shared memory,
// a thread per output pixel with all output channels in registers;
// input channels may come from two planes sets (the concatenation): channels
// [0, cin_a) from inA, [cin_a, cin) from inB; ytanh (a data gradient): the result
// times 1 - ytanh^2
template <int COUT>
__global__ void __launch_bounds__(NTT)
conv3x3_fwd(const float* __restrict__ inA, int cin_a, const float* __restrict__ inB, int cin,
            const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias,
            float* __restrict__ out, int B, int H, int W, int act, int mode_a,
            const float* __restrict__ ytanh) {
  __shared__ float sin_[CCH][TS + 2][TS + 2];
  __shared__ float sw[COUT][CCH][9];
  const int tx = threadIdx.x % TS, ty = threadIdx.x / TS;
  const int x0 = blockIdx.x * TS, y0 = blockIdx.y * TS, b = blockIdx.z;
  const int x = x0 + tx, y = y0 + ty;
  const size_t plane = (size_t)B * H * W;
  const size_t img = (size_t)b * H * W;
  float acc[COUT];
#pragma unroll
  for (int co = 0; co < COUT; ++co) acc[co] = bias ? bias[co] : 0.0f;
  for (int c0 = 0; c0 < cin; c0 += CCH) {
    const int nc = min(CCH, cin - c0);
    __syncthreads();
    for (int e = threadIdx.x; e < CCH * (TS + 2) * (TS + 2); e += NTT) {
      const int cc = e / ((TS + 2) * (TS + 2));
      const int rr = e - cc * (TS + 2) * (TS + 2);
      const int yy = y0 - 1 + rr / (TS + 2), xx = x0 - 1 + rr % (TS + 2);
      float v = 0.0f;
      if (cc < nc && yy >= 0 && yy < H && xx >= 0 && xx < W)
        v = src_at(inA, cin_a, inB, mode_a, c0 + cc, b, B, H, W, yy, xx);
      sin_[cc][rr / (TS + 2)][rr % (TS + 2)] = v;
    }
    for (int e = threadIdx.x; e < COUT * CCH * 9; e += NTT) {
      const int co = e / (CCH * 9), rem = e - co * CCH * 9;
      const int cc = rem / 9, tap = rem - cc * 9;
      sw[co][cc][tap] = cc < nc ? __bfloat162float(w[((size_t)co * cin + c0 + cc) * 9 + tap]) : 0.0f;
    }
    __syncthreads();
    for (int cc = 0; cc < nc; ++cc) {
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        const float v = sin_[cc][ty + tap / 3][tx + tap % 3];
#pragma unroll
        for (int co = 0; co < COUT; ++co) acc[co] = fmaf(sw[co][cc][tap], v, acc[co]);
      }
    }
  }
  if (x < W && y < H) {
#pragma unroll
    for (int co = 0; co < COUT; ++co) {
      float v = act != ACT_NONE ? tanhf(acc[co]) : acc[co];   // exact reference
      const size_t k = (size_t)co * plane + img + (size_t)y * W + x;
      if (ytanh) v *= 1.0f - ytanh[k] * ytanh[k];
      out[k] = v;
    }
  }
}

// Weight and bias gradients of one layer,
//   dW[co][ci][tap] = sum_p dout[co](p) in[ci](p + tap),  dbias[co] = sum_p dout[co](p),
// in float32 on the FMA pipe.  A thread owns one input channel and WG_COT output
// channels with all nine taps in registers and walks the pixels of a WG_TY x
// WG_TX tile: per pixel three new input values (the 3 x 3 window slides along x)
// and one 16-byte load of output gradients (the same address for a warp's
// lanes) feed 9 WG_COT FMAs.  The bias is one more input channel that holds
// ones.  Where a layer has few (channel, channel group) pairs the threads also
// split the tile's row segments (nsl slices) and add their sums in a fixed
// order.  Tiles arrive by cp.async into two buffers.  A CTA keeps its
// accumulators over all its tiles and writes one partial set; wgrad_reduce adds
// the partial sets in order, so the gradients are deterministic.  One thread per
// weight walking the pixels in shared memory with a float atomic per tile, as
// before, was bound by its two shared loads per FMA: the six layers of a
// 64 x 32^2 batch (24, 48) took 1234 us, now 194 and 10 for the reduction (the
// FMA pipe's floor is 35; the copies of the halo tiles are the rest: tiles of
// four rows instead of eight, half of them halo, 201 and 13).
constexpr int WG_TX = 16, WG_TY = 8, WG_SEG = 8;          // tile, pixels per row segment
constexpr int WG_HX = WG_TX + 2, WG_HY = WG_TY + 2;
constexpr int WG_PLANE = WG_HX * WG_HY + 1;               // odd: lanes of a warp hit 32 banks
constexpr int WG_UNITS = WG_TY * (WG_TX / WG_SEG);        // row segments of a tile
constexpr int WG_MAX_THREADS = 320;                       // two CTAs of 96 registers a thread
constexpr int WG_COT = 4;                                 // output channels of a thread
constexpr int WG_SLOTS = 296;                             // partial sets: two CTAs per SM

struct WgShape {
  int ncog, cic, nchunk, nsl, threads, slots;
  size_t smem, part;   // bytes of shared memory; floats of one partial set
};

// the upsampled source of the concatenation layer: tiles of UG_Y x UG_X of its pixels
// and the output gradients around them
constexpr int UG_X = 8, UG_Y = 4, UG_P = UG_X * UG_Y;
constexpr int UG_FX = 2 * UG_X + 2, UG_FY = 2 * UG_Y + 2, UG_FS = UG_FX * UG_FY + 1;
constexpr int UG_THREADS = 288;

// channel groups, input channels per chunk (the ones channel included), slices
// and threads of a layer's CTAs; up: the input channels in front of these that are
// upsampled (conv3x3_wgrad_up's, which fills the same partial sets)
static WgShape wg_shape(int cin, int cout, int B, int H, int W, int up) {
  WgShape g;
  const int cot = cout % WG_COT == 0 ? WG_COT : 1;
  g.ncog = cout / cot;
  const int planes = cin + 1, cmax = WG_MAX_THREADS / g.ncog;
  g.nchunk = (planes + cmax - 1) / cmax;
  g.cic = (planes + g.nchunk - 1) / g.nchunk;
  const int pairs = g.cic * g.ncog;
  g.nsl = std::max(1, std::min(WG_UNITS, WG_MAX_THREADS / pairs));
  g.threads = (pairs * g.nsl + 31) / 32 * 32;
  const long long ntiles = (long long)((W + WG_TX - 1) / WG_TX) * ((H + WG_TY - 1) / WG_TY) * B;
  const long long utiles =
      (long long)((W / 2 + UG_X - 1) / UG_X) * ((H / 2 + UG_Y - 1) / UG_Y) * B;
  // as few partial sets as take the same number of rounds
  const long long nt = up ? utiles : ntiles, rounds = (nt + WG_SLOTS - 1) / WG_SLOTS;
  g.slots = (int)((nt + rounds - 1) / rounds);
  const size_t stage =
      2 * ((((size_t)g.cic * WG_PLANE + 3) & ~(size_t)3) +
           (size_t)WG_TX * WG_TY * (cot > 1 ? cout + 4 : 1));
  const size_t red = g.nsl > 1 ? (size_t)pairs * g.nsl * 9 * cot : 0;
  g.smem = std::max(stage, red) * sizeof(float);
  g.part = (size_t)cout * (up + cin) * 9 + cout;
  return g;
}

__device__ __forceinline__ void cp_async4z(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_u32(dst)), "l"(src),
               "r"(valid ? 4 : 0)
               : "memory");
}

template <int COT>
__global__ void __launch_bounds__(WG_MAX_THREADS, 2)
conv3x3_wgrad(const float* __restrict__ in, int cin, const float* __restrict__ dout, int cout,
              float* __restrict__ part, int up, int B, int H, int W, int mode, int ncog, int cic,
              int nsl) {
  pdl_enter();
  extern __shared__ __align__(16) float wsm[];
  const int nt = blockDim.x, tid = threadIdx.x;
  const int c_lo = blockIdx.y * cic, c_n = min(cic, cin + 1 - c_lo);
  const int c_real = min(c_n, cin - c_lo);   // input channels of this chunk without the ones
  // a staging buffer: input planes, then the output gradients [pixel][dstr]
  // (16-byte rows); two of them, so that a tile's copies land while the one
  // before it is worked on
  const int dstr = COT > 1 ? cout + 4 : 1;
  const int sd_off = (cic * WG_PLANE + 3) & ~3, buf = sd_off + WG_TX * WG_TY * dstr;
  const int pairs = cic * ncog;
  const int sl = tid / pairs, pr = tid - sl * pairs;
  const int cog = pr / cic, ci = pr - cog * cic;
  const bool work = sl < nsl && ci < c_n;
  const size_t plane = (size_t)B * H * W;
  const int tx = (W + WG_TX - 1) / WG_TX, ty = (H + WG_TY - 1) / WG_TY;
  const int ntiles = tx * ty * B;
  if (c_real < c_n)
    for (int e = tid; e < 2 * WG_HX * WG_HY; e += nt) {
      const int k = e / (WG_HX * WG_HY);
      wsm[k * buf + c_real * WG_PLANE + (e - k * (WG_HX * WG_HY))] = 1.0f;
    }
  const int hl = tid & 15, hw = tid >> 4, nhw = nt >> 4;
  auto stage = [&](int t, int k) {
    float* sin_ = wsm + k * buf;
    float* sd = sin_ + sd_off;
    const int b = t / (tx * ty), rt = t - b * (tx * ty);
    const int x0 = (rt % tx) * WG_TX, y0 = (rt / tx) * WG_TY;
    const size_t img = (size_t)b * H * W;
    // a half-warp per row of 16 pixels: the lane's column, plus the two halo
    // columns on lanes 0 and 1
    const int xx = x0 + hl, xh = hl == 0 ? x0 - 1 : x0 + WG_TX;
    const bool xin = xx < W, hin = hl < 2 && xh >= 0 && xh < W;
    const int hcol = hl == 0 ? 0 : WG_HX - 1;
    for (int e = hw; e < c_real * WG_HY; e += nhw) {
      const int cc = e / WG_HY, r = e - cc * WG_HY;
      const int yy = y0 - 1 + r, c = c_lo + cc;
      const bool yin = yy >= 0 && yy < H;
      float* dst = sin_ + cc * WG_PLANE + r * WG_HX;
      if (mode == SRC_POOL) {   // the average is formed, not copied
        dst[1 + hl] =
            (yin && xin) ? src_at(in, cin, nullptr, SRC_POOL, c, b, B, H, W, yy, xx) : 0.0f;
        if (hl < 2)
          dst[hcol] =
              (yin && hin) ? src_at(in, cin, nullptr, SRC_POOL, c, b, B, H, W, yy, xh) : 0.0f;
        continue;
      }
      const float* row = in + (yin ? (size_t)c * plane + img + yy * W : 0);
      cp_async4z(dst + 1 + hl, row + (yin && xin ? xx : 0), yin && xin);
      if (hl < 2) cp_async4z(dst + hcol, row + (yin && hin ? xh : 0), yin && hin);
    }
    for (int e = hw; e < cout * WG_TY; e += nhw) {
      const int c = e / WG_TY, r = e - c * WG_TY;
      const bool in = y0 + r < H && xin;
      cp_async4z(sd + (r * WG_TX + hl) * dstr + c,
                 in ? dout + (size_t)c * plane + img + (y0 + r) * W + xx : dout, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[COT][9];
#pragma unroll
  for (int c = 0; c < COT; ++c)
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[c][k] = 0.0f;
  stage(blockIdx.x, 0);   // gridDim.x <= ntiles
  int k = 0;
#pragma unroll 1
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x, k ^= 1) {
    // the other buffer was read in the previous round, which every thread has
    // left: the barrier below
    if (t + (int)gridDim.x < ntiles) {
      stage(t + gridDim.x, k ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (work) {
      const float* ip = wsm + k * buf + ci * WG_PLANE;
      const float* dp = wsm + k * buf + sd_off + cog * COT;
#pragma unroll 1
      for (int u = sl; u < WG_UNITS; u += nsl) {
        const int yy = u / (WG_TX / WG_SEG), xs = (u % (WG_TX / WG_SEG)) * WG_SEG;
        const float* r0 = ip + yy * WG_HX + xs;
        const float* q = dp + (yy * WG_TX + xs) * dstr;
        float w[9];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          w[3 * a + 1] = r0[a * WG_HX];
          w[3 * a + 2] = r0[a * WG_HX + 1];
        }
#pragma unroll
        for (int x = 0; x < WG_SEG; ++x) {
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            w[3 * a] = w[3 * a + 1];
            w[3 * a + 1] = w[3 * a + 2];
            w[3 * a + 2] = r0[a * WG_HX + x + 2];
          }
          float d[COT];
          if constexpr (COT == 4) {
            const float4 v = *(const float4*)(q + x * dstr);
            d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
          } else {
            d[0] = q[x * dstr];
          }
#pragma unroll
          for (int c = 0; c < COT; ++c)
#pragma unroll
            for (int j = 0; j < 9; ++j) acc[c][j] = fmaf(d[c], w[j], acc[c][j]);
        }
      }
    }
    __syncthreads();
  }
  // slices in order through shared memory: slot [sl][9 COT values][pair]
  if (nsl > 1) {
    __syncthreads();
    if (work)
#pragma unroll
      for (int c = 0; c < COT; ++c)
#pragma unroll
        for (int k = 0; k < 9; ++k) wsm[((size_t)sl * 9 * COT + c * 9 + k) * pairs + pr] = acc[c][k];
    __syncthreads();
    if (!work || sl > 0) return;
    for (int s2 = 1; s2 < nsl; ++s2)
#pragma unroll
      for (int c = 0; c < COT; ++c)
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[c][k] += wsm[((size_t)s2 * 9 * COT + c * 9 + k) * pairs + pr];
  }
  if (!work) return;
  const int gci = c_lo + ci;
  const int ct = up + cin;   // the layer's input channels
  float* out = part + (size_t)blockIdx.x * ((size_t)cout * ct * 9 + cout);
  if (gci < cin) {
#pragma unroll
    for (int c = 0; c < COT; ++c)
#pragma unroll
      for (int k = 0; k < 9; ++k)
        out[(size_t)((cog * COT + c) * 9 + k) * ct + up + gci] = acc[c][k];
  } else {
#pragma unroll
    for (int c = 0; c < COT; ++c) out[(size_t)cout * ct * 9 + cog * COT + c] = acc[c][4];
  }
}

// Weight gradients of the upsampled channels of the concatenation layer (the first cin
// of its cin + direct inputs), at the source's resolution.  in(p + tap - 1) is the
// source's pixel P for p in a 2 x 2 block that depends on the tap, so
//   dW[co][ci][tap] = sum_P in[ci](P) S[co][tap](P),  S = the block's sum of dout:
// a quarter of the products.  A CTA forms S of a tile (32 source pixels) once in shared
// memory; a thread owns one input and four output channels with all nine taps, and per
// pixel one value and nine 16-byte loads (the same address for most of a warp) feed 36
// FMAs.  64 x 32^2, 48 + 24 -> 24 channels: all 72 channels at full resolution 116 us,
// now 30 here and 38 for the other 24.
__global__ void __launch_bounds__(UG_THREADS, 2)
conv3x3_wgrad_up(const float* __restrict__ in, int cin, const float* __restrict__ dout, int cout,
                 float* __restrict__ part, int direct, int B, int H, int W, int nsl) {
  pdl_enter();
  extern __shared__ __align__(16) float wsm[];
  float* S = wsm;                                 // [pixel][tap][cout]
  float* sin_ = S + UG_P * 9 * cout;              // [cin][pixel], odd stride
  float* sd = sin_ + cin * (UG_P + 1);            // [cout][fine pixel], odd stride
  const int tid = threadIdx.x;
  const int h = H / 2, w = W / 2, pairs = cin * (cout / WG_COT);
  const int sl = tid / pairs, pr = tid - sl * pairs;
  const int cog = pr / cin, ci = pr - cog * cin;
  const bool work = sl < nsl;
  const int tx = (w + UG_X - 1) / UG_X, ty = (h + UG_Y - 1) / UG_Y, ntiles = tx * ty * B;
  float acc[WG_COT][9];
#pragma unroll
  for (int c = 0; c < WG_COT; ++c)
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[c][k] = 0.0f;
#pragma unroll 1
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int b = t / (tx * ty), rt = t - b * (tx * ty);
    const int x0 = (rt % tx) * UG_X, y0 = (rt / tx) * UG_Y;
    for (int e = tid; e < cout * UG_FX * UG_FY; e += UG_THREADS) {
      const int c = e / (UG_FX * UG_FY), q = e - c * (UG_FX * UG_FY);
      const int fy = q / UG_FX, yy = 2 * y0 - 1 + fy, xx = 2 * x0 - 1 + q - fy * UG_FX;
      const bool ok = yy >= 0 && yy < H && xx >= 0 && xx < W;
      cp_async4z(sd + c * UG_FS + q,
                 ok ? dout + (((size_t)c * B + b) * H + yy) * W + xx : dout, ok);
    }
    for (int e = tid; e < cin * UG_P; e += UG_THREADS) {
      const int c = e / UG_P, q = e % UG_P, yy = y0 + q / UG_X, xx = x0 + q % UG_X;
      const bool ok = yy < h && xx < w;
      cp_async4z(sin_ + c * (UG_P + 1) + q,
                 ok ? in + (((size_t)c * B + b) * h + yy) * w + xx : in, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int e = tid; e < UG_P * cout; e += UG_THREADS) {
      const int P = e / cout, c = e - P * cout;
      const float* q = sd + c * UG_FS + 2 * (P / UG_X) * UG_FX + 2 * (P % UG_X);
      float r[3][4];   // sums of neighbouring rows
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float a0 = q[x], a1 = q[UG_FX + x], a2 = q[2 * UG_FX + x], a3 = q[3 * UG_FX + x];
        r[0][x] = a0 + a1;
        r[1][x] = a1 + a2;
        r[2][x] = a2 + a3;
      }
#pragma unroll
      for (int k = 0; k < 9; ++k)   // tap (dy, dx): rows and columns 2 - dy, 2 - dx on
        S[(P * 9 + k) * cout + c] = r[2 - k / 3][2 - k % 3] + r[2 - k / 3][3 - k % 3];
    }
    __syncthreads();
    if (work) {
#pragma unroll 1
      for (int P = sl; P < UG_P; P += nsl) {
        const float v = sin_[ci * (UG_P + 1) + P];
        const float* q = S + P * 9 * cout + cog * WG_COT;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          const float4 d = *(const float4*)(q + k * cout);
          acc[0][k] = fmaf(d.x, v, acc[0][k]);
          acc[1][k] = fmaf(d.y, v, acc[1][k]);
          acc[2][k] = fmaf(d.z, v, acc[2][k]);
          acc[3][k] = fmaf(d.w, v, acc[3][k]);
        }
      }
    }
    __syncthreads();
  }
  // slices in order through shared memory
  if (nsl > 1) {
    if (work)
#pragma unroll
      for (int c = 0; c < WG_COT; ++c)
#pragma unroll
        for (int k = 0; k < 9; ++k)
          wsm[((size_t)sl * 9 * WG_COT + c * 9 + k) * pairs + pr] = acc[c][k];
    __syncthreads();
    if (!work || sl > 0) return;
    for (int s2 = 1; s2 < nsl; ++s2)
#pragma unroll
      for (int c = 0; c < WG_COT; ++c)
#pragma unroll
        for (int k = 0; k < 9; ++k)
          acc[c][k] += wsm[((size_t)s2 * 9 * WG_COT + c * 9 + k) * pairs + pr];
  }
  if (!work) return;
  const int ct = cin + direct;
  float* out = part + (size_t)blockIdx.x * ((size_t)cout * ct * 9 + cout);
#pragma unroll
  for (int c = 0; c < WG_COT; ++c)
#pragma unroll
    for (int k = 0; k < 9; ++k) out[(size_t)((cog * WG_COT + c) * 9 + k) * ct + ci] = acc[c][k];
}

// the partial sets of all six layers added in order; a set is [cout][tap][cin], then
// the biases (as [cout][cin][tap] its stores were nine times as many sectors)
struct WgReduce {
  const float* part[6];
  int slots[6], cin[6], nw[6], nb[6], off_w[6], off_b[6], first[7];   // first: entry offsets
};

// A CTA adds 32 entries: warp w takes the sets w, w + 8, ... and the eight sums
// are added in order.
__global__ void __launch_bounds__(NT)
wgrad_reduce(const WgReduce R, float* __restrict__ dw, float* __restrict__ db) {
  pdl_enter();
  __shared__ float sh[NT / 32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;
  int l = 0;
  while (l < 5 && e >= R.first[l + 1]) ++l;
  const int k = e - R.first[l], n = R.nw[l] + R.nb[l];
  float s = 0.0f;
  if (e < R.first[6]) {
    const float* q = R.part[l] + k;
#pragma unroll 8
    for (int i = warp; i < R.slots[l]; i += NT / 32) s += q[(size_t)i * n];
  }
  sh[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || e >= R.first[6]) return;
#pragma unroll
  for (int w = 1; w < NT / 32; ++w) s += sh[w][lane];
  if (k < R.nw[l]) {
    const int row = k / R.cin[l], ci = k - row * R.cin[l], co = row / 9, tap = row - co * 9;
    dw[R.off_w[l] + (co * R.cin[l] + ci) * 9 + tap] = s;
  } else {
    db[R.off_b[l] + k - R.nw[l]] = s;
  }
}

// transposed, flipped weights for the data gradients, wt[ci][co][8 - tap], of
// layers 1 .. 5 (each at its own offset)
struct FlipTab {
  int off[6], cin[6], cout[6];
};

__global__ void flip_weights(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wt,
                             const FlipTab f, int n) {
  pdl_enter();
  for (int e = f.off[1] + blockIdx.x * NT + threadIdx.x; e < n; e += gridDim.x * NT) {
    int l = 1;
    while (l < 5 && e >= f.off[l + 1]) ++l;
    const int k = e - f.off[l], cin = f.cin[l];
    const int co = k / (cin * 9), rem = k - co * cin * 9;
    const int ci = rem / 9, tap = rem - ci * 9;
    wt[f.off[l] + (ci * f.cout[l] + co) * 9 + (8 - tap)] = w[e];
  }
}

// The backward of the layer inputs, each with the tanh derivative 1 - y^2 of the
// activation it reaches (in the convolution's epilogue where the data gradient is
// that input itself).  Separate passes for the pooling, the sum and the derivative
// took 22 us of a 64 x 32^2 batch's step, the upsampling 12.

// gradient of e2: the average pool's (g1 / 4, half resolution) plus the
// concatenation's, then the derivative (C channels of at most 2^31 elements: plane_slice)
__global__ void pool_add_tanh_back(const float* __restrict__ g1, const float* __restrict__ g2,
                                   const float* __restrict__ y, float* __restrict__ gin, int C,
                                   int B, int H, int W) {
  pdl_enter();
  const unsigned n = (unsigned)C * B * H * W, uW = W, uH = H;
  for (unsigned k = blockIdx.x * NT + threadIdx.x; k < n; k += gridDim.x * NT) {
    const unsigned t = k / uW, xx = k - t * uW;
    const unsigned cb = t / uH, yy = t - cb * uH;
    const float yk = y[k];
    gin[k] = (0.25f * g1[((size_t)cb * (uH / 2) + yy / 2) * (uW / 2) + xx / 2] + g2[k]) *
             (1.0f - yk * yk);
  }
}

// gradient of m2 through the nearest upsampling: the 2x2 sum, then the derivative
__global__ void upsample2_tanh_back(const float* __restrict__ gout, const float* __restrict__ y,
                                    float* __restrict__ gin, int C, int B, int H, int W) {
  pdl_enter();
  const unsigned Ho = H / 2, Wo = W / 2, n = (unsigned)C * B * Ho * Wo;
  for (unsigned k = blockIdx.x * NT + threadIdx.x; k < n; k += gridDim.x * NT) {
    const unsigned t = k / Wo, xo = k - t * Wo;
    const unsigned cb = t / Ho, yo = t - cb * Ho;
    const float* q = gout + (size_t)cb * H * W + (size_t)(2 * yo) * W + 2 * xo;
    const float yk = y[k];
    gin[k] = (q[0] + q[1] + q[W] + q[W + 1]) * (1.0f - yk * yk);
  }
}

// one Adam step of the weights (the first n entries) and the biases
struct AdamSet {
  float *w, *m, *v;
  const float* g;
  __nv_bfloat16* wb;
};

__global__ void adam_kernel(const AdamSet W, const AdamSet Bi, int n, int nb, float lr, float b1,
                            float b2, float eps, float c1, float c2) {
  pdl_enter();
  for (int e = blockIdx.x * NT + threadIdx.x; e < n + nb; e += gridDim.x * NT) {
    const AdamSet& S = e < n ? W : Bi;
    const int k = e < n ? e : e - n;
    const float g0 = S.g[k];
    const float gk = isfinite(g0) ? g0 : 0.0f;   // a non-finite entry is skipped
    const float mk = b1 * S.m[k] + (1.0f - b1) * gk;
    const float vk = b2 * S.v[k] + (1.0f - b2) * gk * gk;
    S.m[k] = mk;
    S.v[k] = vk;
    const float wk = S.w[k] - lr * (mk / c1) / (sqrtf(vk / c2) + eps);
    S.w[k] = wk;
    S.wb[k] = __float2bfloat16(wk);
  }
}

}  // namespace unet
}  // namespace zb

// ── features, scaling, patch operator, loss ─────────────────────────────────
namespace zb {
namespace unet {

// per image b: s[b] = sqrt(mean r^2) (tiny floor so a zero residual stays
// zero), as a two-stage deterministic reduction: P partial sums per image
// (grid (P, B)), then one warp per image adds them in a fixed order
constexpr int RMS_PARTS = 1024;   // partial-sum slots in the workspace

// part p of P of image b's sum of squares: a fixed set of cells in a fixed order (the
// first NT threads' sums)
__device__ __forceinline__ void rms_store_part(float acc, float* part, int slot) {
  __shared__ float red[NT / 32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0 && threadIdx.x < NT) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int i = 0; i < NT / 32; ++i) t += red[i];
    part[slot] = t;
  }
}

__global__ void rms_part_kernel(const float* __restrict__ r, size_t npix, int P,
                                float* __restrict__ part) {
  pdl_enter();
  const int b = blockIdx.y, p = blockIdx.x;
  float acc = 0.0f;
#pragma unroll 4
  for (size_t k = (size_t)p * NT + threadIdx.x; k < npix; k += (size_t)P * NT) {
    const float v = r[(size_t)b * npix + k];
    acc += v * v;
  }
  rms_store_part(acc, part, b * P + p);
}

// s of image b from its parts, by a whole warp
__device__ __forceinline__ float rms_of(const float* part, int P, int b, size_t npix) {
  float t = 0.0f;
  for (int p = threadIdx.x & 31; p < P; p += 32) t += part[b * P + p];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return fmaxf(sqrtf(t / (float)npix), 1e-30f);
}

__global__ void rms_final_kernel(const float* __restrict__ part, int P, size_t npix,
                                 float* __restrict__ s) {
  pdl_enter();
  const float v = rms_of(part, P, blockIdx.x, npix);
  if (threadIdx.x == 0) s[blockIdx.x] = v;
}

static int rms_parts(int B, size_t npix) {
  const int P = (int)std::min<size_t>(256, std::max<size_t>(1, npix / (NT * 16)));
  return std::max(1, std::min(P, RMS_PARTS / std::max(1, B)));
}

static int rms(const float* r, int B, size_t npix, float* part, float* s, cudaStream_t st) {
  const int P = rms_parts(B, npix);
  ZB_CUDA_TRY(pdl_launch(rms_part_kernel, dim3(P, B), dim3(NT), 0, st, r, npix, P, part));
  ZB_CUDA_TRY(pdl_launch(rms_final_kernel, dim3(B), dim3(32), 0, st, (const float*)part, P, npix, s));
  return ZB_OK;
}

// cell coefficient of image b's cell (i, j) from its faces: cx (B, H+1, W),
// cy (B, H, W+1)
__device__ __forceinline__ float cell_c(const float* cx, const float* cy, int b, int H, int W,
                                        int i, int j) {
  const float* ax = cx + (size_t)b * (H + 1) * W;
  const float* ay = cy + (size_t)b * H * (W + 1);
  return 0.25f * (ax[(size_t)i * W + j] + ax[(size_t)(i + 1) * W + j] +
                  ay[(size_t)i * (W + 1) + j] + ay[(size_t)i * (W + 1) + j + 1]);
}

__global__ void features_kernel(const float* __restrict__ r, const float* __restrict__ s,
                                const float* __restrict__ cx, const float* __restrict__ cy,
                                int B, int H, int W, float inv_cmax, float* __restrict__ in) {
  pdl_enter();
  const size_t npix = (size_t)H * W, n = (size_t)B * npix;
  for (size_t k = blockIdx.x * (size_t)NT + threadIdx.x; k < n; k += (size_t)gridDim.x * NT) {
    const int b = (int)(k / npix);
    const size_t p = k - (size_t)b * npix;
    const int i = (int)(p / W), j = (int)(p - (size_t)i * W);
    in[k] = r[k] / s[b];
    in[n + k] = cell_c(cx, cy, b, H, W, i, j) * inv_cmax;
  }
}

// the same two input channels of one image as one chunk of the chunked bf16 layout
// (channels 2..7 zero), each rounded as the planar kernel rounds them.  Every block
// adds the P parts of s itself (in rms_final_kernel's order); block 0 stores it.
__global__ void __launch_bounds__(NT)
features_cb8_kernel(const float* __restrict__ r, const float* __restrict__ part, int P,
                    float* __restrict__ s_out, const float* __restrict__ cx,
                    const float* __restrict__ cy, int H, int W, float inv_cmax,
                    uint4* __restrict__ in) {
  pdl_enter();
  __shared__ float sh;
  const unsigned n = (unsigned)H * W, uW = W;
  if (threadIdx.x < 32) {
    const float v = rms_of(part, P, 0, n);
    if (threadIdx.x == 0) {
      sh = v;
      if (blockIdx.x == 0) s_out[0] = v;
    }
  }
  __syncthreads();
  const float s = sh;
#pragma unroll 2
  for (unsigned k = blockIdx.x * NT + threadIdx.x; k < n; k += gridDim.x * NT) {
    const unsigned i = k / uW, j = k - i * uW;
    __align__(16) __nv_bfloat16 v[8];
    v[0] = __float2bfloat16_rn(r[k] / s);
    v[1] = __float2bfloat16_rn(cell_c(cx, cy, 0, H, W, i, j) * inv_cmax);
#pragma unroll
    for (int c = 2; c < 8; ++c) v[c] = __float2bfloat16_rn(0.0f);
    in[k] = *(const uint4*)v;
  }
}

// y = x_in + s dx^2 / c * out   (x_in may be null; y may alias x_in)
__global__ void scale_out_kernel(const float* __restrict__ out, const float* __restrict__ s,
                                 const float* __restrict__ cx, const float* __restrict__ cy,
                                 int B, int H, int W, float dx2, const float* x_in, float* y) {
  pdl_enter();
  const unsigned npix = (unsigned)H * W, n = B * npix, uW = W;
  for (unsigned k = blockIdx.x * NT + threadIdx.x; k < n; k += gridDim.x * NT) {
    const unsigned b = k / npix, p = k - b * npix;
    const int i = (int)(p / uW), j = (int)(p - i * uW);
    const float v = s[b] * dx2 / cell_c(cx, cy, b, H, W, i, j) * out[k];
    y[k] = x_in ? x_in[k] + v : v;
  }
}

__device__ __forceinline__ float xg(const float* x, int H, int W, int i, int j, float self) {
  return (i < 0 || i >= H || j < 0 || j >= W) ? -self : x[(size_t)i * W + j];
}

// f - A x at cell (i, j) of an image whose arrays start at x, ax, ay (Dirichlet
// ghost -x; x null means zero)
__device__ __forceinline__ float residual_at(float f, const float* x, const float* ax_,
                                             const float* ay_, int H, int W, int i, int j,
                                             float idx2) {
  float ax = 0.0f;
  if (x) {
    const float xc = x[(size_t)i * W + j];
    ax = (ax_[(size_t)(i + 1) * W + j] * (xc - xg(x, H, W, i + 1, j, xc)) +
          ax_[(size_t)i * W + j] * (xc - xg(x, H, W, i - 1, j, xc)) +
          ay_[(size_t)i * (W + 1) + j + 1] * (xc - xg(x, H, W, i, j + 1, xc)) +
          ay_[(size_t)i * (W + 1) + j] * (xc - xg(x, H, W, i, j - 1, xc))) * idx2;
  }
  return f - ax;
}

// res = f - A x per image
__global__ void patch_residual(const float* __restrict__ f, const float* __restrict__ x,
                               const float* __restrict__ cx, const float* __restrict__ cy,
                               int B, int H, int W, float idx2, float* __restrict__ res) {
  pdl_enter();
  const unsigned npix = (unsigned)H * W, n = B * npix, uW = W;
  for (unsigned k = blockIdx.x * NT + threadIdx.x; k < n; k += gridDim.x * NT) {
    const unsigned b = k / npix, p = k - b * npix;
    const int i = (int)(p / uW), j = (int)(p - i * uW);
    res[k] = residual_at(f[k], x ? x + (size_t)b * npix : nullptr, cx + (size_t)b * (H + 1) * W,
                         cy + (size_t)b * H * (W + 1), H, W, i, j, idx2);
  }
}

// res = f - A x of one image and the parts of its sum of squares.  The parts are
// rms_part_kernel's, cell for cell and in its order (the same bits), but four
// threads share one of its threads' cells: they leave them in shared memory, 16 at
// a time, and one adds them in order.  Bound by the latency of its loads; 1024^2: 11 us
// and 10 for the separate sum, now 10.7 (one thread per sum: 17.6).
constexpr int RR_SPLIT = 4, RR_CELLS = 16;

__global__ void __launch_bounds__(NT * RR_SPLIT)
residual_rms_kernel(const float* __restrict__ f, const float* __restrict__ x,
                    const float* __restrict__ cx, const float* __restrict__ cy, int H, int W,
                    float idx2, float* __restrict__ res, int P, float* __restrict__ part) {
  pdl_enter();
  __shared__ float sv[RR_CELLS][NT];
  const unsigned n = (unsigned)H * W, uW = W, stride = (unsigned)P * NT;
  const unsigned t = threadIdx.x % NT, q = threadIdx.x / NT;
  float acc = 0.0f;
  for (unsigned k0 = blockIdx.x * NT; k0 < n; k0 += RR_CELLS * stride) {
    float v[RR_CELLS / RR_SPLIT];
#pragma unroll
    for (int u = 0; u < RR_CELLS / RR_SPLIT; ++u) {
      const unsigned k = k0 + t + (RR_SPLIT * u + q) * stride;
      v[u] = 0.0f;   // adds nothing to the sum
      if (k < n) {
        const unsigned i = k / uW;
        v[u] = residual_at(f[k], x, cx, cy, H, W, (int)i, (int)(k - i * uW), idx2);
      }
    }
    __syncthreads();   // the sum of the cells before
#pragma unroll
    for (int u = 0; u < RR_CELLS / RR_SPLIT; ++u) {
      const unsigned k = k0 + t + (RR_SPLIT * u + q) * stride;
      if (k < n) res[k] = v[u];
      sv[RR_SPLIT * u + q][t] = v[u];
    }
    __syncthreads();
    if (q == 0) {
#pragma unroll
      for (int c = 0; c < RR_CELLS; ++c) acc += sv[c][t] * sv[c][t];
    }
  }
  rms_store_part(acc, part, blockIdx.x);
}

// loss terms per image: lnum[b] = a_b . b_b, lden[b] = c_b . d_b (residual
// loss: a = b = res, c = d = r; energy loss: a = res, b = A res, c = e,
// d = A e).  An image whose denominator is not a positive finite number above
// 1e-30 (a patch without signal) is left out of the loss and its gradient.
__global__ void loss_kernel(const float* __restrict__ a_, const float* __restrict__ b_,
                            const float* __restrict__ c_, const float* __restrict__ d_, int B,
                            size_t npix, float* __restrict__ lnum, float* __restrict__ lden) {
  pdl_enter();
  __shared__ float red[2][NT / 32];
  const int b = blockIdx.x;
  float a = 0.0f, c = 0.0f;
  for (size_t k = threadIdx.x; k < npix; k += NT) {
    const size_t q = (size_t)b * npix + k;
    a += a_[q] * b_[q];
    c += c_[q] * d_[q];
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = a; red[1][threadIdx.x >> 5] = c; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float ta = 0.0f, tc = 0.0f;
    for (int i = 0; i < NT / 32; ++i) { ta += red[0][i]; tc += red[1][i]; }
    lnum[b] = ta;
    lden[b] = tc;
  }
}

__device__ __forceinline__ bool loss_counts(float den) { return den > 1e-30f && den < 3e38f; }

// one warp, its lanes' sums added in a fixed order
__global__ void loss_total(const float* lnum, const float* lden, int B, double* out) {
  pdl_enter();
  double t = 0.0;
  for (int b = threadIdx.x; b < B; b += 32)
    if (loss_counts(lden[b])) t += (double)lnum[b] / (double)lden[b];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (threadIdx.x == 0) *out = t / B;
}

// A x per image (Dirichlet ghost -x)
__global__ void patch_apply(const float* __restrict__ x, const float* __restrict__ cx,
                            const float* __restrict__ cy, int B, int H, int W, float idx2,
                            float* __restrict__ out) {
  pdl_enter();
  const unsigned npix = (unsigned)H * W, n = B * npix, uW = W;
  for (unsigned k = blockIdx.x * NT + threadIdx.x; k < n; k += gridDim.x * NT) {
    const unsigned b = k / npix, p = k - b * npix;
    const int i = (int)(p / uW), j = (int)(p - i * uW);
    const float* xb = x + (size_t)b * npix;
    const float* ax_ = cx + (size_t)b * (H + 1) * W;
    const float* ay_ = cy + (size_t)b * H * (W + 1);
    const float xc = xb[p];
    out[k] = (ax_[(size_t)(i + 1) * W + j] * (xc - xg(xb, H, W, i + 1, j, xc)) +
              ax_[(size_t)i * W + j] * (xc - xg(xb, H, W, i - 1, j, xc)) +
              ay_[(size_t)i * (W + 1) + j + 1] * (xc - xg(xb, H, W, i, j + 1, xc)) +
              ay_[(size_t)i * (W + 1) + j] * (xc - xg(xb, H, W, i, j - 1, xc))) * idx2;
  }
}

__global__ void sub_kernel(const float* __restrict__ a, const float* __restrict__ b, size_t n,
                           float* __restrict__ out) {
  pdl_enter();
  for (size_t k = blockIdx.x * (size_t)NT + threadIdx.x; k < n; k += (size_t)gridDim.x * NT)
    out[k] = a[k] - b[k];
}

// dL/dout = -2 (A res)_b / (B den_b) * s_b dx^2 / c   (A symmetric); ar holds
// A res (energy loss) or is null, in which case A res is formed here from res
__global__ void loss_grad_kernel(const float* __restrict__ res, const float* __restrict__ ar_in,
                                 const float* __restrict__ cx, const float* __restrict__ cy,
                                 const float* __restrict__ lden, const float* __restrict__ s,
                                 int B, int H, int W, float idx2, float dx2,
                                 float* __restrict__ dout) {
  pdl_enter();
  const unsigned npix = (unsigned)H * W, n = B * npix, uW = W;
  for (unsigned k = blockIdx.x * NT + threadIdx.x; k < n; k += gridDim.x * NT) {
    const unsigned b = k / npix, p = k - b * npix;
    const int i = (int)(p / uW), j = (int)(p - i * uW);
    float ar;
    if (ar_in) {
      ar = ar_in[k];
    } else {
      const float* rb = res + (size_t)b * npix;
      const float* ax_ = cx + (size_t)b * (H + 1) * W;
      const float* ay_ = cy + (size_t)b * H * (W + 1);
      const float rc = rb[p];
      ar = (ax_[(size_t)(i + 1) * W + j] * (rc - xg(rb, H, W, i + 1, j, rc)) +
            ax_[(size_t)i * W + j] * (rc - xg(rb, H, W, i - 1, j, rc)) +
            ay_[(size_t)i * (W + 1) + j + 1] * (rc - xg(rb, H, W, i, j + 1, rc)) +
            ay_[(size_t)i * (W + 1) + j] * (rc - xg(rb, H, W, i, j - 1, rc))) * idx2;
    }
    const float den = lden[b];
    const float c = cell_c(cx, cy, b, H, W, i, j);
    dout[k] = loss_counts(den) ? -2.0f * ar / ((float)B * den) * s[b] * dx2 / c : 0.0f;
  }
}

// ── network plumbing ────────────────────────────────────────────────────────
struct Net {
  int c1, c2;
  size_t off_w[6], off_b[6];
  int cin[6], cout[6];
  size_t nw, nb;
};

static Net net_layout(int c1, int c2) {
  Net n;
  const int ci[6] = {2, c1, c1, c2, c1 + c2, c1};
  const int co[6] = {c1, c1, c2, c2, c1, 1};
  size_t w = 0, b = 0;
  for (int l = 0; l < 6; ++l) {
    n.cin[l] = ci[l];
    n.cout[l] = co[l];
    n.off_w[l] = w;
    n.off_b[l] = b;
    w += (size_t)co[l] * ci[l] * 9;
    b += (size_t)co[l];
  }
  n.c1 = c1;
  n.c2 = c2;
  n.nw = w;
  n.nb = b;
  return n;
}

// channel pairs with an instantiated convolution for every layer and for the
// data gradient of the concatenation layer (c1 + c2 output channels)
static bool valid_channels(int c1, int c2) {
  return (c1 == 8 && c2 == 16) || (c1 == 16 && c2 == 16) || (c1 == 16 && c2 == 32) ||
         (c1 == 24 && c2 == 48);
}

// which convolution runs the forward and data-gradient passes: 0 = the
// CUDA-core direct convolution (float32 operands, kept as the exactness
// reference); 1 (default) = the tcgen05 implicit GEMM (bf16 operands), the
// smoother application's forward through the chunked bf16 layout
// (conv3x3_cb8) and training through the float32 planar staging
// (conv3x3_tc); 2 = the tcgen05 GEMM with the planar staging everywhere (the
// same bits as 1)
static int g_conv_impl = 1;
static __device__ unsigned g_unet_err;

static unsigned* unet_err_word() {
  static std::atomic<unsigned*> ptrs[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!ptrs[dev].load()) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_unet_err) != cudaSuccess) return nullptr;
    ptrs[dev].store((unsigned*)p);
  }
  return ptrs[dev].load();
}

static int conv_tc_launch(const float* inA, int cin_a, const float* inB, int cin,
                          const __nv_bfloat16* w, const float* bias, float* out, int cout, int B,
                          int H, int W, int act, int mode_a, const float* ytanh,
                          cudaStream_t st) {
  const int cinp = pad16(cin), coutp = pad16(cout);
  if (coutp > 256 || cinp > 256) return ZB_E_UNSUPPORTED;
  int cols = 32;
  while (cols < coutp) cols *= 2;
  static std::atomic<int> sms[64];
  static std::atomic<bool> attr[64];
  int dev = 0;
  ZB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return ZB_E_CUDA;
  if (!sms[dev].load()) {
    int v = 0;
    ZB_CUDA_TRY(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    sms[dev].store(v);
  }
  if (!attr[dev].load()) {
#define ZB_SMEM_ATTR(G)                                                                       \
  ZB_CUDA_TRY(                                                                                 \
      cudaFuncSetAttribute(conv3x3_tc<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024))
    ZB_SMEM_ATTR(1); ZB_SMEM_ATTR(2); ZB_SMEM_ATTR(3); ZB_SMEM_ATTR(5);
#undef ZB_SMEM_ATTR
    attr[dev].store(true);
  }
  // resident CTAs of one SM must never ask for more than its 512 TMEM
  // columns: pad the shared memory so that at most 512 / cols fit
  const int smem_sm = 228 * 1024, per_cta_reserved = 1024;
  const int by_tmem = 512 / cols, by_threads = TC_PER_SM;
  size_t smem = tc_smem_bytes(cinp, coutp);
  if (by_tmem < by_threads) {
    const size_t floor_bytes = (size_t)(smem_sm / (by_tmem + 1) - per_cta_reserved + 16);
    smem = std::max(smem, floor_bytes);
  }
  if (smem > 227 * 1024) return ZB_E_UNSUPPORTED;
  const int fit = std::min(by_threads, (int)(smem_sm / (smem + per_cta_reserved)));
  const long long ntiles =
      (long long)((W + TCX - 1) / TCX) * ((H + TCY - 1) / TCY) * B;
  const int grid = (int)std::max<long long>(1, std::min<long long>(ntiles, (long long)sms[dev] * std::max(1, fit)));
  // channel groups of 16 of the networks' layers (valid_channels)
  switch (cinp / 16) {
#define ZB_TC(G)                                                                               \
  case G:                                                                                      \
    ZB_CUDA_TRY(pdl_launch(conv3x3_tc<G>, dim3(grid), dim3(TC_THREADS), smem, st, inA, cin_a,  \
                           inB, cin, w, bias, out, cout, B, H, W, act, mode_a, ytanh, cols,    \
                           unet_err_word()));                                                  \
    break
    ZB_TC(1); ZB_TC(2); ZB_TC(3); ZB_TC(5);
#undef ZB_TC
    default: return ZB_E_UNSUPPORTED;
  }
  return zb_launch_check();
}

// cuTensorMapEncodeTiled from the driver, fetched once through the runtime
// (no link against the driver library)
static PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
  static std::atomic<void*> fn{nullptr};
  void* f = fn.load();
  if (!f) {
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault,
                                         &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !f)
      return nullptr;
    fn.store(f);
  }
  return (PFN_cuTensorMapEncodeTiled_v12000)f;
}

// The halo-box map of a chunked activation: dimensions (8 channels, W, H,
// chunks x B) with byte strides (16, 16 W, 16 H W), box (8, 18, 18, 1); pixels
// outside the image read as zeros.  The base is 16-byte aligned and every
// stride a multiple of 16, as the encoder requires.
static bool cb8_map(CUtensorMap* m, const uint4* base, int nchunks, int B, int H, int W) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tmap_encoder();
  if (!enc || !base || ((uintptr_t)base & 15u)) return false;
  const cuuint64_t dims[4] = {8, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)nchunks * B};
  const cuuint64_t strides[3] = {16, (cuuint64_t)W * 16, (cuuint64_t)H * W * 16};
  const cuuint32_t box[4] = {8, (cuuint32_t)CHX, (cuuint32_t)CHY, 1};
  const cuuint32_t es[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)base, dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// conv3x3_cb8 over B images H x W (see conv_tc.cuh); resident CTAs are capped
// so that their TMEM columns (two buffers of two M tiles of coutp each) fit in 512
static int conv_cb8_launch(const uint4* inA, int chA, int mode_a, const uint4* inB, int chB,
                           int cin, const __nv_bfloat16* w, const float* bias, void* out,
                           uint4* pool, int cout, int out_form, int B, int H, int W, int act,
                           cudaStream_t st) {
  const int cinp = pad16(cin), coutp = pad16(cout);
  if (4 * coutp > 512 || cinp > 256 || chA + chB > cinp / 8) return ZB_E_UNSUPPORTED;
  int cols = 32;
  while (cols < 4 * coutp) cols *= 2;   // two buffers of two M tiles
  static std::atomic<int> sms[64];
  static std::atomic<bool> attr[64];
  int dev = 0;
  ZB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return ZB_E_CUDA;
  if (!sms[dev].load()) {
    int v = 0;
    ZB_CUDA_TRY(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    sms[dev].store(v);
  }
  if (!attr[dev].load()) {
#define ZB_SMEM_ATTR(G)                                                                        \
  ZB_CUDA_TRY(cudaFuncSetAttribute(conv3x3_cb8<G, CB_NTH>,                                     \
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024)); \
  ZB_CUDA_TRY(cudaFuncSetAttribute(conv3x3_cb8<G, CB_NTH_UP>,                                  \
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024))
    ZB_SMEM_ATTR(1); ZB_SMEM_ATTR(2); ZB_SMEM_ATTR(3); ZB_SMEM_ATTR(5);
#undef ZB_SMEM_ATTR
    attr[dev].store(true);
  }
  const bool up = mode_a == SRC_UP && chA > 0;
  const int nth = up ? CB_NTH_UP : CB_NTH, stages = cb_stages(up);
  const int smem_sm = 228 * 1024, per_cta_reserved = 1024;
  const int by_tmem = 512 / cols, by_threads = cb_per_sm(nth);
  size_t smem = cb8_smem_bytes(cinp, coutp, stages);
  if (by_tmem < by_threads) {
    const size_t floor_bytes = (size_t)(smem_sm / (by_tmem + 1) - per_cta_reserved + 16);
    smem = std::max(smem, floor_bytes);
  }
  if (smem > 227 * 1024) return ZB_E_UNSUPPORTED;
  const int fit = std::max(1, std::min(by_threads, (int)(smem_sm / (smem + per_cta_reserved))));
  const long long nreg = (long long)((W + CBX - 1) / CBX) * ((H + CBY - 1) / CBY) * B;
  // CTAs per SM: the most that leave no SM waiting on a last round
  int per_sm = 1;
  auto rounds = [&](int k) {
    const long long g = (long long)sms[dev] * k;
    return (nreg + g - 1) / g * k;
  };
  for (int k = 2; k <= fit; ++k)
    if (rounds(k) <= rounds(per_sm)) per_sm = k;
  const int grid = (int)std::max<long long>(1, std::min<long long>(nreg, (long long)sms[dev] * per_sm));
  // tensor maps of the sources read as stored (the upsampled source, and one
  // whose map cannot be encoded, stay on the cp.async copies)
  CUtensorMap tm_a, tm_b;
  std::memset(&tm_a, 0, sizeof(tm_a));
  std::memset(&tm_b, 0, sizeof(tm_b));
  const int tma_a = (mode_a == SRC_DIRECT && chA > 0 && cb8_map(&tm_a, inA, chA, B, H, W)) ? 1 : 0;
  const int tma_b = (chB > 0 && cb8_map(&tm_b, inB, chB, B, H, W)) ? 1 : 0;
  switch (cinp / 16) {
#define ZB_CB8(G)                                                                              \
  case G:                                                                                      \
    ZB_CUDA_TRY(pdl_launch(up ? conv3x3_cb8<G, CB_NTH_UP> : conv3x3_cb8<G, CB_NTH>, dim3(grid), dim3(nth), smem, st, inA, chA, mode_a, inB, \
                           chB, cin, w, bias, out, pool, cout, out_form, B, H, W, act, cols,   \
                           stages, unet_err_word(), tm_a, tm_b, tma_a, tma_b));                \
    break
    ZB_CB8(1); ZB_CB8(2); ZB_CB8(3); ZB_CB8(5);
#undef ZB_CB8
    default: return ZB_E_UNSUPPORTED;
  }
  return zb_launch_check();
}

static int conv(const float* inA, int cin_a, const float* inB, int cin,
                const __nv_bfloat16* w, const float* bias, float* out, int cout, int B, int H,
                int W, int act, cudaStream_t st, int mode_a = SRC_DIRECT,
                const float* ytanh = nullptr) {
  if (g_conv_impl >= 1)
    return conv_tc_launch(inA, cin_a, inB, cin, w, bias, out, cout, B, H, W, act, mode_a, ytanh,
                          st);
  dim3 grid((W + TS - 1) / TS, (H + TS - 1) / TS, B);
  switch (cout) {
#define ZB_CONV(N) case N: conv3x3_fwd<N><<<grid, NTT, 0, st>>>(inA, cin_a, inB, cin, w, bias, out, B, H, W, act, mode_a, ytanh); break;
    ZB_CONV(1) ZB_CONV(8) ZB_CONV(16) ZB_CONV(24) ZB_CONV(32) ZB_CONV(48) ZB_CONV(72)
#undef ZB_CONV
    default: return ZB_E_UNSUPPORTED;
  }
  return zb_launch_check();
}

// one layer's partial weight and bias gradients: `up` input channels of the half
// resolution inUp (may be 0), then cin from `in`
static int wgrad(const float* in, int cin, const float* dout, int cout, float* part, int B, int H,
                 int W, cudaStream_t st, int mode = SRC_DIRECT, const float* inUp = nullptr,
                 int up = 0) {
  const WgShape g = wg_shape(cin, cout, B, H, W, up);
  static std::atomic<unsigned> attr{0u};
  int dev = 0;
  ZB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 32 || g.smem > 227 * 1024) return ZB_E_UNSUPPORTED;
  if (!(attr.load() & (1u << dev))) {
    ZB_CUDA_TRY(cudaFuncSetAttribute(conv3x3_wgrad<WG_COT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     227 * 1024));
    ZB_CUDA_TRY(cudaFuncSetAttribute(conv3x3_wgrad<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     227 * 1024));
    ZB_CUDA_TRY(cudaFuncSetAttribute(conv3x3_wgrad_up, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     227 * 1024));
    attr.fetch_or(1u << dev);
  }
  if (up) {
    const int pairs = up * (cout / WG_COT);
    if (cout % WG_COT != 0 || pairs > UG_THREADS) return ZB_E_UNSUPPORTED;
    const int nsl = std::max(1, std::min(8, UG_THREADS / pairs));
    const size_t stage = (size_t)UG_P * 9 * cout + (size_t)up * (UG_P + 1) + (size_t)cout * UG_FS;
    const size_t red = nsl > 1 ? (size_t)pairs * nsl * 9 * WG_COT : 0;
    ZB_CUDA_TRY(pdl_launch(conv3x3_wgrad_up, dim3(g.slots), dim3(UG_THREADS),
                           std::max(stage, red) * sizeof(float), st, inUp, up, dout, cout, part,
                           cin, B, H, W, nsl));
  }
  ZB_CUDA_TRY(pdl_launch(cout % WG_COT == 0 ? conv3x3_wgrad<WG_COT> : conv3x3_wgrad<1>,
                         dim3(g.slots, g.nchunk), dim3(g.threads), g.smem, st, in, cin, dout, cout,
                         part, up, B, H, W, mode, g.ncog, g.cic, g.nsl));
  return zb_launch_check();
}

static int gridn(size_t n) { return (int)std::max<size_t>(1, std::min<size_t>((n + NT - 1) / NT, 148 * 16)); }

// m1 and m2 run at half resolution
static bool layer_half(int l) { return l == 2 || l == 3; }

// the gradient partials' shape of layer l on images H x W (the network's)
static WgShape wg_layer(const Net& n, int l, int B, int H, int W) {
  const int up = l == 4 ? n.c2 : 0;
  return wg_shape(n.cin[l] - up, n.cout[l], B, layer_half(l) ? H / 2 : H,
                  layer_half(l) ? W / 2 : W, up);
}

// activation buffers (floats) for a batch of B images H x W
struct Acts {
  float *in, *e1, *e2, *m1, *m2, *o1, *out, *s, *part;
  // training: gradients and scratch
  float *d_e1, *d_e2, *d_p, *d_m1, *d_m2, *d_cat, *d_o1, *d_out, *res, *lnum, *lden, *tmp;
  __nv_bfloat16* wflip;
  float* wpart[6];   // partial weight gradients of each layer
};

static size_t acts_floats(const Net& n, int B, int H, int W, bool train) {
  const size_t N0 = (size_t)B * H * W, N1 = (size_t)B * (H / 2) * (W / 2);
  // in (2), e1, e2 (c1 each), m1, m2 (c2 each, half resolution), o1 (c1), out
  size_t f = 2 * N0 + 2 * (size_t)n.c1 * N0 + 2 * (size_t)n.c2 * N1 + (size_t)n.c1 * N0 + N0 +
             512 + RMS_PARTS;
  if (train)
    f += 2 * (size_t)n.c1 * N0 + (size_t)n.c1 * N1 + 2 * (size_t)n.c2 * N1 +
         (size_t)(n.c1 + n.c2) * N0 + (size_t)n.c1 * N0 + N0 + N0 + 1024 +
         (size_t)n.c1 * N0 + (n.nw + 64);   // tmp + flipped weights (bf16 fits in floats)
  if (train)
    for (int l = 0; l < 6; ++l) {
      const WgShape g = wg_layer(n, l, B, H, W);
      f += (size_t)g.slots * g.part;
    }
  return f;
}

static Acts acts_split(const Net& n, void* base, int B, int H, int W, bool train) {
  const size_t N0 = (size_t)B * H * W, N1 = (size_t)B * (H / 2) * (W / 2);
  float* f = (float*)base;
  Acts a;
  std::memset(&a, 0, sizeof(a));
  a.in = f; f += 2 * N0;
  a.e1 = f; f += (size_t)n.c1 * N0;
  a.e2 = f; f += (size_t)n.c1 * N0;
  a.m1 = f; f += (size_t)n.c2 * N1;
  a.m2 = f; f += (size_t)n.c2 * N1;
  a.o1 = f; f += (size_t)n.c1 * N0;
  a.out = f; f += N0;
  a.s = f; f += 512;   // per-image RMS, batch <= 512
  a.part = f; f += RMS_PARTS;
  if (train) {
    a.d_e1 = f; f += (size_t)n.c1 * N0;
    a.d_e2 = f; f += (size_t)n.c1 * N0;
    a.d_p = f; f += (size_t)n.c1 * N1;
    a.d_m1 = f; f += (size_t)n.c2 * N1;
    a.d_m2 = f; f += (size_t)n.c2 * N1;
    a.d_cat = f; f += (size_t)(n.c1 + n.c2) * N0;
    a.d_o1 = f; f += (size_t)n.c1 * N0;
    a.d_out = f; f += N0;
    a.res = f; f += N0;
    a.lnum = f; f += 512;
    a.lden = f; f += 512;
    a.tmp = f; f += (size_t)n.c1 * N0;
    a.wflip = (__nv_bfloat16*)f;
    f += n.nw + 64;
    for (int l = 0; l < 6; ++l) {
      const WgShape g = wg_layer(n, l, B, H, W);
      a.wpart[l] = f;
      f += (size_t)g.slots * g.part;
    }
  }
  return a;
}

// forward of the network from a.in; weights bf16, biases float32
static int forward(const Net& n, const Acts& a, const __nv_bfloat16* w, const float* b, int B, int H,
                   int W, cudaStream_t st, int act = ACT_TANH) {
  const int H1 = H / 2, W1 = W / 2;
  int rc;
  if ((rc = conv(a.in, 2, nullptr, 2, w + n.off_w[0], b + n.off_b[0], a.e1, n.c1, B, H, W, act, st))) return rc;
  if ((rc = conv(a.e1, n.c1, nullptr, n.c1, w + n.off_w[1], b + n.off_b[1], a.e2, n.c1, B, H, W, act, st))) return rc;
  // pool(e2) and up(m2) are read through the convolutions' loaders, never stored
  if ((rc = conv(a.e2, n.c1, nullptr, n.c1, w + n.off_w[2], b + n.off_b[2], a.m1, n.c2, B, H1, W1, act, st, SRC_POOL))) return rc;
  if ((rc = conv(a.m1, n.c2, nullptr, n.c2, w + n.off_w[3], b + n.off_b[3], a.m2, n.c2, B, H1, W1, act, st))) return rc;
  if ((rc = conv(a.m2, n.c2, a.e2, n.c2 + n.c1, w + n.off_w[4], b + n.off_b[4], a.o1, n.c1, B, H, W, act, st, SRC_UP))) return rc;
  if ((rc = conv(a.o1, n.c1, nullptr, n.c1, w + n.off_w[5], b + n.off_b[5], a.out, 1, B, H, W, ACT_NONE, st))) return rc;
  return zb_launch_check();
}

// Inference forward in the chunked bf16 layout (conv3x3_cb8), the same bits as
// forward(): the activations live where the float32 ones would (the chunked
// tensors take fewer bytes); e2's epilogue also writes pool(e2), o1 reads
// up(m2) through its loader.  The network output goes to a.out (float32).
struct ActsCB8 {
  uint4 *in, *e1, *e2, *e2p, *m1, *m2, *o1;
};

static bool acts_cb8(const Net& n, const Acts& a, int B, int H, int W, ActsCB8* c) {
  const size_t N0 = (size_t)B * H * W, N1 = (size_t)B * (H / 2) * (W / 2);
  uint4* p = (uint4*)a.in;
  c->in = p; p += N0;
  c->e1 = p; p += (size_t)(n.c1 / 8) * N0;
  c->e2 = p; p += (size_t)(n.c1 / 8) * N0;
  c->e2p = p; p += (size_t)(n.c1 / 8) * N1;
  c->m1 = p; p += (size_t)(n.c2 / 8) * N1;
  c->m2 = p; p += (size_t)(n.c2 / 8) * N1;
  c->o1 = p; p += (size_t)(n.c1 / 8) * N0;
  return (const void*)p <= (const void*)a.out && (((uintptr_t)a.in) & 15u) == 0;
}

static int forward_cb8(const Net& n, const Acts& a, const ActsCB8& c, const __nv_bfloat16* w,
                       const float* b, int B, int H, int W, cudaStream_t st) {
  const int H1 = H / 2, W1 = W / 2, k1 = n.c1 / 8, k2 = n.c2 / 8;
  int rc;
  if ((rc = conv_cb8_launch(c.in, 1, SRC_DIRECT, nullptr, 0, 2, w + n.off_w[0], b + n.off_b[0],
                            c.e1, nullptr, n.c1, CB_OUT_CHUNKED, B, H, W, ACT_TANH_SFU, st))) return rc;
  if ((rc = conv_cb8_launch(c.e1, k1, SRC_DIRECT, nullptr, 0, n.c1, w + n.off_w[1], b + n.off_b[1],
                            c.e2, c.e2p, n.c1, CB_OUT_CHUNKED, B, H, W, ACT_TANH_SFU, st))) return rc;
  if ((rc = conv_cb8_launch(c.e2p, k1, SRC_DIRECT, nullptr, 0, n.c1, w + n.off_w[2], b + n.off_b[2],
                            c.m1, nullptr, n.c2, CB_OUT_CHUNKED, B, H1, W1, ACT_TANH_SFU, st))) return rc;
  if ((rc = conv_cb8_launch(c.m1, k2, SRC_DIRECT, nullptr, 0, n.c2, w + n.off_w[3], b + n.off_b[3],
                            c.m2, nullptr, n.c2, CB_OUT_CHUNKED, B, H1, W1, ACT_TANH_SFU, st))) return rc;
  if ((rc = conv_cb8_launch(c.m2, k2, SRC_UP, c.e2, k1, n.c2 + n.c1, w + n.off_w[4], b + n.off_b[4],
                            c.o1, nullptr, n.c1, CB_OUT_CHUNKED, B, H, W, ACT_TANH_SFU, st))) return rc;
  if ((rc = conv_cb8_launch(c.o1, k1, SRC_DIRECT, nullptr, 0, n.c1, w + n.off_w[5], b + n.off_b[5],
                            a.out, nullptr, 1, CB_OUT_F32, B, H, W, ACT_NONE, st))) return rc;
  return zb_launch_check();
}

// data gradient through conv layer l: din (cin channels) from dout (cout) with the
// flipped weights, times 1 - y^2 where y is given
static int data_grad(const Net& n, int l, const __nv_bfloat16* wflip, const float* dout, float* din,
                     int B, int H, int W, cudaStream_t st, const float* y = nullptr) {
  const int ci = n.cin[l], co = n.cout[l];
  return conv(dout, co, nullptr, co, wflip + n.off_w[l], nullptr, din, ci, B, H, W, ACT_NONE, st,
              SRC_DIRECT, y);
}

}  // namespace unet
}  // namespace zb

using namespace zb;
using namespace zb::unet;

extern "C" {

int zb_unet_conv_impl(int impl) {
  const int prev = g_conv_impl;
  if (impl == 0 || impl == 1 || impl == 2) g_conv_impl = impl;
  return prev;
}

int zb_unet_status(int clear) {
  unsigned* p = unet_err_word();
  if (!p) return ZB_E_CUDA;
  unsigned v = 0;
  ZB_CUDA_TRY(cudaMemcpy(&v, p, sizeof(v), cudaMemcpyDeviceToHost));
  if (clear && v) {
    const unsigned z = 0;
    ZB_CUDA_TRY(cudaMemcpy(p, &z, sizeof(z), cudaMemcpyHostToDevice));
  }
  return (int)v;
}

size_t zb_unet_param_count(int c1, int c2, size_t* n_weights, size_t* n_biases) {
  if (!valid_channels(c1, c2)) return 0;
  const Net n = net_layout(c1, c2);
  if (n_weights) *n_weights = n.nw;
  if (n_biases) *n_biases = n.nb;
  return n.nw + n.nb;
}

size_t zb_smoother_workspace_bytes(int c1, int c2, int nx, int ny) {
  if (!valid_channels(c1, c2) || nx < 2 || ny < 2 || (nx & 1) || (ny & 1)) return 0;
  return acts_floats(net_layout(c1, c2), 1, nx, ny, false) * sizeof(float) + 256;
}

int zb_smoother_apply(const zb_smoother* smo, const float* f, const float* x_in, float* x_out,
                      const float* cx, const float* cy, float* r_scratch, int nx, int ny,
                      double dx, int pre, zb_stream_t stream) {
  (void)pre;
  if (!smo || !f || !x_out || !cx || !cy || !r_scratch) return ZB_E_ARG;
  if (!valid_channels(smo->c1, smo->c2) || (nx & 1) || (ny & 1)) return ZB_E_ARG;
  if (nx > smo->max_nx || ny > smo->max_ny || !smo->act ||
      smo->act_bytes < zb_smoother_workspace_bytes(smo->c1, smo->c2, nx, ny))
    return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const Net n = net_layout(smo->c1, smo->c2);
  const Acts a = acts_split(n, smo->act, 1, nx, ny, false);
  const float idx2 = (float)(1.0 / (dx * dx));
  const size_t N0 = (size_t)nx * ny;
  const int P = rms_parts(1, N0);
  ZB_CUDA_TRY(pdl_launch(residual_rms_kernel, dim3(P), dim3(NT * RR_SPLIT), 0, st, f, x_in, cx, cy, nx, ny,
                         idx2, r_scratch, P, a.part));
  int rc;
  ActsCB8 c;
  if (g_conv_impl == 1 && acts_cb8(n, a, 1, nx, ny, &c)) {
    ZB_CUDA_TRY(pdl_launch(features_cb8_kernel, dim3(std::min(gridn(N0), 148 * 8)), dim3(NT), 0, st,
                           (const float*)r_scratch, (const float*)a.part, P, a.s, cx, cy, nx, ny,
                           1.0f / smo->cmax, c.in));
    rc = forward_cb8(n, a, c, (const __nv_bfloat16*)smo->w, smo->b, 1, nx, ny, st);
  } else {
    ZB_CUDA_TRY(pdl_launch(rms_final_kernel, dim3(1), dim3(32), 0, st, (const float*)a.part, P, N0,
                           a.s));
    ZB_CUDA_TRY(pdl_launch(features_kernel, dim3(gridn(N0)), dim3(NT), 0, st,
                           (const float*)r_scratch, (const float*)a.s, cx, cy, 1, nx, ny,
                           1.0f / smo->cmax, a.in));
    rc = forward(n, a, (const __nv_bfloat16*)smo->w, smo->b, 1, nx, ny, st, ACT_TANH_SFU);
  }
  if (rc) return rc;
  ZB_CUDA_TRY(pdl_launch(scale_out_kernel, dim3(gridn(N0)), dim3(NT), 0, st, (const float*)a.out,
                         (const float*)a.s, cx, cy, 1, nx, ny, (float)(dx * dx), x_in, x_out));
  return zb_launch_check();
}

size_t zb_unet_train_workspace_bytes(int c1, int c2, int batch, int n) {
  if (!valid_channels(c1, c2) || batch < 1 || batch > 512 || n < 4 || (n & 1)) return 0;
  return acts_floats(net_layout(c1, c2), batch, n, n, true) * sizeof(float) + 256;
}

int zb_unet_forward(const zb_unet_trainer* t, const float* r, const float* cx, const float* cy,
                    double dx, float* y, zb_stream_t stream) {
  if (!t || !r || !cx || !cy || !y || !valid_channels(t->c1, t->c2)) return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const Net n = net_layout(t->c1, t->c2);
  const Acts a = acts_split(n, t->act, t->batch, t->n, t->n, true);
  const int B = t->batch, H = t->n, W = t->n;
  const size_t N0 = (size_t)B * H * W;
  int rc = rms(r, B, (size_t)H * W, a.part, a.s, st);
  if (rc) return rc;
  ZB_CUDA_TRY(pdl_launch(features_kernel, dim3(gridn(N0)), dim3(NT), 0, st, r, (const float*)a.s,
                         cx, cy, B, H, W, 1.0f / t->cmax, a.in));
  rc = forward(n, a, (const __nv_bfloat16*)t->w_bf16, t->b_master, B, H, W, st);
  if (rc) return rc;
  ZB_CUDA_TRY(pdl_launch(scale_out_kernel, dim3(gridn(N0)), dim3(NT), 0, st, (const float*)a.out,
                         (const float*)a.s, cx, cy, B, H, W, (float)(dx * dx),
                         (const float*)nullptr, y));
  return zb_launch_check();
}

int zb_unet_backward(const zb_unet_trainer* t, const float* r, const float* target,
                     const float* cx, const float* cy, double dx, double* loss_out,
                     zb_stream_t stream) {
  if (!t || !r || !cx || !cy || !valid_channels(t->c1, t->c2)) return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const Net n = net_layout(t->c1, t->c2);
  const Acts a = acts_split(n, t->act, t->batch, t->n, t->n, true);
  const int B = t->batch, H = t->n, W = t->n, H1 = H / 2, W1 = W / 2;
  const size_t N0 = (size_t)B * H * W, N1 = (size_t)B * H1 * W1;
  const float idx2 = (float)(1.0 / (dx * dx)), dx2 = (float)(dx * dx);
  const __nv_bfloat16* w = (const __nv_bfloat16*)t->w_bf16;
  int rc;
  // forward (keeps activations), y into a.tmp
  if ((rc = zb_unet_forward(t, r, cx, cy, dx, a.tmp, stream))) return rc;
  const dim3 g0(gridn(N0)), nt(NT);
  FlipTab ft;
  for (int l = 0; l < 6; ++l) {
    ft.off[l] = (int)n.off_w[l];
    ft.cin[l] = n.cin[l];
    ft.cout[l] = n.cout[l];
  }
  ZB_CUDA_TRY(pdl_launch(flip_weights, dim3(gridn(n.nw)), nt, 0, st, w, a.wflip, ft, (int)n.nw));
  if (target) {
    // energy loss: res = e - y, (res . A res) / (e . A e); A res -> d_out,
    // A e -> tmp (y is no longer needed once res is formed)
    ZB_CUDA_TRY(pdl_launch(sub_kernel, g0, nt, 0, st, target, (const float*)a.tmp, N0, a.res));
    ZB_CUDA_TRY(pdl_launch(patch_apply, g0, nt, 0, st, (const float*)a.res, cx, cy, B, H, W, idx2,
                           a.d_out));
    ZB_CUDA_TRY(pdl_launch(patch_apply, g0, nt, 0, st, target, cx, cy, B, H, W, idx2, a.tmp));
    ZB_CUDA_TRY(pdl_launch(loss_kernel, dim3(B), nt, 0, st, (const float*)a.res,
                           (const float*)a.d_out, target, (const float*)a.tmp, B, (size_t)H * W,
                           a.lnum, a.lden));
  } else {
    ZB_CUDA_TRY(pdl_launch(patch_residual, g0, nt, 0, st, r, (const float*)a.tmp, cx, cy, B, H, W,
                           idx2, a.res));
    ZB_CUDA_TRY(pdl_launch(loss_kernel, dim3(B), nt, 0, st, (const float*)a.res,
                           (const float*)a.res, r, r, B, (size_t)H * W, a.lnum, a.lden));
  }
  if (loss_out)
    ZB_CUDA_TRY(pdl_launch(loss_total, dim3(1), dim3(32), 0, st, (const float*)a.lnum,
                           (const float*)a.lden, B, loss_out));
  ZB_CUDA_TRY(pdl_launch(loss_grad_kernel, g0, nt, 0, st, (const float*)a.res,
                         (const float*)(target ? a.d_out : nullptr), cx, cy, (const float*)a.lden,
                         (const float*)a.s, B, H, W, idx2, dx2, a.d_out));
  // out = conv(o1)
  if ((rc = wgrad(a.o1, n.c1, a.d_out, 1, a.wpart[5], B, H, W, st))) return rc;
  if ((rc = data_grad(n, 5, a.wflip, a.d_out, a.d_o1, B, H, W, st, a.o1))) return rc;
  // o1 = tanh(conv([u, e2]))
  if ((rc = wgrad(a.e2, n.c1, a.d_o1, n.c1, a.wpart[4], B, H, W, st, SRC_DIRECT, a.m2, n.c2))) return rc;
  if ((rc = data_grad(n, 4, a.wflip, a.d_o1, a.d_cat, B, H, W, st))) return rc;
  // d_cat = [du (c2), de2_b (c1)]
  ZB_CUDA_TRY(pdl_launch(upsample2_tanh_back, dim3(gridn((size_t)n.c2 * N1)), nt, 0, st,
                         (const float*)a.d_cat, (const float*)a.m2, a.d_m2, n.c2, B, H, W));
  if ((rc = wgrad(a.m1, n.c2, a.d_m2, n.c2, a.wpart[3], B, H1, W1, st))) return rc;
  if ((rc = data_grad(n, 3, a.wflip, a.d_m2, a.d_m1, B, H1, W1, st, a.m1))) return rc;
  if ((rc = wgrad(a.e2, n.c1, a.d_m1, n.c2, a.wpart[2], B, H1, W1, st, SRC_POOL))) return rc;
  if ((rc = data_grad(n, 2, a.wflip, a.d_m1, a.d_p, B, H1, W1, st))) return rc;
  const int slice = plane_slice(n.c1, (long long)N0);
  for (int c = 0; c < n.c1; c += slice) {
    const int nc = std::min(slice, n.c1 - c);
    ZB_CUDA_TRY(pdl_launch(pool_add_tanh_back, dim3(gridn((size_t)nc * N0)), nt, 0, st,
                           (const float*)(a.d_p + (size_t)c * N1),
                           (const float*)(a.d_cat + (size_t)(n.c2 + c) * N0),
                           (const float*)(a.e2 + (size_t)c * N0), a.d_e2 + (size_t)c * N0, nc, B,
                           H, W));
  }
  if ((rc = wgrad(a.e1, n.c1, a.d_e2, n.c1, a.wpart[1], B, H, W, st))) return rc;
  if ((rc = data_grad(n, 1, a.wflip, a.d_e2, a.d_e1, B, H, W, st, a.e1))) return rc;
  if ((rc = wgrad(a.in, 2, a.d_e1, n.c1, a.wpart[0], B, H, W, st))) return rc;
  WgReduce R;
  R.first[0] = 0;
  for (int l = 0; l < 6; ++l) {
    const WgShape g = wg_layer(n, l, B, H, W);
    R.part[l] = a.wpart[l];
    R.slots[l] = g.slots;
    R.cin[l] = n.cin[l];
    R.nb[l] = n.cout[l];
    R.nw[l] = n.cout[l] * n.cin[l] * 9;
    R.off_w[l] = (int)n.off_w[l];
    R.off_b[l] = (int)n.off_b[l];
    R.first[l + 1] = R.first[l] + R.nw[l] + R.nb[l];
  }
  ZB_CUDA_TRY(pdl_launch(wgrad_reduce, dim3((R.first[6] + 31) / 32), nt, 0, st, R, t->g_w, t->g_b));
  return zb_launch_check();
}

int zb_unet_adam(const zb_unet_trainer* t, float lr, int step, zb_stream_t stream) {
  if (!t || step < 1 || !valid_channels(t->c1, t->c2)) return ZB_E_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const Net n = net_layout(t->c1, t->c2);
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  // biases stay float32: the bf16 shadow is only written for the weights
  const AdamSet W = {t->w_master, t->m_w, t->v_w, t->g_w, (__nv_bfloat16*)t->w_bf16};
  const AdamSet Bi = {t->b_master, t->m_b, t->v_b, t->g_b, (__nv_bfloat16*)t->b_shadow};
  ZB_CUDA_TRY(pdl_launch(adam_kernel, dim3(gridn(n.nw + n.nb)), dim3(NT), 0, st, W, Bi, (int)n.nw,
                         (int)n.nb, lr, b1, b2, eps, c1, c2));
  return zb_launch_check();
}

}  // extern "C"
