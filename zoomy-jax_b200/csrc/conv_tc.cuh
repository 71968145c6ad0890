// 3x3 convolution as an implicit GEMM on the 5th-generation tensor cores
// (tcgen05.mma, kind::f16 with bf16 operands, float32 accumulation in TMEM).
//
// GEMM view of one output tile: M = 128 pixels (an 8-wide by 16-tall block;
// GEMM row m is pixel (x0 + m % 8, y0 + m / 8)), N = output channels rounded
// up to 16, K = 9 taps x input channels rounded up to 16.  No im2col copy is
// made: the input tile with its one-pixel halo (10 x 18 pixels) is staged once
// in shared memory in the canonical no-swizzle K-major layout,
//   byte(chunk, q) = chunk * (180 * 16) + q * 16,   q = halo pixel (y * 10 + x),
// 8 consecutive channels (one 16-byte core-matrix row) per (chunk, q), so the
// A operand of tap (dy, dx) is the same buffer with its descriptor start moved
// by (dy * 10 + dx) * 16 bytes: rows of one 8-pixel line are 16 bytes apart
// (the core matrix), successive lines 160 bytes apart (stride byte offset),
// the two 8-channel halves of a K=16 step 2880 bytes apart (leading byte
// offset).  The weights sit next to it as [tap][chunk][n][8 channels].  One
// thread issues the 9 * Cin/16 MMAs of a tile and commits them to an
// mbarrier; the warps then read the accumulator rows they own out of TMEM
// (tcgen05.ld 32x32b), add the bias, apply tanh and store float32 planes.
// CTAs are persistent over the tiles; the weights are staged once per CTA.
//
// Every wait is bounded: on a timeout the kernel raises a flag in the error
// word, skips the tile's stores, and still releases its TMEM columns.
#pragma once

#include <cuda.h>   // CUtensorMap (the type only; the encoder is fetched at run time)
#include <cuda_bf16.h>
#include <stdint.h>

namespace zb {
namespace unet {

constexpr int TCX = 8, TCY = 16;            // output tile (M = 128)
constexpr int THX = TCX + 2, THY = TCY + 2; // halo tile
constexpr int THP = THX * THY;              // 180 halo pixels
constexpr int TC_THREADS = 256, TC_PER_SM = 3;   // resident CTAs the registers are bounded for
constexpr unsigned TC_SPIN_LIMIT = 1u << 24;

__host__ __device__ constexpr int pad16(int c) { return (c + 15) & ~15; }

// How input channels [0, cin_a) are read: as stored, as the nearest-neighbour
// 2x upsampling of a half-resolution field (the U-Net's up(m2)), or as the 2x2
// average of a double-resolution field (pool(e2)); the last two replace the
// materialised upsampled / pooled activations.  Channels [cin_a, cin) are read
// as stored from the second source.
enum { SRC_DIRECT = 0, SRC_UP = 1, SRC_POOL = 2 };

__device__ __forceinline__ float src_at(const float* __restrict__ inA, int cin_a,
                                        const float* __restrict__ inB, int mode_a, int ci, int b,
                                        int B, int H, int W, int yy, int xx) {
  if (ci < cin_a) {
    if (mode_a == SRC_UP) {
      const int h = H >> 1, w = W >> 1;
      return inA[((size_t)ci * B + b) * h * w + (size_t)(yy >> 1) * w + (xx >> 1)];
    }
    if (mode_a == SRC_POOL) {
      const int w = 2 * W;
      const float* q = inA + ((size_t)ci * B + b) * (size_t)(2 * H) * w + (size_t)(2 * yy) * w + 2 * xx;
      return 0.25f * (q[0] + q[1] + q[w] + q[w + 1]);
    }
    return inA[((size_t)ci * B + b) * H * W + (size_t)yy * W + xx];
  }
  return inB[((size_t)(ci - cin_a) * B + b) * H * W + (size_t)yy * W + xx];
}

// the values of channels c0 .. c0 + 7 at one pixel, zero outside the image and
// past the source's channels; the eight (SRC_POOL: 32) loads are independent and
// in flight together (one value at a time, each with its own choice of source, the
// staging of 16^2 pooled images took 30 us of a 34 us launch)
__device__ __forceinline__ void tc_gather8(float* f, const float* __restrict__ inA, int cin_a,
                                           const float* __restrict__ inB, int cin, int mode_a,
                                           int c0, int b, int B, int H, int W, int yy, int xx,
                                           bool inside) {
  const bool fromA = c0 < cin_a;
  const int n = inside ? (fromA ? min(cin_a, cin) : cin) - c0 : 0;
  const size_t p0 = (size_t)yy * W + xx;
  if (fromA && mode_a == SRC_POOL) {
    const int w = 2 * W;
    const size_t ps = (size_t)B * 4 * H * W;
    const float* q = inA + (size_t)c0 * ps + (size_t)b * 4 * H * W + (size_t)(2 * yy) * w + 2 * xx;
    float g[8][4];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const bool in = k < n;
      g[k][0] = in ? q[k * ps] : 0.0f;
      g[k][1] = in ? q[k * ps + 1] : 0.0f;
      g[k][2] = in ? q[k * ps + w] : 0.0f;
      g[k][3] = in ? q[k * ps + w + 1] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = 0.25f * (g[k][0] + g[k][1] + g[k][2] + g[k][3]);
    return;
  }
  const bool up = fromA && mode_a == SRC_UP;
  const size_t hw = up ? (size_t)(H >> 1) * (W >> 1) : (size_t)H * W, ps = (size_t)B * hw;
  const float* q = (fromA ? inA + (size_t)c0 * ps : inB + (size_t)(c0 - cin_a) * ps) + (size_t)b * hw +
                   (up ? (size_t)(yy >> 1) * (W >> 1) + (xx >> 1) : p0);
#pragma unroll
  for (int k = 0; k < 8; ++k) f[k] = k < n ? q[k * ps] : 0.0f;
}

__host__ __device__ inline size_t tc_smem_bytes(int cinp, int coutp) {
  return (size_t)cinp * THP * 2 + (size_t)9 * cinp * coutp * 2 + 64;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// canonical K-major, no-swizzle shared-memory matrix descriptor (sm_100)
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;   // descriptor version for sm_100
  // base offset 0, legacy LBO mode, layout type 0 (no swizzle)
  return d;
}

// instruction descriptor: D f32, A and B bf16, both K-major, M = 128, N
__device__ __forceinline__ uint32_t tc_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t dtmem, uint64_t adesc, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
      "}\n"
      :
      : "r"(dtmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}

// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(p));
  return p != 0;
}

// The 9 G MMAs of one 128-pixel tile (G = input channels / 16), issued by one
// thread: a is the staged tile's first pixel (chunk stride CS bytes, HX pixels a
// line), b the weights.  Unrolled over taps and channel groups, so that a step is
// an add to each descriptor's start (with the loops at run time the issue alone
// took longer than the tensor core).
template <int G, int CS, int HX>
__device__ __forceinline__ void tc_issue_tile(uint32_t tmem, uint32_t a, uint32_t b, int coutp,
                                              uint32_t idesc) {
  const uint64_t da = tc_desc(a, CS, HX * 16);
  uint64_t db = tc_desc(b, coutp * 16, 128);
#pragma unroll
  for (int tap = 0; tap < 9; ++tap)
#pragma unroll
    for (int g = 0; g < G; ++g) {
      tc_mma(tmem, da + (uint64_t)((2 * g * CS + ((tap / 3) * HX + tap % 3) * 16) >> 4), db, idesc,
             tap + g > 0 ? 1u : 0u);
      db += (uint64_t)(2 * coutp);
    }
}

// Weights of a layer into shared memory as [tap][chunk][n][8] bf16, zero outside
// (cout, cin).  A thread takes the 8 channels x 9 taps of one (n, chunk): 144
// contiguous bytes, nine 16-byte loads where they are aligned (element by
// element, 72 loads of two bytes 18 bytes apart, the staging took a few
// microseconds of every CTA).
__device__ __forceinline__ void tc_stage_weights(unsigned char* sB,
                                                 const __nv_bfloat16* __restrict__ w, int cin,
                                                 int cout, int nch, int coutp, int tid, int nth) {
  for (int e = tid; e < nch * coutp; e += nth) {
    const int ch = e / coutp, n = e - ch * coutp;
    const __nv_bfloat16* src = w + ((size_t)n * cin + ch * 8) * 9;
    __align__(16) unsigned short v[72];
    if (n < cout && ch * 8 + 8 <= cin && ((uintptr_t)src & 15u) == 0) {
#pragma unroll
      for (int i = 0; i < 9; ++i) ((uint4*)v)[i] = ((const uint4*)src)[i];
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int tap = 0; tap < 9; ++tap)
          v[k * 9 + tap] = n < cout && ch * 8 + k < cin
                               ? ((const unsigned short*)src)[k * 9 + tap] : (unsigned short)0;
    }
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      __align__(16) unsigned short o[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = v[k * 9 + tap];
      *(uint4*)(sB + ((size_t)(tap * nch + ch) * coutp + n) * 16) = *(const uint4*)o;
    }
  }
}

__device__ __forceinline__ void tc_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               :
               : "r"(mbar)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(mbar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Activation of the tensor-core epilogues: act 0 none, 1 tanhf, 2 tanh on the
// SFU (tanh.approx.f32), whose maximum relative error, about 2^-11 per the PTX
// ISA, sits below the bf16 rounding every activation takes before the next
// layer reads it.  The smoother application uses 2; training keeps 1, so its
// gradients stay those of the exact activation.
__device__ __forceinline__ float tanh_sfu(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// out[co][b][y][x] = act(bias[co] + sum_ci sum_tap w[co][ci][tap] in[ci][b][y+dy-1][x+dx-1])
// with the input channels [0, cin_a) from inA (read per mode_a, see src_at)
// and [cin_a, cin) from inB, the input rounded to bf16, zero padding at the
// image border.  err (may be null)
// receives 1 when an mbarrier wait timed out.
template <int G>
__global__ void __launch_bounds__(TC_THREADS, TC_PER_SM)
conv3x3_tc(const float* __restrict__ inA, int cin_a, const float* __restrict__ inB, int cin,
           const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias,
           float* __restrict__ out, int cout, int B, int H, int W, int act, int mode_a,
           const float* __restrict__ ytanh, int tmem_cols, unsigned* err) {
  extern __shared__ __align__(128) unsigned char tc_sm[];
  const int cinp = pad16(cin), coutp = pad16(cout);
  const int nch = cinp / 8;
  unsigned char* sA = tc_sm;
  unsigned char* sB = tc_sm + (size_t)cinp * THP * 2;
  unsigned long long* mbar = (unsigned long long*)(sB + (size_t)9 * cinp * coutp * 2);
  uint32_t* tmem_slot = (uint32_t*)(mbar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  tc_stage_weights(sB, w, cin, cout, nch, coutp, tid, TC_THREADS);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :
                 : "r"(smem_u32(tmem_slot)), "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // The weights were read above, before this wait: the launch directly before this one must
  // not write them, and each of its CTAs must wait for its own predecessor before it lets
  // this one start.  Between adam_kernel or flip_weights and the first convolution that
  // reads their result stand at least the features' or the loss's launches.
  pdl_enter();
  const uint32_t tmem = *tmem_slot;
  const uint32_t mbar_a = smem_u32(mbar);
  const uint32_t sA_a = smem_u32(sA), sB_a = smem_u32(sB);
  const uint32_t idesc = tc_idesc(coutp);
  const size_t plane = (size_t)B * H * W;
  const int tiles_x = (W + TCX - 1) / TCX, tiles_y = (H + TCY - 1) / TCY;
  const int ntiles = tiles_x * tiles_y * B;
  uint32_t parity = 0;
  bool failed = false;

  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int b = t / (tiles_x * tiles_y);
    const int r = t - b * tiles_x * tiles_y;
    const int x0 = (r % tiles_x) * TCX, y0 = (r / tiles_x) * TCY;
    const size_t img = (size_t)b * H * W;
    // halo tile: one thread per (chunk, halo pixel), 8 channels -> 16 bytes
    for (int e = tid; e < nch * THP; e += TC_THREADS) {
      const int q = e % THP, ch = e / THP;
      const int yy = y0 - 1 + q / THX, xx = x0 - 1 + q % THX;
      __align__(16) __nv_bfloat16 v[8];
      const bool inside = yy >= 0 && yy < H && xx >= 0 && xx < W;
      // a chunk is all of A or all of B (cin_a is a multiple of 8 where B follows)
      float f[8];
      tc_gather8(f, inA, cin_a, inB, cin, mode_a, ch * 8, b, B, H, W, yy, xx, inside);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = __float2bfloat16_rn(f[k]);
      *(uint4*)(sA + ((size_t)ch * THP + q) * 16) = *(const uint4*)v;
    }
    // make the generic-proxy stores visible to the tensor core's async proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0 && elect_one()) {
      tc_issue_tile<G, THP * 16, THX>(tmem, sA_a, sB_a, coutp, idesc);
      tc_commit(mbar_a);
    }
    // the activations that a data gradient is multiplied with, on their way while
    // the MMAs run (read in the epilogue one by one they doubled the launch)
    const int m = (warp & 3) * 32 + lane;
    const int x = x0 + (m % TCX), y = y0 + (m / TCX);
    const bool store = x < W && y < H;
    const size_t pix = img + (size_t)y * W + x;
    float yv[16];
    auto load_y = [&](int c0) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        yv[i] = store && c0 + i < cout ? ytanh[(size_t)(c0 + i) * plane + pix] : 0.0f;
    };
    if (ytanh) load_y((warp >> 2) * 16);
    // wait for the tile's MMAs (bounded); the CTA agrees on the outcome so
    // every warp takes the same path through the collective TMEM loads
    bool done = false;
    for (unsigned it = 0; it < TC_SPIN_LIMIT; ++it) {
      if (mbar_try_wait(mbar_a, parity)) { done = true; break; }
    }
    parity ^= 1u;
    if (__syncthreads_or(done ? 0 : 1)) {
      failed = true;
      if (err && tid == 0) atomicExch(err, 1u);
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // epilogue: warps w and w + 4 own accumulator rows (pixels) 32w .. 32w+31 and
    // take every second group of 16 channels
    for (int c0 = (warp >> 2) * 16; c0 < coutp; c0 += 32) {
      float v[16];
      __syncwarp();
      tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int co = c0 + i;
        if (store && co < cout) {
          float s = v[i] + (bias ? bias[co] : 0.0f);
          if (act == 1) s = tanhf(s);
          else if (act == 2) s = tanh_sfu(s);
          if (ytanh) s *= 1.0f - yv[i] * yv[i];   // a data gradient into a tanh
          out[(size_t)co * plane + pix] = s;
        }
      }
      if (ytanh && c0 + 32 < coutp) load_y(c0 + 32);
    }
    // TMEM reads and smem reads of this tile complete before the next tile
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (failed) {
    // give an in-flight MMA a bounded chance to land before releasing TMEM
    for (unsigned it = 0; it < TC_SPIN_LIMIT; ++it)
      if (mbar_try_wait(mbar_a, parity ^ 1u)) break;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(tmem_cols)
                 : "memory");
  }
}

// ── the chunked bf16 activation layout (inference) ──────────────────────────
// An activation of C channels (C a multiple of 8) on B images H x W is stored
// as C / 8 chunks, chunk-major: byte ((chunk * B + b) * H * W + y * W + x) * 16
// holds channels 8 chunk .. 8 chunk + 7 of pixel (b, y, x) as bf16.  A pixel's
// chunk is then one 16-byte core-matrix row of the MMA's A operand, and a row
// of pixels is contiguous, so a tile's halo is staged with coalesced 16-byte
// cp.async copies (zero-filled outside the image) instead of per-thread
// float32 gathers; the producing layer writes it in its epilogue.  Values are
// the float32 activations rounded to bf16 once (the rounding the planar
// kernel applies when it stages them), so a network run through this layout
// gives the same bits as through conv3x3_tc.
constexpr int CBX = 16, CBY = 16;            // output region: two 8 x 16 M tiles
constexpr int CHX = CBX + 2, CHY = CBY + 2;  // halo region
constexpr int CHP = CHX * CHY;               // 324 halo pixels
// one staged chunk: the 18 x 18 halo pixels x 16 bytes, its stride rounded up
// to 128 bytes (the alignment of a tensor-copy destination)
constexpr int CB_CHUNK_BYTES = CHP * 16;                            // 5184
constexpr int CB_CHUNK_STRIDE = ((CB_CHUNK_BYTES + 127) / 128) * 128;  // 5248

// Roles of conv3x3_cb8's warps: 0 .. 15 epilogue (two groups of eight that take
// every second region each; warp w of a group reads TMEM lane quarter w % 4 of M
// tile w / 4), 16 tensor copies, 17 MMA issue, 18 .. 21 (launched for the upsampled
// source only) 16-byte copies.
constexpr int CB_EPI = 16, CB_NTH = 32 * (CB_EPI + 2), CB_NTH_UP = CB_NTH + 128;
// stages of a region's chunks: four hide a tensor copy's latency (two: 299 us the
// application below, four: 268); the wide layer with cp.async copies has room for
// three
constexpr int CB_MAX_STAGES = 4;
__host__ __device__ constexpr int cb_stages(bool up) { return up ? 3 : 4; }
// resident CTAs that the registers are bounded for
__host__ __device__ constexpr int cb_per_sm(int nth) { return nth == CB_NTH ? 2 : 1; }

// weights, staged chunks, biases, mbarriers, the TMEM slot and the failure flag
__host__ __device__ inline size_t cb8_smem_bytes(int cinp, int coutp, int stages) {
  return (size_t)stages * (cinp / 8) * CB_CHUNK_STRIDE + (size_t)9 * cinp * coutp * 2 +
         (size_t)coutp * 4 + 192;
}

// TMA: a 4-D tiled tensor copy of one chunk's halo box into shared memory,
// completing on an mbarrier (no multicast)
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                            int c2, int c3, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];"
      :
      : "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
        "r"(mbar)
      : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
               "r"(src_bytes)
               : "memory");
}

// Output forms of conv3x3_cb8.
enum { CB_OUT_CHUNKED = 0, CB_OUT_F32 = 1 };

// out = act(bias + conv3x3(in)) with in = [A (chA chunks; mode_a SRC_DIRECT
// at H x W or SRC_UP: the nearest 2x upsampling of an H/2 x W/2 field), then
// B (chB chunks at H x W)], cin real channels (the rest of the chunks and the
// padding to 16 read as zeros).  out_form CB_OUT_CHUNKED: out holds cout / 8
// chunks; pool (may be null) also receives the 2x2 average of the float32
// activation (H/2 x W/2 chunks, the average of conv3x3_tc's SRC_POOL loader,
// in its summation order).  CB_OUT_F32: out is float32 planes [co][b][y][x].
// H and W even.  act != 0: tanh on the SFU (the inference activation, act 2
// of conv3x3_tc).
// Staging: the chunks read as stored (A in SRC_DIRECT mode when tma_a, B when
// tma_b) arrive by TMA, one 4-D box (8 channels x 18 x 18 pixels x 1 image
// chunk) per chunk on the maps tm_a / tm_b (out-of-image pixels are filled
// with zeros by the copy), issued by one thread and completed on an mbarrier;
// the upsampled chunks of SRC_UP keep 16-byte cp.async copies (their address
// map is not a box); the padding chunks are zeroed once.  Staged chunk ch of
// stage s sits at (s nch + ch) * CB_CHUNK_STRIDE from the start of dynamic shared
// memory; a CTA whose dynamic shared memory does not start on 128 bytes (the
// alignment a tensor copy's destination needs) stages everything by cp.async.
//
// The CTA is a pipeline of warp roles over its regions, because a region's chain
// (copies, 18 G MMAs, accumulator load, tanh, stores) is long and the tensor core
// busy for a tenth of it: copies run a stage or two ahead of the MMAs, the MMAs an
// accumulator buffer ahead of the epilogue.  empty / full_t / full_c[s]: stage s
// free, its tensor copies landed, its cp.async copies landed; acc_full /
// acc_free[k]: accumulator buffer k.  With all warps in step (stage, MMA,
// epilogue) and several CTAs per SM to overlap, one application on 1024^2 (24, 48)
// took 429 us, now 242 (convolutions 415 -> 226): the wide layer (o1) 143 -> 83, which
// is the 32 cycles that each of a region's 180 MMAs (M = 128, N = 32) takes, e1 44 ->
// 27, e2 68 -> 41, m1 35 -> 19, m2 63 -> 22, out 47 -> 34.  Lines of 128 pixels as
// tiles, the three rows of taps in one MMA (N = 96, a third of the MMAs), gave 218 us
// for the application: an MMA takes about N cycles in every form, and as an output's
// accumulator then moves from line to line, the lines wait for one another.
//
// Every wait is bounded: on a timeout the role raises the CTA's failure flag (which
// ends every other wait) and the error word, waits, bounded, for its own copies or
// MMAs in flight, and the CTA releases its TMEM columns.
template <int G, int NTH>
__global__ void __launch_bounds__(NTH, cb_per_sm(NTH))
conv3x3_cb8(const uint4* __restrict__ inA, int chA, int mode_a, const uint4* __restrict__ inB,
            int chB, int cin, const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias,
            void* __restrict__ out, uint4* __restrict__ pool, int cout, int out_form, int B,
            int H, int W, int act, int tmem_cols, int stages, unsigned* err,
            const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
            int tma_a_req, int tma_b_req) {
  extern __shared__ __align__(1024) unsigned char tc_sm[];
  constexpr int nch = 2 * G;
  constexpr uint32_t STAGE = (uint32_t)nch * CB_CHUNK_STRIDE;
  const int coutp = pad16(cout);
  unsigned char* sA = tc_sm;
  unsigned char* sB = sA + (size_t)stages * STAGE;
  float* sbias = (float*)(sB + (size_t)9 * 16 * G * coutp * 2);
  unsigned long long* bars = (unsigned long long*)(sbias + coutp);
  uint32_t* tmem_slot = (uint32_t*)(bars + 3 * CB_MAX_STAGES + 5);
  volatile uint32_t* fail = tmem_slot + 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool tma_aligned = (smem_u32(tc_sm) & 127u) == 0u;
  const int tma_a = tma_a_req && tma_aligned, tma_b = tma_b_req && tma_aligned;
  const int ntma = (tma_a ? chA : 0) + (tma_b ? chB : 0);
  const int cp_lo = tma_a ? chA : 0, cp_hi = chA + (tma_b ? 0 : chB);   // chunks by cp.async
  // cp.async copies: the warps for them, or (the fallback) the tensor-copy warp
  const int ncpt = cp_hi > cp_lo ? (NTH > CB_NTH ? NTH - CB_NTH : 32) : 0;

  // Weights and biases are read before the wait for the launch before this one, which must
  // not write them and all of whose CTAs must wait before they let this one start (the
  // residual and the features' launches stand between a writer and the first convolution)
  for (int st = 0; st < stages; ++st)
    for (int e = tid; e < (nch - chA - chB) * (CB_CHUNK_STRIDE / 16); e += NTH)
      ((uint4*)(sA + st * STAGE + (size_t)(chA + chB) * CB_CHUNK_STRIDE))[e] =
          make_uint4(0u, 0u, 0u, 0u);
  tc_stage_weights(sB, w, cin, cout, nch, coutp, tid, NTH);
  for (int e = tid; e < coutp; e += NTH) sbias[e] = bias && e < cout ? bias[e] : 0.0f;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :
                 : "r"(smem_u32(tmem_slot)), "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t b_empty = bar0, b_full_t = bar0 + 8 * CB_MAX_STAGES,
                 b_full_c = bar0 + 16 * CB_MAX_STAGES, b_acc_full = bar0 + 24 * CB_MAX_STAGES,
                 b_acc_free = b_acc_full + 16, b_drain = b_acc_full + 32;
  if (tid == 0) {
    auto init = [](uint32_t b, unsigned n) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(n) : "memory");
    };
    for (int s = 0; s < CB_MAX_STAGES; ++s) {
      init(b_empty + 8 * s, 1);
      init(b_full_t + 8 * s, 1);
      init(b_full_c + 8 * s, ncpt > 0 ? ncpt : 1);
    }
    for (int k = 0; k < 2; ++k) {
      init(b_acc_full + 8 * k, 1);
      init(b_acc_free + 8 * k, CB_EPI / 2);
    }
    init(b_drain, 1);
    *fail = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the zeroed padding chunks and the weights, for the tensor core's async proxy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_enter();
  const uint32_t tmem = *tmem_slot;
  const uint32_t sA_a = smem_u32(sA), sB_a = smem_u32(sB);
  const size_t npix = (size_t)B * H * W;
  const int H2 = H >> 1, W2 = W >> 1;
  const int rx = (W + CBX - 1) / CBX, ry = (H + CBY - 1) / CBY;
  const int nreg = rx * ry * B, step = (int)gridDim.x;
  // bounded wait for a barrier's phase; false after the limit or another role's failure
  auto wait = [&](uint32_t b, uint32_t parity) {
    for (unsigned it = 0; it < TC_SPIN_LIMIT; ++it) {
      if (mbar_try_wait(b, parity)) return true;
      if (*fail) return false;
    }
    return false;
  };
  auto give_up = [&]() {
    *fail = 1u;
    if (err) atomicExch(err, 1u);
  };
  auto arrive = [](uint32_t b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory");
  };

  if (warp == CB_EPI || warp >= CB_EPI + 2) {
    // ── copies ──
    const bool cp = ncpt > 0 && (NTH > CB_NTH ? warp >= CB_EPI + 2 : warp == CB_EPI);
    const int ct = warp >= CB_EPI + 2 ? tid - CB_NTH : lane;
    int s = 0, sp = 0;          // this region's stage, the one before
    uint32_t par = 1;
    bool pending = false, ok = true;
    auto signal = [&]() {       // the previous region's copies have landed
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      arrive(b_full_c + 8 * sp);
    };
    for (int t = blockIdx.x; t < nreg; t += step) {
      const int b = t / (rx * ry);
      const int rr = t - b * rx * ry;
      const int x0 = (rr % rx) * CBX, y0 = (rr / rx) * CBY;
      if (!wait(b_empty + 8 * s, par)) { ok = false; break; }
      const uint32_t dst = sA_a + (uint32_t)s * STAGE;
      // one box per chunk; it starts one pixel up and left of the region (the
      // innermost coordinate, the channel, is always 0)
      if (warp == CB_EPI && lane == 0 && ntma > 0) {
        mbar_expect_tx(b_full_t + 8 * s, (uint32_t)ntma * CB_CHUNK_BYTES);
        if (tma_a)
          for (int ch = 0; ch < chA; ++ch)
            tma_load_4d(dst + (uint32_t)ch * CB_CHUNK_STRIDE, &tm_a, 0, x0 - 1, y0 - 1,
                        ch * B + b, b_full_t + 8 * s);
        if (tma_b)
          for (int ch = 0; ch < chB; ++ch)
            tma_load_4d(dst + (uint32_t)(chA + ch) * CB_CHUNK_STRIDE, &tm_b, 0, x0 - 1, y0 - 1,
                        ch * B + b, b_full_t + 8 * s);
      }
      if (cp) {
        for (int q = ct; q < CHP; q += ncpt) {
          const int qy = q / CHX, yy = y0 - 1 + qy, xx = x0 - 1 + q - qy * CHX;
          const bool inside = yy >= 0 && yy < H && xx >= 0 && xx < W;
          const uint32_t bytes = inside ? 16u : 0u;
          const bool up = mode_a == SRC_UP;
          const size_t pa = !inside ? 0
                            : up    ? ((size_t)b * H2 + (yy >> 1)) * W2 + (xx >> 1)
                                    : ((size_t)b * H + yy) * W + xx;
          const size_t ca = (size_t)B * (up ? (size_t)H2 * W2 : (size_t)H * W);
          const size_t pb = inside ? ((size_t)b * H + yy) * W + xx : 0;
          for (int ch = cp_lo; ch < cp_hi; ++ch)
            cp_async16(dst + (uint32_t)ch * CB_CHUNK_STRIDE + (uint32_t)q * 16,
                       ch < chA ? inA + ch * ca + pa : inB + (ch - chA) * npix + pb, bytes);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (pending) {
          asm volatile("cp.async.wait_group 1;" ::: "memory");
          signal();
        }
        pending = true;
        sp = s;
      }
      if (++s == stages) { s = 0; par ^= 1u; }
    }
    if (cp) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (pending) signal();
    }
    // The last regions' commits have arrived at `empty` before the CTA gives its shared
    // memory back: the epilogue waits for the ones at acc_full alone.
    if (ok && warp == CB_EPI) {
      int k = s;
      uint32_t kpar = par;
      for (int n = 0; n < stages; ++n) {
        ok = ok && wait(b_empty + 8 * k, kpar);
        if (++k == stages) { k = 0; kpar ^= 1u; }
      }
    }
    if (!ok) {
      give_up();
      // tensor copies still in flight: the stages issued before this one (a phase
      // that has completed returns at once)
      if (warp == CB_EPI && lane == 0 && ntma > 0) {
        for (int k = 0; k < stages; ++k) {
          // stage k's last issued phase: before `s` in this lap, else the lap before
          const uint32_t lap = par ^ 1u;            // parity of this lap's fills
          const uint32_t ph = k < s ? lap : lap ^ 1u;
          for (unsigned it = 0; it < TC_SPIN_LIMIT; ++it)
            if (mbar_try_wait(b_full_t + 8 * k, ph)) break;
        }
      }
    }
  } else if (warp == CB_EPI + 1) {
    // ── MMA issue ──
    const uint32_t idesc = tc_idesc(coutp);
    int s = 0, k = 0;
    uint32_t par = 0, kpar = 1;
    bool ok = true;
    for (int t = blockIdx.x; t < nreg; t += step) {
      ok = (ntma == 0 || wait(b_full_t + 8 * s, par)) && (ncpt == 0 || wait(b_full_c + 8 * s, par)) &&
           wait(b_acc_free + 8 * k, kpar);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        // M tile i: pixels x0 + 8 i .. x0 + 8 i + 7 of the region's 16 rows,
        // accumulator columns [(2 k + i) coutp, (2 k + i + 1) coutp)
#pragma unroll 1
        for (int i = 0; i < 2; ++i)
          tc_issue_tile<G, CB_CHUNK_STRIDE, CHX>(tmem + (uint32_t)((2 * k + i) * coutp),
                                                 sA_a + (uint32_t)s * STAGE + (uint32_t)(8 * i) * 16,
                                                 sB_a, coutp, idesc);
        tc_commit(b_empty + 8 * s);
        tc_commit(b_acc_full + 8 * k);
      }
      __syncwarp();
      if (++s == stages) { s = 0; par ^= 1u; }
      if (++k == 2) { k = 0; kpar ^= 1u; }
    }
    if (!ok) {
      give_up();
      // MMAs in flight
      if (elect_one()) {
        tc_commit(b_drain);
        for (unsigned it = 0; it < TC_SPIN_LIMIT; ++it)
          if (mbar_try_wait(b_drain, 0)) break;
      }
      __syncwarp();
    }
  } else {
    // ── epilogue: 32 pixels of an M tile, one per lane ──
    const int k = warp >> 3;   // group and accumulator buffer
    const int i = (warp >> 2) & 1, m = (warp & 3) * 32 + lane;
    const int px = lane & 1, py = (lane >> 3) & 1;   // place in the 2x2 block
    uint32_t kpar = 0;
    for (int t = blockIdx.x + k * step; t < nreg; t += 2 * step) {
      const int b = t / (rx * ry);
      const int rr = t - b * rx * ry;
      const int x = (rr % rx) * CBX + 8 * i + (m % 8), y = (rr / rx) * CBY + m / 8;
      const bool store = x < W && y < H;
      const size_t pix = (size_t)b * H * W + (size_t)y * W + x;
      const size_t ppix = (size_t)b * H2 * W2 + (size_t)(y >> 1) * W2 + (x >> 1);
      const bool ok = wait(b_acc_full + 8 * k, kpar);
      if (!__all_sync(0xffffffffu, ok)) {
        give_up();
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int c0 = 0; c0 < coutp; c0 += 16) {
        float v[16];
        __syncwarp();
        tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) +
                      (uint32_t)((2 * k + i) * coutp + c0), v);
        if (c0 + 16 >= coutp) {   // the buffer is read: the MMAs may have it
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive(b_acc_free + 8 * k);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int chunk = c0 / 8 + h;
          if (chunk * 8 >= cout) continue;   // padding columns; uniform
          float a[8];
#pragma unroll
          for (int j = 0; j < 8; j += 4) {
            const float4 bi = *(const float4*)(sbias + chunk * 8 + j);
            a[j] = v[8 * h + j] + bi.x;
            a[j + 1] = v[8 * h + j + 1] + bi.y;
            a[j + 2] = v[8 * h + j + 2] + bi.z;
            a[j + 3] = v[8 * h + j + 3] + bi.w;
          }
          if (act) {   // the inference kernel: tanh on the SFU
#pragma unroll
            for (int j = 0; j < 8; ++j) a[j] = tanh_sfu(a[j]);
          }
          if (out_form == CB_OUT_F32) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (store && chunk * 8 + j < cout)
                ((float*)out)[(size_t)(chunk * 8 + j) * npix + pix] = a[j];
            continue;
          }
          __align__(16) __nv_bfloat16 o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = __float2bfloat16_rn(a[j]);
          if (store) ((uint4*)out)[(size_t)chunk * npix + pix] = *(const uint4*)o;
          if (pool) {
            // the 2x2 average ((a00 + a01) + a10) + a11: the block's four lanes take
            // two channels each (8 exchanges instead of 24).  Left and right
            // neighbours swap four channels, then rows swap: the lower row gives its
            // pairs of the upper row's two channels, the upper row the sums of the
            // lower row's.
            float l[4], r[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float own = px ? a[4 + j] : a[j];
              const float got = __shfl_xor_sync(0xffffffffu, px ? a[j] : a[4 + j], 1);
              l[j] = px ? got : own;
              r[j] = px ? own : got;
            }
            const float s2 = l[2] + r[2], s3 = l[3] + r[3];
            const float g0 = __shfl_xor_sync(0xffffffffu, py ? l[0] : s2, 8);
            const float g1 = __shfl_xor_sync(0xffffffffu, py ? r[0] : s3, 8);
            const float g2 = __shfl_xor_sync(0xffffffffu, l[1], 8);
            const float g3 = __shfl_xor_sync(0xffffffffu, r[1], 8);
            const float p0 = py ? (g0 + l[2]) + r[2] : ((l[0] + r[0]) + g0) + g1;
            const float p1 = py ? (g1 + l[3]) + r[3] : ((l[1] + r[1]) + g2) + g3;
            if (store)
              ((__nv_bfloat162*)(pool + (size_t)chunk * B * H2 * W2 + ppix))[2 * px + py] =
                  __halves2bfloat162(__float2bfloat16_rn(0.25f * p0),
                                     __float2bfloat16_rn(0.25f * p1));
          }
        }
      }
      kpar ^= 1u;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(tmem_cols)
                 : "memory");
  }
}

}  // namespace unet
}  // namespace zb
