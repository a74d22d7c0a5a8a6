// Learned closure, training side: the coarse-grained samples of a fine run,
// the 3x3 convolution layers forward and backward, the loss and the Adam
// update, each as a plain CUDA kernel behind the C ABI of include/lbm_cnn.h.
//
// Layout: activations [N, C, H, W] f32, weights [Cout, Cin, 3, 3], zero
// padding outside the image.  Multiply-adds are written as explicit fmaf (the
// library is compiled with contraction off for the lattice kernels).  Every
// reduction (weight gradients, loss) is two-stage with fixed order, so
// results are deterministic run to run.
#include <cuda_runtime.h>
#include <cstdarg>
#include <cmath>
#include <cstdio>
#include <type_traits>

#include "../../include/lbm_cnn.h"
#include "lbm_device.cuh"

namespace lbm_internal {
void set_last_error(const char* msg);
}

namespace {

int cfail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  lbm_internal::set_last_error(buf);
  return code;
}

#define CCK(call)                                                                              \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) return cfail(LBM_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

constexpr int kRow = 128;          // pixels per block in the per-pixel kernels
constexpr int kTile = 64;          // pixels of a row in a convolution tile
constexpr int kTileS = 72;         // a staged row: columns x0 - 4 .. x0 + 67 of the tile at x0, whole 16-byte words
constexpr int kTile0 = 4;          // index of column x0 in it
constexpr int kChunk = 8;          // input channels staged at a time
constexpr int kWBlocks = 304;      // weight-gradient blocks (2 per SM)
constexpr int kMaxC = 32;          // channels handled by the templates
constexpr int kLossBlocks = 608;   // loss partial sums (4 per SM)

inline cudaStream_t as_stream(void* s) { return (cudaStream_t)s; }

__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }

// Asynchronous 4-byte copy to shared memory, zero where `in` is false (the
// address is then not read).
__device__ __forceinline__ void copy4(float* dst, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0)
               : "memory");
}
// One staged row by one warp: columns x0 - 1 .. x0 + 64 of the image row at
// `src` (zero where row_in is false or outside [0, W)).  `wide` (W a multiple of
// four, 16-byte aligned rows): 18 copies of four columns, each wholly inside or outside.
__device__ __forceinline__ void stage_row(float* dst, const float* src, bool row_in, int x0, int W, bool wide) {
  const int lane = threadIdx.x & 31;
  if (wide) {
    const int xx = x0 - kTile0 + 4 * lane;
    const bool in = row_in && xx >= 0 && xx < W;
    if (lane < kTileS / 4) copy16(dst + 4 * lane, src + (in ? xx : 0), in);
    return;
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int j = lane + 32 * k, xx = x0 - 1 + j;
    const bool in = row_in && xx >= 0 && xx < W;
    if (j < kTile + 2) copy4(dst + kTile0 - 1 + j, src + (in ? xx : 0), in);
  }
}
__host__ __device__ __forceinline__ bool wide_rows(const float* p, const float* q, int W) {
  return W % 4 == 0 && (((uintptr_t)p | (uintptr_t)q) & 15u) == 0;
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Starts the copies of rows y0 - 1 .. y0 + rows of channels c0 .. c0 + nc - 1
// of image n into `sx` [nc][rows + 2][kTileS].  mask_staged visits the same
// elements by the same threads, so a thread may use what it copied itself
// without a barrier.
__device__ __forceinline__ void stage_rows(const float* __restrict__ x, int n, int C, int c0, int nc, int H, int W,
                                           int x0, int y0, int rows, bool wide, float* sx) {
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int r = warp; r < nc * (rows + 2); r += warps) {
    const int c = r / (rows + 2), yy = y0 - 1 + r % (rows + 2);
    const bool row_in = yy >= 0 && yy < H;
    stage_row(sx + r * kTileS, x + (((size_t)n * C + c0 + c) * H + (row_in ? yy : 0)) * W, row_in, x0, W, wide);
  }
}
// ReLU mask of staged gradients: zero where the staged output `sa` is not positive.
__device__ __forceinline__ void mask_staged(float* sx, const float* sa, int nc, int rows, bool wide) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int r = warp; r < nc * (rows + 2); r += warps) {
    float* v = sx + r * kTileS;
    const float* m = sa + r * kTileS;
    if (wide) {
      if (lane < kTileS / 4) {
        float4 g = ((float4*)v)[lane];
        const float4 q = ((const float4*)m)[lane];
        if (!(q.x > 0.0f)) g.x = 0.0f;
        if (!(q.y > 0.0f)) g.y = 0.0f;
        if (!(q.z > 0.0f)) g.z = 0.0f;
        if (!(q.w > 0.0f)) g.w = 0.0f;
        ((float4*)v)[lane] = g;
      }
      continue;
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int j = lane + 32 * k + kTile0 - 1;
      if (lane + 32 * k < kTile + 2 && !(m[j] > 0.0f)) v[j] = 0.0f;
    }
  }
}

// ---- 3x3 convolution to 32 channels -------------------------------------------------
// Forward (BWD false): y = act(conv(x) + b) from C input channels.  Input
// gradient (BWD true): the same sum over the C output channels of the layer
// with the pixels of the taps mirrored, of the gradient masked by the layer's ReLU output.
// A warp owns 64 pixels of one row and all 32 channels: lane (pixel group
// lane & 7, channel group lane >> 3) holds eight pixels (4 g .. 4 g + 3 and 32
// further on, so that 16-byte reads do not conflict) times eight channels as
// channel pairs on the packed multiply-add, which one pixel value and one
// weight pair feed: per input channel and kernel row 288 multiply-adds for
// four reads of pixels and six of weights, where one thread per pixel read
// eight times as many weights and was bound by those reads.  Per output the
// terms are added in the order channel, row, column of the weights, starting
// from the bias.
// The next channels are copied while the current ones are summed (loading them
// between two barriers took half the time).  4 images of 256 x 512, 32 to 32
// channels: 195 us forward and 230 us backward; one thread per pixel took three
// times that.  The packed multiply-adds keep their pipe 70 % busy; what is left
// is the operand reads of three-operand forms and the pixel pairs' moves.
constexpr int kWStride = 36;  // floats per (channel, tap) row of 32 weights: 16-byte multiple, off the bank period
template <bool BWD>
__global__ void __launch_bounds__(256, 2) k_conv32(const float* __restrict__ x, const float* __restrict__ a, int C,
                                                   int H, int W, const float* __restrict__ w,
                                                   const float* __restrict__ b, int relu, float* __restrict__ y) {
  extern __shared__ float4 smem4[];
  // channels staged at a time: with a mask half as many, and their ReLU outputs
  constexpr int kStep = BWD ? kChunk / 2 : kChunk;
  float* sw = (float*)smem4;               // [C * 9][kWStride]
  float* sbuf = sw + C * 9 * kWStride;     // two times [kChunk][rows + 2][kTileS]
  const int rows = blockDim.x >> 5, row_tiles = (H + rows - 1) / rows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pg = lane & 7, cg = lane >> 3;
  const int n = blockIdx.y / row_tiles, y0 = (blockIdx.y % row_tiles) * rows, x0 = blockIdx.x * kTile;
  for (int i = threadIdx.x; i < kMaxC * C * 9; i += blockDim.x) {
    int o, r;
    if (BWD) {  // w [c][o][tap]
      const int c = i / (kMaxC * 9), k = i % 9;
      o = (i / 9) % kMaxC;
      r = c * 9 + k;
    } else {  // w [o][c][tap]
      o = i / (C * 9);
      r = i % (C * 9);
    }
    copy4(sw + r * kWStride + o, w + i, true);
  }
  float2 acc[8][4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float2 b2 = BWD ? make_float2(0.0f, 0.0f) : make_float2(b[8 * cg + 2 * c], b[8 * cg + 2 * c + 1]);
#pragma unroll
    for (int p = 0; p < 8; p++) acc[p][c] = b2;
  }
  const bool wide = wide_rows(x, a, W);
  const int buf = kChunk * (rows + 2) * kTileS, masked = kStep * (rows + 2) * kTileS;
  auto stage = [&](int c0) {
    float* to = sbuf + (c0 / kStep & 1) * buf;
    const int nc = min(kStep, C - c0);
    stage_rows(x, n, C, c0, nc, H, W, x0, y0, rows, wide, to);
    if (BWD && a) stage_rows(a, n, C, c0, nc, H, W, x0, y0, rows, wide, to + masked);
    copies_commit();
  };
  stage(0);
  for (int c0 = 0; c0 < C; c0 += kStep) {
    const int nc = min(kStep, C - c0);
    float* sx = sbuf + (c0 / kStep & 1) * buf;
    if (c0 + kStep < C) {
      stage(c0 + kStep);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    if (BWD && a) mask_staged(sx, sx + masked, nc, rows, wide);
    __syncthreads();
    for (int ci = 0; ci < nc; ci++) {
#pragma unroll
      for (int ky = 0; ky < 3; ky++) {
        const float* row = sx + (ci * (rows + 2) + warp + (BWD ? 2 - ky : ky)) * kTileS + kTile0 + 4 * pg;
        float v[2][6];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const float4 q = *(const float4*)(row + 32 * h);
          v[h][0] = row[32 * h - 1];
          v[h][1] = q.x; v[h][2] = q.y; v[h][3] = q.z; v[h][4] = q.w;
          v[h][5] = row[32 * h + 4];
        }
#pragma unroll
        for (int kx = 0; kx < 3; kx++) {
          const float4* wr = (const float4*)(sw + ((c0 + ci) * 9 + ky * 3 + kx) * kWStride + 8 * cg);
          const float4 wa = wr[0], wb = wr[1];
          const float2 wp[4] = {make_float2(wa.x, wa.y), make_float2(wa.z, wa.w), make_float2(wb.x, wb.y),
                                make_float2(wb.z, wb.w)};
#pragma unroll
          for (int p = 0; p < 8; p++) {
            const float2 xv = dup(v[p >> 2][(p & 3) + (BWD ? 2 - kx : kx)]);
#pragma unroll
            for (int c = 0; c < 4; c++) acc[p][c] = __ffma2_rn(xv, wp[c], acc[p][c]);
          }
        }
      }
    }
    __syncthreads();  // this buffer takes the channels after the next
  }
  const int py = y0 + warp;
  if (py >= H) return;
  const size_t plane = (size_t)H * W;
  const bool wide_out = wide_rows(y, nullptr, W);
#pragma unroll
  for (int c = 0; c < 8; c++) {
    float* out = y + ((size_t)n * kMaxC + 8 * cg + c) * plane + (size_t)py * W;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int px = x0 + 32 * h + 4 * pg;
      float r[4];
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const float2 q = acc[4 * h + p][c >> 1];
        r[p] = (c & 1) ? q.y : q.x;
        if (!BWD && relu) r[p] = fmaxf(r[p], 0.0f);
      }
      if (wide_out && px < W) {
        *(float4*)(out + px) = make_float4(r[0], r[1], r[2], r[3]);
      } else {
#pragma unroll
        for (int p = 0; p < 4; p++)
          if (px + p < W) out[px + p] = r[p];
      }
    }
  }
}

// ---- forward to one channel: four pixels of a row per thread ------------------------
// Bound by reading the input once: 16 threads cover a tile's row, 8 rows a
// block, staged as above; 18 values serve 36 multiply-adds.
__global__ void __launch_bounds__(kTile / 4 * 8) k_conv1(const float* __restrict__ x, int C, int H, int W,
                                                         const float* __restrict__ w, const float* __restrict__ b,
                                                         int relu, float* __restrict__ y) {
  constexpr int kRows = 8;
  __shared__ __align__(16) float sbuf[2][kChunk * (kRows + 2) * kTileS];
  __shared__ float sw[kMaxC * 9];
  const int row_tiles = (H + kRows - 1) / kRows, g = threadIdx.x % (kTile / 4), r = threadIdx.x / (kTile / 4);
  const int n = blockIdx.y / row_tiles, y0 = (blockIdx.y % row_tiles) * kRows, x0 = blockIdx.x * kTile;
  for (int i = threadIdx.x; i < C * 9; i += blockDim.x) sw[i] = w[i];
  float acc[4] = {b[0], b[0], b[0], b[0]};
  const bool wide = wide_rows(x, nullptr, W);
  auto stage = [&](int c0) {
    stage_rows(x, n, C, c0, min(kChunk, C - c0), H, W, x0, y0, kRows, wide, sbuf[c0 / kChunk & 1]);
    copies_commit();
  };
  stage(0);
  for (int c0 = 0; c0 < C; c0 += kChunk) {
    const int nc = min(kChunk, C - c0);
    const float* sx = sbuf[c0 / kChunk & 1];
    if (c0 + kChunk < C) {
      stage(c0 + kChunk);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncthreads();
    for (int ci = 0; ci < nc; ci++)
#pragma unroll
      for (int ky = 0; ky < 3; ky++) {
        const float* row = sx + (ci * (kRows + 2) + r + ky) * kTileS + kTile0 + 4 * g;
        const float4 q = *(const float4*)row;
        const float v[6] = {row[-1], q.x, q.y, q.z, q.w, row[4]};
#pragma unroll
        for (int kx = 0; kx < 3; kx++) {
          const float wk = sw[(c0 + ci) * 9 + ky * 3 + kx];
#pragma unroll
          for (int p = 0; p < 4; p++) acc[p] = fmaf(v[p + kx], wk, acc[p]);
        }
      }
    __syncthreads();
  }
  if (y0 + r >= H) return;
  float* out = y + ((size_t)n * H + y0 + r) * W;
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const int px = x0 + 4 * g + p;
    if (px < W) out[px] = relu ? fmaxf(acc[p], 0.0f) : acc[p];
  }
}

// ---- backward, weight gradient --------------------------------------------------
// gw[co][ci][k] = sum over pixels of g[co] x[ci] shifted by tap k, with
// g = ga * (a > 0) when the layer has a ReLU.  kWBlocks blocks stride over tiles
// of 64 pixels of a row and leave partial sums; in a block every sum is one
// chain over its pixels in order and the partials are added in block order, so
// the result does not depend on how the threads share the sums.  A lane holds
// one input channel (CINP 4: and one of eight groups of output channels), a
// thread four output channels (the packed multiply-add takes two of them, which
// lie side by side once g is masked and transposed, and one pixel of x) and KY
// kernel rows: per four pixels of 32 to 32 channels 72 packed multiply-adds for
// four reads of g, the same for the whole warp, and three of x.  The next tile
// is copied while the current one is summed.  4 images of 256 x 512: 32 to 32
// channels 287 us (a thread with 36 scalar sums, 1300), bound by the packed
// multiply-adds' pipe; 4 to 32 97 us and 32 to 1 148 us, bound by the copies of
// their few warps.  With the pixels of a tile shared out over more threads the
// three took 300, 72 and 56 us, but sums in another order than before: an ulp in
// some weights after a step.
template <int CINP, int KY> struct WGeom {
  static constexpr int kCO = CINP == 32 && KY == 1 ? 4 : 32;  // output channels
  static constexpr int kThreads = KY == 3 ? 256 : 96;         // warps: groups of four output channels, or kernel rows
  static constexpr int kGR = kTile + 4;                       // floats of a staged row of g: 17 (odd) 16-byte words
  static constexpr int kXC = 3 * kTileS + 4;                  // floats of a channel of x: 55 16-byte words
  static constexpr int kG = kCO * kGR, kX = CINP * kXC;       // floats of one tile's g, x
  static constexpr int kBuf = 2 * kG + kX;                    // g, the ReLU output, x
  static constexpr size_t kSmem = (size_t)(2 * kBuf + kTile * kCO) * sizeof(float);
};
template <int CINP, int KY>
__global__ void __launch_bounds__(WGeom<CINP, KY>::kThreads, 2)
    k_conv_bwd_weight(const float* __restrict__ x, const float* __restrict__ ga, const float* __restrict__ a, int N,
                      int CIN, int COUT, int H, int W, float* __restrict__ partial) {
  using Geo = WGeom<CINP, KY>;
  constexpr int kCO = Geo::kCO, kThreads = Geo::kThreads;
  extern __shared__ float4 smem4[];
  float* smem = (float*)smem4;
  float* gt = smem + 2 * Geo::kBuf;  // g of the tile in work, [pixel][output channel]
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int ci = lane % CINP, cog = KY == 3 ? warp : lane / CINP, ky0 = KY == 3 ? 0 : warp;
  // the bias sums: four channels a warp, or all of them in the first
  const int bias_co = KY == 3 ? 4 * warp + (lane & 3) : lane % kCO;
  const bool bias = KY == 3 || warp == 0;
  float2 acc[2][KY][3];
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int k = 0; k < KY * 3; k++) acc[j][k / 3][k % 3] = make_float2(0.0f, 0.0f);
  float accb = 0.0f;
  const size_t plane = (size_t)H * W;
  const int tiles_x = (W + kTile - 1) / kTile;
  const long long tiles = (long long)N * H * tiles_x;
  const bool wide = wide_rows(ga, a, W) && wide_rows(x, nullptr, W);
  auto stage = [&](long long tile, float* G) {
    float* A = G + Geo::kG;
    float* X = A + Geo::kG;
    const int x0 = (int)(tile % tiles_x) * kTile;
    const long long rowi = tile / tiles_x;
    const int n = (int)(rowi / H), py = (int)(rowi % H);
    if (wide) {
      for (int i = t; i < kCO * (kTile / 4); i += kThreads) {
        const int c = i / (kTile / 4), p = 4 * (i % (kTile / 4));
        const bool in = c < COUT && x0 + p < W;
        const size_t o = in ? ((size_t)n * COUT + c) * plane + (size_t)py * W + x0 + p : 0;
        copy16(G + c * Geo::kGR + p, ga + o, in);
        if (a) copy16(A + c * Geo::kGR + p, a + o, in);
      }
    } else {
      for (int i = t; i < kCO * kTile; i += kThreads) {
        const int c = i / kTile, p = i % kTile;
        const bool in = c < COUT && x0 + p < W;
        const size_t o = in ? ((size_t)n * COUT + c) * plane + (size_t)py * W + x0 + p : 0;
        copy4(G + c * Geo::kGR + p, ga + o, in);
        if (a) copy4(A + c * Geo::kGR + p, a + o, in);
      }
    }
    for (int r = warp; r < CINP * 3; r += kThreads / 32) {
      const int c = r / 3, yy = py + r % 3 - 1;
      const bool row_in = c < CIN && yy >= 0 && yy < H;
      stage_row(X + c * Geo::kXC + (r % 3) * kTileS, x + (row_in ? ((size_t)n * CIN + c) * plane + (size_t)yy * W : 0),
                row_in, x0, W, wide);
    }
    copies_commit();
  };
  int turn = 0;
  if (blockIdx.x < tiles) stage(blockIdx.x, smem);
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x, turn ^= 1) {
    const float* G = smem + turn * Geo::kBuf;
    const float* X = G + 2 * Geo::kG;
    if (tile + gridDim.x < tiles) {
      stage(tile + gridDim.x, smem + (turn ^ 1) * Geo::kBuf);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncthreads();
    for (int i = t; i < kCO * (kTile / 4); i += kThreads) {
      const int co = i % kCO, p = 4 * (i / kCO);
      float4 g = *(const float4*)(G + co * Geo::kGR + p);
      if (a) {
        const float4 q = *(const float4*)(G + Geo::kG + co * Geo::kGR + p);
        if (!(q.x > 0.0f)) g.x = 0.0f;
        if (!(q.y > 0.0f)) g.y = 0.0f;
        if (!(q.z > 0.0f)) g.z = 0.0f;
        if (!(q.w > 0.0f)) g.w = 0.0f;
      }
      gt[p * kCO + co] = g.x;
      gt[(p + 1) * kCO + co] = g.y;
      gt[(p + 2) * kCO + co] = g.z;
      gt[(p + 3) * kCO + co] = g.w;
    }
    __syncthreads();
    const float* gp = gt + 4 * cog;
    const float* xp = X + ci * Geo::kXC + ky0 * kTileS + kTile0;
    float before[KY];  // pixel p - 1 of each row
    float4 now[KY];    // pixels p .. p + 3
#pragma unroll
    for (int ky = 0; ky < KY; ky++) {
      before[ky] = xp[ky * kTileS - 1];
      now[ky] = *(const float4*)(xp + ky * kTileS);
    }
#pragma unroll 1
    for (int p = 0; p < kTile; p += 4) {
      float4 g[4];
#pragma unroll
      for (int i = 0; i < 4; i++) g[i] = *(const float4*)(gp + (p + i) * kCO);
      if (bias) {
#pragma unroll
        for (int i = 0; i < 4; i++) accb += gt[(p + i) * kCO + bias_co];
      }
#pragma unroll
      for (int ky = 0; ky < KY; ky++) {
        const float4 next = *(const float4*)(xp + ky * kTileS + p + 4);
        const float v[6] = {before[ky], now[ky].x, now[ky].y, now[ky].z, now[ky].w, next.x};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int kx = 0; kx < 3; kx++) {
            const float2 xv = dup(v[i + kx]);
            acc[0][ky][kx] = __ffma2_rn(xv, make_float2(g[i].x, g[i].y), acc[0][ky][kx]);
            acc[1][ky][kx] = __ffma2_rn(xv, make_float2(g[i].z, g[i].w), acc[1][ky][kx]);
          }
        before[ky] = now[ky].w;
        now[ky] = next;
      }
    }
    __syncthreads();  // this buffer takes the tile after the next
  }
  const int nw = COUT * CIN * 9;
  float* part = partial + (size_t)blockIdx.x * (nw + COUT);
  if (ci < CIN) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int co = 4 * cog + j;
      if (co >= COUT) break;
#pragma unroll
      for (int ky = 0; ky < KY; ky++)
#pragma unroll
        for (int kx = 0; kx < 3; kx++)
          part[(co * CIN + ci) * 9 + (ky0 + ky) * 3 + kx] = (j & 1) ? acc[j >> 1][ky][kx].y : acc[j >> 1][ky][kx].x;
    }
  }
  if (bias && lane < (KY == 3 ? 4 : kCO) && bias_co < COUT) part[nw + bias_co] = accb;
}

// Sum the per-block partials [nblocks][nw + nb] in block order into the weight
// gradient (first nw entries) and the bias gradient (last nb): eight warps
// fetch 32 entries of all blocks, and one lane per entry adds them.
__global__ void __launch_bounds__(256) k_sum_partials(const float* __restrict__ partial, int nblocks, int nw, int nb,
                                                      float* __restrict__ gw, float* __restrict__ gb) {
  __shared__ float sh[kWBlocks][32];
  const int lane = threadIdx.x & 31, i = blockIdx.x * 32 + lane, n = nw + nb;
  if (i < n) {
#pragma unroll 8
    for (int bl = threadIdx.x >> 5; bl < nblocks; bl += 8) sh[bl][lane] = partial[(size_t)bl * n + i];
  }
  __syncthreads();
  if (threadIdx.x >= 32 || i >= n) return;
  float s = 0.0f;
#pragma unroll 8
  for (int bl = 0; bl < nblocks; bl++) s += sh[bl][lane];
  if (i < nw) gw[i] = s;
  else gb[i - nw] = s;
}

// ---- loss ----------------------------------------------------------------------------
__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

// Per cell A dt^2 - 2 B dt + C with dt = dt_max * sigmoid(z): partial sums
// per block (f64) and, when gz is given, dL/dz scaled by inv_norm.
__global__ void __launch_bounds__(256) k_closure_loss(const float* __restrict__ z, const float* __restrict__ coef,
                                                      long long cells_per_image, int N, float dt_max, float inv_norm,
                                                      float* __restrict__ gz, double* __restrict__ partial) {
  __shared__ double sh[256];
  double s = 0.0;
  const long long total = cells_per_image * N;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
    const long long n = i / cells_per_image, c = i % cells_per_image;
    const float* cf = coef + n * 3 * cells_per_image + c;
    const float A = cf[0], B = cf[cells_per_image], C = cf[2 * cells_per_image];
    const float sg = sigmoid(z[i]);
    const float dt = dt_max * sg;
    s += (double)fmaf(dt, fmaf(dt, A, -2.0f * B), C);
    if (gz) gz[i] = (2.0f * fmaf(dt, A, -B)) * inv_norm * dt_max * sg * (1.0f - sg);
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// One warp: each lane adds every 32nd partial, then the lanes in a fixed tree.
__global__ void k_sum_double(const double* __restrict__ partial, int n, double scale, double* __restrict__ out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 32) s += partial[i];
  for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
  if (threadIdx.x == 0) *out = s * scale;
}

// ---- Adam ------------------------------------------------------------------------------
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// ---- coarse-grained samples of a fine run ------------------------------------------
// Pass 1, per coarse cell: Favre block averages over the fluid fine cells of
// its F x F block -> (rho, Ux, Uy, tau_xx, tau_xy, tau_yy) planes, and the
// coarse solid flag (fewer than half the cells fluid).  FIXED: the factor, its
// block's moments kept in registers between the two sweeps (every population is
// then read once, F at a time); 0: any factor, read twice.  Bound by memory (36
// bytes a fine cell).
template <int FIXED>
__global__ void k_coarsen(const float* __restrict__ pops, const uint8_t* __restrict__ solid_f, int Hf, int Wf,
                          int factor, float* __restrict__ avg, uint8_t* __restrict__ solid_c) {
  const int F = FIXED ? FIXED : factor;
  const int W = Wf / F, H = Hf / F;
  const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y;
  if (X >= W) return;
  const size_t planef = (size_t)Hf * Wf, planec = (size_t)H * W, oc = (size_t)Y * W + X;
  constexpr int K = FIXED ? FIXED : 1;
  float kr[K][K], kx[K][K], ky[K][K];
  bool ks[K][K];
  auto cell = [&](size_t o, float& rho, float& jx, float& jy) {
    rho = jx = jy = 0.0f;
#pragma unroll
    for (int q = 0; q < 9; q++) {
      const float f = pops[q * planef + o];
      rho += f;
      jx += (float)lbm::cx(q) * f;
      jy -= (float)lbm::cy(q) * f;
    }
  };
  if constexpr (FIXED != 0) {
    using V = std::conditional_t<FIXED == 4, float4, float2>;
#pragma unroll
    for (int dy = 0; dy < K; dy++) {
      const size_t o = (size_t)(Y * F + dy) * Wf + X * F;
#pragma unroll
      for (int dx = 0; dx < K; dx++) {
        ks[dy][dx] = solid_f[o + dx] != 0;
        kr[dy][dx] = kx[dy][dx] = ky[dy][dx] = 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 9; q++) {
        const V v = *reinterpret_cast<const V*>(pops + q * planef + o);
        const float* f = reinterpret_cast<const float*>(&v);
#pragma unroll
        for (int dx = 0; dx < K; dx++) {
          kr[dy][dx] += f[dx];
          kx[dy][dx] += (float)lbm::cx(q) * f[dx];
          ky[dy][dx] -= (float)lbm::cy(q) * f[dx];
        }
      }
    }
  }
  // calls use(rho, jx, jy) for the block's fluid cells in row order
  auto sweep = [&](auto use) {
    if constexpr (FIXED != 0) {
#pragma unroll
      for (int dy = 0; dy < K; dy++)
#pragma unroll
        for (int dx = 0; dx < K; dx++)
          if (!ks[dy][dx]) use(kr[dy][dx], kx[dy][dx], ky[dy][dx]);
    } else {
      for (int dy = 0; dy < F; dy++)
        for (int dx = 0; dx < F; dx++) {
          const size_t o = (size_t)(Y * F + dy) * Wf + X * F + dx;
          if (solid_f[o]) continue;
          float rho, jx, jy;
          cell(o, rho, jx, jy);
          use(rho, jx, jy);
        }
    }
  };
  // two sweeps: the Favre mean, then the density-weighted spread around it
  // (no cancellation between <rho u u> and U U)
  float R = 0.0f, Jx = 0.0f, Jy = 0.0f;
  int nf = 0;
  sweep([&](float rho, float jx, float jy) {
    nf++;
    R += rho;
    Jx += jx;
    Jy += jy;
  });
  const float Rs = nf > 0 ? R : 1.0f;
  const float Ux = Jx / Rs, Uy = Jy / Rs;
  float Sxx = 0.0f, Sxy = 0.0f, Syy = 0.0f;
  sweep([&](float rho, float jx, float jy) {
    const float vx = jx / rho - Ux, vy = jy / rho - Uy;
    Sxx = fmaf(rho * vx, vx, Sxx);
    Sxy = fmaf(rho * vx, vy, Sxy);
    Syy = fmaf(rho * vy, vy, Syy);
  });
  avg[oc] = nf > 0 ? R / (float)nf : 0.0f;
  avg[planec + oc] = Ux;
  avg[2 * planec + oc] = Uy;
  avg[3 * planec + oc] = Sxx / Rs;
  avg[4 * planec + oc] = Sxy / Rs;
  avg[5 * planec + oc] = Syy / Rs;
  solid_c[oc] = 2 * nf < F * F ? 1 : 0;
}

// Pass 2: features and the eddy-viscosity loss coefficients of each coarse cell.
__global__ void k_sample(const float* __restrict__ avg, const uint8_t* __restrict__ solid_c, int H, int W,
                         float* __restrict__ feat, float* __restrict__ coef) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y;
  if (X >= W) return;
  const size_t plane = (size_t)H * W, o = (size_t)Y * W + X;
  const int xl = max(X - 1, 0), xr = min(X + 1, W - 1);
  const int yu = Y == 0 ? H - 1 : Y - 1, yd = Y == H - 1 ? 0 : Y + 1;  // north / south rows, periodic
  const bool fluid = solid_c[o] == 0;
  const bool valid = fluid && X > 0 && X < W - 1 && !solid_c[(size_t)Y * W + xl] && !solid_c[(size_t)Y * W + xr] &&
                     !solid_c[(size_t)yu * W + X] && !solid_c[(size_t)yd * W + X];
  const float* Ux = avg + plane;
  const float* Uy = avg + 2 * plane;
  const float dUx_dx = 0.5f * (Ux[(size_t)Y * W + xr] - Ux[(size_t)Y * W + xl]);
  const float dUy_dx = 0.5f * (Uy[(size_t)Y * W + xr] - Uy[(size_t)Y * W + xl]);
  const float dUx_dy = 0.5f * (Ux[(size_t)yu * W + X] - Ux[(size_t)yd * W + X]);  // y points north
  const float dUy_dy = 0.5f * (Uy[(size_t)yu * W + X] - Uy[(size_t)yd * W + X]);
  const float sxx = 0.5f * (dUx_dx - dUy_dy), sxy = 0.5f * (dUx_dy + dUy_dx);
  const float txx = avg[3 * plane + o], txy = avg[4 * plane + o], tyy = avg[5 * plane + o];
  const float dxx = 0.5f * (txx - tyy);
  const float v = valid ? 1.0f : 0.0f;
  feat[o] = fluid ? (avg[o] - 1.0f) * LBM_CNN_S_RHO : 0.0f;
  feat[plane + o] = fluid ? Ux[o] * LBM_CNN_S_U : 0.0f;
  feat[2 * plane + o] = fluid ? Uy[o] * LBM_CNN_S_U : 0.0f;
  feat[3 * plane + o] = fluid ? 0.0f : 1.0f;
  coef[o] = v * (8.0f / 9.0f) * fmaf(sxx, sxx, sxy * sxy);
  coef[plane + o] = v * (-4.0f / 3.0f) * fmaf(dxx, sxx, txy * sxy);
  coef[2 * plane + o] = v * 2.0f * fmaf(dxx, dxx, txy * txy);
}

bool bad_shape(int N, int C, int H, int W) { return N < 1 || C < 1 || H < 1 || W < 1 || (long long)N * H > 65535ll * 1024; }

// Launch of k_conv32 over N images: eight rows a block where that fills the
// multiprocessors twice, else fewer (a block's rows share its staged weights).
int launch_conv32(bool bwd, const float* x, const float* a, int n, int C, int h, int w, const float* weight,
                         const float* bias, int relu, float* y, cudaStream_t s) {
  if ((long long)n * h > 65535) return cfail(LBM_ERR_CUDA, "convolution: n h = %lld above 65535", (long long)n * h);
  const int tx = (w + kTile - 1) / kTile;
  int rows = 8;
  while (rows > 2 && (long long)tx * n * ((h + rows - 1) / rows) < 304) rows /= 2;
  const size_t smem = ((size_t)C * 9 * kWStride + 2 * (size_t)kChunk * (rows + 2) * kTileS) * sizeof(float);
  dim3 grid(tx, n * ((h + rows - 1) / rows));
  auto kern = bwd ? k_conv32<true> : k_conv32<false>;
  CCK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<grid, 32 * rows, smem, s>>>(x, a, C, h, w, weight, bias, relu, y);
  CCK(cudaGetLastError());
  return LBM_OK;
}

template <int CINP, int KY>
int launch_bwd_weight(const float* in, const float* grad_out, const float* out, int n, int cin, int cout, int h, int w,
                      float* scratch, int blocks, cudaStream_t s) {
  using Geo = WGeom<CINP, KY>;
  constexpr size_t smem = Geo::kSmem;
  auto kern = k_conv_bwd_weight<CINP, KY>;
  CCK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<blocks, Geo::kThreads, smem, s>>>(in, grad_out, out, n, cin, cout, h, w, scratch);
  CCK(cudaGetLastError());
  return LBM_OK;
}

}  // namespace

extern "C" {

int lbm_cnn_conv_forward(const float* x, int n, int cin, int h, int w, const float* weight, const float* bias,
                         int cout, int relu, float* y, void* stream) {
  if (!x || !weight || !bias || !y) return cfail(LBM_ERR_ARG, "null pointer");
  if (bad_shape(n, cin, h, w) || cin > kMaxC || (cout != kMaxC && cout != 1))
    return cfail(LBM_ERR_ARG, "conv forward: shape n=%d cin=%d h=%d w=%d cout=%d", n, cin, h, w, cout);
  if (cout == kMaxC)
    return launch_conv32(false, x, nullptr, n, cin, h, w, weight, bias, relu, y, as_stream(stream));
  if ((long long)n * h > 65535) return cfail(LBM_ERR_CUDA, "convolution: n h = %lld above 65535", (long long)n * h);
  dim3 grid((w + kTile - 1) / kTile, n * ((h + 7) / 8));
  k_conv1<<<grid, kTile / 4 * 8, 0, as_stream(stream)>>>(x, cin, h, w, weight, bias, relu, y);
  CCK(cudaGetLastError());
  return LBM_OK;
}

int lbm_cnn_conv_backward_data(const float* grad_out, const float* out, int n, int cin, int h, int w,
                               const float* weight, int cout, float* grad_in, void* stream) {
  if (!grad_out || !weight || !grad_in) return cfail(LBM_ERR_ARG, "null pointer");
  if (bad_shape(n, cin, h, w) || cin != kMaxC || cout < 1 || cout > kMaxC)
    return cfail(LBM_ERR_ARG, "conv backward data: shape n=%d cin=%d h=%d w=%d cout=%d", n, cin, h, w, cout);
  return launch_conv32(true, grad_out, out, n, cout, h, w, weight, nullptr, 0, grad_in, as_stream(stream));
}

int lbm_cnn_conv_backward_weight(const float* in, const float* grad_out, const float* out, int n, int cin, int h,
                                 int w, int cout, float* grad_weight, float* grad_bias, float* scratch,
                                 size_t scratch_bytes, void* stream) {
  if (!in || !grad_out || !grad_weight || !grad_bias || !scratch) return cfail(LBM_ERR_ARG, "null pointer");
  if (bad_shape(n, cin, h, w) || cin > kMaxC || cout < 1 || cout > kMaxC)
    return cfail(LBM_ERR_ARG, "conv backward weight: shape n=%d cin=%d h=%d w=%d cout=%d", n, cin, h, w, cout);
  const int nw = cout * cin * 9, per = nw + cout;
  if (scratch_bytes < (size_t)kWBlocks * per * sizeof(float))
    return cfail(LBM_ERR_ARG, "scratch needs %zu bytes", (size_t)kWBlocks * per * sizeof(float));
  cudaStream_t s = as_stream(stream);
  const long long tiles = (long long)n * h * ((w + kTile - 1) / kTile);
  const int blocks = (int)(tiles < kWBlocks ? tiles : kWBlocks);
  const int rc = cin <= 4    ? launch_bwd_weight<4, 1>(in, grad_out, out, n, cin, cout, h, w, scratch, blocks, s)
                 : cout <= 4 ? launch_bwd_weight<32, 1>(in, grad_out, out, n, cin, cout, h, w, scratch, blocks, s)
                             : launch_bwd_weight<32, 3>(in, grad_out, out, n, cin, cout, h, w, scratch, blocks, s);
  if (rc) return rc;
  k_sum_partials<<<(per + 31) / 32, 256, 0, s>>>(scratch, blocks, nw, cout, grad_weight, grad_bias);
  CCK(cudaGetLastError());
  return LBM_OK;
}

size_t lbm_cnn_weight_scratch_bytes(int cin, int cout) {
  return (size_t)kWBlocks * (cout * cin * 9 + cout) * sizeof(float);
}

int lbm_cnn_closure_loss(const float* z, const float* coef, int n, int h, int w, float norm, float* grad_z,
                         double* scratch, double* loss_out, void* stream) {
  if (!z || !coef || !scratch || !loss_out) return cfail(LBM_ERR_ARG, "null pointer");
  if (bad_shape(n, 1, h, w) || !(norm > 0.0f)) return cfail(LBM_ERR_ARG, "closure loss: bad argument");
  cudaStream_t s = as_stream(stream);
  k_closure_loss<<<kLossBlocks, 256, 0, s>>>(z, coef, (long long)h * w, n, LBM_CNN_DT_MAX, 1.0f / norm, grad_z,
                                             scratch);
  CCK(cudaGetLastError());
  k_sum_double<<<1, 32, 0, s>>>(scratch, kLossBlocks, 1.0 / (double)norm, loss_out);
  CCK(cudaGetLastError());
  return LBM_OK;
}

int lbm_cnn_adam(float* param, const float* grad, float* m, float* v, int n, int t, float lr, float beta1,
                 float beta2, float eps, void* stream) {
  if (!param || !grad || !m || !v || n < 0 || t < 1) return cfail(LBM_ERR_ARG, "adam: bad argument");
  if (n == 0) return LBM_OK;
  const float c1 = (float)(1.0 - pow((double)beta1, t)), c2 = (float)(1.0 - pow((double)beta2, t));
  k_adam<<<(n + 255) / 256, 256, 0, as_stream(stream)>>>(param, grad, m, v, n, lr, beta1, beta2, eps, c1, c2);
  CCK(cudaGetLastError());
  return LBM_OK;
}

int lbm_cnn_closure_sample(const float* pops, const uint8_t* solid_fine, int hf, int wf, int factor, float* feat,
                           float* coef, float* scratch, uint8_t* solid_coarse, void* stream) {
  if (!pops || !solid_fine || !feat || !coef || !scratch || !solid_coarse) return cfail(LBM_ERR_ARG, "null pointer");
  if (factor < 1 || hf < 3 * factor || wf < 3 * factor || hf > 65535 * factor)
    return cfail(LBM_ERR_ARG, "closure sample: bad shape");
  const int H = hf / factor, W = wf / factor;
  cudaStream_t s = as_stream(stream);
  dim3 grid((W + kRow - 1) / kRow, H);
  // rows of whole blocks, read as 8- or 16-byte words
  const bool words = wf % factor == 0 && ((uintptr_t)pops & 15u) == 0;
  auto coarsen = words && factor == 4 ? k_coarsen<4> : (words && factor == 2 ? k_coarsen<2> : k_coarsen<0>);
  coarsen<<<grid, kRow, 0, s>>>(pops, solid_fine, hf, wf, factor, scratch, solid_coarse);
  CCK(cudaGetLastError());
  k_sample<<<grid, kRow, 0, s>>>(scratch, solid_coarse, H, W, feat, coef);
  CCK(cudaGetLastError());
  return LBM_OK;
}

}  // extern "C"
