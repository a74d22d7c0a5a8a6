// The one-step kernel of reference mode (f32 and 16-bit storage): two adjacent
// cells per lane, one row per warp, straight from global memory.
//
// Every cell of a reference-mode lattice collides, solids with their own
// previous values, and column 0, column nx - 1 and the first and last row
// follow rules of their own.  The staged kernel resolves those cells one row
// after another inside its row loop, each behind two global-memory latencies;
// here every row is another warp's, the cells on the lattice's edge go to CTAs
// of their own, one per lane and first in the grid, and the pair's collision
// runs on the packed operations.  Bound by latency on small lattices, by L2 and
// the arithmetic on lattices that fit it, by HBM above.  f32, us per step, against
// the staged kernel: 256 x 128 3.9 against 6.1, 600 x 400 4.7 against 8.0,
// 1100 x 700 7.6 against 18.2, 2048 x 1024 26.3 against 40.4, 4096 x 2048 96.6
// against 158.7 (6090 GB/s).  f16 (bf16 the same within 3 %), alone / three
// lattices at once: 256 x 128 8.6 / 3.0 against 9.7 / 3.9, 600 x 400 8.1 / 3.2
// against 11.6 / 6.1, 1100 x 700 9.3 / 4.8 against 28.5 / 13.5, 2048 x 1024 14.1 /
// 15.4 against 65.8 / 34.9, 4096 x 2048 64 / 61 against 260 / 130, 8192 x 4096 245 /
// 243 against 993 / 497; with stochastic rounding a tenth more on both sides.
#pragma once
#include "lbm_multi.cuh"

namespace lbm {

constexpr int kPairWarps = 4;  // rows per CTA

template <class S, class C> struct PairArgs {
  StepArgs<S, C> a;
  float one;       // 1 (see Ones)
  int edge_ctas;   // CTAs that take the edge cells
  int cols;        // CTAs side by side: columns / 64
};

template <class St, int KM, bool SR>
__device__ __forceinline__ void pair_step(const PairArgs<typename St::S, typename St::C>& m, int x0, int y) {
  using S = typename St::S;
  using Pr = Pair<St>;
  using P = typename Pr::P;
  const StepArgs<S, typename St::C>& a = m.a;
  const Layout& L = a.L;
  bool in[2];  // cells off the edge columns
#pragma unroll
  for (int j = 0; j < 2; j++) in[j] = x0 + j >= 1 && x0 + j <= L.nx - 2;
  const uint32_t pitch = (uint32_t)L.pitch, r0 = (uint32_t)y * pitch + (uint32_t)x0;
  // (columns outside the lattice read neighbouring rows or the padding: dropped)
  P f[9];
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const S* base = q == 4 ? a.rest : a.srcp[slot(q)];
    const S* p = base + (long long)(int)(cy(q) < 0 ? r0 + pitch : (cy(q) > 0 ? r0 - pitch : r0)) - cx(q);
    if (cx(q) == 0) f[q] = Pr::lds(p);
    else f[q] = Pr::make(__ldg(p), __ldg(p + 1));
  }
  // solid bits of columns x0 - 1 .. x0 + 2 in the three rows
  const int bit = x0 - 1, k = bit >> 5, b = bit & 31;
  uint32_t w[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const uint32_t* row = a.mask + (long long)(y - 1 + i) * L.mw + k;
    w[i] = __funnelshift_r(__ldg(row), __ldg(row + 1), b) & 15u;
  }
  if (!(in[0] || in[1])) return;
  if (w[0] | w[1] | w[2]) {
    // every word that may be needed at once: one more latency, not one per direction
    P opp[9], old[9];
    const bool solid = (w[1] & 6u) != 0u;
#pragma unroll
    for (int q = 0; q < 9; q++) {
      if (q == 4) continue;
      opp[q] = Pr::lds(a.srcp[slot(8 - q)] + (long long)(int)r0);
      if (solid) old[q] = Pr::lds(a.dstp[slot(q)] + (long long)(int)r0);
    }
#pragma unroll
    for (int q = 0; q < 9; q++) {
      if (q == 4) continue;
      const uint32_t wr = w[1 - cy(q)];
      const P r = Pr::template bounce<KM>(opp[q], q, a.ref);  // half-way bounce-back
#pragma unroll
      for (int j = 0; j < 2; j++) {
        if ((wr >> (j + 1 - cx(q))) & 1u) f[q] = Pr::take(f[q], r, j);
        if (solid && ((w[1] >> (j + 1)) & 1u)) f[q] = Pr::take(f[q], old[q], j);  // its own previous value
      }
    }
  }
  float2 g[9], rho, aux, jx, jy;
#pragma unroll
  for (int q = 0; q < 9; q++) g[q] = Pr::val(f[q]);
  const Ones ones{dup2(m.one), dup2(-m.one)};
  Pr::template moments<KM>(g, rho, aux, jx, jy, a.ref, ones);
  const float sum = (in[0] ? rho.x : 0.0f) + (in[1] ? rho.y : 0.0f);
  if (!(sum - sum == 0.0f)) atomicOr(a.flag, 1);
  if (a.rho_out) {
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (in[j]) {
        a.rho_out[r0 + j] = j ? rho.y : rho.x;
        a.jx_out[r0 + j] = j ? jx.y : jx.x;
        a.jy_out[r0 + j] = j ? jy.y : jy.x;
      }
  }
  Pr::template relax_uniform<KM>(g, rho, aux, jx, jy, St::omega_consts(a.omega), a.ref, ones);
  if (SR) {
    const uint32_t kp = sr_pair_key(sr_row_key(sr_step_key(a.sr), y, a.sr), x0);
#pragma unroll
    for (int q = 0; q < 9; q++) f[q] = Pr::word_sr(g[q], sr_bits(kp, q));
  } else {
#pragma unroll
    for (int q = 0; q < 9; q++) f[q] = Pr::word(g[q]);
  }
  if (in[0] && in[1]) {
#pragma unroll
    for (int q = 0; q < 9; q++) Pr::store((q == 4 ? a.rest : a.dstp[slot(q)]) + r0, f[q]);
  } else {
    const int j = in[0] ? 0 : 1;
#pragma unroll
    for (int q = 0; q < 9; q++) (q == 4 ? a.rest : a.dstp[slot(q)])[r0 + j] = Pr::half(f[q], j);
  }
}

template <class St, bool SR>
__global__ void __launch_bounds__(32 * kPairWarps)
    k_step_pair(const __grid_constant__ PairArgs<typename St::S, typename St::C> m) {
  const StepArgs<typename St::S, typename St::C>& a = m.a;
  const int nx = a.L.nx, ny = a.L.ny;
  if ((int)blockIdx.x < m.edge_ctas) {  // rows 0 and ny - 1, then the other cells of columns 0 and nx - 1
    int i = blockIdx.x * blockDim.x + threadIdx.x, x, y;
    if (i < 2 * nx) {
      x = i < nx ? i : i - nx;
      y = i < nx ? 0 : ny - 1;
    } else {
      i -= 2 * nx;
      if (i >= 2 * (ny - 2)) return;
      x = (i & 1) ? nx - 1 : 0;
      y = 1 + (i >> 1);
    }
    if (y >= a.row0 && y < a.row_end) step_cell<St, EDGE_REF>(a, x, y);
    return;
  }
  const int block = blockIdx.x - m.edge_ctas, by = block / m.cols;
  const int x0 = 64 * (block - by * m.cols) + 2 * (threadIdx.x & 31);
  const int y = a.row0 + by * kPairWarps + (threadIdx.x >> 5);
  if (y >= a.row_end || x0 >= nx || y == 0 || y == ny - 1) return;
  if (St::kDev && m.a.ref.shift) pair_step<St, 1, SR>(m, x0, y);
  else pair_step<St, 0, SR>(m, x0, y);
}

}  // namespace lbm
