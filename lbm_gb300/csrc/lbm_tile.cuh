// Three steps in one launch for small lattices, with or without the learned
// closure (channel mode, f32 and 16-bit storage).
//
// A small lattice's steps are bound by latency: 512 x 256 cells give each
// multiprocessor 860, and a launch of one step spends most of its 4 us on the
// launch, the first loads and the drain.  Here a CTA takes a tile of 60
// columns and `rows` rows through three steps: one warp per row, two columns
// per lane, the first step pulled from global memory, the next ones from shared
// memory with one barrier between them (k_step_multi, whose warps walk down
// their rows one after the other, is the better one where there are enough
// rows to fill the multiprocessors).  The first step covers two rows more on
// each side, the second one more; columns shrink by one per step on each
// side of a warp's 64.
//
// Cells are advanced and rounded exactly as by one-step launches.  The rest
// plane is read from `rest` and written to `rest_out`, as in k_step_multi.
#pragma once
#include "lbm_multi.cuh"

namespace lbm {

constexpr int kTileRows = 8;                              // rows a CTA stores, at most
constexpr int kTileWarps = kTileRows + 2 * (kMultiSteps - 1);
constexpr int kTilePad = 4;                               // elements around a level's buffer: lane 0 reads one to its left

template <class S> constexpr int tile_level_elems(int rows) { return 9 * rows * 64 + 2 * kTilePad; }
template <class S> constexpr size_t tile_smem(int rows) {  // the outputs of levels 1 and 2
  return (size_t)(tile_level_elems<S>(rows + 4) + tile_level_elems<S>(rows + 2)) * sizeof(S);
}

template <class St, int KM, bool SR, bool CL>
__device__ __forceinline__ void tile_steps(const MultiArgs<typename St::S, typename St::C>& m, int xb, int y0, int y1,
                                           unsigned char* smem, unsigned char (*wins)[32]) {
  using S = typename St::S;
  using Pr = Pair<St>;
  using P = typename Pr::P;
  constexpr int T = kMultiSteps;
  const StepArgs<S, typename St::C>& a = m.a;
  const Layout& L = a.L;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = a.rows;  // (y1 - y0 is less in the last band)
  const int x0 = xb - kMultiHalo + 2 * lane;
  const bool inner = lane >= 1 && lane <= 30;
  bool out[2], cell[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    out[j] = x0 + j == L.nx - 1;
    cell[j] = inner && x0 + j >= 1 && x0 + j <= L.nx - 1;
  }
  const bool inlet = x0 == 0;
  const Ones ones{dup2(m.one), dup2(-m.one)};
  const typename St::Om om = St::omega_consts(a.omega);
  // the levels' outputs: level 1 rows y0 - 2 .., level 2 rows y0 - 1 ..
  S* buf[2];
  buf[0] = reinterpret_cast<S*>(smem) + kTilePad;
  buf[1] = buf[0] + tile_level_elems<S>(rows + 4);
  auto wrap = [&](int y) { return y < 0 ? y + L.ny : (y >= L.ny ? y - L.ny : y); };
  // this lane's pair of direction q, row r of a level's buffer of n rows
  auto at = [&](S* b, int n, int q, int r) -> S* { return b + (q * n + r) * 64 + 2 * lane; };

  // level 1's pulls first (they do not need the mask), then the solid bits
  const int ya = y0 - (T - 1) + warp;
  const bool row_on = warp < y1 - y0 + 2 * (T - 1);
  const uint32_t pitch = (uint32_t)L.pitch;
  P f[9];
  uint32_t rm = 0, r0 = 0, rp = 0;  // element offsets of this lane's pair in rows ya - 1, ya, ya + 1
  if (row_on) {
    // (columns outside the lattice read neighbouring rows or the padding: dropped)
    rm = (uint32_t)wrap(ya - 1) * pitch + (uint32_t)x0;
    r0 = (uint32_t)wrap(ya) * pitch + (uint32_t)x0;
    rp = (uint32_t)wrap(ya + 1) * pitch + (uint32_t)x0;
#pragma unroll
    for (int q = 0; q < 9; q++) {
      const S* base = q == 4 ? a.rest : a.srcp[slot(q)];
      const S* p = base + (long long)(int)(cy(q) < 0 ? rp : (cy(q) > 0 ? rm : r0));
      if (q == 4) {
        f[q] = Pr::lds(p);
      } else {
        S v[2];
#pragma unroll
        for (int j = 0; j < 2; j++) v[j] = __ldg(p + j + (cx(q) > 0 ? -1 : (cx(q) < 0 && !out[j] ? 1 : 0)));
        f[q] = Pr::make(v[0], v[1]);
      }
    }
  }
  for (int r = warp; r < y1 - y0 + 2 * T; r += blockDim.x >> 5) {  // rows y0 - 3 ..
    const int bit = x0 - 1, k = bit >> 5, b = bit & 31;
    const uint32_t* w = a.mask + (long long)wrap(y0 - T + r) * L.mw + k;
    wins[r][lane] = (unsigned char)(__funnelshift_r(__ldg(w), __ldg(w + 1), b) & 15u);
  }
  uint32_t key[T] = {};
  if constexpr (SR) {
#pragma unroll
    for (int l = 0; l < T; l++) {
      SrArgs s = a.sr;
      s.t += (uint32_t)l;
      key[l] = sr_step_key(s);
    }
  }
  __syncthreads();

  auto wall = [&](P v, P own, int q, uint32_t w) -> P {
    const P r = Pr::template bounce<KM>(own, q, a.ref);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int up = cx(q) > 0 ? j : (cx(q) < 0 ? (out[j] ? j + 1 : j + 2) : j + 1);
      if ((w >> up) & 1u) v = Pr::take(v, r, j);
    }
    return v;
  };
  float rho_sum = 0.0f;
  uint32_t fallbacks = 0;
  // collide the pulled pairs of row y at level l + 1 (w: its solid bits) and round them
  auto advance = [&](int l, int y, uint32_t w, bool own_row) {
    float2 g[9], rho;
#pragma unroll
    for (int q = 0; q < 9; q++) g[q] = Pr::val(f[q]);
    if constexpr (CL) {
      const long long o = (long long)wrap(y) * L.pitch + x0;
      float2 jx, jy, aux;
      Pr::template moments<KM>(g, rho, aux, jx, jy, a.ref, ones);
      float2 w2;
      bool fb[2];
      w2.x = closure_omega(a, a.closure[o], rho.x, jx.x, jy.x, fb[0]);
      w2.y = closure_omega(a, a.closure[o + 1], rho.y, jx.y, jy.y, fb[1]);
#pragma unroll
      for (int j = 0; j < 2; j++)
        fallbacks += (fb[j] && own_row && cell[j] && !((w >> (j + 1)) & 1u)) ? 1u : 0u;
      Pr::relax(g, rho, aux, jx, jy, w2, a.ref, ones);
    } else {
      Pr::template collide_checked<KM>(g, rho, om, a.ref, ones);
    }
    if (SR) {
      const uint32_t kp = sr_pair_key(sr_row_key(key[l], wrap(y), a.sr), x0);
#pragma unroll
      for (int q = 0; q < 9; q++) f[q] = Pr::word_sr(g[q], sr_bits(kp, q));
    } else {
#pragma unroll
      for (int q = 0; q < 9; q++) f[q] = Pr::word(g[q]);
    }
    if (l == T - 1) {
      if (cell[0] && !((w >> 1) & 1u)) rho_sum += rho.x;
      if (cell[1] && !((w >> 2) & 1u)) rho_sum += rho.y;
    }
  };

  if (row_on) {  // ---- level 1, row ya = window row warp + 1
    const uint32_t wm = wins[warp][lane], w0 = wins[warp + 1][lane], wp = wins[warp + 2][lane];
    const bool own_row = ya >= y0 && ya < y1;
    const bool near_solid = __any_sync(0xffffffffu, (wm | w0 | wp) != 0u);
    if (near_solid) {
#pragma unroll
      for (int q = 0; q < 9; q++)
        if (q != 4)
          f[q] = wall(f[q], Pr::lds(a.srcp[slot(8 - q)] + (long long)(int)r0), q, cy(q) < 0 ? wp : (cy(q) > 0 ? wm : w0));
    }
    // inert cells keep their rest value in the other rest plane
    if (own_row) {
#pragma unroll
      for (int j = 0; j < 2; j++)
        if ((cell[j] && ((w0 >> (j + 1)) & 1u)) || (j == 0 && inlet)) m.rest_out[r0 + j] = Pr::half(f[4], j);
    }
    advance(0, ya, w0, own_row);
    if (inlet) {  // the inlet column keeps its stored words
#pragma unroll
      for (int q = 0; q < 9; q++)
        f[q] = Pr::take(f[q], Pr::lds((q == 4 ? a.rest : a.srcp[slot(q)]) + (long long)(int)r0), 0);
    }
#pragma unroll
    for (int q = 0; q < 9; q++) Pr::store(at(buf[0], rows + 4, q, warp), f[q]);
  }
#pragma unroll
  for (int l = 1; l < T; l++) {  // ---- levels 2 and 3
    __syncthreads();
    const int n = rows + 2 * (T - l);  // rows of the source buffer
    S* src = buf[l - 1];
    const int y = y0 - (T - 1 - l) + warp;
    if (warp >= y1 - y0 + 2 * (T - 1 - l)) continue;
    const bool own_row = y >= y0 && y < y1;
    // source rows warp .. warp + 2 are y - 1 .. y + 1; windows are one row per level further in
    const uint32_t wm = wins[warp + l][lane], w0 = wins[warp + l + 1][lane], wp = wins[warp + l + 2][lane];
    const bool near_solid = __any_sync(0xffffffffu, (wm | w0 | wp) != 0u);
#pragma unroll
    for (int q = 0; q < 9; q++) {
      const S* p = at(src, n, q, warp + 1 - cy(q));
      f[q] = cx(q) > 0 ? Pr::lds_left(p) : (cx(q) < 0 ? Pr::lds_right(p) : Pr::lds(p));
      if (cx(q) < 0) {
        if (out[0]) f[q] = Pr::take(f[q], Pr::lds(p), 0);
        if (out[1]) f[q] = Pr::take(f[q], Pr::lds(p), 1);
      }
    }
    if (near_solid) {
#pragma unroll
      for (int q = 0; q < 9; q++)
        if (q != 4) f[q] = wall(f[q], Pr::lds(at(src, n, 8 - q, warp + 1)), q, cy(q) < 0 ? wp : (cy(q) > 0 ? wm : w0));
    }
    advance(l, y, w0, own_row);
    if (l < T - 1) {
      if (inlet) {
#pragma unroll
        for (int q = 0; q < 9; q++) f[q] = Pr::take(f[q], Pr::lds(at(src, n, q, warp + 1)), 0);
      }
#pragma unroll
      for (int q = 0; q < 9; q++) Pr::store(at(buf[l], rows + 2 * (T - 1 - l), q, warp), f[q]);
    } else {
      const uint32_t o = (uint32_t)y * pitch + (uint32_t)x0;
      const bool c0 = cell[0] && !((w0 >> 1) & 1u), c1 = cell[1] && !((w0 >> 2) & 1u);
      if (c0 && c1) {
#pragma unroll
        for (int q = 0; q < 9; q++) Pr::store((q == 4 ? m.rest_out : a.dstp[slot(q)]) + o, f[q]);
      } else if (c0 || c1) {
        const int j = c0 ? 0 : 1;
#pragma unroll
        for (int q = 0; q < 9; q++) (q == 4 ? m.rest_out : a.dstp[slot(q)])[o + j] = Pr::half(f[q], j);
      }
    }
  }
  if (!(rho_sum - rho_sum == 0.0f)) atomicOr(a.flag, 1);
  if constexpr (CL) {
    const uint32_t total = __reduce_add_sync(0xffffffffu, fallbacks);
    if (a.fallback && lane == 0 && total) atomicAdd(a.fallback, (unsigned long long)total);
  }
}

template <class St, bool SR, bool CL>
__global__ void __launch_bounds__(32 * kTileWarps, 2)
    k_step_tile(const __grid_constant__ MultiArgs<typename St::S, typename St::C> m) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ unsigned char wins[kTileRows + 2 * kMultiSteps][32];
  const int xb = blockIdx.x * kMultiCols, y0 = blockIdx.y * m.a.rows, y1 = min(y0 + m.a.rows, m.a.row_end);
  if (St::kDev && m.a.ref.shift) tile_steps<St, 1, SR, CL>(m, xb, y0, y1, smem, wins);
  else tile_steps<St, 0, SR, CL>(m, xb, y0, y1, smem, wins);
}

}  // namespace lbm
