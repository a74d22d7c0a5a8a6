// Three steps in one launch (channel mode, f32 and 16-bit storage).
//
// A single step moves 72 bytes per cell (f32) through HBM for about 110
// floating-point operations, so the one-step kernel runs at the copy
// bandwidth with the arithmetic units mostly idle.  This kernel reads the
// state once, takes kMultiSteps steps on chip and writes it once: a third of
// the traffic per step.  The price is cells advanced twice: the levels of a band
// of h rows cover h + 4, h + 2 and h rows, 2 / h more (8 % at 24 rows, 17 % at
// 12, 25 % at 8), and 64 columns are advanced for 60 stored (7 %).
//
// A CTA is one warp, which owns 64 columns, two per lane, and walks down a
// band of rows by itself: it fills its own ring of staged rows in shared
// memory with bulk copies (one lane issues them), so there is no producer
// warp and no barrier.  (CTAs of several such warps were slower, 157 against
// 140 us a launch at 4096 x 2048 in f32: with one warp all its row arithmetic
// is uniform and runs outside the vector pipes, and a finished warp's place is
// taken at once.)  Level 1
// (the first step) pulls from the ring as the one-step kernel does.  The later levels never touch memory:
// when level l - 1 has produced row r, level l can complete row r - 1, and
// what it needs of rows r - 2 and r - 1 is kept in registers (per cell three
// south-moving values already pulled, the pulled e / w and the rest value,
// and the cell's own three south-moving values for bounce-back).  Columns
// move between lanes by shuffle.  The outermost lane on each side computes
// values that go stale by one column per level and never stores; with two
// columns per lane that covers the two columns the levels after the first use
// up.
//
// Cells are advanced by the same operations in the same order as in three
// one-step launches, and 16-bit words are rounded after every level, so the
// stored state is the same to the bit.
//
// The rest plane is read by neighbouring CTAs (halo cells are advanced
// redundantly), so it cannot be updated in place: it is read from `rest` and
// written to `rest_out`, inert cells included.
#pragma once
#include <cuda.h>
#include <type_traits>
#include "lbm_stage.cuh"

namespace lbm {

constexpr int kMultiSteps = 3;                      // odd: the buffer parity after a launch is that of single steps
constexpr int kMultiHalo = 2;                       // columns per side used up by the levels after the first
constexpr int kMultiCols = 64 - 2 * kMultiHalo;     // columns a warp stores
constexpr int kMultiOcc = 16;                       // CTAs (of one warp) per multiprocessor: 128 registers each

// a / b for b in a moderate range, correctly rounded, sharing the reciprocal
// between the quotients of one denominator: y = 1 / b to the nearest (an
// approximation within one ulp and one Newton step with fused operations), then
// q = a y corrected once by its exact remainder (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990).  The
// method makes one exception for y, a mantissa of all ones (1 - 2^-24 is such a
// density): 1 / b then lies just above a tie, and the step rounds to the nearest
// only from an approximation above it.  rcp.approx gives that one: over all 2^23
// mantissas at eight exponents from 2^-57 to 2^63 every y equalled 1 / b, and
// sixteen quotients by each equalled a / b.  Quotients too small for an exact
// remainder (|a| < 2^-100) may be off in the last place; with b of at least
// 2^-63 they are velocities below 2^-37, added to 1, and only a tie of a later
// rounding could tell.
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Sums and differences as a fused multiply-add by 1 and -1, which rounds as
// they do.  The assembler contracts a packed product and a packed sum into
// one fused operation even where both carry their rounding and contraction is
// off, which would change the last bit; it cannot do so through a factor that
// it does not know, so the two factors are kernel arguments.
struct Ones {
  float2 p, m;  // (1, 1), (-1, -1)
  __device__ __forceinline__ float2 add(float2 a, float2 b) const { return fma2(b, p, a); }
  __device__ __forceinline__ float2 sub(float2 a, float2 b) const { return fma2(b, m, a); }
};
__device__ __forceinline__ float2 recip_rn2(float2 b, float2 nb) {
  const float2 y = make_float2(rcp_approx(b.x), rcp_approx(b.y));
  return fma2(fma2(nb, y, dup2(1.0f)), y, y);
}
__device__ __forceinline__ float2 quot2(float2 a, float2 nb, float2 y) {
  const float2 q = mul2(a, y);
  return fma2(fma2(nb, q, a), y, q);
}
// What a tile remembers of two cells' quotients: they are the rounded ones
// where every denominator lay in [2^-63, 2^65) and every quotient's square was
// finite.  Otherwise the tile is advanced again with plain divisions.
struct QuotRange {
  uint32_t x = 0, y = 0;
  float2 u2 = make_float2(0.0f, 0.0f);
  __device__ __forceinline__ bool ok_x() const { return (x & 0xC0000000u) == 0u && u2.x - u2.x == 0.0f; }
  __device__ __forceinline__ bool ok_y() const { return (y & 0xC0000000u) == 0u && u2.y - u2.y == 0.0f; }
};

// moments<float> and bgk<float> of two cells on the packed f32x2 operations:
// every operation rounds each component as the scalar one does, so the pair
// gives what two scalar evaluations give.
__device__ __forceinline__ void moments_f32_2(const float2 f[9], float2& rho, float2& jx, float2& jy, const Ones& k) {
  const float2 a = add2(f[2], f[8]);
  const float2 ux_c = k.sub(k.sub(a, f[0]), f[6]);
  const float2 uy_c = k.sub(k.sub(add2(f[2], f[0]), f[8]), f[6]);
  const float2 rho_c = add2(add2(a, f[0]), f[6]);
  jx = add2(ux_c, k.sub(f[5], f[3]));
  jy = add2(uy_c, k.sub(f[1], f[7]));
  rho = add2(add2(rho_c, add2(add2(add2(f[5], f[1]), f[7]), f[3])), f[4]);
}
// Relaxation towards the equilibrium of velocity (ux, uy), u2 = |u|^2, at rates w2.
__device__ __forceinline__ void relax_f32_2(float2 f[9], float2 rho, float2 ux, float2 uy, float2 ux2, float2 uy2,
                                            float2 u2, float2 w2, const Ones& k) {
  const float2 c45 = dup2(4.5f);
  const float2 ux3 = mul2(dup2(3.0f), ux), uy3 = mul2(dup2(3.0f), uy);
  const float2 uxuy2 = mul2(mul2(dup2(2.0f), ux), uy);
  const float2 u215 = mul2(dup2(1.5f), u2);
  const float2 r36 = mul2(dup2(1.0f / 36.0f), rho), r9 = mul2(dup2(1.0f / 9.0f), rho);
  const float2 sp = mul2(c45, k.add(u2, uxuy2)), sm = mul2(c45, k.sub(u2, uxuy2));
  const float2 sx = mul2(c45, ux2), sy = mul2(c45, uy2);
  const float2 px = k.add(k.p, ux3), mx = k.sub(k.p, ux3);
  // f + w (r (c - u215) - f)
  auto relax = [&](int q, float2 r, float2 c) {
    const float2 eq = mul2(r, k.sub(c, u215));
    f[q] = k.add(f[q], mul2(w2, fma2(f[q], k.m, eq)));
  };
  relax(2, r36, k.add(k.add(px, uy3), sp));
  relax(8, r36, k.add(k.sub(px, uy3), sm));
  relax(0, r36, k.add(k.add(mx, uy3), sm));
  relax(6, r36, k.add(k.sub(mx, uy3), sp));
  relax(4, mul2(dup2(4.0f / 9.0f), rho), k.p);
  relax(5, r9, k.add(px, sx));
  relax(3, r9, k.add(mx, sx));
  relax(1, r9, k.add(k.add(k.p, uy3), sy));
  relax(7, r9, k.add(k.sub(k.p, uy3), sy));
}
// NEAR: quotients by division on request, solid cells not in `range`.
template <bool NEAR>
__device__ __forceinline__ void bgk_f32_2(float2 f[9], float2 rho, float2 jx, float2 jy, float w, const Ones& k,
                                          bool divide, QuotRange& range, uint32_t solid) {
  const float2 nb = mul2(rho, k.m), y = recip_rn2(rho, nb);
  float2 ux = quot2(jx, nb, y), uy = quot2(jy, nb, y);
  if (NEAR && divide) {
    ux = make_float2(jx.x / rho.x, jx.y / rho.y);
    uy = make_float2(jy.x / rho.x, jy.y / rho.y);
  }
  const float2 ux2 = mul2(ux, ux), uy2 = mul2(uy, uy);
  const float2 u2 = k.add(ux2, uy2);
  {  // (solid cells hold whatever words they were given and are never stored)
    const bool sx = NEAR && (solid & 2u), sy = NEAR && (solid & 4u);
    range.x |= sx ? 0u : __float_as_uint(rho.x) - 0x20000000u;
    range.y |= sy ? 0u : __float_as_uint(rho.y) - 0x20000000u;
    range.u2 = k.add(range.u2, NEAR ? make_float2(sx ? 0.0f : u2.x, sy ? 0.0f : u2.y) : u2);
  }
  relax_f32_2(f, rho, ux, uy, ux2, uy2, u2, dup2(w), k);
}
// The same with the quotients checked at once and rates of two cells.
__device__ __forceinline__ void bgk_f32_2_checked(float2 f[9], float2 rho, float2 jx, float2 jy, float2 w2,
                                                  const Ones& k) {
  const float2 nb = mul2(rho, k.m), y = recip_rn2(rho, nb);
  float2 ux = quot2(jx, nb, y), uy = quot2(jy, nb, y);
  float2 ux2 = mul2(ux, ux), uy2 = mul2(uy, uy), u2 = k.add(ux2, uy2);
  QuotRange range;
  range.x = __float_as_uint(rho.x) - 0x20000000u;
  range.y = __float_as_uint(rho.y) - 0x20000000u;
  range.u2 = u2;
  if (!(range.ok_x() && range.ok_y())) {
    ux = make_float2(jx.x / rho.x, jx.y / rho.y);
    uy = make_float2(jy.x / rho.x, jy.y / rho.y);
    ux2 = mul2(ux, ux);
    uy2 = mul2(uy, uy);
    u2 = k.add(ux2, uy2);
  }
  relax_f32_2(f, rho, ux, uy, ux2, uy2, u2, w2, k);
}

// Two adjacent columns of one direction as the levels keep them: a pair of
// floats, or two 16-bit words in one register.
template <class St> struct Pair {  // 16-bit storage
  using S = typename St::S;
  using P = uint32_t;
  __device__ static P lds(const S* p) { return *reinterpret_cast<const uint32_t*>(p); }
  // the pair one column to the left / right of `e` in a staged row
  __device__ static P lds_left(const S* p) { return __byte_perm(lds(p - 2), lds(p), 0x5432); }
  __device__ static P lds_right(const S* p) { return __byte_perm(lds(p), lds(p + 2), 0x5432); }
  __device__ static P from_left(P a) { return __byte_perm(__shfl_up_sync(0xffffffffu, a, 1), a, 0x5432); }
  __device__ static P from_right(P a) { return __byte_perm(a, __shfl_down_sync(0xffffffffu, a, 1), 0x5432); }
  __device__ static float2 val(P a) {
    float2 v;
    load_pair((const S*)nullptr, a, v.x, v.y);
    return v;
  }
  __device__ static P word(float2 v) {
    S h[2] = {St::store(v.x, 0), St::store(v.y, 0)};
    uint32_t u;
    memcpy(&u, h, 4);
    return u;
  }
  __device__ static P word_sr(float2 v, uint32_t R) { return St::store2_sr(v.x, v.y, R); }
  __device__ static S half(P a, int j) {
    const uint16_t b = (uint16_t)(j ? a >> 16 : a & 0xffffu);
    S s;
    memcpy(&s, &b, 2);
    return s;
  }
  // `a` with column j replaced by column j of `b`
  __device__ static P take(P a, P b, int j) { return j ? __byte_perm(a, b, 0x7610) : __byte_perm(a, b, 0x3254); }
  // own opposite population bounced back into direction q
  template <int KM> __device__ static P bounce(P own, int q, const StoreRef& R) {
    if (!shifted<KM>(R)) return own;
    const float2 v = val(own);
    return word(make_float2(v.x + R.bb[q], v.y + R.bb[q]));
  }
  __device__ static P make(S lo, S hi) {
    S h[2] = {lo, hi};
    uint32_t u;
    memcpy(&u, h, 4);
    return u;
  }
  template <int KM>
  __device__ static void moments(const float2 f[9], float2& rho, float2& aux, float2& jx, float2& jy, const StoreRef& R,
                                 const Ones&) {
    St::template moments2<KM>(f, rho, aux, jx, jy, R);
  }
  // relaxation at a rate of its own per cell
  __device__ static void relax(float2 f[9], float2 rho, float2 aux, float2 jx, float2 jy, float2 w, const StoreRef& R,
                               const Ones&) {
    float g[9];
#pragma unroll
    for (int q = 0; q < 9; q++) g[q] = f[q].x;
    St::collide(g, rho.x, aux.x, jx.x, jy.x, w.x, R);
#pragma unroll
    for (int q = 0; q < 9; q++) {
      f[q].x = g[q];
      g[q] = f[q].y;
    }
    St::collide(g, rho.y, aux.y, jx.y, jy.y, w.y, R);
#pragma unroll
    for (int q = 0; q < 9; q++) f[q].y = g[q];
  }
  template <int KM>
  __device__ static void relax_uniform(float2 f[9], float2 rho, float2 aux, float2 jx, float2 jy,
                                       const typename St::Om& om, const StoreRef& R, const Ones&) {
    St::template collide_u2<KM>(f, rho, aux, jx, jy, om, R);
  }
  template <int KM>
  __device__ static void collide_checked(float2 f[9], float2& rho, const typename St::Om& om, const StoreRef& R,
                                         const Ones& k) {
    QuotRange range;
    collide<KM, false>(f, rho, om, R, k, false, range, 0u);
  }
  template <int KM, bool NEAR>
  __device__ static void collide(float2 f[9], float2& rho, const typename St::Om& om, const StoreRef& R, const Ones&,
                                 bool, QuotRange&, uint32_t) {
    float2 aux, jx, jy;
    St::template moments2<KM>(f, rho, aux, jx, jy, R);
    St::template collide_u2<KM>(f, rho, aux, jx, jy, om, R);
  }
  __device__ static void store(S* p, P a) { *reinterpret_cast<uint32_t*>(p) = a; }
};
template <> struct Pair<StF32> {
  using S = float;
  using P = float2;
  __device__ static P lds(const S* p) { return *reinterpret_cast<const float2*>(p); }
  __device__ static P lds_left(const S* p) { return make_float2(p[-1], p[0]); }
  __device__ static P lds_right(const S* p) { return make_float2(p[1], p[2]); }
  __device__ static P from_left(P a) { return make_float2(__shfl_up_sync(0xffffffffu, a.y, 1), a.x); }
  __device__ static P from_right(P a) { return make_float2(a.y, __shfl_down_sync(0xffffffffu, a.x, 1)); }
  __device__ static float2 val(P a) { return a; }
  __device__ static P word(float2 v) { return v; }
  __device__ static P word_sr(float2 v, uint32_t) { return v; }
  __device__ static S half(P a, int j) { return j ? a.y : a.x; }
  __device__ static P take(P a, P b, int j) { return j ? make_float2(a.x, b.y) : make_float2(b.x, a.y); }
  template <int KM> __device__ static P bounce(P own, int, const StoreRef&) { return own; }
  __device__ static P make(S lo, S hi) { return make_float2(lo, hi); }
  template <int KM>
  __device__ static void moments(const float2 f[9], float2& rho, float2&, float2& jx, float2& jy, const StoreRef&,
                                 const Ones& k) {
    moments_f32_2(f, rho, jx, jy, k);
  }
  __device__ static void relax(float2 f[9], float2 rho, float2, float2 jx, float2 jy, float2 w, const StoreRef&,
                               const Ones& k) {
    bgk_f32_2_checked(f, rho, jx, jy, w, k);
  }
  template <int KM>
  __device__ static void relax_uniform(float2 f[9], float2 rho, float2, float2 jx, float2 jy, const float& om,
                                       const StoreRef&, const Ones& k) {
    bgk_f32_2_checked(f, rho, jx, jy, dup2(om), k);
  }
  template <int KM>
  __device__ static void collide_checked(float2 f[9], float2& rho, const float& om, const StoreRef&, const Ones& k) {
    float2 jx, jy;
    moments_f32_2(f, rho, jx, jy, k);
    bgk_f32_2_checked(f, rho, jx, jy, dup2(om), k);
  }
  template <int KM, bool NEAR>
  __device__ static void collide(float2 f[9], float2& rho, const float& om, const StoreRef&, const Ones& k, bool divide,
                                 QuotRange& range, uint32_t solid) {
    float2 jx, jy;
    moments_f32_2(f, rho, jx, jy, k);
    bgk_f32_2<NEAR>(f, rho, jx, jy, om, k, divide, range, solid);
  }
  __device__ static void store(S* p, P a) { *reinterpret_cast<float2*>(p) = a; }
};

// Shared-memory layout of one staged row of a warp: 8 moving planes (one
// tensor copy: the planes are the outer dimension of a [8][ny][pitch] map) and
// the rest plane, from the 16-byte boundary at or before column xb - 4 to
// column xb + 63, then 8 mask words.
template <class S> struct MultiGeom {
  static constexpr int kAlign = 16 / (int)sizeof(S);
  static constexpr int kSeg = (kAlign - 4 + 4 + kMultiCols + 4 + kAlign - 1) / kAlign * kAlign;
  static constexpr uint32_t kSegBytes = kSeg * sizeof(S);
  static constexpr uint32_t kMaskOff = 9 * kSegBytes;
  static constexpr uint32_t kCopied = kMaskOff + 32;
  static constexpr uint32_t kBytes = (kCopied + 127) / 128 * 128;  // tensor copies land on 128-byte boundaries
  // kMultiOcc CTAs per multiprocessor: 14 KB of ring each
  static constexpr int kStages = sizeof(S) == 4 ? 5 : 8;
  static_assert(kSegBytes % 16 == 0 && 8 * kSegBytes % 16 == 0, "bulk-copy alignment");
};

// Box {kSeg, 1, 8} of the tensor map at column x, row y, every plane.  x is a
// multiple of 16 bytes; columns outside the map read as zero.
__device__ __forceinline__ void tensor_g2s(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(0), "r"(bar)
      : "memory");
}

// Before the first copy through a tensor map that lies in global memory and was
// written by a copy: later tensor copies of this lane see the map's present
// contents, not what a freed map at the same address held.  (A map passed as a
// __grid_constant__ argument needs none.)
__device__ __forceinline__ void acquire_map(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
}

template <class S, class C> struct MultiArgs {
  StepArgs<S, C> a;
  S* rest_out;
  float one;  // 1 (see Ones)
  int wcols;  // warps side by side: columns / 60
};

// One warp's tile: columns [xb, xb + 60) of rows [y0, y1).  EDGE: the tile
// holds the inlet column, the outflow column or columns past it.
template <class St, int KM, bool SR, bool EDGE>
__device__ __forceinline__ void multi_tile(const MultiArgs<typename St::S, typename St::C>& m, const CUtensorMap* map,
                                           int xb, int y0, int y1, unsigned char* smem, uint64_t* full) {
  using S = typename St::S;
  using Pr = Pair<St>;
  using P = typename Pr::P;
  using G = MultiGeom<S>;
  constexpr int T = kMultiSteps, NS = G::kStages;
  const StepArgs<S, typename St::C>& a = m.a;
  const Layout& L = a.L;
  const int lane = threadIdx.x & 31;
  const int n_stage = y1 - y0 + 2 * T;           // staged rows y0 - T .. y1 + T - 1
  const int iters = y1 - y0 + 2 * (T - 1);
  const int xs = (xb - 4) & ~(G::kAlign - 1);    // first staged column
  const int mw0 = ((xb - 4) >> 5) & ~3;          // first staged mask word (16-byte boundary)
  // columns x0, x0 + 1 per lane; lanes 1 .. 30 store
  const int x0 = xb - kMultiHalo + 2 * lane;
  const int e = x0 - xs;
  const int bit = x0 - 1 - 32 * mw0, k = bit >> 5, b = bit & 31;  // mask bit of column x0 - 1 in the staged words
  const bool inner = lane >= 1 && lane <= 30;
  bool out[2], cell[2];  // the outflow column; columns this lane advances and stores
#pragma unroll
  for (int j = 0; j < 2; j++) {
    out[j] = EDGE && x0 + j == L.nx - 1;
    cell[j] = inner && (!EDGE || (x0 + j >= 1 && x0 + j <= L.nx - 1));
  }
  const bool inlet = EDGE && x0 == 0;  // (x0 is even: column 0 is some lane's first)
  const typename St::Om om = St::omega_consts(a.omega);
  const Ones ones{dup2(m.one), dup2(-m.one)};
  uint32_t key[T] = {};
  if constexpr (SR) {
#pragma unroll
    for (int l = 0; l < T; l++) {
      SrArgs s = a.sr;
      s.t += (uint32_t)l;
      key[l] = sr_step_key(s);
    }
  }
  // staged row i into ring slot s (every lane calls it, one issues the copies)
  auto stage = [&](int i, int s) {
    int rr = y0 - T + i;
    rr = rr < 0 ? rr + L.ny : (rr >= L.ny ? rr - L.ny : rr);
    if (elect_one()) {
      const uint32_t st = smem_addr(smem + (size_t)s * G::kBytes), bar = smem_addr(&full[s]);
      mbar_arrive_expect_tx(bar, G::kCopied);
      tensor_g2s(st, map, xs, rr, bar);
      bulk_g2s(st + 8 * G::kSegBytes, a.rest + ((long long)rr * L.pitch + xs), G::kSegBytes, bar);
      bulk_g2s(st + G::kMaskOff, a.mask + (long long)rr * L.mw + mw0, 32u, bar);
    }
    __syncwarp();
  };
  auto win = [&](const unsigned char* st) -> uint32_t {  // solid bits of columns x0 - 1 .. x0 + 2
    const uint32_t* w = reinterpret_cast<const uint32_t*>(st + G::kMaskOff);
    return __funnelshift_r(w[k], w[k + 1], b) & 15u;
  };
  auto staged = [&](const unsigned char* st, int q) -> const S* {  // this lane's pair of direction q in a staged row
    return reinterpret_cast<const S*>(st + (q == 4 ? 8 : slot(q)) * G::kSegBytes) + e;
  };
  auto outflow = [&](P pulled, P own) -> P {  // the outflow column pulls its x + 1 populations from itself
    if (out[0]) pulled = Pr::take(pulled, own, 0);
    if (out[1]) pulled = Pr::take(pulled, own, 1);
    return pulled;
  };
  // pulled pair of direction q from the pair `v` of the upstream row
  auto pull = [&](P v, int q) -> P {
    if (cx(q) > 0) return Pr::from_left(v);
    if (cx(q) < 0) return EDGE ? outflow(Pr::from_right(v), v) : Pr::from_right(v);
    return v;
  };
  // bounce-back: columns of `v` whose upstream cell (in the row with solid
  // bits w) is solid take the cell's own opposite population
  auto wall = [&](P v, P own, int q, uint32_t w) -> P {
    const P r = Pr::template bounce<KM>(own, q, a.ref);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int up = cx(q) > 0 ? j : (cx(q) < 0 ? (out[j] ? j + 1 : j + 2) : j + 1);
      if ((w >> up) & 1u) v = Pr::take(v, r, j);
    }
    return v;
  };

  QuotRange range;
  float rho_sum = 0.0f;  // finite exactly when every density of the last level was
  // what level l keeps between rows (index l - 2)
  P sp[T - 1][3], so[T - 1][3], ew[T - 1][3];
  uint32_t hist = 0;  // solid bits, 4 per row: the newest staged row lowest
  uint32_t own = 0;   // this lane's first cell in the row the last level completes

  // One row of every level: level 1 at row y from the staged rows y - 1 (sm),
  // y (s0), y + 1 (st), level l at row y - (l - 1).  The general form (a lane
  // has a solid cell in reach, the levels are filling: level l + 1 runs from
  // it = 2 l on, or quotients by division) and the straight-line form that
  // almost every row takes: two bodies, as more of them miss the instruction cache.
  auto row = [&](auto near_c, int it, const unsigned char* sm, const unsigned char* s0, const unsigned char* st,
                 bool divide) {
    constexpr bool NEAR = decltype(near_c)::value;
    const int y = y0 - (T - 1) + it;
    float2 rho;
    // collide the pulled pairs of row t at level l + 1 and round them as the step stores them
    auto advance = [&](P f[9], int l, int t, uint32_t w) {
      float2 g[9];
#pragma unroll
      for (int q = 0; q < 9; q++) g[q] = Pr::val(f[q]);
      Pr::template collide<KM, NEAR>(g, rho, om, a.ref, ones, divide, range, w);
      if (SR) {
        const uint32_t kp = sr_pair_key(sr_row_key(key[l], t < 0 ? t + L.ny : (t >= L.ny ? t - L.ny : t), a.sr), x0);
#pragma unroll
        for (int q = 0; q < 9; q++) f[q] = Pr::word_sr(g[q], sr_bits(kp, q));
      } else {
#pragma unroll
        for (int q = 0; q < 9; q++) f[q] = Pr::word(g[q]);
      }
    };
    auto keep_inlet = [&](P f[9], const unsigned char* s) {  // the inlet column keeps its stored words
      if (inlet) {
#pragma unroll
        for (int q = 0; q < 9; q++) f[q] = Pr::take(f[q], Pr::lds(staged(s, q)), 0);
      }
    };
    P f[9];
#pragma unroll
    for (int q = 0; q < 9; q++) {
      const S* p = staged(cy(q) < 0 ? st : (cy(q) > 0 ? sm : s0), q);
      f[q] = cx(q) > 0 ? Pr::lds_left(p) : (cx(q) < 0 ? Pr::lds_right(p) : Pr::lds(p));
      if (EDGE && cx(q) < 0) f[q] = outflow(f[q], Pr::lds(p));
    }
    if (NEAR) {
#pragma unroll
      for (int q = 0; q < 9; q++)
        if (q != 4) f[q] = wall(f[q], Pr::lds(staged(s0, 8 - q)), q, hist >> (cy(q) < 0 ? 0 : (cy(q) > 0 ? 8 : 4)));
    }
    if ((NEAR || EDGE) && y >= y0 && y < y1) {  // inert cells keep their rest value in the other rest plane
      const P r = Pr::lds(staged(s0, 4));
#pragma unroll
      for (int j = 0; j < 2; j++)
        if ((cell[j] && ((hist >> (4 + j + 1)) & 1u)) || (j == 0 && inlet))
          m.rest_out[(uint32_t)y * (uint32_t)L.pitch + (uint32_t)(x0 + j)] = Pr::half(r, j);
    }
    advance(f, 0, y, hist >> 4);
    keep_inlet(f, s0);
#pragma unroll
    for (int l = 0; l < T - 1; l++) {  // level l + 2 from row r = y - l of level l + 1
      P g[9];
      P(&SP)[3] = sp[l];
      P(&SO)[3] = so[l];
      P(&EW)[3] = ew[l];
      const uint32_t wr = hist >> (4 * (l + 1)), wt = hist >> (4 * (l + 2));  // solid bits of rows r and r - 1
#pragma unroll
      for (int q = 0; q < 3; q++) {
        g[q] = pull(f[q], q);
        if (NEAR) g[q] = wall(g[q], SO[2 - q], q, wr);
        g[3 + q] = EW[q];
        g[6 + q] = SP[q];
      }
      // keep what the next row needs
#pragma unroll
      for (int i = 0; i < 3; i++) {
        SP[i] = pull(SO[i], 6 + i);
        EW[i] = pull(f[3 + i], 3 + i);
        if (NEAR) {
          SP[i] = wall(SP[i], f[2 - i], 6 + i, wt);
          if (i != 1) EW[i] = wall(EW[i], f[5 - i], 3 + i, wr);
        }
      }
#pragma unroll
      for (int i = 0; i < 3; i++) SO[i] = f[6 + i];
      if (NEAR && it < 2 * (l + 1)) return;
      const int t = y - (l + 1);
      advance(g, l + 1, t, wt);
      if (l < T - 2) keep_inlet(g, sm);  // (level 2's row is still staged)
#pragma unroll
      for (int q = 0; q < 9; q++) f[q] = g[q];
      if (l == T - 2) {  // complete
        // a density that went non-finite at an earlier level still is: the
        // cell's rest value, which never leaves it, was set from that density
        const bool c0 = cell[0] && !(NEAR && ((wt >> 1) & 1u)), c1 = cell[1] && !(NEAR && ((wt >> 2) & 1u));
        if (c0) rho_sum += rho.x;
        if (c1) rho_sum += rho.y;
        if (c0 && c1) {
#pragma unroll
          for (int q = 0; q < 9; q++) Pr::store((q == 4 ? m.rest_out : a.dstp[slot(q)]) + own, f[q]);
        } else if (c0 || c1) {
          const int j = c0 ? 0 : 1;
#pragma unroll
          for (int q = 0; q < 9; q++) (q == 4 ? m.rest_out : a.dstp[slot(q)])[own + j] = Pr::half(f[q], j);
        }
      }
    }
  };
  using Yes = std::integral_constant<bool, true>;
  using No = std::integral_constant<bool, false>;

  bool ok = true;
  for (bool divide = false;; divide = true) {
    if (lane == 0) {
      for (int i = 0; i < NS; i++) mbar_init(smem_addr(&full[i]), 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    int issued = min(NS, n_stage);  // staged rows whose copies were issued
    for (int i = 0; i < issued; i++) stage(i, i);
#pragma unroll
    for (int l = 0; l < T - 1; l++)
#pragma unroll
      for (int i = 0; i < 3; i++) sp[l][i] = so[l][i] = ew[l][i] = P{};
    own = (uint32_t)(y0 - 2 * (T - 1)) * (uint32_t)L.pitch + (uint32_t)x0;
    ok = mbar_wait(smem_addr(&full[0]), 0u) && mbar_wait(smem_addr(&full[1]), 0u);
    if (ok) hist = (win(smem) << 4) | win(smem + G::kBytes);
    int slot_m = 0, slot_0 = 1, slot_p = 2;
    uint32_t parity_p = 0u;
    for (int it = 0; it < iters && ok; it++, own += (uint32_t)L.pitch) {
      if (!mbar_wait(smem_addr(&full[slot_p]), parity_p)) { ok = false; break; }
      const unsigned char* sm = smem + slot_m * (int)G::kBytes;
      const unsigned char* s0 = smem + slot_0 * (int)G::kBytes;
      const unsigned char* st = smem + slot_p * (int)G::kBytes;
      hist = (hist << 4) | win(st);
      const bool near_solid = __any_sync(0xffffffffu, (hist & 0xffffu) != 0u);
      if (divide || near_solid || it < 2 * (T - 1)) row(Yes{}, it, sm, s0, st, divide);
      else row(No{}, it, sm, s0, st, false);
      __syncwarp();  // every lane has read the oldest staged row: refill its slot
      if (issued < n_stage) stage(issued++, slot_m);
      slot_m = slot_0;
      slot_0 = slot_p;
      if (++slot_p == NS) { slot_p = 0; parity_p ^= 1u; }
    }
    if (!ok) {  // a wait ran out: no copy may be in flight at exit
      if (lane == 0) atomicOr(a.flag, 2);
      for (int i = max(0, issued - NS); i < issued; i++) mbar_wait(smem_addr(&full[i % NS]), (uint32_t)(i / NS) & 1u);
      break;
    }
    // the halo lanes' cells count too: their neighbours are stored (columns 0
    // and outside the lattice hold whatever was pulled and feed nothing)
    const bool in0 = !EDGE || (x0 >= 1 && x0 < L.nx), in1 = !EDGE || (x0 >= 0 && x0 + 1 < L.nx);
    if (divide || __all_sync(0xffffffffu, (range.ok_x() || !in0) && (range.ok_y() || !in1))) break;
    rho_sum = 0.0f;
    __syncwarp();
    if (lane == 0)
      for (int i = 0; i < NS; i++) mbar_inval(smem_addr(&full[i]));
    __syncwarp();
  }
  if (!(rho_sum - rho_sum == 0.0f)) atomicOr(a.flag, 1);
}

// One warp's tile by the lattice's storage reference and the tile's edges
// (the halo lanes advance the next two columns too, by their own rules).
template <class St, bool SR>
__device__ __forceinline__ void multi_dispatch(const MultiArgs<typename St::S, typename St::C>& m,
                                               const CUtensorMap* map, int xb, int y0, int y1, unsigned char* smem,
                                               uint64_t* full) {
  const bool edge = xb == 0 || xb + kMultiCols + kMultiHalo >= m.a.L.nx;
  if (St::kDev && m.a.ref.shift) {
    if (edge) multi_tile<St, 1, SR, true>(m, map, xb, y0, y1, smem, full);
    else multi_tile<St, 1, SR, false>(m, map, xb, y0, y1, smem, full);
  } else {
    if (edge) multi_tile<St, 0, SR, true>(m, map, xb, y0, y1, smem, full);
    else multi_tile<St, 0, SR, false>(m, map, xb, y0, y1, smem, full);
  }
}

template <class St, bool SR>
__global__ void __launch_bounds__(32, kMultiOcc)
    k_step_multi(const __grid_constant__ CUtensorMap map,  // the 8 planes of `src`
                 const __grid_constant__ MultiArgs<typename St::S, typename St::C> m) {
  using G = MultiGeom<typename St::S>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[G::kStages];
  const int band = blockIdx.x / m.wcols;
  const int xb = (blockIdx.x - band * m.wcols) * kMultiCols;
  const int y0 = band * m.a.rows, y1 = min(y0 + m.a.rows, m.a.row_end);
  if (y0 >= y1) return;
  multi_dispatch<St, SR>(m, &map, xb, y0, y1, smem, full);
}

// Host side: the tensor map of a buffer set's 8 planes, for the kernels' copies.
template <class S> bool encode_planes(CUtensorMap* map, const Layout& L, void* planes) {
  using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult found;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess ||
      !fn)
    return false;
  const cuuint64_t dim[3] = {(cuuint64_t)L.pitch, (cuuint64_t)L.ny, 8};
  const cuuint64_t stride[2] = {(cuuint64_t)L.pitch * sizeof(S), (cuuint64_t)L.ps * sizeof(S)};
  const cuuint32_t box[3] = {(cuuint32_t)MultiGeom<S>::kSeg, 1, 8}, step[3] = {1, 1, 1};
  return ((EncodeTiled)fn)(map, sizeof(S) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 3,
                           planes, dim, stride, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace lbm
