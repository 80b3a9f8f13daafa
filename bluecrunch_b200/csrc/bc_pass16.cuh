// bc_pass16.cuh — outer column passes with 16 points per thread.
//
// Same arithmetic and data layout as k2_outer_fwd / k2_outer_inv
// (bc_pipe.cuh); the column transform is organised differently.  An L-point
// column (L = 16 R, R in {4, 8, 16}) is held by R threads with 16 points
// each, point t + R i in register i of thread t.  The transform is the
// four-step split L = 16 x R:
//   1. a 16-point DFT in registers over i (constant twiddles),
//   2. the twiddle e^{-+2 pi i t k2 / L},
//   3. ONE exchange through shared memory,
//   4. DFT-R over t for the 16/R values of k2 = t + R j a thread owns.
// Outputs land in the same register contract (frequency t + R i in register
// i), so the pass reads digits / tiles and writes results exactly as the
// 8-points-per-thread kernels do, with one exchange and two barriers per
// column transform instead of two exchanges and four barriers, and twice
// the independent work per thread between barriers.
#pragma once
#include "bc_pipe.cuh"
#include "bc_rows_warp.cuh"

namespace bc {

constexpr int P16 = 16;

// 16-point DFT in registers, natural order in and out: n = n1 + 4 n2,
// k = k2 + 4 k1; DFT-4 over n2, twiddle w16^(n1 k2), DFT-4 over n1.
template <bool INV>
__device__ __forceinline__ void dft16(double2 (&a)[P16]) {
#pragma unroll
  for (int n1 = 0; n1 < 4; n1++) {
    dft4<INV>(a[n1], a[n1 + 4], a[n1 + 8], a[n1 + 12]);  // a[n1 + 4 k2] = y[n1][k2]
#pragma unroll
    for (int k2 = 1; k2 < 4; k2++) a[n1 + 4 * k2] = rot32<INV>(a[n1 + 4 * k2], 2 * n1 * k2);
  }
  double2 o[P16];
#pragma unroll
  for (int k2 = 0; k2 < 4; k2++) {
    double2 b0 = a[4 * k2], b1 = a[4 * k2 + 1], b2 = a[4 * k2 + 2], b3 = a[4 * k2 + 3];
    dft4<INV>(b0, b1, b2, b3);
    o[k2] = b0;
    o[k2 + 4] = b1;
    o[k2 + 8] = b2;
    o[k2 + 12] = b3;
  }
#pragma unroll
  for (int k = 0; k < P16; k++) a[k] = o[k];
}

template <int R, bool INV>
__device__ __forceinline__ void dft_small16(double2 (&x)[R]) {
  static_assert(R == 4 || R == 8 || R == 16, "second-stage radix");
  if constexpr (R == 4) dft4<INV>(x[0], x[1], x[2], x[3]);
  else if constexpr (R == 8) dft8<INV>(x);
  else dft16<INV>(x);
}

// Shared-memory twiddles of block16: tw[k2*R + t] = e^{-2 pi i t k2 / L},
// t < R = L/16, k2 < 16, from the flat table flat[m] = e^{-2 pi i m/L}
// (m < 3L/4; above that e^{-2 pi i m/L} = -e^{-2 pi i (m - L/2)/L}).  The
// threads of a warp hold four or more neighbouring t of one k2: consecutive
// entries, one pass over the banks (k2 fastest put them 256 bytes apart, four
// passes).  All NT threads; the caller's next barrier publishes the table.
template <int L, int NT>
__device__ __forceinline__ void tw16_build(double2 *dst, const double2 *__restrict__ flat) {
  constexpr int R = L / P16;
#pragma unroll
  for (int q = 0; q < L / NT; q++) {
    const int i = threadIdx.x + q * NT, m = (i % R) * (i / R);
    const double2 w = __ldg(&flat[m < 3 * L / 4 ? m : m - L / 2]);
    dst[i] = m < 3 * L / 4 ? w : make_double2(-w.x, -w.y);
  }
  static_assert(L % NT == 0, "whole rounds");
}

// L-point transforms of W columns by R = L/16 threads per column.  On entry
// and exit v[i] = x[t + R i] of column s (natural order).  sm is the tile's
// shared memory (L x W, the swizzled layout of sidx); tw the table of
// tw16_build.  Ends past a barrier, so the CTA may reuse sm.
template <int L, int W, bool INV>
__device__ __forceinline__ void block16(double2 (&v)[P16], int t, int s, double2 *sm, const double2 *tw) {
  constexpr int R = L / P16, J = P16 / R;
  dft16<INV>(v);  // v[k2] = Y[t][k2]
#pragma unroll
  for (int k2 = 1; k2 < P16; k2++) v[k2] = ctw<INV>(v[k2], tw[k2 * R + t]);
#pragma unroll
  for (int k2 = 0; k2 < P16; k2++) sm[sidx<L, W>(k2 * R + t, s)] = v[k2];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < J; j++) {
    const int k2 = t + R * j;
    double2 x[R];
#pragma unroll
    for (int tp = 0; tp < R; tp++) x[tp] = sm[sidx<L, W>(k2 * R + tp, s)];
    dft_small16<R, INV>(x);
#pragma unroll
    for (int k1 = 0; k1 < R; k1++) v[j + J * k1] = x[k1];  // frequency k2 + 16 k1 = t + R (j + J k1)
  }
  __syncthreads();
}

// Tile geometry of the 16-point passes: same tiles as PassTile<L> (L rows x
// W columns, W = pass_tile_w(L)), R = L/16 threads per column.
template <int L> struct Pass16 {
  static constexpr int W = pass_tile_w(L);
  static constexpr int R = L / P16;
  static constexpr int NT = R * W;
  static_assert(L == 64 || L == 128 || L == 256, "16-point passes cover L1 = 64, 128, 256");
  // twelve warps per SM (at most 170 registers per thread)
  static constexpr int MINB = 384 / NT;
  // dynamic shared memory
  static constexpr size_t TWB = (size_t)L * 16;  // block16 twiddles
  static constexpr size_t SMEM_INV = 2 * (size_t)L * W * 16 + TWB + (size_t)L * 16 + 2 * 38 * 16 + 1024;
};

// Outer-pass twiddles e^{-2 pi i col (4 k1 - 1)/(4M)} of one thread, for
// k1 = t + R i (i = 0..15) and col = tile W + s, as four runs of 4 (a base
// and a step, then products).  With T(m) = e^{-2 pi i m/(4M)} (m signed) and
// T(col x) = T(tile W x) T(s x):
//   base of run 0      T(col (4t - 1))          = F_t * T(s (4t - 1))
//   step               T(col 4R)                = G * T(s 4R)
//   base of run j      that of run j - 1 or 0 times T(col 16R j), j = 1, 2
//   T(col 16R) = J * T(s 16R), T(col 32R) = H * T(s 32R)
// The tile factors F_t (t < 16), G, J, H come from the two-level table, T(m) =
// lo * hi: both entries of each are copied to shared memory one unit ahead
// (cp.async), each thread multiplies the four pairs it needs.  The column
// factors depend only on the thread (s, t fixed by tid) and stay in registers.
// Computing the tile factors by sincospi took 130 instructions in every warp
// of every unit, a tenth of the pass's issue slots, and at the start of a CTA
// 2 us.  The runs are short because a table product's error is above
// sincospi's and grows along a run: with two runs of 8 the rounding error of a
// 2^24-limb product grew from 0.0142 to 0.0158, with four of 4 it is 0.0127.
// (Steps per column straight from the table, one product each, 0.0135, took
// 64 entries a unit and the inverse pass from 0.233 to 0.247 ms.)
constexpr int TILE_TW = 19;             // tile factors per unit
constexpr int TILE_TW_N = 2 * TILE_TW;  // their table entries (lo, hi)

// Index of T(m) = e^{-2 pi i m/(4M)} in the two-level table, |m| < 4M.
__device__ __forceinline__ unsigned long long t4m_index(long long m, int M) {
  return (unsigned long long)(m < 0 ? m + 4ll * M : m);
}

struct ColTw16 {
  double2 c0, cst, cj, ch;
};
template <int R>
__device__ __forceinline__ ColTw16 col_tw16(int s, int t, const Tw2 &T, int M) {
  ColTw16 c;
  c.c0 = tw2_get(T, t4m_index((long long)s * (4 * t - 1), M));
  c.cst = tw2_get(T, (unsigned long long)s * 4 * R);
  c.cj = tw2_get(T, (unsigned long long)s * 16 * R);
  c.ch = tw2_get(T, (unsigned long long)s * 32 * R);
  return c;
}

// Copies the table entries of tile's factors to fac (lo of factor j at j, hi
// at TILE_TW + j: F_0..F_15, G, J, H); the caller commits, waits and
// synchronises.
template <int R, int W>
__device__ __forceinline__ void tile_tw16(double2 *fac, int tile, const Tw2 &T, int M) {
  const int k = threadIdx.x;
  if (k < TILE_TW_N) {
    const int j = k < TILE_TW ? k : k - TILE_TW;
    const long long x = j < 16 ? 4 * j - 1 : (j == 16 ? 4 * R : (j == 17 ? 16 * R : 32 * R));
    const unsigned long long m = t4m_index((long long)tile * W * x, M);
    cp_async16(fac + k, k < TILE_TW ? &T.lo[m & T.mask] : &T.hi[m >> T.h], 16);
  }
}

// The bases of the four runs and the step.
struct OuterRun16 {
  double2 b[4], st;
};
template <int R>
__device__ __forceinline__ OuterRun16 outer_run16(const double2 *fac, const ColTw16 &c, int t) {
  auto factor = [&](int j) { return cmul(fac[j], fac[TILE_TW + j]); };
  OuterRun16 o;
  const double2 j = cmul(factor(17), c.cj);
  o.b[0] = cmul(factor(t), c.c0);
  o.b[1] = cmul(o.b[0], j);
  o.b[2] = cmul(o.b[0], cmul(factor(18), c.ch));
  o.b[3] = cmul(o.b[2], j);
  o.st = cmul(factor(16), c.cst);
  return o;
}

// ------------------------------------------------------------------ outer forward (pack)
// Units: (item, operand, column tile), as k2_outer_fwd.  One limb stage: the
// next unit's words are copied (cp.async) as soon as this unit's digits are
// cut, and land while this unit is transformed and stored.
// PARTS: 1 when no operand of the class has digits at M or above (products of
// operands of about one length): the limb stage then holds one part, and
// sixteen warps of 128 registers fit an SM instead of twelve (L = 64 would
// spill): 0.380 -> 0.360 ms at 2^25 points (L = 256).
// TW: columns of a tile.  At L = 128, 16 where that still gives every SM two
// units (256-byte segments, fewer limb copies per digit: whole 2^21-point
// product 0.112 -> 0.108 ms), else 8 (2^15 points 0.045 -> 0.043 ms a call).
// At L = 256 always 8: a CTA of 256 threads lost more than it gained (2^23
// points 0.394 -> 0.405 ms).
template <int L, int PARTS, int TW> struct Fwd16 {
  static constexpr int W = TW;
  static constexpr int R = L / P16, NT = R * W;
  static constexpr int MINB = (PARTS == 1 && L > 64 ? 512 : 384) / NT;
  using Stage = PackTile<L, W>;
  static constexpr int STAGE_WORDS = Stage::STAGE_WORDS / 2 * PARTS;
  static constexpr size_t SMEM = (size_t)L * W * 16 + (size_t)STAGE_WORDS * 4 + 2 * (size_t)L * 16 +
                                 2 * TILE_TW_N * 16 + 1024;
};

template <int L, int PARTS, int TW>
__global__ void __launch_bounds__(Fwd16<L, PARTS, TW>::NT, Fwd16<L, PARTS, TW>::MINB)
    k3_outer_fwd(const __grid_constant__ ClassParams p) {
  pdl_trigger();  // the first pass of a class: launched normally, lets the next one start early
  using T = Fwd16<L, PARTS, TW>;
  using K = typename T::Stage;
  constexpr int W = T::W, R = T::R, NT = T::NT;
  extern __shared__ unsigned char smraw[];
  double2 *tile = align1024(smraw);
  uint32_t *stg = reinterpret_cast<uint32_t *>(tile + L * W);  // one stage: L segments per part
  double2 *twS = reinterpret_cast<double2 *>(stg + T::STAGE_WORDS);
  double2 *pwS = twS + L;
  double2 *fac = pwS + L;  // tile factors of a unit, of the units in turn at fac + par * TILE_TW_N
  const int tid = threadIdx.x, s = tid % W, t = tid / W;
  const int tiles = (int)p.fd_fwd.d;
  const unsigned nA = fwd_units_a(p, (unsigned)tiles);
  const unsigned total = nA + fwd_units_b(p, (unsigned)tiles);  // far below 2^32
  // limb staging: as k2_outer_fwd (every row segment of a tile shares one
  // alignment below a 16-byte boundary)
  auto seg_shift = [&](int tl, int b, bool al16) -> int {
    return al16 ? (int)((((long long)tl * W * b >> 5) - 1) & 3) : 0;
  };
  // the unit's limb words and, to the set `par`, its tile factors (the threads
  // still at the unit before read the other set)
  auto stage_copy = [&](unsigned u, int par) {
    const FwdUnit f = fwd_unit(p, u, nA, p.fd_fwd, (unsigned)tiles);
    const int tl = (int)f.rest;
    tile_tw16<R, W>(fac + par * TILE_TW_N, tl, p.tw4M, p.M);
    const FwdOperand it = fwd_operand(p, f.item, f.op);
    const uint32_t *X = it.X;
    const int XL = it.XL;
    const int b = it.b;
    const bool al16 = it.al16;
    const int RW = words_below(p.S1, b), PW = words_below(p.M, b);
    const int wbase = ((tl * W * b) >> 5) - 1 - seg_shift(tl, b, al16);
    const int parts = PARTS == 2 && it.nd > (unsigned)p.M ? 2 : 1;
    if (al16) {
      // the chunks up to the last digit's last bit (the second word that its
      // cut reads may lie beyond: those bits are masked away)
      constexpr int CH = K::SEGW4 / 4;
      const int NCH = parts * L * CH;
      const int need = ((32 * (1 + seg_shift(tl, b, true)) + ((tl * W * b) & 31) + W * b - 1) >> 5) / 4 + 1;
      for (int idx = tid; idx < NCH; idx += NT) {
        const int segi = idx / CH, k = idx - segi * CH;
        const int part = segi >= L, row = segi - (part ? L : 0);
        const int w = row * RW + (part ? PW : 0) + wbase + 4 * k;  // multiple of 4
        int nv = XL - w;
        nv = nv < 0 ? 0 : (nv > 4 ? 4 : nv);
        if (w < 0) nv = 0;
        if (k < need) cp_async16(stg + segi * K::SEGW4 + 4 * k, X + (nv ? w : 0), nv * 4);
      }
    } else {
      for (int idx = tid; idx < parts * (K::STAGE_WORDS / 2); idx += NT) {
        const int segi = idx / K::SEGW4, k = idx - segi * K::SEGW4;
        const int part = segi >= L, row = segi - (part ? L : 0);
        const int w = row * RW + (part ? PW : 0) + wbase + k;
        const bool in = w >= 0 && w < XL;
        cp_async4(stg + idx, X + (in ? w : 0), in ? 4 : 0);
      }
    }
  };
  unsigned u = blockIdx.x;
  if (u < total) stage_copy(u, 0);
  cp_async_commit();
  first_kernel_setup(p);
  // while the first unit's words cross: the tables and this thread's factors
  tw16_build<L, NT>(twS, p.twL1);
  table_to_smem<L, NT>(pwS, p.pw_fwd);
  const ColTw16 ct = col_tw16<R>(s, t, p.tw4M, p.M);
  for (int par = 0; u < total; u += gridDim.x, par ^= 1) {
    const FwdUnit f = fwd_unit(p, u, nA, p.fd_fwd, (unsigned)tiles);
    const int tl = (int)f.rest;
    const FwdOperand it = fwd_operand(p, f.item, f.op);
    const int col = tl * W + s;
    cp_async_wait<0>();
    __syncthreads();  // the stage (every thread's copies) has landed
    const unsigned nd = it.nd;
    double2 *gbuf = it.buf;
    const int b = it.b;
    const bool al16 = it.al16;
    const unsigned rel = 32u * (1u + (unsigned)seg_shift(tl, b, al16)) + (unsigned)((tl * W * b) & 31) +
                         (unsigned)(s * b);  // bit of digit j0+s in its staged segment
    const unsigned wi = (rel - 1) >> 5, sh = (rel - 1) & 31;
    const unsigned mask = (1u << b) - 1;
    const bool imag = PARTS == 2 && nd > (unsigned)p.M;
    auto digit = [&](int part, int n1) -> double {
      const unsigned j = (unsigned)n1 * (unsigned)p.S1 + col + (part ? (unsigned)p.M : 0u);
      const uint32_t *rw = stg + (part * L + n1) * K::SEGW4 + wi;
      const unsigned x = __funnelshift_r(rw[0], rw[1], sh);
      const int r = (int)((x >> 1) & mask);
      const int top = (j + 1 >= nd) ? 0 : (r >> (b - 1));
      return j < nd ? (double)(r - (top << b) + (int)(x & 1u)) : 0.0;
    };
    double2 v[P16];
    if (imag) {
#pragma unroll
      for (int i = 0; i < P16; i++) {
        const int n1 = t + i * R;
        v[i] = cmul(make_double2(digit(0, n1), digit(1, n1)), pwS[n1]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < P16; i++) {
        const int n1 = t + i * R;
        const double d = digit(0, n1);
        const double2 w = pwS[n1];
        v[i] = make_double2(d * w.x, d * w.y);
      }
    }
    __syncthreads();  // every thread has cut its digits: the stage is free
    const unsigned un = u + gridDim.x;
    if (un < total) stage_copy(un, par ^ 1);
    cp_async_commit();
    block16<L, W, false>(v, t, s, tile, twS);
    const OuterRun16 tw = outer_run16<R>(fac + par * TILE_TW_N, ct, t);
    double2 w = tw.b[0];
#pragma unroll
    for (int i = 0; i < P16; i++) {
      if (i % 4 == 0) w = tw.b[i / 4];
      gbuf[(unsigned)(t + i * R) * (unsigned)p.S1 + col] = cmul(v[i], w);
      w = cmul(w, tw.st);
    }
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------ outer inverse
// Units: (item, column tile), as k2_outer_inv; tiles by TMA one unit ahead.
template <int L>
__global__ void __launch_bounds__(Pass16<L>::NT, Pass16<L>::MINB)
    k3_outer_inv(ClassParams p, const __grid_constant__ CUtensorMap mA) {
  using T = Pass16<L>;
  constexpr int W = T::W, R = T::R, NT = T::NT, G = W / 8;
  extern __shared__ unsigned char smraw[];
  __shared__ uint64_t bars[2];
  double2 *const buf0 = align1024(smraw);  // stage st's tile at buf0 + st * L * W
  double2 *twS = buf0 + 2 * L * W;
  double2 *pwS = twS + L;
  double2 *fac = pwS + L;  // tile factors of unit parity st at fac + st * TILE_TW_N
  const int tid = threadIdx.x, s = tid % W, t = tid / W;
  const FastDiv fd_tiles = p.fd_outer;
  const unsigned tiles = fd_tiles.d;
  const unsigned total = (unsigned)p.nitems * tiles;  // far below 2^32
  if (blockIdx.x < total) tile_tw16<R, W>(fac, (int)(blockIdx.x - fd_tiles.div(blockIdx.x) * tiles), p.tw4M, p.M);
  cp_async_commit();
  tw16_build<L, NT>(twS, p.twL1);
  table_to_smem<L, NT>(pwS, p.pw_inv);
  const ColTw16 ct = col_tw16<R>(s, t, p.tw4M, p.M);
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    fence_mbar_init();
  }
  cp_async_wait<0>();
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  // largest rounding error of this thread's units of the current item,
  // published (one atomic per warp) when the item changes and at the end
  double err_acc = 0.0;
  int err_item = -1;
  unsigned phases = 0;  // bit st: parity to wait for on bars[st]
  int st = 0;
  unsigned u = blockIdx.x;
  if (tid == 0 && u < total) {
    fence_proxy_async_smem();
    const unsigned q0 = fd_tiles.div(u);
    tile_load_3d<L, W>(buf0, &mA, &bars[0], (int)(u - q0 * tiles) * W, (int)q0);
  }
  for (; u < total; u += gridDim.x) {
    const unsigned un = u + gridDim.x;
    if (tid == 0 && un < total) {
      fence_proxy_async_smem();
      const unsigned qn = fd_tiles.div(un);
      tile_load_3d<L, W>(buf0 + (st ^ 1) * L * W, &mA, &bars[st ^ 1], (int)(un - qn * tiles) * W, (int)qn);
    }
    const int item = (int)fd_tiles.div(u), tile = (int)(u - (unsigned)item * tiles);
    if (item != err_item) {  // uniform over the CTA: every thread is on unit u
      if (err_item >= 0) atomic_max_err(p.items[err_item].err, err_acc);
      err_acc = 0.0;
      err_item = item;
    }
    const ItemDesc &it = p.items[item];
    const unsigned par = (phases >> st) & 1u;
    const bool ok = mbar_wait(&bars[st], par);
    phases ^= 1u << st;
    double2 *bf = buf0 + st * L * W;
    double2 v[P16];
    {
      const OuterRun16 tw = outer_run16<R>(fac + st * TILE_TW_N, ct, t);
      double2 w = tw.b[0];
#pragma unroll
      for (int i = 0; i < P16; i++) {
        if (i % 4 == 0) w = tw.b[i / 4];
        v[i] = cmulc(bf[bidx<L>(t + i * R, s)], w);
        w = cmul(w, tw.st);
      }
    }
    if (__syncthreads_or(!ok)) {  // a wait gave up: flag, drain, leave
      if (tid == 0) {
        atomicOr(it.flags, FLAG_TIMEOUT);
        mbar_drain(&bars[st], par);
        if (un < total) mbar_drain(&bars[st ^ 1], (phases >> (st ^ 1)) & 1u);
      }
      return;
    }
    // the next unit's tile factors (landed and published by this unit's last barriers)
    if (un < total) tile_tw16<R, W>(fac + (st ^ 1) * TILE_TW_N, (int)(un - fd_tiles.div(un) * tiles), p.tw4M, p.M);
    cp_async_commit();
    block16<L, W, true>(v, t, s, bf, twS);
#pragma unroll
    for (int i = 0; i < P16; i++) {
      const int n1 = t + i * R;
      double2 z = cmul(v[i], pwS[n1]);
      double re = rint(z.x), im = rint(z.y);
      err_acc = fmax(err_acc, round_check(z, re, im));
      bf[bidx<L>(n1, s)] = make_double2(re, im);
    }
    cp_async_wait<0>();
    __syncthreads();
    // run records: one 8-column group of one row per (thread, q); L*G rows x
    // groups over NT threads
#pragma unroll
    for (int q = 0; q < (L * G) / NT; q++) {
      const int idx = tid + q * NT, row = idx % L, gi = idx / L;
      double cre[8], cim[8];
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const double2 z = bf[bidx<L>(row, 8 * gi + c)];
        cre[c] = z.x;
        cim[c] = z.y;
      }
      const unsigned n0 = (unsigned)row * (unsigned)p.S1 + (unsigned)tile * W + 8 * gi;
      store_rec(&it.rec[n0 >> 3], make_run(cre, it.b));
      store_rec(&it.rec[(n0 + p.M) >> 3], make_run(cim, it.b));
    }
    static_assert((L * G) % NT == 0, "run pairs per thread");
    __syncthreads();  // the tile buffer is reloaded next iteration
    st ^= 1;
  }
  if (err_item >= 0) atomic_max_err(p.items[err_item].err, err_acc);
}

}  // namespace bc
