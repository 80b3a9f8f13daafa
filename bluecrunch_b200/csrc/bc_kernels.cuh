// bc_kernels.cuh — shared pieces of the exact FFT multiply (sm_100a): item
// and class descriptors, rounding check, the carry kernel and the one-CTA
// kernel for short transforms.
//
// A product class has complex length M = L1 * S1 (two levels, S1 = Lr) or
// M = L1 * L2 * Lr (three levels).  Point n of operand X holds the balanced
// digits n and n+M weighted by e^{i pi n/(2M)}.  Passes (one launch each,
// every launch covers all items of the class; the pass kernels are in
// bc_pipe.cuh):
//
//   k2_outer_fwd  digits -> pre-weight -> L1-point DFT down each column of the
//                 L1 x S1 matrix -> twiddle e^{-2 pi i s(4k1-1)/(4M)} (the
//                 column's weight factor folded in) -> buffer
//   k2_mid<L,0>   (3 levels) L2-point DFT down columns of each L2 x Lr block,
//                 twiddle e^{-2 pi i s k2/(L2 Lr)}
//   k2_rows       per row of Lr points: forward DFT of A and B, pointwise
//                 product (or square), inverse DFT — the spectrum never
//                 leaves the chip (rows of 1024 points: k2_rows_w1024, one
//                 warp per row, bc_rows_warp.cuh)
//   k2_mid<L,1>   (3 levels) inverse of k2_mid<L,0>
//   k2_outer_inv  conjugate twiddle -> inverse L1-point DFT -> un-weight and
//                 1/M -> round (max |x - round(x)| recorded) -> run records:
//                 8 consecutive coefficients -> (H, C), value H + C*2^{8b}
//   k_carry       decoupled-lookback scan of run carries -> output words
//
// k_small does all of it in one CTA for M <= 5120, k_cluster (bc_cluster.cuh)
// in one cluster of CTAs.
//
// Reference correspondence: the whole pipeline computes what _fft_mul
// computes (bigfloat/mul.c:108-174): the exact C = A*B mod 2^{32 CL}.
#pragma once
#include <cuda/atomic>

#include "bc_async.cuh"
#include "bc_device.cuh"

namespace bc {

enum : unsigned { FLAG_TIMEOUT = 1u, FLAG_TOPCARRY = 2u };

struct ItemDesc {
  const uint32_t *A;
  const uint32_t *B;
  uint32_t *C;
  unsigned long long AL, BL, CL;  // AL, BL already clamped to CL
  unsigned long long ndA, ndB;    // number of balanced digits
  double2 *bufA;
  double2 *bufB;                  // null when squaring
  RunRec *rec;                    // 2M/8 run records
  uint32_t *status;               // lookback tile status, zeroed before k_carry
  unsigned long long nwords;      // words written by k_carry (the rest are 0)
  unsigned long long nruns;       // runs needed to cover nwords
  unsigned long long tile0;       // first k_carry tile of this item (class-wide numbering)
  unsigned long long *err;        // max rounding error as double bits (atomicMax)
  unsigned int *flags;
  int b;
  int square;
  int a16, b16;                   // operand A / B starts on a 16-byte boundary
  unsigned long long *outcome;    // three words of pinned host memory: err, flags, and flags of a carry wait that gave up
  int bslot;                      // slot of B's transform in the class's B slab (shared by items with the same B)
};

struct ClassParams {
  int M;
  int L1, S1;      // outer pass: L1-point DFTs with stride S1 = M/L1
  int L2, Lr;      // 3 levels: L2-point DFTs with stride Lr; 2 levels: L2 = 1, Lr = S1
  // Forward-pass units: the A transform of every item, then the B slab's
  // slots (nb of them; slot j is B of item bowner[j], null: item j).  Items
  // with the same B share one slot, so their B is packed and transformed
  // once.  fwd_ops restricts the outer forward pass to A (1) or B (2)
  // units; 0 covers both.
  int fwd_ops;
  int nb;
  const int *bowner;
  Tw2 tw4M;        // e^{-2 pi i m/(4M)}
  const double2 *pw_fwd;  // e^{+i pi n1/(2 L1)}
  const double2 *pw_inv;  // e^{-i pi n1/(2 L1)} / M
  const double2 *twL1, *twL2, *twLr;  // e^{-2 pi i m/L}
  const ItemDesc *items;
  int nitems;
  int sq;                 // every item of the class squares (one operand)
  int parts;              // 2 when an operand of the class has digits at M or above (imaginary parts), else 1
  unsigned int *counter;  // k_carry dynamic tile counter (zeroed before launch)
  unsigned long long carry_tiles;  // total k_carry tiles over the class
  // fused middle pass (three levels): per block (nitems * L1 of them) the
  // count of finished column items, then of finished row items; zeroed
  // before launch.  Null: the middle runs as separate passes.
  unsigned int *blkdone;
  // divisions of unit numbers: by the column tiles of the outer passes (forward,
  // inverse), the
  // units of one operand and the column tiles of a block in the middle passes,
  // and the rows of an item (launch_class fills them in)
  FastDiv fd_fwd, fd_outer, fd_op, fd_mid, fd_rows;
  double2 *slabA, *slabB;          // the class's A and B slabs (item i at slab + i*slab_elems)
  unsigned long long slab_elems;
  // A product alone in its call: its descriptor comes with the first kernel's
  // parameters (single = 1) and that kernel stores it to items[0] for the
  // others and clears the zero_n 16-byte words at `zero` (errors, flags,
  // counters, lookback status), instead of a copy and a memset before it.
  int single;
  unsigned zero_n;
  uint4 *zero;
  ItemDesc one;
};

// Limb words below digit n of an operand cut in digits of b bits, n a multiple
// of 32.  Divided first: n b reaches 2^32 from transforms of 2^28 points on
// (width 16), while n / 32 b stays below 2^30 for n up to 2^30 and b up to 24.
__host__ __device__ __forceinline__ int words_below(int n, int b) { return n / 32 * b; }

// Run records of a transform of M points: its 2M coefficients in runs of 8.
// (2M itself does not fit an int at 2^30 points.)
__host__ __device__ __forceinline__ unsigned long long run_records(int M) { return (unsigned long long)M / 4; }

// What the outer forward pass reads of an item's operand, by value: from the
// parameters' constant bank for a product alone in its call.
struct FwdOperand {
  const uint32_t *X;
  double2 *buf;
  int XL, b;
  unsigned nd;  // below 2^30
  bool al16;
};
__device__ __forceinline__ FwdOperand fwd_operand(const ClassParams &p, int item, int op) {
  FwdOperand o;
  if (p.single) {
    o.X = op ? p.one.B : p.one.A;
    o.buf = op ? p.one.bufB : p.one.bufA;
    o.XL = (int)(op ? p.one.BL : p.one.AL);
    o.nd = (unsigned)(op ? p.one.ndB : p.one.ndA);
    o.b = p.one.b;
    o.al16 = op ? p.one.b16 : p.one.a16;
  } else {
    const ItemDesc &it = p.items[item];
    o.X = op ? it.B : it.A;
    o.buf = op ? it.bufB : it.bufA;
    o.XL = (int)(op ? it.BL : it.AL);
    o.nd = (unsigned)(op ? it.ndB : it.ndA);
    o.b = it.b;
    o.al16 = op ? it.b16 : it.a16;
  }
  return o;
}

// The first kernel's part for a product alone in its call (see ClassParams);
// what the call's later kernels read is complete when this one has ended.
__device__ __forceinline__ void first_kernel_setup(const ClassParams &p) {
  if (!p.single) return;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < p.zero_n; i += gridDim.x * blockDim.x)
    p.zero[i] = make_uint4(0, 0, 0, 0);
  constexpr unsigned N = sizeof(ItemDesc) / 8;
  static_assert(sizeof(ItemDesc) % 8 == 0, "copied by 8-byte words");
  if (blockIdx.x == 0)
    for (unsigned i = threadIdx.x; i < N; i += blockDim.x)
      reinterpret_cast<unsigned long long *>(const_cast<ItemDesc *>(p.items))[i] =
          reinterpret_cast<const unsigned long long *>(&p.one)[i];
}

// An item's outcome to the host (posted writes), once what sets its error and
// flags is done and visible, by the thread that knows of a carry out of the
// product.
__device__ __forceinline__ void publish_outcome(const ItemDesc &it, unsigned more_flags = 0) {
  if (!it.outcome) return;
  const unsigned long long e = *reinterpret_cast<volatile const unsigned long long *>(it.err);
  const unsigned f = *reinterpret_cast<volatile const unsigned *>(it.flags);
  it.outcome[0] = e;
  it.outcome[1] = f | more_flags;
}

// One unit of a forward pass: operand `op` of item `item` (for B, the owner
// of slot `slot`), and the unit's index `rest` inside that operand's
// per_op units.  Units [0, nA) are A's (item-major), the rest B's
// (slot-major).
struct FwdUnit {
  int item, op, slot;
  unsigned rest;
};
__device__ __forceinline__ FwdUnit fwd_unit(const ClassParams &p, unsigned u, unsigned nA, const FastDiv &fd_op,
                                            unsigned per_op) {
  FwdUnit f;
  if (u < nA) {
    const unsigned i = fd_op.div(u);
    f.item = (int)i;
    f.slot = (int)i;
    f.op = 0;
    f.rest = u - i * per_op;
  } else {
    const unsigned v = u - nA, j = fd_op.div(v);
    f.slot = (int)j;
    f.item = p.bowner ? p.bowner[j] : (int)j;
    f.op = 1;
    f.rest = v - j * per_op;
  }
  return f;
}
// A and B unit counts of a forward pass with per_op units per operand.
__device__ __forceinline__ unsigned fwd_units_a(const ClassParams &p, unsigned per_op) {
  return p.fwd_ops != 2 ? (unsigned)p.nitems * per_op : 0u;
}
__device__ __forceinline__ unsigned fwd_units_b(const ClassParams &p, unsigned per_op) {
  return (!p.sq && p.fwd_ops != 1) ? (unsigned)p.nb * per_op : 0u;
}

// Nearest integer of |z| < 2^51 (ties to even, as rint): added to 1.5 2^52 the
// fraction is rounded off.  Above that the result stays near z, so the check
// below still sees a value too large.
__device__ __forceinline__ double round_near(double z) { return (z + 6755399441055744.0) - 6755399441055744.0; }

// Rounding check of one point: max |x - round(x)| of its two coefficients,
// or 1.0 when a coefficient reaches 2^50 — beyond that the distance to the
// nearest integer stops measuring the error (doubles near 2^53 hold no
// fractions), so the product must be redone with narrower digits.
__device__ __forceinline__ double round_check(double2 z, double re, double im) {
  const double big = 1125899906842624.0;  // 2^50
  double e = fmax(fabs(z.x - re), fabs(z.y - im));
  return (fabs(re) >= big || fabs(im) >= big) ? 1.0 : e;
}

__device__ __forceinline__ void atomic_max_err(unsigned long long *p, double e) {
  // non-negative doubles order like their bit patterns
  unsigned long long bits = (unsigned long long)__double_as_longlong(e);
  for (int o = 16; o; o >>= 1) {
    unsigned long long t = __shfl_xor_sync(~0u, bits, o);
    bits = t > bits ? t : bits;
  }
  if ((threadIdx.x & 31) == 0 && bits) atomicMax(p, bits);
}

// ------------------------------------------------------------------ runs
// Low 32 bits of (hi:lo) >> s and high 32 bits of (hi:lo) << s, 0 <= s < 32.
__host__ __device__ __forceinline__ uint32_t shf_r(uint32_t lo, uint32_t hi, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, s);
#else
  return (uint32_t)((((unsigned long long)hi << 32) | lo) >> s);
#endif
}
__host__ __device__ __forceinline__ uint32_t shf_l(uint32_t lo, uint32_t hi, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (uint32_t)(((((unsigned long long)hi << 32) | lo) << s) >> 32);
#endif
}

// An integer held in a double, |c| < 2^51, as 64 bits: added to 1.5 2^52 it
// sits in the low bits of the sum (one add and one subtraction instead of
// the conversion instruction, whose rate is a quarter of theirs).
__host__ __device__ __forceinline__ long long int_of(double c) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(c + 6755399441055744.0) - 0x4338000000000000ll;
#else
  return (long long)c;
#endif
}

// 8 consecutive rounded coefficients c_u (exact integers held in doubles) ->
// H = sum (bits of the running carry) and C = final signed carry.  The digits
// cut from the running carry (b <= 24 bits each) are packed from the top down,
// H = H 2^b + digit, on 32-bit words: only the words that can be nonzero after
// so many digits are shifted.
__host__ __device__ __forceinline__ RunRec make_run(const double *c, int b) {
  uint32_t d[8];
  uint32_t lo = 0, hi = 0;  // the running carry, signed 64 bits
  const uint32_t mask = (1u << b) - 1;
#pragma unroll
  for (int u = 0; u < 8; u++) {
    const unsigned long long acc =
        (((unsigned long long)hi << 32) | lo) + (unsigned long long)int_of(c[u]);
    lo = (uint32_t)acc;
    hi = (uint32_t)(acc >> 32);
    d[u] = lo & mask;
    lo = shf_r(lo, hi, b);
    hi = (uint32_t)((int32_t)hi >> b);  // arithmetic: floor division
  }
  RunRec r;
  r.c = (long long)(((unsigned long long)hi << 32) | lo);
  if (b == 16) {  // constant places
    r.h0 = (unsigned long long)(d[0] | d[1] << 16) | (unsigned long long)(d[2] | d[3] << 16) << 32;
    r.h1 = (unsigned long long)(d[4] | d[5] << 16) | (unsigned long long)(d[6] | d[7] << 16) << 32;
    r.h2 = 0;
    return r;
  }
  uint32_t w[6] = {d[7], 0, 0, 0, 0, 0};
#pragma unroll
  for (int u = 6; u >= 0; u--) {
    const int top = (24 * (8 - u) - 1) / 32;  // highest word after this digit
#pragma unroll
    for (int k = 5; k > 0; k--)
      if (k <= top) w[k] = shf_l(w[k - 1], w[k], b);
    w[0] = w[0] << b | d[u];
  }
  r.h0 = (unsigned long long)w[1] << 32 | w[0];
  r.h1 = (unsigned long long)w[3] << 32 | w[2];
  r.h2 = (unsigned long long)w[5] << 32 | w[4];
  return r;
}

// A record is 32 bytes on a 32-byte boundary: one 256-bit access.  In the
// outer inverse pass every lane's record lies in another row, so each store
// instruction is 32 passes over the L1 data path, its busiest unit; one
// instead of two of them took the pass from 0.252 to 0.219 ms at 2^25 points.
__device__ __forceinline__ void store_rec(RunRec *dst, const RunRec &r) {
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(dst), "l"(r.h0), "l"(r.h1), "l"(r.h2), "l"(r.c)
               : "memory");
}

__device__ __forceinline__ RunRec load_rec(const RunRec *src) {
  RunRec r;
  asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(r.h0), "=l"(r.h1), "=l"(r.h2), "=l"(r.c) : "l"(src)
               : "memory");
  return r;
}

// ------------------------------------------------------------------ scan helper
// Exclusive scan of transfer functions over a CTA of NT threads (earliest
// thread first).  sw needs 65 words.  Returns the exclusive prefix; *total
// receives the composition over the whole CTA.
template <int NT>
__device__ __forceinline__ uint32_t block_scan_fn(uint32_t f, uint32_t *sw, uint32_t *total) {
  static_assert(NT % 32 == 0 && NT <= 1024, "scan CTA size");
  constexpr int NW = NT / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t inc = f;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t o = __shfl_up_sync(~0u, inc, d);
    if (lane >= d) inc = fn_compose(o, inc);
  }
  uint32_t ex = __shfl_up_sync(~0u, inc, 1);
  if (lane == 0) ex = FN_ID;
  if (lane == 31) sw[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    uint32_t x = lane < NW ? sw[lane] : FN_ID;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t o = __shfl_up_sync(~0u, x, d);
      if (lane >= d) x = fn_compose(o, x);
    }
    uint32_t wx = __shfl_up_sync(~0u, x, 1);
    if (lane == 0) wx = FN_ID;
    if (lane < NW) sw[32 + lane] = wx;
    if (lane == 31) sw[64] = x;
  }
  __syncthreads();
  const uint32_t r = fn_compose(sw[32 + wid], ex);
  *total = sw[64];
  __syncthreads();
  return r;
}

// ------------------------------------------------------------------ carry
// Tiles of 1024 runs.  The carry map of a run is constant unless the run is
// all zeros or all ones, so the carry into a run is nearly always known from
// the run before it alone: each warp loads 32 neighbouring records a time
// (32 bytes a lane, coalesced), takes the C below by shuffle, and the carry in
// from the map of the lane below; the tile's first run is preceded by one more
// map that thread 0 computes from the two records before the tile.  Only a
// tile that holds a map that is not constant scans its maps, and only one
// whose predecessor's last map is not constant looks back over the tiles'
// status words: 0 = not ready, (1<<30)|fn = aggregate, (2<<30)|(delta+1) =
// inclusive.  A status word carries all that it says, so it is stored and read
// without ordering other memory.
// What bounds it: HBM, 32 bytes read and b bytes written per run.  Staging
// each tile in shared memory, scanning every tile and looking back for every
// one took 0.138 ms for the 2^24-limb product's 2^26 coefficients (2.9 TB/s);
// this form takes 0.070 ms (5.8 TB/s).
constexpr int CARRY_NT = 256;
constexpr int CARRY_RPT = 4;                            // runs per thread, CARRY_NT apart
constexpr int CARRY_TILE_RUNS = CARRY_NT * CARRY_RPT;   // runs per tile
constexpr unsigned ST_AGG = 1u << 30, ST_INC = 2u << 30;
constexpr int LOOKBACK_SPINS = 1 << 22;

__device__ __forceinline__ U192 rec_h(const RunRec &r) { U192 h = {{r.h0, r.h1, r.h2}}; return h; }

// The words of a run of nbits >= 64 bits that starts at bit bit0: put(w, x)
// for every word w that starts inside the run; a word that straddles into the
// next run takes its high bits from `next`, that run's low 32 bits.
template <class Put>
__host__ __device__ __forceinline__ void run_words(unsigned long long bit0, int nbits, const U192 &h, uint32_t next,
                                          const Put &put) {
  const unsigned long long w0 = (bit0 + 31) >> 5;
  const int o = (int)((w0 << 5) - bit0);  // bit of the run where word w0 starts, below 32
  const uint32_t W[7] = {(uint32_t)h.w[0], (uint32_t)(h.w[0] >> 32), (uint32_t)h.w[1], (uint32_t)(h.w[1] >> 32),
                         (uint32_t)h.w[2], (uint32_t)(h.w[2] >> 32), 0u};
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const int off = o + 32 * k;
    if (off < nbits) {
      uint32_t x = shf_r(W[k], W[k + 1], o);
      if (off + 32 > nbits) x |= next << (nbits - off);
      put(w0 + k, x);
    }
  }
}

// Words of run r (bits [r nbits, (r+1) nbits)) below nwords; a word that
// straddles into run r+1 takes its high bits from hn.
__device__ __forceinline__ void write_run_words(uint32_t *C, unsigned long long nwords, unsigned long long r,
                                                int nbits, const U192 &h, const U192 &hn) {
  run_words(r * (unsigned long long)nbits, nbits, h, (uint32_t)hn.w[0], [&](unsigned long long w, uint32_t x) {
    if (w < nwords) C[w] = x;
  });
}

// Carry into tile `tile` (> 0) by its status words, nearest first; *timed_out
// when the bounded wait gave up.
__device__ __forceinline__ int carry_lookback(uint32_t *status, unsigned long long tile, bool *timed_out) {
  uint32_t acc = FN_ID;  // maps of the tiles passed so far (nearest applied last)
  long long prev = (long long)tile - 1;
  int spins = 0;
  for (;;) {
    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> st(status[prev]);
    const uint32_t v = st.load(cuda::memory_order_relaxed);
    if (v & ST_INC) return fn_apply(acc, (int)(v & 3u) - 1);
    if (v & ST_AGG) {
      acc = fn_compose(v & 0x3fu, acc);
      prev--;  // tile 0 publishes an inclusive value, so prev stays at 0 or above
    } else {
      if (++spins > LOOKBACK_SPINS) { *timed_out = true; return 0; }
      if (spins > 64) __nanosleep(32);
    }
  }
}

// NB = 128: every item of the class has width 16 (runs of 128 bits), so the
// run arithmetic below is specialised at compile time; NB = 0: any width.
// Tiles are claimed from a counter (the first before the pass before this one
// has ended, each further one while the tile before it is worked on), so a
// lookback waits only for tiles that running CTAs hold.
template <int NB>
__global__ void __launch_bounds__(CARRY_NT, 4) k_carry(ClassParams p) {
  constexpr int NW = CARRY_NT / 32;
  __shared__ __align__(16) uint32_t words[CARRY_TILE_RUNS * (NB ? 4 : 6)];  // the tile's words, unless they go to C at once
  __shared__ uint32_t low[NB ? 4 : CARRY_TILE_RUNS + 1];  // low word of each corrected run, and of the run after them
  __shared__ uint32_t lastf[CARRY_RPT * NW];   // map of each warp's last run
  __shared__ uint8_t fm[CARRY_TILE_RUNS];      // all maps, then the carries + 1 (only when the tile is scanned)
  __shared__ uint32_t sw[65];
  __shared__ unsigned s_unit[2];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // Before the wait: the counter was cleared two or more launches ago (by the
  // class's first kernel or a copy before it), and every pass between waits
  // before it triggers, so what came before the previous pass is complete here.
  if (tid == 0) s_unit[0] = atomicAdd(p.counter, 1u);
  pdl_wait();
  pdl_trigger();
  __syncthreads();
  for (int par = 0;; par ^= 1) {
    const unsigned long long unit = s_unit[par];
    if (unit >= p.carry_tiles) break;
    if (tid == 0) s_unit[par ^ 1] = atomicAdd(p.counter, 1u);  // read after the tile's last barrier
    // find the item owning this tile (items are ordered by tile0)
    int lo = 0, hi = p.nitems - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (p.items[mid].tile0 <= unit) lo = mid; else hi = mid - 1;
    }
    const ItemDesc &it = p.items[lo];
    const unsigned long long tile = unit - it.tile0;
    const unsigned long long rt = tile * CARRY_TILE_RUNS;  // first run of the tile
    const unsigned long long nruns = it.nruns, nwords = it.nwords;
    const int nr = (int)min((unsigned long long)CARRY_TILE_RUNS, nruns - rt);  // runs of this tile
    const int nbits = NB ? NB : 8 * it.b;
    const unsigned long long nrec = run_records(p.M);
    const RunRec *const rec = it.rec + rt;
    // ---- records: run q*CARRY_NT + tid in slot q
    U192 h[CARRY_RPT];
    long long c[CARRY_RPT], cp[CARRY_RPT];
    uint32_t f[CARRY_RPT];
#pragma unroll
    for (int q = 0; q < CARRY_RPT; q++) {
      const int k = q * CARRY_NT + tid;
      RunRec r = {0, 0, 0, 0};
      if (k < nr) r = load_rec(&rec[k]);
      h[q] = rec_h(r);
      c[q] = r.c;
      cp[q] = 0;
      if (lane == 0 && k < nr && rt + k > 0) cp[q] = rec[k - 1].c;
    }
    // the carry into the tile, when the map of the run before it tells
    int din = 0;
    bool known = true;
    if (tid == 0 && rt > 0) {
      const RunRec r1 = load_rec(&rec[-1]);
      U192 h1 = rec_h(r1);
      const uint32_t f1 = run_transfer(h1, rt > 1 ? rec[-2].c : 0, nbits);
      known = fn_is_const(f1);
      din = fn_apply(f1, 0);
    }
    bool odd = !known;
#pragma unroll
    for (int q = 0; q < CARRY_RPT; q++) {
      const long long up = __shfl_up_sync(~0u, c[q], 1);
      f[q] = FN_ID;
      if (q * CARRY_NT + tid < nr) {
        f[q] = run_transfer(h[q], lane ? up : cp[q], nbits);
        odd = odd || !fn_is_const(f[q]);
      }
      if (lane == 31) lastf[q * NW + wid] = f[q];
    }
    const bool scan = __syncthreads_or(odd);
    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> me(it.status[tile]);
    int d[CARRY_RPT];  // carry into each run
    if (!scan) {
#pragma unroll
      for (int q = 0; q < CARRY_RPT; q++) {
        const uint32_t up = __shfl_up_sync(~0u, f[q], 1);
        const int k = q * CARRY_NT + tid;
        d[q] = k == 0 ? din : fn_apply(lane ? up : lastf[q * NW + wid - 1], 0);
        if (k + 1 == nr) me.store(ST_INC | (uint32_t)(fn_apply(f[q], 0) + 1), cuda::memory_order_relaxed);
      }
    } else {
#pragma unroll
      for (int q = 0; q < CARRY_RPT; q++) fm[q * CARRY_NT + tid] = (uint8_t)f[q];
      __syncthreads();
      uint32_t F = FN_ID;  // the thread's four neighbouring runs
#pragma unroll
      for (int j = 0; j < CARRY_RPT; j++) F = fn_compose(F, fm[CARRY_RPT * tid + j]);
      uint32_t agg;
      const uint32_t ex = block_scan_fn<CARRY_NT>(F, sw, &agg);
      if (tid == 0) {
        const bool fixed = fn_is_const(agg);
        if (fixed || known) me.store(ST_INC | (uint32_t)(fn_apply(agg, din) + 1), cuda::memory_order_relaxed);
        else me.store(ST_AGG | agg, cuda::memory_order_relaxed);
        if (!known) {
          bool timed_out = false;
          din = carry_lookback(it.status, tile, &timed_out);
          if (timed_out) {
            atomicOr(it.flags, FLAG_TIMEOUT);
            if (it.outcome) it.outcome[2] = FLAG_TIMEOUT;
          }
          if (!fixed) me.store(ST_INC | (uint32_t)(fn_apply(agg, din) + 1), cuda::memory_order_relaxed);
        }
        sw[0] = (uint32_t)(din + 1);
      }
      __syncthreads();
      int dd = fn_apply(ex, (int)sw[0] - 1);
#pragma unroll
      for (int j = 0; j < CARRY_RPT; j++) {
        const uint32_t fj = fm[CARRY_RPT * tid + j];
        fm[CARRY_RPT * tid + j] = (uint8_t)(dd + 1);
        dd = fn_apply(fj, dd);
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < CARRY_RPT; q++) d[q] = (int)fm[q * CARRY_NT + tid] - 1;
    }
    // ---- corrected runs: each one's four words straight to C (runs of 128
    // bits, every word of the tile inside the product, C on a 16-byte
    // boundary), or through shared memory
    const bool whole = nbits == 128 && (reinterpret_cast<uintptr_t>(it.C) & 15) == 0 &&
                       4ull * (rt + (unsigned long long)nr) <= nwords;
#pragma unroll
    for (int q = 0; q < CARRY_RPT; q++) {
      const int k = q * CARRY_NT + tid;
      if (k < nr) {
        u192_add_delta(h[q], d[q], nbits);
        if (whole) {
          *reinterpret_cast<uint4 *>(it.C + 4 * (rt + (unsigned long long)k)) =
              make_uint4((uint32_t)h[q].w[0], (uint32_t)(h[q].w[0] >> 32), (uint32_t)h[q].w[1],
                         (uint32_t)(h[q].w[1] >> 32));
        } else if (NB) {  // 128 bits: no word straddles two runs
          reinterpret_cast<uint4 *>(words)[k] = make_uint4((uint32_t)h[q].w[0], (uint32_t)(h[q].w[0] >> 32),
                                                           (uint32_t)h[q].w[1], (uint32_t)(h[q].w[1] >> 32));
        } else {
          low[k] = (uint32_t)h[q].w[0];
        }
        if (k + 1 == nr) {
          const int dout = fn_apply(f[q], d[q]);
          const unsigned long long r = rt + k;
          if (!NB) {
            // the run after the tile's last one, for a word that straddles it:
            // inside this item only when the item ends inside this tile
            low[nr] = nr < CARRY_TILE_RUNS && r + 1 < nrec
                          ? (uint32_t)(rec[k + 1].h0 + (unsigned long long)(c[q] + dout)) : 0u;
          }
          unsigned top = 0;
          if (r + 1 == nrec && c[q] + dout != 0) {
            top = FLAG_TOPCARRY;
            atomicOr(it.flags, top);
          }
          // the item's last run: its error and the flags of the passes before
          // are complete, so this thread tells the host
          if (r + 1 == nruns) publish_outcome(it, top);
        }
      }
    }
    if (!whole) {  // uniform over the CTA
      __syncthreads();
      if (!NB) {
        // the tile starts on a word boundary (1024 runs of 8b bits)
#pragma unroll
        for (int q = 0; q < CARRY_RPT; q++) {
          const int k = q * CARRY_NT + tid;
          if (k < nr)
            run_words((unsigned long long)(k * nbits), nbits, h[q], low[k + 1],
                      [&](unsigned long long w, uint32_t x) { words[w] = x; });
        }
        __syncthreads();
      }
      const unsigned long long w0 = rt * (unsigned long long)nbits / 32;
      const unsigned long long wend = min(nwords, w0 + ((unsigned long long)nr * nbits + 31) / 32);
      const int nw = wend > w0 ? (int)(wend - w0) : 0;
      uint32_t *const out = it.C + w0;
      if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
        for (int i = tid; i < nw / 4; i += CARRY_NT)
          reinterpret_cast<uint4 *>(out)[i] = reinterpret_cast<const uint4 *>(words)[i];
        if (tid < (nw & 3)) out[(nw & ~3) + tid] = words[(nw & ~3) + tid];
      } else {
        for (int i = tid; i < nw; i += CARRY_NT) out[i] = words[i];
      }
    }
    // zero any words beyond the product (CL > product length)
    if (tile == 0) {
      for (unsigned long long w = nwords + tid; w < it.CL; w += CARRY_NT) it.C[w] = 0;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ small
// Whole product in one CTA of M/8 threads (M <= 5120): pack, FFT, product,
// inverse, round, runs, in-CTA carry scan, words.
template <int M, bool SQ>
__global__ void __launch_bounds__(M / PTS, 1) k_small(ClassParams p) {
  extern __shared__ double2 sm[];
  constexpr int TC = M / PTS, NR = M / 8;  // NR real runs, NR imaginary runs
  static_assert(TC % 32 == 0, "k_small needs M >= 256");
  __shared__ uint32_t sw[65];
  const int t = threadIdx.x;
  RunRec *srec = reinterpret_cast<RunRec *>(sm);  // reused after the FFTs
  for (int item = blockIdx.x; item < p.nitems; item += gridDim.x) {
    const ItemDesc &it = p.items[item];
    double2 va[PTS], v[PTS];
#pragma unroll
    for (int i = 0; i < PTS; i++) {
      const int n = t + i * TC;
      double2 z = make_double2(digit_at(it.A, it.AL, it.b, n, it.ndA), digit_at(it.A, it.AL, it.b, n + M, it.ndA));
      va[i] = cmul(z, __ldg(&p.pw_fwd[n]));
    }
    block_fft<M, 1, false>(va, t, 0, sm, p.twL1);
    if (SQ) {
#pragma unroll
      for (int i = 0; i < PTS; i++) v[i] = cmul(va[i], va[i]);
    } else {
#pragma unroll
      for (int i = 0; i < PTS; i++) {
        const int n = t + i * TC;
        double2 z = make_double2(digit_at(it.B, it.BL, it.b, n, it.ndB), digit_at(it.B, it.BL, it.b, n + M, it.ndB));
        v[i] = cmul(z, __ldg(&p.pw_fwd[n]));
      }
      block_fft<M, 1, false>(v, t, 0, sm, p.twL1);
#pragma unroll
      for (int i = 0; i < PTS; i++) v[i] = cmul(va[i], v[i]);
    }
    block_fft<M, 1, true>(v, t, 0, sm, p.twL1);
    double err = 0.0;
#pragma unroll
    for (int i = 0; i < PTS; i++) {
      const int n = t + i * TC;
      double2 z = cmul(v[i], __ldg(&p.pw_inv[n]));
      double re = rint(z.x), im = rint(z.y);
      err = fmax(err, round_check(z, re, im));
      sm[sidx<M, 1>(n, 0)] = make_double2(re, im);
    }
    atomic_max_err(it.err, err);
    __syncthreads();
    double cre[8], cim[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      double2 z = sm[sidx<M, 1>(8 * t + u, 0)];
      cre[u] = z.x; cim[u] = z.y;
    }
    RunRec rre = make_run(cre, it.b), rim = make_run(cim, it.b);
    __syncthreads();
    srec[t] = rre;
    srec[NR + t] = rim;
    __syncthreads();
    const int nbits = 8 * it.b;
    // transfer functions
    U192 hre = rec_h(rre), him = rec_h(rim);
    const long long cprev_re = t ? srec[t - 1].c : 0;
    const long long cprev_im = srec[NR + t - 1].c;
    const uint32_t fre = run_transfer(hre, cprev_re, nbits);
    const uint32_t fim = run_transfer(him, cprev_im, nbits);
    uint32_t tot_re, tot_im;
    const uint32_t ex_re = block_scan_fn<TC>(fre, sw, &tot_re);
    const uint32_t ex_im = block_scan_fn<TC>(fim, sw, &tot_im);
    const int din_re = fn_apply(ex_re, 0);
    const int d_half = fn_apply(tot_re, 0);
    const int din_im = fn_apply(ex_im, d_half);
    u192_add_delta(hre, din_re, nbits);
    u192_add_delta(him, din_im, nbits);
    const int dout_im = fn_apply(fim, din_im);
    __syncthreads();
    srec[t].h0 = hre.w[0]; srec[t].h1 = hre.w[1]; srec[t].h2 = hre.w[2];
    srec[NR + t].h0 = him.w[0]; srec[NR + t].h1 = him.w[1]; srec[NR + t].h2 = him.w[2];
    __syncthreads();
    const U192 zero = {{0, 0, 0}};
    const U192 nre = rec_h(srec[t + 1 < 2 * NR ? t + 1 : t]);
    const U192 nim = (NR + t + 1 < 2 * NR) ? rec_h(srec[NR + t + 1]) : zero;
    write_run_words(it.C, it.nwords, (unsigned long long)t, nbits, hre, nre);
    write_run_words(it.C, it.nwords, (unsigned long long)(NR + t), nbits, him, nim);
    if (t == TC - 1 && rim.c + dout_im != 0) atomicOr(it.flags, FLAG_TOPCARRY);
    for (unsigned long long w = it.nwords + t; w < it.CL; w += TC) it.C[w] = 0;
    __threadfence();  // the warps' error and flag updates, before thread 0 reads them
    __syncthreads();
    if (t == 0) publish_outcome(it);
  }
}

}  // namespace bc
