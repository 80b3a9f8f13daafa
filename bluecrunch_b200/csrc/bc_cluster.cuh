// bc_cluster.cuh — short products (one kernel each) on a cluster of CTAs.
//
// A transform of M points is split M = NC x S over the NC CTAs of a cluster:
// point n = s + S i (i < NC), and CTA c transforms row c of S points.
//
//   forward  row c, point s:  e^{i pi s/(2M)} e^{-2 pi i s c/M} *
//            sum_i d[s + S i] e^{i pi i/(2 NC)} e^{-2 pi i i c/NC}
//            then an S-point DFT.  The column DFT of length NC is a sum of NC
//            digits times constants of the CTA (the right-angle weight is
//            inside them), so every CTA cuts the digits it needs itself and
//            nothing is exchanged.  A and B run side by side in two groups of
//            S/8 threads.
//   product, inverse S-point DFT, conjugate twiddle: Y_c[s] in shared memory.
//   inverse  CTA c takes the columns s of its S/NC wide share, reads their NC
//            values from the CTAs of the cluster (distributed shared memory;
//            each starts at its own, so no CTA is read by all at once), an
//            NC-point DFT per thread, un-weight, round.
//   carry    its columns are 2 NC segments of the product (real and imaginary
//            part of every i).  It also computes the 8 columns before and
//            after its share (the neighbours' runs), so the run carries need no
//            exchange; the segments' composed carry maps are pushed to every
//            CTA, one warp scans all of them.
//
// What bounds it: latency, a chain of phases of one to three thousand cycles.
// One CTA for the whole product (k_small, M/8 threads) leaves 147 SMs idle and
// does the FP64 work of three transforms on one SM: 12.6 us of it at M = 5120
// at the full FP64 rate.  The cluster divides that work by NC and waits on the
// others twice per product.  GPU time of one product, k_small -> this kernel:
// 14.6 -> 10.5 us at M = 256, 16.8 -> 12.4 at 1024, 26.8 -> 16.9 at 2560,
// 45.6 -> 20.4 at 5120 (B200; 16.6, 18.8, 29 and 48 us with the run packing
// that k_small had before).
#pragma once
#include <cooperative_groups.h>

#include "bc_kernels.cuh"

namespace bc {

template <int M> struct ClusterShape {
  // eight CTAs where every CTA's share of the columns is whole runs of 8
  static constexpr int NC = (M % 512 == 0) ? 8 : 4;
  static constexpr int S = M / NC;           // row of one CTA
  static constexpr int P = S / NC;           // its share of the columns
  static constexpr int TC = S / PTS;         // threads of one row transform
  // a point of A or B each in the packing.  512 threads leave 128 registers,
  // which the row transforms (NF threads) exceed where S is 3 or 5 times a
  // power of two: 1,280, 1,536, 2,560, 3,072 and 5,120 points spill 160 to 350
  // bytes a thread, 768 points (384 threads) 88.
  static constexpr int NT = 2 * S < 512 ? 2 * S : 512;
  static constexpr int NF = (2 * TC + 31) / 32 * 32;    // threads that run the row transforms
  static constexpr int NG = (NF + TC - 1) / TC;  // their groups (two in use, the rest idle along)
  static constexpr int SEG = 2 * NC;         // segments of the product per CTA
  static constexpr int RUNS = P / 8;         // runs per segment
  static constexpr int SLOTS = RUNS + 2;     // with the neighbours' runs
  static constexpr int COLS = P + 16;
  static_assert(M % NC == 0 && P % 8 == 0 && S % 64 == 0, "columns in whole runs");
  static_assert(SEG * RUNS <= NT && COLS <= NT && NF <= NT && NT % 32 == 0, "threads cover the phases");
  // limb words of both operands (their digits number at most 2M + 1 of at
  // most 24 bits: at most 3M/2 words) with a zero word below, two above and
  // up to three for alignment each
  static constexpr int LIMBS = 3 * M / 2 + 48;
  static constexpr int TWN = StagedTw<S>::entries();
  static constexpr size_t O_ROWS = 0;                                  // NG rows; row 1 later holds Y
  static constexpr size_t O_FLAT = O_ROWS + (size_t)NG * S * 16;
  static constexpr size_t O_STG = O_FLAT + (size_t)tw_entries<S>() * 16;
  static constexpr size_t O_TWC = O_STG + (size_t)TWN * 16;
  static constexpr size_t O_REC = O_TWC + (size_t)S * 16;
  static constexpr size_t O_COEF = O_REC + (size_t)SEG * SLOTS * sizeof(RunRec);
  static constexpr size_t O_LIMB = O_COEF + (size_t)SEG * COLS * 8;
  static constexpr size_t SMEM = O_LIMB + (size_t)LIMBS * 4;
};

// Exact conversion of a small integer without the quarter-rate I2F: the bits
// of 2^52 + 2^31 + d, minus that constant.
__device__ __forceinline__ double small_to_double(int d) {
  return __hiloint2double(0x43300000, (int)((unsigned)d ^ 0x80000000u)) - 4503601774854144.0;
}

// XL limbs into dst[0..XL+2]: a zero word (below the first digit), the limbs
// (dst + 1 on a 16-byte boundary), two zero words; all threads, asynchronous,
// 16 bytes at a time where the operand starts on a 16-byte boundary.
__device__ __forceinline__ void stage_limbs(uint32_t *dst, const uint32_t *__restrict__ X, int XL) {
  if ((reinterpret_cast<uintptr_t>(X) & 15) == 0) {
    for (int i = 4 * threadIdx.x; i < XL; i += 4 * blockDim.x)
      cp_async16(dst + 1 + i, X + i, 4 * min(4, XL - i));  // zeros past the last limb
  } else {
    for (int i = threadIdx.x; i < XL; i += blockDim.x) cp_async4(dst + 1 + i, X + i, 4);
  }
  if (threadIdx.x < 3) dst[threadIdx.x == 0 ? 0 : XL + (int)threadIdx.x] = 0u;
}

template <int M, bool SQ>
__global__ void __cluster_dims__(ClusterShape<M>::NC, 1, 1) __launch_bounds__(ClusterShape<M>::NT, 1)
    k_cluster(const __grid_constant__ ClassParams p) {
  namespace cg = cooperative_groups;
  using T = ClusterShape<M>;
  constexpr int NC = T::NC, S = T::S, P = T::P, TC = T::TC, NT = T::NT, NF = T::NF;
  constexpr int SEG = T::SEG, RUNS = T::RUNS, SLOTS = T::SLOTS, COLS = T::COLS;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ uint32_t fm[SEG * RUNS];      // carry map of each run
  __shared__ uint32_t segmap[SEG * NC];    // composed map of every segment of the product, in order
  __shared__ int segd[SEG];                // delta into this CTA's segments
  __shared__ double2 K[NC];                // e^{i pi i/(2 NC)} e^{-2 pi i i c/NC}
  __shared__ double2 Ki[NC];               // e^{-i pi i/(2 NC)} / M * e^{+2 pi i i c/NC}
  double2 *const rows = reinterpret_cast<double2 *>(smraw + T::O_ROWS);
  double2 *const flat = reinterpret_cast<double2 *>(smraw + T::O_FLAT);
  double2 *const stg = reinterpret_cast<double2 *>(smraw + T::O_STG);
  double2 *const twc = reinterpret_cast<double2 *>(smraw + T::O_TWC);
  RunRec *const rec = reinterpret_cast<RunRec *>(smraw + T::O_REC);
  double *const coef = reinterpret_cast<double *>(smraw + T::O_COEF);
  uint32_t *const limb = reinterpret_cast<uint32_t *>(smraw + T::O_LIMB);
  cg::cluster_group cl = cg::this_cluster();
  const int c = (int)cl.block_rank();
  const int tid = threadIdx.x;
  double2 *const Y = rows + S;
  const int nclus = gridDim.x / NC;
  bool tables = false;
  if (c == 0) {  // before the cluster's first barrier; nothing here is used before it
    if (p.single)
      for (unsigned i = tid; i < p.zero_n; i += NT) p.zero[i] = make_uint4(0, 0, 0, 0);
  }
  for (int item = blockIdx.x / NC; item < p.nitems; item += nclus) {
    const ItemDesc &it = p.single ? p.one : p.items[item];
    const int AL = (int)it.AL, BL = (int)it.BL, b = it.b;
    uint32_t *const limbA = limb + 3, *const limbB = limbA + ((AL + 3 + 3) & ~3);
    stage_limbs(limbA, it.A, AL);
    if (!SQ) stage_limbs(limbB, it.B, BL);
    cp_async_commit();
    if (!tables) {  // while the limbs cross
      tables = true;
      for (int m = tid; m < tw_entries<S>(); m += NT) flat[m] = __ldg(&p.twL1[m * NC]);
      for (int s = tid; s < S; s += NT) twc[s] = cmul(__ldg(&p.pw_fwd[s]), __ldg(&p.twL1[s * c]));
      staged_tw_build<S, NC>(stg, p.twL1);
      if (tid < NC) {
        K[tid] = cmul(__ldg(&p.pw_fwd[tid * S]), __ldg(&p.twL1[((tid * c) % NC) * S]));
        Ki[tid] = cmulc(__ldg(&p.pw_inv[tid * S]), __ldg(&p.twL1[((tid * c) % NC) * S]));
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    // ---- digits, column sums, twiddle: one point of A or B per thread and step
    for (int k = tid; k < (SQ ? S : 2 * S); k += NT) {
      const bool opB = k >= S;
      const int s = opB ? k - S : k;
      const int nd = (int)(opB ? it.ndB : it.ndA);
      // digit s + S i: its bits start at ((s + S i) b) of the limbs; one bit
      // below it, past the zero word, sits at bit `sh` of word w (S b is a
      // multiple of 32, so sh is the same for every i)
      const unsigned pos = (unsigned)(s * b) + 31u, sh = pos & 31u;
      const uint32_t *x0 = opB ? limbB : limbA, *w = x0 + (pos >> 5);
      const int step = S / 32 * b, up = 31 - b, down = 32 - b;
      // all NC digits at once (independent loads); a digit at nd or above is
      // zero and reads word 0 of its operand.  Sign-extended b bits plus the
      // top bit of the digit below; the most significant digit (j = nd - 1)
      // stays unsigned.
      auto cut = [&](int i0, double (&d)[NC]) {
#pragma unroll
        for (int i = 0; i < NC; i++) {
          const int j = s + S * (i0 + i);
          const uint32_t *wj = j < nd ? w + (i0 + i) * step : x0;
          const unsigned x = __funnelshift_r(wj[0], wj[1], sh);
          int r = ((int)(x << up) >> down);
          if (j + 1 == nd) r = (int)((x << up) >> down);
          d[i] = small_to_double(j < nd ? r + (int)(x & 1u) : 0);
        }
      };
      double2 a = make_double2(0.0, 0.0);
      double d[NC];
      cut(0, d);
#pragma unroll
      for (int i = 0; i < NC; i++) {
        a.x = fma(d[i], K[i].x, a.x);
        a.y = fma(d[i], K[i].y, a.y);
      }
      if (nd > M) {  // digits M and up: the imaginary parts
        cut(NC, d);
#pragma unroll
        for (int i = 0; i < NC; i++) {
          a.x = fma(-d[i], K[i].y, a.x);
          a.y = fma(d[i], K[i].x, a.y);
        }
      }
      rows[opB ? S + sidx<S, 1>(s, 0) : sidx<S, 1>(s, 0)] = cmul(a, twc[s]);
    }
    __syncthreads();
    // ---- row transforms (A and B in step), product, inverse
    if (tid < NF) {
      const GroupSync<NF> fs{1};
      const int grp = tid / TC, t = tid - grp * TC;
      double2 *const myrow = rows + grp * S;
      double2 v[PTS];
      load_regs<S, 1>(v, t, 0, myrow);
      fs();
      block_fft<S, 1, false, GroupSync<NF>, true>(v, t, 0, myrow, flat, fs, stg);
      if (SQ) {
#pragma unroll
        for (int k = 0; k < PTS; k++) v[k] = cmul(v[k], v[k]);
        fs();
      } else {
        if (grp == 1) {
#pragma unroll
          for (int k = 0; k < PTS; k++) myrow[sidx<S, 1>(t + k * TC, 0)] = v[k];
        }
        fs();
        if (grp == 0) {
#pragma unroll
          for (int k = 0; k < PTS; k++) v[k] = cmul(v[k], rows[S + sidx<S, 1>(t + k * TC, 0)]);
        }
        fs();  // row 1 is read: the groups' exchanges may use it again
      }
      block_fft<S, 1, true, GroupSync<NF>, true>(v, t, 0, myrow, flat, fs, stg);
      fs();
      if (grp == 0) {
#pragma unroll
        for (int k = 0; k < PTS; k++) Y[t + k * TC] = cmulc(v[k], twc[t + k * TC]);
      }
    }
    cl.sync();
    // ---- this CTA's columns (and 8 on either side): inverse column DFT, round
    double err = 0.0;
    if (tid < COLS) {
      const int cc = tid;
      int s = c * P - 8 + cc, dq = 0;  // values of column s land in segment i + dq
      if (s < 0) { s += S; dq = 1; }
      else if (s >= S) { s -= S; dq = -1; }
      double2 x[NC];
#pragma unroll
      for (int k = 0; k < NC; k++) x[k] = cl.map_shared_rank(Y, (k + c) % NC)[s];  // from c up: Ki turns it back
      dftR<NC, true>(x);
#pragma unroll
      for (int i = 0; i < NC; i++) {
        const double2 z = cmul(x[i], Ki[i]);
        const double re = round_near(z.x), im = round_near(z.y);
        err = fmax(err, round_check(z, re, im));
        const int q = i + dq, qi = NC + i + dq;
        if (q >= 0) coef[q * COLS + cc] = re;
        if (qi < SEG) coef[qi * COLS + cc] = im;
      }
    }
    if (tid < (COLS + 31) / 32 * 32) atomic_max_err(it.err, err);
    __syncthreads();
    // ---- runs of 8 coefficients; slot 0 and the last one are the neighbours'
    for (int k = tid; k < SEG * SLOTS; k += NT) {
      const int q = k / SLOTS, sl = k - q * SLOTS;
      const bool none = (q == 0 && sl == 0 && c == 0) || (q == SEG - 1 && sl == SLOTS - 1 && c == NC - 1);
      double cr[8];
#pragma unroll
      for (int u = 0; u < 8; u++) cr[u] = none ? 0.0 : coef[q * COLS + 8 * sl + u];
      rec[k] = make_run(cr, b);
    }
    __syncthreads();
    // ---- carry map of each run
    const int nbits = 8 * b;
    const bool has = tid < SEG * RUNS;
    const int q = has ? tid / RUNS : 0, rr = has ? tid - q * RUNS : 0;
    const RunRec me = rec[q * SLOTS + rr + 1];
    U192 h = rec_h(me);
    uint32_t f = FN_ID;
    if (has) {
      f = run_transfer(h, rec[q * SLOTS + rr].c, nbits);
      fm[tid] = f;
    }
    __syncthreads();
    // ---- composed map of each segment: the maps from its last run back to the
    // nearest constant one (nearly always the last), to every CTA
    if (tid < SEG) {
      int k = RUNS - 1;
      uint32_t F = fm[tid * RUNS + k];
      while (k > 0 && !fn_is_const(F)) F = fn_compose(fm[tid * RUNS + --k], F);
#pragma unroll
      for (int k2 = 0; k2 < NC; k2++) cl.map_shared_rank(segmap, k2)[tid * NC + c] = F;
    }
    cl.sync();
    // ---- delta into each segment: back from the one before it to the nearest
    // constant map
    if (tid < SEG) {
      int g = tid * NC + c;  // this segment's place in the product
      uint32_t F = FN_ID;
      while (g > 0 && !fn_is_const(F)) F = fn_compose(segmap[--g], F);
      segd[tid] = fn_apply(F, 0);
    }
    __syncthreads();
    // ---- carries into each run, words
    if (has) {
      int k = rr;
      uint32_t F = FN_ID;
      while (k > 0 && !fn_is_const(F)) F = fn_compose(fm[q * RUNS + --k], F);
      const int din = fn_apply(F, segd[q]);
      const int dout = fn_apply(f, din);
      u192_add_delta(h, din, nbits);
      // the low word of the next run, for a word that straddles it
      U192 hn = {{rec[q * SLOTS + rr + 2].h0 + (unsigned long long)(me.c + dout), 0, 0}};
      const unsigned long long r = (unsigned long long)((q * S + c * P) / 8 + rr);
      write_run_words(it.C, it.nwords, r, nbits, h, hn);
      if (q == SEG - 1 && c == NC - 1 && rr == RUNS - 1 && me.c + dout != 0) {
        atomicOr(it.flags, FLAG_TOPCARRY);
        __threadfence();
      }
    }
    for (unsigned long long w = it.nwords + (unsigned)(c * NT + tid); w < it.CL; w += NC * NT) it.C[w] = 0;
    __syncthreads();  // the limbs, runs and maps are free for the next product
    // the errors were published before the second cluster barrier, the flag of
    // a carry out of the product by this CTA
    if (tid == 0 && c == NC - 1) publish_outcome(it);
    // ---- end
  }
}

}  // namespace bc
