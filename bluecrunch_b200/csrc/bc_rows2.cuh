// bc_rows2.cuh — the row pass for rows of P1 x P2 points (128, 192, 256, 320,
// 384, 640, 768), each stage one transform in registers.
//
// Same arithmetic contract as k2_rows (bc_pipe.cuh): every row r of the class
// gets A_r <- IDFT(DFT(A_r) . DFT(B_r)) (or the square), unscaled.  With
// n = j + P2 i and k = k1 + P1 k2:
//   forward  thread j (< P2): DFT-P1 over i, twiddle e^{-2 pi i j k1/L};
//            one exchange through the row's buffer;
//            thread k1 (< P1): DFT-P2 over j: X[k1 + P1 k2] in w[k2].
//   inverse  the same steps backwards: thread k1 inverse DFT-P2, exchange,
//            thread j conjugate twiddle, inverse DFT-P1, points j + P2 i.
// A and B meet in registers.  Up to 256 points B's spectrum stays there while A
// is transformed, from 320 on it waits in B's buffer.  A row is held by
// max(P1, P2) threads; rows whose threads divide a warp (16 of them up to 256
// points, 32 at 640 and 768) are private to it, others synchronise over the CTA.
//
// What bounds it: shared memory and FP64 about alike.  k2_rows exchanges two
// or three times per transform (and stores the odd radix's points back
// first), 8 points per thread: at 24 ps per point it was a third of every
// product whose length is 3 or 5 times a power of two, 2.5 times the 9.5 ps of
// the 512-point rows.  Rows of 320 points at 5*2^22: 0.496 -> 0.264 ms, of 384
// at 3*2^23: 0.618 -> 0.337, of 192 squared at 3*2^21: 0.080 -> 0.049.
//
// Exchange entries (k1, j) lie at k1 * (P2 | 1) + j: the odd pitch keeps both
// the lines of consecutive j and the columns of consecutive k1 on distinct
// banks.
#pragma once
#include "bc_pass16.cuh"

namespace bc {

// DFT of N1 x N2 points, N1 and N2 coprime, in registers, natural order in
// and out (Good's prime factor map: n = N2 n1 + N1 n2, k = e1 k1 + e2 k2 mod N
// with e1 = 1 mod N1, 0 mod N2 and e2 the other way round; no twiddles).
__host__ __device__ constexpr int crt_unit(int n1, int n2) {  // 1 mod n1, 0 mod n2
  for (int e = n2; e < n1 * n2; e += n2)
    if (e % n1 == 1) return e;
  return 0;
}
template <int N1, int N2, bool INV>
__device__ __forceinline__ void dft_coprime(double2 (&x)[N1 * N2]) {
  constexpr int N = N1 * N2, E1 = crt_unit(N1, N2), E2 = crt_unit(N2, N1);
  double2 y[N];
#pragma unroll
  for (int n2 = 0; n2 < N2; n2++) {
    double2 a[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) a[n1] = x[(N2 * n1 + N1 * n2) % N];
    dftR<N1, INV>(a);
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) y[k1 * N2 + n2] = a[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < N1; k1++) {
    double2 a[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) a[n2] = y[k1 * N2 + n2];
    dftR<N2, INV>(a);
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) x[(E1 * k1 + E2 * k2) % N] = a[k2];
  }
}
template <int N, bool INV>
__device__ __forceinline__ void dft_regs(double2 (&x)[N]) {
  if constexpr (N == 8) dft8<INV>(x);
  else if constexpr (N == 12) dft_coprime<3, 4, INV>(x);
  else if constexpr (N == 16) dft16<INV>(x);
  else if constexpr (N == 20) dft_coprime<5, 4, INV>(x);
  else if constexpr (N == 24) dft_coprime<3, 8, INV>(x);
  else dft32<INV>(x);
  static_assert(N == 8 || N == 12 || N == 16 || N == 20 || N == 24 || N == 32, "lengths in registers");
}

template <int L> struct Rows2 {
  static constexpr int P2 = L == 128 ? 8 : (L == 192 ? 12 : (L <= 384 ? 16 : 32));
  static constexpr int P1 = L / P2;
  static constexpr int TR = P1 > P2 ? P1 : P2;      // threads per row
  static constexpr int NR = L == 640 ? 4 : 8;       // rows per unit
  static constexpr int NT = NR * TR;
  static constexpr bool WARP = 32 % TR == 0;        // rows private to a warp
  static constexpr int PITCH = P2 | 1;
  static constexpr int ROW = (P1 * PITCH > L ? P1 * PITCH : L);  // entries of a row's buffer
  // ten or twelve warps per SM, at most 168 registers (640 and 768 points:
  // eight, 255); B's spectrum stays in registers where that leaves room, else
  // in B's buffer.  168 are too few for 384 points, which spill 228 bytes a
  // thread (squares 116); 192 points spill 32, the others nothing.
  static constexpr int MINB = L == 768 ? 1 : (L == 640 || NT != 128 ? 2 : 3);
  static constexpr bool PARK = L >= 320;
  static constexpr size_t SMEM = (size_t)(2 * NR * ROW + L) * 16;
  static_assert(NT % 32 == 0, "whole warps");
};

template <int L, bool SQ>
__global__ void __launch_bounds__(Rows2<L>::NT, Rows2<L>::MINB)
    k5_rows(ClassParams p, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap) {
  using T = Rows2<L>;
  constexpr int P1 = T::P1, P2 = T::P2, TR = T::TR, NR = T::NR, NT = T::NT, PITCH = T::PITCH, ROW = T::ROW;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ uint64_t bars[2];
  double2 *const twS = reinterpret_cast<double2 *>(smraw);  // twS[k1*P2 + j] = e^{-2 pi i j k1/L}
  double2 *const bufA = twS + L, *const bufB = bufA + NR * ROW;
  const int tid = threadIdx.x, rl = tid / TR, u = tid % TR;
#pragma unroll
  for (int q = 0; q < (L + NT - 1) / NT; q++) {
    const int i = tid + q * NT, m = (i / P2) * (i % P2);  // below L
    if (i < L) twS[i] = __ldg(&p.twLr[m]);
  }
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  const FastDiv fd_rows = p.fd_rows;
  const unsigned rows_item = fd_rows.d;
  const unsigned total = (unsigned)p.nitems * rows_item / NR;  // units of the class; NR divides rows_item
  auto row_base = [&](unsigned row, bool opB) -> double2 * {
    const unsigned item = fd_rows.div(row);
    const ItemDesc &it = p.items[item];
    return (opB ? it.bufB : it.bufA) + (size_t)(row - item * rows_item) * L;
  };
  // thread 0, after a barrier behind the buffer's last use: a unit's NR rows
  // (neighbours in memory), each to its own place
  auto fetch = [&](double2 *dst, uint64_t *bar, unsigned un, bool opB) {
    fence_proxy_async_smem();
    mbar_expect_tx(bar, NR * L * 16);
    const double2 *src = row_base(un * NR, opB);
#pragma unroll
    for (int r = 0; r < NR; r++) bulk_load(dst + r * ROW, src + r * L, L * 16, bar);
  };
  auto sync = [] {
    if (T::WARP) __syncwarp();
    else __syncthreads();
  };
  // the threads beyond a stage's count do its last thread's work again and
  // store nothing (a branch around it would keep both sides' registers)
  const bool jt = u < P2, kt = u < P1;
  const int uj = jt ? u : P2 - 1, uk = kt ? u : P1 - 1;
  // forward transform of this thread's row, whose points lie in b[0..L)
  auto forward = [&](double2 (&w)[P2], double2 *b) {
    double2 v[P1];
#pragma unroll
    for (int i = 0; i < P1; i++) v[i] = b[uj + P2 * i];
    sync();  // the points are read: b serves the exchange
    dft_regs<P1, false>(v);
#pragma unroll
    for (int k1 = 1; k1 < P1; k1++) v[k1] = cmul(v[k1], twS[k1 * P2 + uj]);
    if (jt) {
#pragma unroll
      for (int k1 = 0; k1 < P1; k1++) b[k1 * PITCH + u] = v[k1];
    }
    sync();
#pragma unroll
    for (int j = 0; j < P2; j++) w[j] = b[uk * PITCH + j];
    dft_regs<P2, false>(w);
  };
  unsigned un = blockIdx.x;
  if (tid == 0 && un < total) {
    if (!SQ) fetch(bufB, &bars[1], un, true);
    fetch(bufA, &bars[0], un, false);
  }
  unsigned par = 0;
  double2 *const ra = bufA + rl * ROW, *const rb = bufB + rl * ROW;
  for (; un < total; un += gridDim.x, par ^= 1u) {
    const bool more = un + gridDim.x < total;
    bool bad = false;
    double2 sb[P2], w[P2];
    if (!SQ) {
      bad = !mbar_wait(&bars[1], par);
      forward(sb, rb);
      if (T::PARK) {  // in place of the exchange entries it came from, read back by this thread only
        if (kt) {
#pragma unroll
          for (int j = 0; j < P2; j++) rb[u * PITCH + j] = sb[j];
        }
      } else {
        __syncthreads();  // every row is done with B's buffer
        if (more && tid == 0) fetch(bufB, &bars[1], un + gridDim.x, true);
      }
    }
    bad |= !mbar_wait(&bars[0], par);
    forward(w, ra);
#pragma unroll
    for (int j = 0; j < P2; j++) {
      if (!SQ && T::PARK) sb[j] = rb[uk * PITCH + j];
      w[j] = SQ ? cmul(w[j], w[j]) : cmul(w[j], sb[j]);
    }
    dft_regs<P2, true>(w);
    sync();  // the forward exchange is read
    if (kt) {
#pragma unroll
      for (int j = 0; j < P2; j++) ra[u * PITCH + j] = w[j];
    }
    sync();
    double2 v[P1];
#pragma unroll
    for (int k1 = 0; k1 < P1; k1++) v[k1] = k1 ? cmulc(ra[k1 * PITCH + uj], twS[k1 * P2 + uj]) : ra[uj];
    const unsigned row0 = un * NR;
    if (__syncthreads_or(bad)) {
      // a wait gave up: flag the item, issue nothing more, let the copies in
      // flight land, leave
      if (tid == 0) {
        atomicOr(p.items[fd_rows.div(row0)].flags, FLAG_TIMEOUT);
        mbar_drain(&bars[0], par);
        if (!SQ) {
          mbar_drain(&bars[1], par);
          if (more && !T::PARK) mbar_drain(&bars[1], par ^ 1u);
        }
      }
      return;
    }
    if (more && tid == 0) {
      fetch(bufA, &bars[0], un + gridDim.x, false);
      if (!SQ && T::PARK) fetch(bufB, &bars[1], un + gridDim.x, true);
    }
    dft_regs<P1, true>(v);
    if (jt) {
      double2 *const out = row_base(row0, false) + rl * L;
#pragma unroll
      for (int i = 0; i < P1; i++) out[u + P2 * i] = v[i];
    }
  }
}

}  // namespace bc
