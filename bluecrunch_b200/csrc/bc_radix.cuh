// bc_radix.cuh — leaves of the binary-to-decimal conversion on the GPU.
//
// A leaf turns a fraction y (len limbs below the point, base 2^32) into k
// base-10^9 digits by k rounds of "multiply by 10^9, take the limb that
// crosses the point", on a window of limbs that drops the low limbs which can
// no longer reach the digit (the reference's convert_trunc,
// bigfloat/radix.c:41-91).  In absolute limb positions (limb len is an extra
// zero), round i works on [lo_i, hi_i): lo_1 = 0, hi_1 = len + 1, and
// lo_i = floor(alpha*(i-1)), hi_i = n + 1 for i >= 2, with alpha =
// log(10^9)/log(2^32) as the caller computes it.  Before the multiply the
// window's top limb is zero; the carry out of the window is dropped; the
// digit is limb n after the multiply and lands in s[k - i].
//
// One warp per leaf, RS limbs per lane in registers, laid out so that limb n
// is the last limb of lane 31 (lane l holds limbs base + l*RS ... base +
// (l+1)*RS - 1, base = n + 1 - 32*RS): the digit is then one fixed register,
// and the window's top limb, which enters each round after the first as
// zero, is that same register.  Limbs above n are not held: carries only move
// up, so they never reach limb n (in the first round the window reaches limb
// len >= n, but what it computes above n is dropped with the carry out).
//
// What bounds it: the instructions of one round after the other, some hundreds
// of rounds, with about one warp per scheduler when leaves are few.  So no
// round has a carry chain: limb q holds s_q < 2^33, its low word plus the high
// word of the limb below, and the next round multiplies that (33 x 30 bits fit
// 64); a lane's last limb keeps 32 bits and hands bit 32 on with its high
// word.  Exact values are needed in two places only.  The digit: limb n plus
// the carry out of limb n - 1, known from that limb's bit 32 unless its low
// word is all ones (then, one round in 2^32, every carry is resolved).  And a
// limb that the window's low end passes (at most one a round, alpha < 1; the
// same register for every lane): nothing lies below it, so its bit 32 is the
// carry that it hands to the next limb before it is cleared.  (A larger alpha
// passes several limbs a round, one after the other; the window is empty above
// limb n and the loop ends there, so a leaf never takes more than n + 1 of
// these steps.  Stopping it by a minimum with n + 1 cost 40 of 360 us for 512
// leaves, by this condition 2.)  512 leaves of
// 830 digits: 0.40 ms, 16,384 of them 4.8 ms; with a carry chain through every
// limb and round 0.47 ms for the former at best, with the clearing by a mask
// over the registers 0.56, on four warps each (eight limbs per lane, a barrier
// per round) 0.41 and 8.2 ms.
#pragma once
#include <cstdint>

namespace bc {

constexpr int RS = 32;                   // limbs per lane
constexpr int RADIX_WINDOW = 32 * RS;    // limbs a leaf window may span
constexpr int RADIX_WARPS = 4;           // warps per CTA
constexpr uint32_t DEC_BASE = 1000000000u;

struct RadixLeaf {
  const uint32_t *y;   // device: len limbs of the fraction
  uint32_t *s;         // device: k digits
  uint32_t len, n, k, pad;
};

// All carries of a leaf's limbs: every s_q below 2^32 but lane 31's last one
// (limb n).  Bounded: a carry passes at most 32 lanes.
__device__ __forceinline__ void radix_resolve(unsigned long long (&s)[RS], int lane) {
  unsigned long long c = 0;
  for (int round = 0; round <= 32; round++) {
#pragma unroll
    for (int q = 0; q < RS; q++) {
      s[q] += c;
      c = 0;
      if (q + 1 < RS || lane != 31) {
        c = s[q] >> 32;
        s[q] &= 0xffffffffull;
      }
    }
    c = __shfl_up_sync(~0u, (uint32_t)c, 1);
    if (lane == 0) c = 0;
    if (!__any_sync(~0u, c != 0)) break;
  }
}

// Limb q of a lane leaves the window: its carry to the limb above (a lane's
// last limb has 32 bits), then zero.  By a switch over the registers: an index
// would put them in local memory.
template <int q>
__device__ __forceinline__ void radix_drop(unsigned long long (&s)[RS], bool mine) {
  if (mine) {
    if constexpr (q + 1 < RS) s[q + 1] += s[q] >> 32;
    s[q] = 0;
  }
}

__global__ void __launch_bounds__(32 * RADIX_WARPS, 2) k_radix_leaves(const RadixLeaf *leaves, int count, double alpha,
                                                                    unsigned *flags) {
  __shared__ uint32_t stage[RADIX_WARPS][RADIX_WINDOW + RADIX_WINDOW / 32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  uint32_t *sm = stage[wib];
  const int warps = gridDim.x * RADIX_WARPS;
  for (int li = blockIdx.x * RADIX_WARPS + wib; li < count; li += warps) {
    const RadixLeaf lf = leaves[li];
    const uint32_t L = lf.len + 1;
    if (L > (uint32_t)RADIX_WINDOW || lf.n + 1 > (uint32_t)RADIX_WINDOW || lf.n + 1 > L + 1) {
      if (lane == 0) atomicOr(flags, 1u);
      continue;
    }
    // limb j sits at index j - base (base = n + 1 - RADIX_WINDOW <= 0): a
    // coalesced load into shared memory (one pad word per 32), then each lane
    // takes its RS consecutive indices
    const int base = (int)lf.n + 1 - RADIX_WINDOW;
    for (int t = lane; t < RADIX_WINDOW; t += 32) {
      const int j = t + base;
      sm[t + (t >> 5)] = (j >= 0 && j < (int)lf.len) ? lf.y[j] : 0u;
    }
    __syncwarp();
    unsigned long long x[RS];  // s_q
#pragma unroll
    for (int q = 0; q < RS; q++) {
      const int t = lane * RS + q;
      x[q] = sm[t + (t >> 5)];
    }
    __syncwarp();
    int lo = 0;    // low end of the round's window
    int ends = 0;  // floor(alpha (i - 1)) of 32 rounds i, one per lane
    for (uint32_t i = 1; i <= lf.k; i++) {
      // limbs that have just left the window (limbs below base are not held)
      if (((i - 1) & 31) == 0) ends = (int)floor(alpha * (double)((i - 1) + (uint32_t)lane));
      const int lo_now = i == 1 ? 0 : __shfl_sync(~0u, ends, (int)((i - 1) & 31));
      for (; lo < lo_now && lo - base < RADIX_WINDOW; lo++) {  // up to limb n
        const int g = lo - base;
        const bool mine = lane == (g >> 5);
        switch (g & 31) {
#define RADIX_DROP(q) case q: radix_drop<q>(x, mine); break;
          RADIX_DROP(0) RADIX_DROP(1) RADIX_DROP(2) RADIX_DROP(3) RADIX_DROP(4) RADIX_DROP(5) RADIX_DROP(6)
          RADIX_DROP(7) RADIX_DROP(8) RADIX_DROP(9) RADIX_DROP(10) RADIX_DROP(11) RADIX_DROP(12) RADIX_DROP(13)
          RADIX_DROP(14) RADIX_DROP(15) RADIX_DROP(16) RADIX_DROP(17) RADIX_DROP(18) RADIX_DROP(19) RADIX_DROP(20)
          RADIX_DROP(21) RADIX_DROP(22) RADIX_DROP(23) RADIX_DROP(24) RADIX_DROP(25) RADIX_DROP(26) RADIX_DROP(27)
          RADIX_DROP(28) RADIX_DROP(29) RADIX_DROP(30) RADIX_DROP(31)
#undef RADIX_DROP
        }
      }
      // multiply the window [lo, n] by 10^9
      uint32_t h = 0;  // high word of the limb below
#pragma unroll
      for (int q = 0; q < RS; q++) {
        const unsigned long long v = (unsigned long long)(uint32_t)x[q] * DEC_BASE;
        const uint32_t hi = (uint32_t)(v >> 32) + (uint32_t)(x[q] >> 32) * DEC_BASE;
        x[q] = (unsigned long long)(uint32_t)v + h;
        h = hi;
      }
      if (lane != 31) {  // limb n's high word is dropped
        h += (uint32_t)(x[RS - 1] >> 32);
        x[RS - 1] &= 0xffffffffull;
      }
      const uint32_t up = __shfl_up_sync(~0u, h, 1);
      if (lane != 0) x[0] += up;
      if (__any_sync(~0u, lane == 31 && (uint32_t)x[RS - 2] == 0xffffffffu)) radix_resolve(x, lane);
      // the digit: limb n with the carry out of the limb below, which then
      // holds 32 bits
      if (lane == 31) {
        lf.s[lf.k - i] = (uint32_t)(x[RS - 1] + (x[RS - 2] >> 32));
        x[RS - 2] &= 0xffffffffull;
        x[RS - 1] = 0;  // the window's top limb enters the next round as zero
      }
    }
  }
}

// ------------------------------------------------------------------ merges
// An internal node's digits from its children's (the reference's merge,
// bigfloat/radix.c:277-316): if the high part's lowest digit is 10^9 - 1 and
// the low part's top digit is 0, add 1 to the high part (base 10^9, carry
// past its top dropped); then the low kl digits are the low part's, or zero
// when the high part's lowest digit is 0 and the low part's top digit is
// 10^9 - 1; above them come the high part's digits from its second on.  No
// other carry can arise: the sum in the reference adds the low part into
// zeros.
struct MergeDesc {
  uint32_t *sh;        // kh digits of the high child (fixed in place)
  const uint32_t *sl;  // kl digits of the low child
  uint32_t *s;         // kh - 1 + kl digits of the node
  unsigned long long kh, kl;
  unsigned long long off;  // first copy unit of this node (batch-wide numbering)
};

// One thread per node: the +1 fix-up and the low-part decision (flag[i]).
__global__ void k_merge_fix(MergeDesc *d, int n, unsigned *flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  MergeDesc m = d[i];
  if (m.sh[0] == DEC_BASE - 1 && m.sl[m.kl - 1] == 0) {
    unsigned long long carry = 1;
    for (unsigned long long q = 0; q < m.kh && carry; q++) {
      const unsigned long long v = (unsigned long long)m.sh[q] + carry;
      carry = v / DEC_BASE;
      m.sh[q] = (uint32_t)(v % DEC_BASE);
    }
  }
  flag[i] = (m.sh[0] == 0 && m.sl[m.kl - 1] == DEC_BASE - 1) ? 1u : 0u;
}

// The copies, MERGE_UNIT digits per unit, units of all nodes in one grid.  A
// depth of 400,000 digits in units of 4096 kept 98 CTAs with 16 rounds each
// busy for 12 us; in units of 1024 it spreads over the SMs.
constexpr int MERGE_UNIT = 1024;
__global__ void k_merge_copy(const MergeDesc *d, int n, unsigned long long units, const unsigned *flag) {
  for (unsigned long long u = blockIdx.x; u < units; u += gridDim.x) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (d[mid].off <= u) lo = mid; else hi = mid - 1;
    }
    const MergeDesc &m = d[lo];
    const bool zero_low = flag[lo] != 0;
    const unsigned long long len = m.kh - 1 + m.kl;
    const unsigned long long i0 = (u - m.off) * MERGE_UNIT;
    for (unsigned long long i = i0 + threadIdx.x; i < i0 + MERGE_UNIT && i < len; i += blockDim.x)
      m.s[i] = i < m.kl ? (zero_low ? 0u : m.sl[i]) : m.sh[i - m.kl + 1];
  }
}

}  // namespace bc
