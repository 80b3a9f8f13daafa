// bc_bsr.cuh — device kernels of the binary-splitting sum for e.
//
// The reference builds P(a,b), Q(a,b) with P/Q = sum_{j=a+1}^{b} 1/((a+1)(a+2)..j)
// and Q = (a+1)(a+2)..b by recursion on the host (main.c:63-109): leaves
// P = 1, Q = b, and P = P0*Q1 + P1, Q = Q0*Q1 at each node.  These integers
// do not depend on where the range is split, so the device version uses its
// own tree: leaves of up to 1024 consecutive terms computed one per warp
// (P(a,k+1) = P(a,k)*(k+1) + 1, Q(a,k+1) = Q(a,k)*(k+1)), then levels that
// pair neighbouring nodes, with both products of a level in one batched FFT
// multiply and the additions in k_add below.
#pragma once
#include <cuda/atomic>

#include "bc_kernels.cuh"
#include "bc_lanes.cuh"

namespace bc {

// Wide leaves, one warp each: up to WLEAF_CAP limbs per value, lane l holding
// limbs [32l, 32l+32) in registers.  Per term k both values are multiplied
// by k (P also gets +1 at limb 0; bc_lanes.cuh).  A carry out of the top lane
// means the leaf was too wide for the capacity: flagged, never written past
// the buffer.  1,661 leaves of 1,024 terms: 1.80 -> 0.61 ms.
constexpr int WLEAF_LPL = LANE_LIMBS;            // limbs per lane
constexpr int WLEAF_CAP = 32 * WLEAF_LPL;        // limbs per value
constexpr int WLEAF_STRIDE = WLEAF_CAP + 2;      // limbs per stored value
constexpr int WLEAF_WARPS = 4;                   // warps per CTA

// Leaf j covers terms (a + j*T, min(b, a + (j+1)*T)]; values go to
// out + (2j)*WLEAF_STRIDE (P) and out + (2j+1)*WLEAF_STRIDE (Q), lengths to
// len[2j], len[2j+1]; flags bit 0 on a capacity overflow.
__global__ void __launch_bounds__(32 * WLEAF_WARPS) k_bsr_leaves_wide(uint32_t a, uint32_t b, uint32_t T,
                                                                     uint32_t nleaf, uint32_t *out, uint32_t *len,
                                                                     unsigned *flags) {
  const int lane = threadIdx.x & 31;
  const uint32_t j = blockIdx.x * WLEAF_WARPS + (threadIdx.x >> 5);
  if (j >= nleaf) return;  // whole warps leave together
  const uint32_t a0 = a + j * T;
  const uint32_t b0 = min(b, a0 + T);
  uint32_t P[WLEAF_LPL], Q[WLEAF_LPL];
#pragma unroll
  for (int q = 0; q < WLEAF_LPL; q++) P[q] = Q[q] = 0;
  if (lane == 0) {
    P[0] = 1;
    Q[0] = a0 + 1;
  }
  unsigned ovf = 0;
  for (uint32_t k = a0 + 2; k <= b0; k++) {
    const uint32_t cp = warp_mul_word(P, k, 1u, lane), cq = warp_mul_word(Q, k, 0u, lane);
    if (lane == 31) ovf |= cp | cq;
  }
  // lengths: highest nonzero limb + 1
  int hp = -1, hq = -1;
#pragma unroll
  for (int q = 0; q < WLEAF_LPL; q++) {
    if (P[q]) hp = lane * WLEAF_LPL + q;
    if (Q[q]) hq = lane * WLEAF_LPL + q;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    hp = max(hp, __shfl_xor_sync(~0u, hp, o));
    hq = max(hq, __shfl_xor_sync(~0u, hq, o));
  }
  uint32_t *oP = out + (size_t)(2 * j) * WLEAF_STRIDE, *oQ = oP + WLEAF_STRIDE;
#pragma unroll
  for (int q = 0; q < WLEAF_LPL; q++) {
    const int i = lane * WLEAF_LPL + q;
    if (i <= hp) oP[i] = P[q];
    if (i <= hq) oQ[i] = Q[q];
  }
  if (lane == 0) {
    len[2 * j] = (uint32_t)(hp + 1);
    len[2 * j + 1] = (uint32_t)(hq + 1);
  }
  if (__any_sync(~0u, ovf != 0) && lane == 0) atomicOr(flags, 1u);
}

// R = X + Y for a batch of items: n = max(lx, ly) limbs of sum, then the
// carry out as limb n (len = n + carry).  X is a product of lx limbs whose
// operands had nonzero top limbs, so its top limb alone may be zero: the
// kernel takes lx - 1 then, and it also gives the significant length of a
// second product q of ql limbs (the lengths would otherwise be a kernel and a
// trip to the host of their own per tree level).  An item has max(lx, ly) /
// ADD_TILE + 1 tiles of ADD_TILE limbs (the one that holds limb n is among
// them; one beyond it may stay empty); the carry into a tile is found by a
// decoupled lookback over the tiles of the item, with the carry maps {0,1} ->
// {0,1} kept in the {-1,0,1} map encoding of the multiply's carry scan
// (fn_make / fn_compose).  A status word carries all that it says, so it needs
// no ordering of other memory.
constexpr int ADD_NT = 256, ADD_PT = 8, ADD_TILE = ADD_NT * ADD_PT;

struct AddDesc {
  const uint32_t *x;
  const uint32_t *y;
  uint32_t *r;
  const uint32_t *q;
  unsigned long long lx, ly, ql;
  unsigned long long tile0;  // first tile of this item (batch-wide numbering)
};

// Limbs of a product of CL limbs without its top limb if that is zero.
__device__ __forceinline__ unsigned long long product_len(const uint32_t *C, unsigned long long CL) {
  return CL - (CL > 1 && C[CL - 1] == 0 ? 1 : 0);
}

struct AddParams {
  const AddDesc *items;
  int nitems;
  unsigned long long tiles;
  unsigned int *counter;       // zeroed before launch
  uint32_t *status;            // one word per tile, zeroed before launch
  unsigned long long *len;     // per item: n + carry out, length of q
  unsigned int *flags;         // bit 0: a lookback wait ran out
};

__global__ void __launch_bounds__(ADD_NT) k_add(AddParams p) {
  __shared__ uint32_t sw[65];
  __shared__ unsigned long long s_unit;
  __shared__ int s_cin;
  const int tid = threadIdx.x;
  for (;;) {
    if (tid == 0) s_unit = atomicAdd(p.counter, 1u);
    __syncthreads();
    const unsigned long long unit = s_unit;
    if (unit >= p.tiles) break;
    int lo = 0, hi = p.nitems - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (p.items[mid].tile0 <= unit) lo = mid; else hi = mid - 1;
    }
    const AddDesc &it = p.items[lo];
    const unsigned long long tile = unit - it.tile0;
    const unsigned long long lx = product_len(it.x, it.lx), n = lx > it.ly ? lx : it.ly;
    if (tile == 0 && tid == 0) p.len[2 * lo + 1] = product_len(it.q, it.ql);
    const unsigned long long i0 = tile * ADD_TILE + (unsigned long long)tid * ADD_PT;
    uint32_t s[ADD_PT];
    unsigned c = 0;
    bool ones = true;
#pragma unroll
    for (int q = 0; q < ADD_PT; q++) {
      const unsigned long long i = i0 + q;
      const uint32_t xv = i < lx ? it.x[i] : 0u, yv = i < it.ly ? it.y[i] : 0u;
      const unsigned long long v = (unsigned long long)xv + yv + c;
      s[q] = (uint32_t)v;
      c = (unsigned)(v >> 32);
      if (i < n) ones = ones && s[q] == 0xffffffffu;
    }
    // carry out of this thread's limbs given its carry in: c, or c | ones
    const int c0 = (int)c, c1 = (int)(c | (ones ? 1u : 0u));
    const uint32_t f = fn_make(c0, c0, c1);
    uint32_t agg;
    const uint32_t ex = block_scan_fn<ADD_NT>(f, sw, &agg);
    if (tid == 0) {
      cuda::atomic_ref<uint32_t, cuda::thread_scope_device> me(p.status[it.tile0 + tile]);
      int cin = 0;
      if (tile == 0) {
        me.store(ST_INC | (uint32_t)(fn_apply(agg, 0) + 1), cuda::memory_order_relaxed);
      } else {
        if (fn_is_const(agg)) me.store(ST_INC | (uint32_t)(fn_apply(agg, 0) + 1), cuda::memory_order_relaxed);
        else me.store(ST_AGG | agg, cuda::memory_order_relaxed);
        uint32_t acc = FN_ID;
        long long prev = (long long)tile - 1;
        int spins = 0;
        bool timed_out = false;
        for (;;) {
          cuda::atomic_ref<uint32_t, cuda::thread_scope_device> st(p.status[it.tile0 + prev]);
          const uint32_t v = st.load(cuda::memory_order_relaxed);
          if (v & ST_INC) {
            cin = fn_apply(acc, (int)(v & 3u) - 1);
            break;
          } else if (v & ST_AGG) {
            const uint32_t fv = v & 0x3fu;
            if (fn_is_const(fv)) { cin = fn_apply(acc, fn_apply(fv, 0)); break; }
            acc = fn_compose(fv, acc);
            prev--;
          } else {
            if (++spins > LOOKBACK_SPINS) { timed_out = true; break; }
            if (spins > 64) __nanosleep(32);
          }
        }
        if (timed_out) {
          atomicOr(p.flags, 1u);
          cin = 0;
        }
        if (!fn_is_const(agg)) me.store(ST_INC | (uint32_t)(fn_apply(agg, cin) + 1), cuda::memory_order_relaxed);
      }
      s_cin = cin;
    }
    __syncthreads();
    unsigned cc = (unsigned)fn_apply(ex, s_cin);  // carry into this thread's limbs
    uint32_t top = 0;
    bool has_top = false;
#pragma unroll
    for (int q = 0; q < ADD_PT; q++) {
      const unsigned long long i = i0 + q;
      const unsigned long long v = (unsigned long long)s[q] + cc;
      cc = (unsigned)(v >> 32);
      if (i < n) it.r[i] = (uint32_t)v;
      else if (i == n) { top = (uint32_t)v; has_top = true; }
    }
    // limb n (inside the item's last tile) is the carry out of limb n-1
    if (has_top) {
      it.r[n] = top;
      p.len[2 * lo] = n + top;
    }
    __syncthreads();
  }
}

}  // namespace bc
