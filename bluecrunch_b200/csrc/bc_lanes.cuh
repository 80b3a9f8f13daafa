// bc_lanes.cuh — a long integer spread over a warp, 32 limbs per lane in
// registers (lane l holds limbs 32 l .. 32 l + 31), times one word.
//
// What bounds it: latency, one warp per number.  The 32 products of a lane are
// independent; only the carries are a chain, so they are added in one chain of
// 32-bit add-with-carry instructions, and a lane's carry word goes only into
// the next lane's lowest limb (a carry out of that limb, one in 2^32, ripples
// in a loop that the warp else skips).  Multiplying limb after limb with the
// carry in each product's addend, and then adding the carry word through all
// 32 limbs, took 1,500 cycles a word; this takes some 300.
#pragma once
#include <cstdint>

namespace bc {

constexpr int LANE_LIMBS = 32;

// r[0..7] = t[0..7] + h[0..7] + c (c 0 or 1); returns the carry out.
__device__ __forceinline__ uint32_t add8(uint32_t *r, const uint32_t *t, const uint32_t *h, uint32_t c) {
  uint32_t o;
  asm("{\n\t.reg .u32 z;\n\t"
      "add.cc.u32 z, %25, 0xffffffff;\n\t"  // the carry flag from c
      "addc.cc.u32 %0, %9, %17;\n\t"
      "addc.cc.u32 %1, %10, %18;\n\t"
      "addc.cc.u32 %2, %11, %19;\n\t"
      "addc.cc.u32 %3, %12, %20;\n\t"
      "addc.cc.u32 %4, %13, %21;\n\t"
      "addc.cc.u32 %5, %14, %22;\n\t"
      "addc.cc.u32 %6, %15, %23;\n\t"
      "addc.cc.u32 %7, %16, %24;\n\t"
      "addc.u32 %8, 0, 0;\n\t}"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]),
        "=&r"(o)
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]), "r"(h[0]), "r"(h[1]),
        "r"(h[2]), "r"(h[3]), "r"(h[4]), "r"(h[5]), "r"(h[6]), "r"(h[7]), "r"(c));
  return o;
}

// The number times k, plus add (below 2^32) at limb 0.  Returns the carry
// word out of lane 31 (the value of the other lanes' return is no use).
__device__ __forceinline__ uint32_t warp_mul_word(uint32_t (&x)[LANE_LIMBS], uint32_t k, uint32_t add, int lane) {
  uint32_t t[LANE_LIMBS], h[LANE_LIMBS];  // h[q]: the high word that is added at limb q
  h[0] = 0;
  uint32_t out = 0;
#pragma unroll
  for (int q = 0; q < LANE_LIMBS; q++) {
    const unsigned long long v = (unsigned long long)x[q] * k;
    t[q] = (uint32_t)v;
    if (q + 1 < LANE_LIMBS) h[q + 1] = (uint32_t)(v >> 32);
    else out = (uint32_t)(v >> 32);
  }
  uint32_t c = 0;
#pragma unroll
  for (int q = 0; q < LANE_LIMBS; q += 8) c = add8(x + q, t + q, h + q, c);
  out += c;  // a product's high word is at most 2^32 - 2
  uint32_t cin = __shfl_up_sync(~0u, out, 1);
  if (lane == 0) cin = add;
  x[0] += cin;
  uint32_t o = x[0] < cin ? 1u : 0u;
  for (int round = 0; round < 32 && __any_sync(~0u, o != 0); round++) {  // rare
#pragma unroll
    for (int q = 1; q < LANE_LIMBS; q++) {
      x[q] += o;
      o = x[q] < o ? 1u : 0u;
    }
    if (lane == 31) out += o;
    o = __shfl_up_sync(~0u, o, 1);
    if (lane == 0) o = 0;
    x[0] += o;
    o = x[0] < o ? 1u : 0u;
  }
  return out;
}

}  // namespace bc
