// Philox4x32-10 with its per-seed, per-ordinal and per-shot work hoisted.
#pragma once
#include "common.cuh"

namespace sdim {

// Philox4x32-10 (the function of philox4x32_10) with its round keys
// precomputed from the seed.  In a phase-pass warp the seed is uniform, so
// the keys sit in uniform registers and each round is two 32x32->64
// multiplies and two three-input xors.
struct PhiloxKeys {
  uint32_t k0[10], k1[10];
  __device__ explicit PhiloxKeys(unsigned long long seed) {
    uint32_t a = (uint32_t)seed, b = (uint32_t)(seed >> 32);
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      k0[r] = a;
      k1[r] = b;
      a += 0x9E3779B9u;
      b += 0xBB67AE85u;
    }
  }
  __device__ __forceinline__ uint4 block(uint4 c) const {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      unsigned long long p0, p1;  // one 32x32->64 multiply each
      asm("mul.wide.u32 %0, %1, %2;" : "=l"(p0) : "r"(c.x), "r"(0xD2511F53u));
      asm("mul.wide.u32 %0, %1, %2;" : "=l"(p1) : "r"(c.z), "r"(0xCD9E8D57u));
      c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ k0[r], (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ k1[r],
                     (uint32_t)p0);
    }
    return c;
  }
};

// Philox rounds shared between many (ordinal, shot) pairs.
// With the counter (ordinal, shot_lo, shot_hi, domain) the first round's
// multiplies see the ordinal and shot_hi alone, the second's the shot alone and
// the ordinal alone, and one of the third's the ordinal alone: five of a
// block's twenty multiplies, which are what bounds the pass.  They are made
// once per ordinal (CoinOrdinal, in shared memory) and once per shot.
struct CoinOrdinal {
  uint32_t c3;      // what the ordinal adds to c2 of round 3
  uint32_t r0, r2;  // what it adds to round 3's first and third word
  uint32_t r3;      // round 3's fourth word
};
__device__ __forceinline__ CoinOrdinal coin_ordinal(const PhiloxKeys& K, uint32_t ord, uint32_t shot_hi, uint32_t domain) {
  const uint32_t kM0 = 0xD2511F53u, kM1 = 0xCD9E8D57u;
  const uint32_t c2 = __umulhi(kM0, ord) ^ domain ^ K.k1[0];           // round 1
  const uint32_t c0 = __umulhi(kM1, c2) ^ (kM1 * shot_hi) ^ K.k0[1];   // round 2
  CoinOrdinal o;
  o.c3 = (kM0 * ord) ^ K.k1[1];
  o.r0 = (kM1 * c2) ^ K.k0[2];
  o.r2 = __umulhi(kM0, c0) ^ K.k1[2];
  o.r3 = kM0 * c0;
  return o;
}
// The shot's part: (hi, lo) of round 2's product.
__device__ __forceinline__ uint2 coin_shot(const PhiloxKeys& K, uint32_t shot_lo, uint32_t shot_hi) {
  const uint32_t c0 = __umulhi(0xCD9E8D57u, shot_hi) ^ shot_lo ^ K.k0[0];
  return make_uint2(__umulhi(0xD2511F53u, c0), 0xD2511F53u * c0);
}
// Block (ordinal, shot): rounds 3 (one multiply) to 10.
__device__ __forceinline__ uint4 coin_block(const PhiloxKeys& K, const CoinOrdinal& o, uint2 sh) {
  unsigned long long p0, p1;
  asm("mul.wide.u32 %0, %1, %2;" : "=l"(p1) : "r"(sh.x ^ o.c3), "r"(0xCD9E8D57u));
  uint4 c = make_uint4((uint32_t)(p1 >> 32) ^ o.r0, (uint32_t)p1, o.r2 ^ sh.y, o.r3);
#pragma unroll
  for (int r = 3; r < 10; ++r) {
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(p0) : "r"(c.x), "r"(0xD2511F53u));
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(p1) : "r"(c.z), "r"(0xCD9E8D57u));
    c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ K.k0[r], (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ K.k1[r],
                   (uint32_t)p0);
  }
  return c;
}

}  // namespace sdim
