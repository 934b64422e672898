// Records of a 32-shot group from bits to bytes.
#pragma once
#include "common.cuh"

namespace sdim {

// Four bytes from four bits: byte i = bit i.
__device__ __forceinline__ uint32_t spread4(uint32_t bits) { return (bits * 0x00204081u) & 0x01010101u; }

// The group's records are one contiguous piece of the output, gout, rows x nm
// bytes: each lane cuts 16 of them at a time out of the bits, whatever rows
// they belong to, and stores them at once.  Plane p of shot s is the words
// bits[(32 p + s) S + w], bit k % 32 of word k / 32 = measurement k; det flags
// the deterministic measurements (bit 7 of a record byte).  Rows and det have
// a word to spare behind the last.
template <int PLANES>
__device__ __forceinline__ void store_records(uint8_t* __restrict__ gout, int rows, int nm, int lane,
                                              const uint32_t* bits, int S, const uint32_t* det) {
  const int total = rows * nm;
  const int head = min(total, (int)((0u - (uint32_t)reinterpret_cast<size_t>(gout)) & 15u));
  const int body = (total - head) & ~15, tail = total - head - body;
  if (lane < head + tail) {  // at most 30 bytes outside the 16-byte boundaries
    const int o = lane < head ? lane : body + lane, r = o / nm, k = o - r * nm, w = k >> 5;
    uint32_t v = (det[w] >> (k & 31)) << 7;
#pragma unroll
    for (int p = 0; p < PLANES; ++p) v |= ((bits[(32 * p + r) * S + w] >> (k & 31)) & 1u) << p;
    gout[o] = (uint8_t)v;
  }
  int r = (head + 16 * lane) / nm, k = head + 16 * lane - r * nm;
  const int dr = 512 / nm, dk = 512 - dr * nm;
  for (int o = 16 * lane; o < body; o += 512) {
    const int w = k >> 5;
    uint32_t d = __funnelshift_r(det[w], det[w + 1], k & 31), v[PLANES];
#pragma unroll
    for (int p = 0; p < PLANES; ++p) {
      const uint32_t* b = bits + (32 * p + r) * S + w;
      v[p] = __funnelshift_r(b[0], b[1], k & 31);
    }
    for (int at = nm - k, rr = r + 1; at < 16; at += nm, ++rr) {  // the next rows' first bits
      const uint32_t m = (1u << at) - 1u;
      d = (d & m) | (det[0] << at);
#pragma unroll
      for (int p = 0; p < PLANES; ++p) v[p] = (v[p] & m) | (bits[(32 * p + rr) * S] << at);
    }
    uint32_t q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      q[i] = spread4((d >> (4 * i)) & 15u) << 7;
#pragma unroll
      for (int p = 0; p < PLANES; ++p) q[i] |= spread4((v[p] >> (4 * i)) & 15u) << p;
    }
    *reinterpret_cast<uint4*>(gout + head + o) = make_uint4(q[0], q[1], q[2], q[3]);
    r += dr;
    k += dk;
    if (k >= nm) {
      k -= nm;
      ++r;
    }
  }
}

}  // namespace sdim
