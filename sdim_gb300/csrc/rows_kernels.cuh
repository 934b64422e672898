// Row form of the x / z pass (rows.cuh), device side: the raw, chain and extra
// passes.  Instantiated for d = 2, 3, 5 and 7 in k_rows_<d>.cu.
#pragma once
#include "follow.cuh"
#include "philox.cuh"
#include "planes3.cuh"
#include "record_out.cuh"
#include "rows.cuh"
#include "trace_split_u8.cuh"
#include "variants.cuh"

#include <type_traits>

namespace sdim {
namespace {

constexpr int L = kRowLanes;

// ---------------------------------------------------------------- elements
// T: the residues of 32 generators in bit planes (rows.cuh).  Every operation
// is a few three-input logic instructions for all 32.

__device__ __forceinline__ uint32_t mux(uint32_t m, uint32_t a, uint32_t b) { return (m & a) | (~m & b); }
__device__ __forceinline__ uint32_t maj(uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (a & c) | (b & c); }
// Bitwise function of three words by its truth table (bit 4 a + 2 b + c of F).
template <int F>
__device__ __forceinline__ uint32_t logic3(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(r) : "r"(a), "r"(b), "r"(c), "n"(F));
  return r;
}
__device__ __forceinline__ uint32_t lane_mask(bool b) { return b ? 0xffffffffu : 0u; }

// Three planes (d = 5, 7): bit 0 in x, bit 1 in y, bit 2 in z; w unused.
template <int D>
struct El {
  using T = uint4;
  static __device__ __forceinline__ T zero() { return make_uint4(0u, 0u, 0u, 0u); }
  // d = 7 keeps 0 as 000 or 111: a sum is a three-bit one with its carry added
  // back in, a negative the complement, twice a value its rotation
  static __device__ __forceinline__ uint32_t nzw(T a) {
    const uint32_t any = a.x | a.y | a.z;
    return D == 7 ? any & ~(a.x & a.y & a.z) : any;
  }
  static __device__ __forceinline__ T add(T a, T b) {
    const uint32_t s0 = a.x ^ b.x, c0 = a.x & b.x;
    const uint32_t s1 = a.y ^ b.y ^ c0, c1 = maj(a.y, b.y, c0);
    const uint32_t s2 = a.z ^ b.z ^ c1, c2 = maj(a.z, b.z, c1);
    if constexpr (D == 7) {
      const uint32_t k = s0 & c2;
      return make_uint4(s0 ^ c2, s1 ^ k, s2 ^ (s1 & k), 0u);
    } else {  // the sum is at most 8: subtract 5 from 5 on
      const uint32_t ge = c2 | (s2 & (s1 | s0));
      return make_uint4(s0 ^ ge, mux(ge, (s1 & s0) | c2, s1), s2 & ~ge, 0u);
    }
  }
  static __device__ __forceinline__ T neg(T a) {
    if constexpr (D == 7) return make_uint4(~a.x, ~a.y, ~a.z, 0u);
    return make_uint4(a.z | (a.y & ~a.x), a.y, a.x & ~a.y, 0u);
  }
  static __device__ __forceinline__ T dbl(T a) {
    if constexpr (D == 7) return make_uint4(a.z, a.x, a.y, 0u);
    return make_uint4((a.x & a.y) | a.z, (a.x & ~a.y) | a.z, a.y & ~a.x, 0u);
  }
  static __device__ __forceinline__ T mulc(T a, int c) {  // c uniform
    switch (c) {
      case 0: return zero();
      case 1: return a;
      case 2: return dbl(a);
      case 3: return D == 7 ? neg(dbl(dbl(a))) : neg(dbl(a));
      case 4: return D == 7 ? dbl(dbl(a)) : neg(a);
      case 5: return neg(dbl(a));
      default: return neg(a);
    }
  }
  // v + c f with c a lane's own
  static __device__ __forceinline__ T muladd(T v, T f, int c) {
    const uint32_t nz = lane_mask(c != 0);
    if constexpr (D == 7) {  // c = +- 2^k: 1 2 4 | 6 5 3
      const uint32_t m1 = lane_mask(c == 2 || c == 5), m2 = lane_mask(c == 4 || c == 3);
      const uint32_t mn = lane_mask(c == 3 || c >= 5);
      const uint32_t x = mux(m1, f.z, mux(m2, f.y, f.x)), y = mux(m1, f.x, mux(m2, f.z, f.y)),
                     z = mux(m1, f.y, mux(m2, f.x, f.z));
      return add(v, make_uint4((x ^ mn) & nz, (y ^ mn) & nz, (z ^ mn) & nz, 0u));
    } else {
      const uint32_t md = lane_mask(c == 2 || c == 3), mn = lane_mask(c >= 3);
      const T g = dbl(f);
      const T t = make_uint4(mux(md, g.x, f.x) & nz, mux(md, g.y, f.y) & nz, mux(md, g.z, f.z) & nz, 0u);
      const T u = neg(t);
      return add(v, make_uint4(mux(mn, u.x, t.x), t.y, mux(mn, u.z, t.z), 0u));
    }
  }
  // A sum under way, carries saved: the planes s and c (of the same weights)
  // count together.  d = 7 counts mod 7, d = 5 mod 15 in four planes, so that a
  // carry out of the last plane is one into the first, a negative is the
  // complement and twice a value its rotation: a term costs a full adder, two
  // instructions, per plane, where a whole addition mod d takes half as many
  // again (d = 7) to twice as many.
  struct Sum {
    static constexpr int P = D == 7 ? 3 : 4;
    uint32_t s[P], c[P];
    __device__ __forceinline__ explicit Sum(T v) {
      s[0] = v.x;
      s[1] = v.y;
      s[2] = v.z;
      if constexpr (P == 4) s[3] = 0u;
#pragma unroll
      for (int i = 0; i < P; ++i) c[i] = 0u;
    }
    // + C f, f = 0 for none
    template <int C>
    __device__ __forceinline__ void add(T f) {
      constexpr bool kNeg = C > D / 2;
      constexpr int A = kNeg ? D - C : C, R = D == 7 && A == 3 ? 2 : A - 1;  // 3 = -4 mod 7
      constexpr bool kInv = D == 7 && A == 3 ? !kNeg : kNeg;
      const uint32_t g[4] = {f.x, f.y, f.z, 0u};
      uint32_t m[P];
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const uint32_t a = kInv ? ~g[(i + P - R) % P] : g[(i + P - R) % P];
        m[i] = maj(s[i], c[i], a);
        s[i] ^= c[i] ^ a;
      }
#pragma unroll
      for (int i = 0; i < P; ++i) c[(i + 1) % P] = m[i];
    }
    __device__ __forceinline__ T value() const {
      if constexpr (D == 7) return El::add(make_uint4(s[0], s[1], s[2], 0u), make_uint4(c[0], c[1], c[2], 0u));
      uint32_t r[4], k = 0u;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        r[i] = s[i] ^ c[i % P] ^ k;
        k = maj(s[i], c[i % P], k);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // the carry back in
        const uint32_t t = r[i] & k;
        r[i] ^= k;
        k = t;
      }
      // 0 .. 15 mod 5: by the low three planes for either value of the high one
      return make_uint4(mux(r[3], logic3<0x29>(r[2], r[1], r[0]), logic3<0x4a>(r[2], r[1], r[0])),
                        mux(r[3], logic3<0x31>(r[2], r[1], r[0]), logic3<0x8c>(r[2], r[1], r[0])),
                        mux(r[3], logic3<0x42>(r[2], r[1], r[0]), logic3<0x10>(r[2], r[1], r[0])), 0u);
    }
  };
  static __device__ __forceinline__ int get(T a, int j) {
    const int v = (int)((a.x >> j) & 1u) | (int)(((a.y >> j) & 1u) << 1) | (int)(((a.z >> j) & 1u) << 2);
    return D == 7 && v == 7 ? 0 : v;
  }
  static __device__ __forceinline__ T set(T a, int j, int v) {
    const uint32_t m = ~(1u << j);
    return make_uint4((a.x & m) | ((uint32_t)(v & 1) << j), (a.y & m) | ((uint32_t)((v >> 1) & 1) << j),
                      (a.z & m) | ((uint32_t)(v >> 2) << j), 0u);
  }
  static __device__ __forceinline__ T pick(uint32_t m, T a, T b) {  // m ? a : b
    return make_uint4(mux(m, a.x, b.x), mux(m, a.y, b.y), mux(m, a.z, b.z), 0u);
  }
  // lanes m set to v
  static __device__ __forceinline__ T put_at(T a, uint32_t m, int v) {
    return make_uint4(mux(m, lane_mask(v & 1), a.x), mux(m, lane_mask(v & 2), a.y), mux(m, lane_mask(v & 4), a.z), 0u);
  }
  static __device__ __forceinline__ int dot(T a, T b) {  // sum of the products (d = 7: mod 7)
    const int p0 = __popc(a.x & b.x), p1 = __popc(a.x & b.y) + __popc(a.y & b.x);
    const int p2 = __popc(a.x & b.z) + __popc(a.y & b.y) + __popc(a.z & b.x);
    const int p3 = __popc(a.y & b.z) + __popc(a.z & b.y), p4 = __popc(a.z & b.z);
    return p0 + 2 * p1 + 4 * p2 + 8 * p3 + 16 * p4;
  }
  static __device__ __forceinline__ T shfl(T a, int l) {
    return make_uint4(__shfl_sync(0xffffffffu, a.x, l), __shfl_sync(0xffffffffu, a.y, l),
                      __shfl_sync(0xffffffffu, a.z, l), 0u);
  }
  static __device__ __forceinline__ T shfl_xor(T a, int o) {
    return make_uint4(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o),
                      __shfl_xor_sync(0xffffffffu, a.z, o), 0u);
  }
  static __device__ __forceinline__ void clear(T* p, int j) {
    atomicAnd(&p->x, ~(1u << j));
    atomicAnd(&p->y, ~(1u << j));
    atomicAnd(&p->z, ~(1u << j));
  }
  static __device__ __forceinline__ void put(T* p, int j, int v) {
    if (v & 1) atomicOr(&p->x, 1u << j);
    if (v & 2) atomicOr(&p->y, 1u << j);
    if (v & 4) atomicOr(&p->z, 1u << j);
  }
};

template <>
struct El<3> {  // two planes (planes3.cuh)
  using T = uint2;
  static __device__ __forceinline__ P3 p(T a) { return p3(a.x, a.y); }
  static __device__ __forceinline__ T t(P3 a) { return make_uint2(a.p0, a.p1); }
  static __device__ __forceinline__ T zero() { return make_uint2(0u, 0u); }
  static __device__ __forceinline__ uint32_t nzw(T a) { return a.x | a.y; }
  static __device__ __forceinline__ T add(T a, T b) { return t(p3_add(p(a), p(b))); }
  static __device__ __forceinline__ T neg(T a) { return make_uint2(a.y, a.x); }
  static __device__ __forceinline__ T mulc(T a, int c) { return c == 0 ? zero() : c == 1 ? a : neg(a); }
  static __device__ __forceinline__ T muladd(T v, T f, int c) {
    const uint32_t m1 = lane_mask(c == 1), m2 = lane_mask(c == 2);
    return add(v, make_uint2((f.x & m1) | (f.y & m2), (f.y & m1) | (f.x & m2)));
  }
  struct Sum {  // mod 3 in two planes, as El<D>::Sum
    uint32_t s[2], c[2];
    __device__ __forceinline__ explicit Sum(T v) : s{v.x, v.y}, c{0u, 0u} {}
    template <int C>
    __device__ __forceinline__ void add(T f) {
      const uint32_t a = C == 1 ? f.x : f.y, b = C == 1 ? f.y : f.x;
      const uint32_t m = maj(s[0], c[0], a), n = maj(s[1], c[1], b);
      s[0] ^= c[0] ^ a;
      s[1] ^= c[1] ^ b;
      c[0] = n;
      c[1] = m;
    }
    __device__ __forceinline__ T value() const {
      const uint32_t a = s[0] ^ c[0], k = s[0] & c[0], b = s[1] ^ c[1] ^ k, m = maj(s[1], c[1], k);
      const uint32_t x = a ^ m, y = b ^ (a & m);
      return make_uint2(x & ~y, y & ~x);  // 3 is 0
    }
  };
  static __device__ __forceinline__ int get(T a, int j) { return p3_get(p(a), j); }
  static __device__ __forceinline__ T set(T a, int j, int v) { return t(p3_set(p(a), j, v)); }
  static __device__ __forceinline__ T pick(uint32_t m, T a, T b) {
    return make_uint2(mux(m, a.x, b.x), mux(m, a.y, b.y));
  }
  static __device__ __forceinline__ T put_at(T a, uint32_t m, int v) {
    return make_uint2(mux(m, lane_mask(v == 1), a.x), mux(m, lane_mask(v == 2), a.y));
  }
  static __device__ __forceinline__ int dot(T a, T b) { return p3_rsum(p3_mul(p(a), p(b))); }
  static __device__ __forceinline__ T shfl(T a, int l) {
    return make_uint2(__shfl_sync(0xffffffffu, a.x, l), __shfl_sync(0xffffffffu, a.y, l));
  }
  static __device__ __forceinline__ T shfl_xor(T a, int o) {
    return make_uint2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
  }
  static __device__ __forceinline__ void clear(T* q, int j) {
    atomicAnd(&q->x, ~(1u << j));
    atomicAnd(&q->y, ~(1u << j));
  }
  static __device__ __forceinline__ void put(T* q, int j, int v) {
    if (v == 1) atomicOr(&q->x, 1u << j);
    if (v == 2) atomicOr(&q->y, 1u << j);
  }
};

template <>
struct El<2> {  // one plane
  using T = uint32_t;
  static __device__ __forceinline__ T zero() { return 0u; }
  static __device__ __forceinline__ uint32_t nzw(T a) { return a; }
  static __device__ __forceinline__ T add(T a, T b) { return a ^ b; }
  static __device__ __forceinline__ T neg(T a) { return a; }
  static __device__ __forceinline__ T mulc(T a, int c) { return c ? a : 0u; }
  static __device__ __forceinline__ T muladd(T v, T f, int c) { return v ^ (f & (0u - (uint32_t)c)); }
  static __device__ __forceinline__ int get(T a, int j) { return (int)((a >> j) & 1u); }
  static __device__ __forceinline__ T set(T a, int j, int v) { return (a & ~(1u << j)) | ((uint32_t)v << j); }
  static __device__ __forceinline__ T pick(uint32_t m, T a, T b) { return mux(m, a, b); }
  static __device__ __forceinline__ T put_at(T a, uint32_t m, int v) { return mux(m, lane_mask(v), a); }
  static __device__ __forceinline__ int dot(T a, T b) { return __popc(a & b); }
  static __device__ __forceinline__ T shfl(T a, int l) { return __shfl_sync(0xffffffffu, a, l); }
};

// Rows written by one CTA of a cluster and read by another in the same launch:
// past L1, which is not coherent between SMs.
__device__ __forceinline__ uint32_t ldc(const uint32_t* p) { return __ldcg(p); }
__device__ __forceinline__ uint2 ldc(const uint2* p) { return __ldcg(p); }
__device__ __forceinline__ uint4 ldc(const uint4* p) { return __ldcg(p); }
__device__ __forceinline__ void stc(uint32_t* p, uint32_t v) { __stcg(p, v); }
__device__ __forceinline__ void stc(uint2* p, uint2 v) { __stcg(p, v); }
__device__ __forceinline__ void stc(uint4* p, uint4 v) { __stcg(p, v); }

template <int D>
__device__ __forceinline__ int inverse(int x) {  // of x in [1, D)
  if constexpr (D == 2) return 1;
  if constexpr (D == 3) return x;
  if constexpr (D == 5) return (0x42310 >> (4 * x)) & 15;    // 1, 3, 2, 4
  return (0x6325410 >> (4 * x)) & 15;                         // 1, 4, 5, 2, 3, 6
}

__device__ __forceinline__ int find_tile(const RowDesc* descs, int nd, int b, bool extra) {
  int lo = 0, hi = nd - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((extra ? descs[mid].x_begin : descs[mid].tile_begin) <= b) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------- raw pass

// A column word of one qudit's row x_q or z_q.  Odd d: an element.  d = 2: the
// S and T words of one position (x, y) and the row's sign exponent as far as
// these words make it (z): a product of rows adds twice the parity of T . S'.
template <int D>
struct Unit : El<D> {
  using T = typename El<D>::T;
  static __device__ __forceinline__ T mask(T a, uint32_t m) {
    a.x &= m;
    a.y &= m;
    if constexpr (D != 3) a.z &= m;
    return a;
  }
  static __device__ __forceinline__ T bump(T a, int v) {  // the constant lane
    return El<D>::set(a, 0, (El<D>::get(a, 0) + v) % D);
  }
};
template <>
struct Unit<2> {
  using T = uint4;
  static __device__ __forceinline__ T zero() { return make_uint4(0u, 0u, 0u, 0u); }
  static __device__ __forceinline__ T add(T a, T b) {
    return make_uint4(a.x ^ b.x, a.y ^ b.y, a.z + b.z + 2u * (uint32_t)__popc(a.y & b.x), 0u);
  }
  static __device__ __forceinline__ T neg(T a) { return a; }
  static __device__ __forceinline__ T mask(T a, uint32_t m) { return make_uint4(a.x & m, a.y & m, a.z & m, 0u); }
  static __device__ __forceinline__ T pick(uint32_t m, T a, T b) {
    return make_uint4(mux(m, a.x, b.x), mux(m, a.y, b.y), mux(m, a.z, b.z), 0u);
  }
  static __device__ __forceinline__ T bump(T a, int v) { return make_uint4(a.x, a.y, a.z + (uint32_t)v, 0u); }
};

// Element of extra row r at unit u.
template <int D>
__device__ __forceinline__ void dump_extra(const RowDesc& rd, int r, int u, typename Unit<D>::T v) {
  using T = typename El<D>::T;
  T* row = reinterpret_cast<T*>(rd.xraw) + (size_t)r * (rd.E + rd.EK);
  if constexpr (D == 2) {
    row[u] = v.x;
  } else {
    if (u < rd.E) row[u] = v;
    else if (u >= 2 * rd.E) row[u - rd.E] = v;
  }
}

// One op (rows.cuh: RowProgram) on unit u, the CTA's unit c (of 2^lg) of every
// qudit.  The gates are one formula without branches -- nx = H ? +-z : x, nz =
// H ? +-x : z + t, x_t += +-x with t = +-x (P) or +-z_t (CNOT) or 0 -- since
// the lanes of a warp hold different gates.
template <int D>
__device__ __forceinline__ void raw_op(const RowDesc& rd, const uint4* o, int u, int c, int lg,
                                       typename Unit<D>::T* x, typename Unit<D>::T* z, bool konst) {
  using U = Unit<D>;
  using T = typename U::T;
  const uint32_t w = o->x;
  const int i = ((int)(w & 0x7ffu) << lg) + c, j = ((int)((w >> 11) & 0x7ffu) << lg) + c;
  const T xa = x[i], za = z[i], xb = x[j], zb = z[j];
  const uint32_t mh = lane_mask(w & (kRopH | kRopHInv)), mc = lane_mask(w & (kRopC | kRopCInv));
  const uint32_t mt = lane_mask(w & (kRopC | kRopCInv | kRopP | kRopPInv));
  T nx, nz, nt;
  if constexpr (D == 2) {
    nt = U::add(U::mask(xa, mc), xb);  // A_c A_t and B_c B_t, B A for a P
    const T t = U::mask(U::pick(mc, zb, xa), mt);
    nz = U::pick(mh, xa, U::add(za, t));
    nx = U::pick(mh, za, xa);
  } else {
    const uint32_t mneg = lane_mask(w & (kRopC | kRopPInv));
    const T t0 = U::pick(mc, zb, xa);
    const T t = U::mask(U::pick(mneg, U::neg(t0), t0), mt);
    const T xn = U::neg(xa), zn = U::neg(za);
    nt = U::add(xb, U::mask(U::pick(lane_mask(w & kRopCInv), xn, xa), mc));
    nz = U::pick(mh, U::pick(lane_mask(w & kRopHInv), xn, xa), U::add(za, t));
    nx = U::pick(mh, U::pick(lane_mask(w & kRopH), zn, za), xa);
  }
  if (konst && (w & kRopK)) {
    nx = U::bump(nx, (int)(o->y & 7u));
    nz = U::bump(nz, (int)((o->y >> 3) & 7u));
  }
  if (w & kRopM) {  // a measurement dumps its row, and leaves the generator Z_q
    using E = typename El<D>::T;
    const int m = (int)o->y;
    E* row = reinterpret_cast<E*>(rd.raw) + (size_t)m * (2 * rd.E + rd.EK);
    const int kbase = D == 2 ? rd.E : 2 * rd.E;
    if constexpr (D == 2) {
      if (u < rd.E) {
        row[u] = nx.x;
        row[rd.E + u] = nx.y;
        rd.kpart[(size_t)m * rd.E + u] = (uint8_t)(nx.z & 3u);
        if (u == 0) rd.ksign[m] = 0;
      } else {
        row[rd.E + u] = nx.x;
      }
    } else {
      row[u] = nx;
    }
    const int v = m + (D == 2 ? 0 : 1);
    if (m < rd.nk && u == kbase + v / L) {
      if constexpr (D == 2)
        nz.x |= 1u << (v % L);
      else
        nz = El<D>::set(nz, v % L, 1);
    }
    if (w & kRopReset) dump_extra<D>(rd, (int)o->z - 1, u, nz);
  }
  x[i] = nx;
  z[i] = nz;
  if (mc) x[j] = nt;
  if (w & kRopN) {  // N1 rows of the qudit, of a CNOT's target
    const uint32_t r = (w & kRopM) ? o->w : o->z;
    if (r) {
      dump_extra<D>(rd, (int)r - 1, u, nx);
      dump_extra<D>(rd, (int)r, u, nz);
    }
    if (mc && o->w) {
      dump_extra<D>(rd, (int)o->w - 1, u, nt);
      dump_extra<D>(rd, (int)o->w, u, zb);
    }
  }
}

// Gates move no data between column words, so a CTA walks the layers on its
// 2^lg units (u0 on) of every qudit alone; a layer's ops are on disjoint
// qudits, so its (op, unit) tasks run in any order and one barrier ends it.
// Bound by the chain of layers (a shared-memory read, a gate, its dumps and a
// barrier each), 600 to 1,000 cycles a layer, so the ops come from global memory
// a window ahead and, for d = 2, from shared memory a layer ahead.
// Threads 0 .. nt - 1 of the block; mem: raw_bytes(n, lg).
constexpr int kRawOps = 768, kRawLayers = 255;

template <int D>
__host__ __device__ inline size_t raw_bytes(int n, int lg) {
  return 2 * ((size_t)n << lg) * sizeof(typename Unit<D>::T) + 2 * kRawOps * sizeof(uint4) + 4 * (kRawLayers + 2);
}

template <int D>
__device__ void raw_program(const RowDesc& rd, int u0, int lg, int nt, uint8_t* mem) {
  using UT = typename Unit<D>::T;
  const int t = threadIdx.x;
  if (t >= nt) return;
  const int n = rd.n, E = rd.E, cw = 1 << lg;
  const int units = (D == 2 ? E : 2 * E) + rd.EK;
  uint4* wops = reinterpret_cast<uint4*>(mem);
  UT* x = reinterpret_cast<UT*>(wops + 2 * kRawOps);
  UT* z = x + ((size_t)n << lg);
  uint32_t* wlay = reinterpret_cast<uint32_t*>(z + ((size_t)n << lg));
  auto sync = [&]() { asm volatile("bar.sync 2, %0;" ::"r"(nt) : "memory"); };
  // stabilizer g = Z_g, destabilizer n + g = X_g
  for (int i = t; i < (n << lg); i += nt) {
    const int q = i >> lg, u = u0 + (i & (cw - 1)), g = q / L;
    UT xv = Unit<D>::zero(), zv = Unit<D>::zero();
    if constexpr (D == 2) {
      if (u == g) xv.y = zv.x = 1u << (q % L);
    } else {
      if (u == E + g) xv = El<D>::set(xv, q % L, 1);
      if (u == g) zv = El<D>::set(zv, q % L, 1);
    }
    x[i] = xv;
    z[i] = zv;
  }
  const int c = t & (cw - 1), u = u0 + c, k0 = t >> lg, dk = nt >> lg;
  const bool mine = u < units, konst = u == (D == 2 ? 0 : 2 * E);
  // the ops of the layers that fit the window, in shared memory (a layer that
  // does not fit by itself is read in place), the next window's on their way
  const uint32_t all = (uint32_t)rd.nops;
  auto stage = [&](uint32_t w, int b) {
    const uint32_t cnt = min(all - w, (uint32_t)kRawOps);
    for (uint32_t i = t; i < cnt; i += nt) {
      const unsigned dst = (unsigned)__cvta_generic_to_shared(wops + b * kRawOps + i);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(rd.ops + w + i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int buf = 0;
  stage(0u, 0);
  for (int l = 0; l < rd.nlayers; l += kRawLayers) {
    const int nl = min(kRawLayers, rd.nlayers - l);
    for (int i = t; i <= nl; i += nt) wlay[i] = __ldg(rd.lay + l + i);
    sync();
    for (int i = 0; i < nl;) {
      const uint32_t w0 = wlay[i];
      int ie = i;  // layers [i, ie) fit
      for (bool more = true; more;) {
        const int q = ie + 1 + (t & 31);
        const uint32_t fit = __ballot_sync(0xffffffffu, q <= nl && wlay[q] <= w0 + kRawOps);
        ie += __popc(fit);
        more = fit == 0xffffffffu;
      }
      const bool whole = ie > i;
      if (!whole) ie = i + 1;
      stage(wlay[ie], buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      sync();
      const uint4* win = wops + buf * kRawOps - w0;
      uint32_t b = w0;
      if (!whole) {
        const uint32_t e = wlay[ie];
        if (mine)
          for (uint32_t k = b + k0; k < e; k += dk) raw_op<D>(rd, rd.ops + k, u, c, lg, x, z, konst);
        i = ie;
        sync();
      }
      if constexpr (D == 2) {  // (odd d: more registers, 100 cycles a layer slower so)
        uint32_t e = wlay[i + 1];
        uint4 ahead = make_uint4(0u, 0u, 0u, 0u);
        if (i < ie && b + k0 < e) ahead = win[b + k0];
        for (; i < ie; ++i) {
          uint4 o = ahead;
          const uint32_t e2 = i + 1 < ie ? wlay[i + 2] : e;
          if (e + k0 < e2) ahead = win[e + k0];
          if (mine)
            for (uint32_t k = b + k0; k < e;) {
              raw_op<D>(rd, &o, u, c, lg, x, z, konst);
              if ((k += dk) < e) o = win[k];
            }
          b = e;
          e = e2;
          sync();
        }
      }
      for (; i < ie; ++i) {
        const uint32_t e = wlay[i + 1];
        if (mine)
          for (uint32_t k = b + k0; k < e; k += dk) raw_op<D>(rd, win + k, u, c, lg, x, z, konst);
        b = e;
        sync();
      }
      buf ^= 1;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int D>
__global__ void __launch_bounds__(256) k_rows_raw(const RowDesc* __restrict__ descs, int nd, int lg) {
  extern __shared__ __align__(16) uint8_t smem[];
  const RowDesc rd = descs[find_tile(descs, nd, (int)blockIdx.x, false)];
  raw_program<D>(rd, ((int)blockIdx.x - rd.tile_begin) << lg, lg, (int)blockDim.x, smem);
}

// ---------------------------------------------------------------- panels

// x mod D for x in [0, 36 * 32 + 6], without a division.
template <int D>
__device__ __forceinline__ int small_mod(int x) {
  constexpr uint32_t m = (65536u + D - 1) / D;  // exact: the error x (m D - 65536) / (65536 D) stays below 1 / D
  return x - D * (int)(((uint32_t)x * m) >> 16);
}

// The updates of one panel, staged in shared memory.
struct PanelOps {
  int nops;
  int p[32], e[32], mord[32];
  int dup[32];   // the last earlier op of the panel with the same pivot, -1 for none
  int last[32];  // 1 when no later op of the panel has this pivot
  uint8_t G[32][32];  // extra pass: G[h][k], what op h's factor adds at op k's pivot (0 where it does not count)
  // chain pass: byte h of Wt[k] = W[h][k] with a = a0 W, a0 the row's entries
  // at the pivots before the panel: W = (1 - G)^-1
  __align__(16) uint32_t Wt[32][8];
};

// cnt elements from global memory (past L1), several loads in flight a thread.
template <class T, class Put>
__device__ __forceinline__ void copy_elems(const T* src, int cnt, int t, int nt, Put put) {
  constexpr int U = sizeof(T) == 16 ? 4 : 8;
  for (int i0 = t; i0 < cnt; i0 += U * nt) {
    T v[U];
#pragma unroll
    for (int j = 0; j < U; ++j)
      if (i0 + j * nt < cnt) v[j] = ldc(src + i0 + j * nt);
#pragma unroll
    for (int j = 0; j < U; ++j)
      if (i0 + j * nt < cnt) put(i0 + j * nt, v[j]);
  }
}

// The panel's factor rows (whole rows, kFull, or their stabilizer halves)
// into Fs[h][cnt], cnt = 2 E or E, with the columns that a later op of the
// panel replaces cleared (odd d), so that a row's update by the whole panel is
// one linear combination of these rows.  The extra pass gets the pivot
// products G first, the chain pass the matrix W from the panel's elimination.
template <int D, bool kFull>
__device__ void stage_panel(PanelOps& po, typename El<D>::T* Fs, const RowDesc& rd, int panel, int first,
                            int nops) {
  using E_ = El<D>;
  using T = typename E_::T;
  const int t = threadIdx.x, nt = blockDim.x;
  const int E = rd.E, cnt = kFull ? 2 * E : E;
  const T* opf = reinterpret_cast<const T*>(rd.opf) + (size_t)first * 2 * E;
  if (t == 0) po.nops = nops;
  if (t < nops) {
    const int4 m = __ldcg(rd.opm + first + t);
    po.p[t] = m.x;
    po.e[t] = m.y;
    po.mord[t] = m.z;
    po.dup[t] = (m.w & 63) - 1;
    po.last[t] = m.w >> 6;
  }
  if constexpr (kFull) {
    if constexpr (D != 2) {
      const uint32_t* w = rd.opw + (size_t)panel * 256;
      for (int i = t; i < nops * 8; i += nt) (&po.Wt[0][0])[i] = ldc(w + i);
    }
    copy_elems(opf, nops * cnt, t, nt, [&](int i, T v) { Fs[i] = v; });
  } else {
    for (int h = t >> 5; h < nops; h += nt >> 5)
      copy_elems(opf + (size_t)h * 2 * E, E, t & 31, 32, [&](int i, T v) { Fs[h * E + i] = v; });
  }
  __syncthreads();
  if constexpr (D != 2) {
    if constexpr (!kFull) {
      for (int i = t; i < 1024; i += nt) {
        const int h = i >> 5, k = i & 31;
        int g = 0;
        if (h < k && k < nops && h > po.dup[k]) g = E_::get(Fs[h * cnt + po.p[k] / L], po.p[k] % L);
        po.G[h][k] = (uint8_t)g;
      }
      __syncthreads();
    }
    // op h keeps nothing at the pivots of ops k >= h: those entries are
    // replaced after it (its own are zero already)
    for (int i = t; i < 1024; i += nt) {
      const int h = i >> 5, k = i & 31;
      if (h >= k || k >= nops) continue;
      const int pe = po.p[k] / L, pl = po.p[k] % L;
#pragma unroll
      for (int half = 0; half < (kFull ? 2 : 1); ++half) {
        E_::clear(&Fs[h * cnt + (half ? E + pe : pe)], pl);
      }
    }
  }
  __syncthreads();
}

// fn(integral_constant<int, c>) for c = 1 .. D - 1.
template <int D, int C = 1, class Fn>
__device__ __forceinline__ void each_multiple(Fn fn) {
  if constexpr (C < D) {
    fn(std::integral_constant<int, C>());
    each_multiple<D, C + 1>(fn);
  }
}

// Odd d: buf[0, cnt) += sum of the panel's factor rows times av (lane h: op h),
// a lane to an element; where a turn's elements leave lanes over, K of them
// share one, each with every K-th op, and the partial sums meet by shuffles.
// The ops are taken multiple by multiple (ord: 32 bytes for their order), so
// that a term is a carry-saving add of fixed form without a branch.
// Bound by its logic instructions.  A panel of 31 rows: 256 qudits of d = 5 11.7k
// cycles with additions mod d behind a branch per term, 6.6k so; 517 of d = 7
// 12.8k and 9k; the step of 384 uneven programs 3534 us and 3423.
template <int D>
__device__ __forceinline__ void combine_row(const typename El<D>::T* Fs, typename El<D>::T* buf, int cnt, int av,
                                            uint8_t* ord) {
  using E_ = El<D>;
  using T = typename E_::T;
  const int lane = threadIdx.x & 31;
  int n[D] = {}, first = 0;
  each_multiple<D>([&](auto c) {
    constexpr int C = c.value;
    const uint32_t m = __ballot_sync(0xffffffffu, av == C);
    n[C] = __popc(m);
    if (av == C) ord[first + __popc(m & ((1u << lane) - 1u))] = (uint8_t)lane;
    first += n[C];
  });
  __syncwarp();
  for (int e0 = 0; e0 < cnt; e0 += 32) {
    int G = 32;
    while (G > 1 && (G >> 1) >= cnt - e0) G >>= 1;
    const int K = 32 / G, part = lane / G, e = e0 + (lane & (G - 1));
    const bool in = e < cnt;
    typename E_::Sum sum(in && part == 0 ? buf[e] : E_::zero());
    const uint8_t* o = ord + part;
    each_multiple<D>([&](auto c) {
      constexpr int C = c.value;
#pragma unroll 2
      for (int i = 0; i < n[C]; i += K) {
        T f = E_::zero();
        if (in && i + part < n[C]) f = Fs[o[i] * cnt + e];
        sum.template add<C>(f);
      }
      o += n[C];
    });
    T v = sum.value();
    for (int p = G; p < 32; p <<= 1) v = E_::add(v, E_::shfl_xor(v, p));
    if (in && part == 0) buf[e] = v;
  }
  __syncwarp();
}

// Odd d, one warp: a whole row in buf[0, 2 E) (shared memory) through the
// panel's ops; kraw: its raw K elements, ab: 32 ints and 32 bytes of this warp.
template <int D>
__device__ __forceinline__ void update_row(const PanelOps& po, const typename El<D>::T* Fs,
                                           typename El<D>::T* buf, const typename El<D>::T* kraw, int E, int nk,
                                           int* ab) {
  using E_ = El<D>;
  const int lane = threadIdx.x & 31;
  const int nops = po.nops;
  int a0 = 0, om = 0;
  if (lane < nops) {
    const int v = po.mord[lane] + 1;
    if (v <= nk) om = E_::get(ldc(kraw + v / L), v % L);
  }
  const int dup = lane < nops ? po.dup[lane] : -1;
  const int omd = __shfl_sync(0xffffffffu, om, dup < 0 ? 0 : dup);
  if (lane < nops) a0 = dup < 0 ? E_::get(buf[po.p[lane] / L], po.p[lane] % L) : omd;
  uint8_t* a0b = reinterpret_cast<uint8_t*>(ab + 32);
  a0b[lane] = (uint8_t)a0;
  __syncwarp();
  int av = 0;
  if (lane < nops) {
    const uint4* x = reinterpret_cast<const uint4*>(a0b);
    const uint4* w = reinterpret_cast<const uint4*>(po.Wt[lane]);
    const uint4 x0 = x[0], x1 = x[1], w0 = w[0], w1 = w[1];
    uint32_t s = 0u;
    s = __dp4a(x0.x, w0.x, s);
    s = __dp4a(x0.y, w0.y, s);
    s = __dp4a(x0.z, w0.z, s);
    s = __dp4a(x0.w, w0.w, s);
    s = __dp4a(x1.x, w1.x, s);
    s = __dp4a(x1.y, w1.y, s);
    s = __dp4a(x1.z, w1.z, s);
    s = __dp4a(x1.w, w1.w, s);
    av = small_mod<D>((int)s);
    // the replaced entries: S[p] from measurement h's K column, T[p] = e a
    if (po.last[lane]) {
      const int pe = po.p[lane] / L, pl = po.p[lane] % L;
      E_::clear(buf + pe, pl);
      E_::put(buf + pe, pl, om);
      E_::clear(buf + E + pe, pl);
      E_::put(buf + E + pe, pl, small_mod<D>(po.e[lane] * av));
    }
  }
  __syncwarp();
  combine_row<D>(Fs, buf, 2 * E, av, a0b);
}

// The same for the stabilizer half alone, through the panel's ops with
// ordinal below `after` (the first `non` ops).
template <int D>
__device__ __forceinline__ void update_half_row(const PanelOps& po, const typename El<D>::T* Fs,
                                                typename El<D>::T* buf, const typename El<D>::T* kraw, int E, int nk,
                                                int after, int* ab) {
  using E_ = El<D>;
  const int lane = threadIdx.x & 31;
  const int nops = po.nops;
  const unsigned onm = __ballot_sync(0xffffffffu, lane < nops && po.mord[lane] < after);
  const int non = __popc(onm);
  int av = 0, om = 0;
  if (lane < non) {
    const int v = po.mord[lane] + 1;
    if (v <= nk) om = E_::get(ldc(kraw + v / L), v % L);
  }
  const int dup = lane < nops ? po.dup[lane] : -1;
  const int omd = __shfl_sync(0xffffffffu, om, dup < 0 ? 0 : dup);
  if (lane < nops) av = dup < 0 ? E_::get(buf[po.p[lane] / L], po.p[lane] % L) : omd;
  __syncwarp();
  // a_h = the row's entry at op h's pivot once the ops before it are applied
  for (int h = 0; h < non; ++h) {
    const int a = small_mod<D>(__shfl_sync(0xffffffffu, av, h));
    av = lane == h ? a : av + a * po.G[h][lane];
  }
  // S[p] from measurement h's K column.  An op past `after` replaces nothing,
  // but its pivot's entry is missing in the combination below (cleared): it is
  // the value gathered above.
  if (lane < non ? po.last[lane] != 0 : lane < nops && dup < non) {
    const int pe = po.p[lane] / L, pl = po.p[lane] % L;
    E_::clear(buf + pe, pl);
    E_::put(buf + pe, pl, lane < non ? om : small_mod<D>(av));
  }
  __syncwarp();
  combine_row<D>(Fs, buf, E, lane < non ? av : 0, reinterpret_cast<uint8_t*>(ab));
}

// d = 2: lanes of a row's group (a power of two of at least E words, at most
// a warp), each holding the words gl, gl + G, ...
__host__ __device__ inline int row_group(int E) {
  int g = 1;
  while (g < E && g < 32) g <<= 1;
  return g;
}
constexpr int kRowGroupWords = 2;  // words per lane: n <= 2048

// d = 2: the words of a row (S, T) in a group's registers through the panel's
// ops with ordinal below `after`, in order; kword: the row's raw K bits of the
// panel's ordinals (m0 on); returns what the row's sign exponent gains (T only).
template <bool kFull>
__device__ __forceinline__ int update_row2(const PanelOps& po, const uint32_t* Fs, uint32_t (&S)[kRowGroupWords],
                                           uint32_t (&T)[kRowGroupWords], uint32_t kword, int m0, int E, int cnt,
                                           int after, int gl, int G) {
  uint32_t acc = 0u;
  int kk = 0;
  for (int h = 0; h < po.nops; ++h) {
    const int mord = po.mord[h];
    const int p = po.p[h], pw = p >> 5;
    const uint32_t sw = pw >= G ? S[1] : S[0];
    const uint32_t word = __shfl_sync(0xffffffffu, sw, pw & (G - 1), G);
    if (mord >= after) continue;  // uniform over the group only: the shuffle comes first
    const uint32_t a = (word >> (p & 31)) & 1u, om = (kword >> (mord - m0)) & 1u, mk = 0u - a;
#pragma unroll
    for (int i = 0; i < kRowGroupWords; ++i) {
      const int w = gl + i * G;
      if (w >= E) break;
      S[i] ^= Fs[h * cnt + w] & mk;
      if constexpr (kFull) {
        const uint32_t ft = Fs[h * cnt + E + w] & mk;
        T[i] ^= ft;
        acc ^= S[i] & ft;
      }
      if (w == pw) {
        S[i] = El<2>::set(S[i], p & 31, (int)om);
        if constexpr (kFull) T[i] = El<2>::set(T[i], p & 31, (int)a);
      }
    }
    if constexpr (kFull) kk += (int)a * ((po.e[h] >> 8) + 2 * (int)om);
  }
  if constexpr (kFull) {
    int par = __popc(acc) & 1;
    for (int o = G >> 1; o > 0; o >>= 1) par ^= __shfl_xor_sync(0xffffffffu, par, o);
    kk += 2 * par;
  }
  return kk;
}

// d = 2: bits [m0, m0 + 31) of a row's raw K words.
__device__ __forceinline__ uint32_t k_bits(const uint32_t* kraw, int EK, int m0) {
  const int q = m0 >> 5;
  const uint32_t lo = q < EK ? ldc(kraw + q) : 0u, hi = q + 1 < EK ? ldc(kraw + q + 1) : 0u;
  return __funnelshift_r(lo, hi, m0 & 31);
}

// ---------------------------------------------------------------- chain pass

template <int D>
struct ChainSmem {
  using T = typename El<D>::T;
  // rows of the panel 2 E + 1 apart, so that a warp reading one word of all of
  // them meets no bank twice
  static __host__ __device__ size_t rows(int E) { return round_up((size_t)32 * (2 * E + 1) * sizeof(T), 16); }
  static __host__ __device__ size_t staged(int E) { return round_up((size_t)kRowPanel * 2 * E * sizeof(T), 16); }
  static __host__ __device__ size_t total(int E, int warps) {
    return rows(E) + staged(E) + (size_t)E * sizeof(T) + warps * 40 * sizeof(int) + 64;
  }
};

// State of a panel while it is eliminated.
struct PanelState {
  uint32_t rand;  // its random rows
  int pv[32];     // pivot | its residue << 16 of a random row
  int orow[32];   // the random rows in order: the panel's ops
  int dup[32], last[32];  // of an op, as in PanelOps
  int kk[32];     // constant lane (odd d), sign exponent (d = 2)
  int kq[32];     // d = 2: parities that the updates add to it
  int tp[32];     // d = 2: parity of S . T of a random row
  int dsum[32];   // T . V of a deterministic row
  uint32_t info[32];  // minfo
  uint8_t om[32][32];  // om[j][i]: raw entry of row i in row j's K column
  // what a warp offers for the next random row, by parity: the first
  // generator of the row in the warp's words (x: | residue << 16, -1 for none)
  // and its rows with a non-zero S (y), all rows' entries at that generator,
  // d = 2: the row's parities
  int2 cp[2][kRowWarps];
  int ct[2][kRowWarps];
  uint8_t ca[2][kRowWarps][32];
  __align__(16) uint32_t Wt[32][8];  // as PanelOps::Wt
  __align__(16) uint32_t Gt[32][8];  // byte h of Gt[o]: G[h][o]
};

__device__ __forceinline__ void bar_threads(int n) { asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); }

// The panel's rows (P, row i at i (2 E + 1), up to date) one after the other:
// lane i holds words of row i and lane 31 those of V, so one update serves all
// rows after a random one and V alike; warp w the words [w CE, (w + 1) CE) of
// S and of T.  Before the barrier of a step every warp offers what it knows of
// the next row, should that be random: its first generator there and all rows'
// entries at it; after it the first warp with one has the pivot.  When that
// row turns out deterministic and a later one is random, one more barrier
// offers that one.  Deterministic rows cost a dot product and no step.
// kSolo: one warp holds whole rows (E <= CE) and needs neither offers nor
// barriers.
// Bound by the step's chain of dependent instructions, then by their number
// (integer logic issues at half rate).  Panels of 31 rows: 17k to 27k cycles at
// 256 qudits of d = 5, 52k at 517 of d = 7, 27k at 451 qubits.  A pivot's warp
// running on alone with the others behind it took twice that.
template <int D, int CE, bool kSolo>
__device__ __forceinline__ void eliminate(const RowDesc& rd, int cnt, typename El<D>::T* P, typename El<D>::T* V,
                                          PanelState& ps) {
  using E_ = El<D>;
  using T = typename E_::T;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int E = rd.E, nw = kSolo ? 1 : (E + CE - 1) / CE, e0 = kSolo ? 0 : warp * CE;
  if (warp >= nw) return;
  T s[CE], t[CE];
#pragma unroll
  for (int i = 0; i < CE; ++i) {
    const int e = e0 + i;
    s[i] = t[i] = E_::zero();
    if (e < E && lane < cnt) {
      s[i] = P[(size_t)lane * (2 * E + 1) + e];
      t[i] = P[(size_t)lane * (2 * E + 1) + E + e];
    }
    if (e < E && lane == 31) s[i] = V[e];
  }
  int kb = lane < cnt ? ps.kk[lane] : 0;
  uint32_t kacc = 0u;  // d = 2: words whose parity the sign exponent gains
  uint32_t randm = 0u;
  int j = -1, buf = 0;
  const uint32_t live = cnt >= 32 ? 0xffffffffu : (1u << cnt) - 1u;
  // this lane's first generator in the warp's words, -1 for none
  auto first = [&]() {
    int k = -1;
#pragma unroll
    for (int i = CE - 1; i >= 0; --i) {
      const uint32_t x = E_::nzw(s[i]);
      k = x ? 32 * i + __ffs(x) - 1 : k;
    }
    return k;
  };
  // this lane's entry at generator k (uniform) of the warp's words
  auto entry = [&](int k) {
    T x = s[0];  // by masks: an index would put s into local memory
#pragma unroll
    for (int i = 1; i < CE; ++i) x = E_::pick(lane_mask((k >> 5) == i), s[i], x);
    return E_::get(x, k & 31);
  };
  // d = 2: parity of S . T | parity of kacc << 1, of row r
  auto parities = [&](int r) {
    int w = 0;
    if constexpr (D == 2) {
      uint32_t x = 0u;
#pragma unroll
      for (int i = 0; i < CE; ++i) x ^= s[i] & t[i];
      w = __shfl_sync(0xffffffffu, (__popc(x) & 1) | ((__popc(kacc) & 1) << 1), r);
    }
    return w;
  };
  auto offer = [&](int key, uint32_t nzm, int r) {
    const int k = __shfl_sync(0xffffffffu, key, r);
    const int a = entry(k & 0x7ff);
    ps.ca[buf][warp][lane] = (uint8_t)a;
    const int v = __shfl_sync(0xffffffffu, a, r), ct = parities(r);
    if (lane == 0) {
      ps.cp[buf][warp] = make_int2(k < 0 ? -1 : (e0 * 32 + k) | (v << 16), (int)nzm);
      if constexpr (D == 2) ps.ct[buf][warp] = ct;
    }
    bar_threads(32 * nw);
  };
  for (int step = 0; step <= cnt; ++step) {  // a random row each, the last without one
    const uint32_t after = j < 0 ? 0xffffffffu : ~((2u << j) - 1u);
    const int key = first();
    const uint32_t nzm = __ballot_sync(0xffffffffu, key >= 0) & live;
    uint32_t rnd;
    int2 got = make_int2(-1, 0);  // lane w: warp w's offer
    if constexpr (kSolo) {
      rnd = nzm & after;
    } else {
      offer(key, nzm, (j + 1) & 31);
      got = lane < nw ? ps.cp[buf][lane] : make_int2(-1, 0);
      rnd = __reduce_or_sync(0xffffffffu, (uint32_t)got.y) & after;
    }
    const int jn = rnd ? __ffs(rnd) - 1 : cnt;
    if (jn > j + 1) {  // deterministic rows up to it: T . V
      int d = 0;
#pragma unroll
      for (int i = 0; i < CE; ++i) d += E_::dot(t[i], E_::shfl(s[i], 31));
      if (lane > j && lane < jn) atomicAdd(&ps.dsum[lane], d);
    }
    if (jn >= cnt) break;
    if (!kSolo && jn > j + 1) {
      buf ^= 1;
      offer(key, nzm, jn);
      got = lane < nw ? ps.cp[buf][lane] : make_int2(-1, 0);
    }
    int p, val, a, tp = 0, kpar = 0;
    if constexpr (kSolo) {
      p = __shfl_sync(0xffffffffu, key, jn);
      a = entry(p);
      val = __shfl_sync(0xffffffffu, a, jn);
      if constexpr (D == 2) {
        const int w = parities(jn);
        tp = w & 1;
        kpar = w >> 1;
      }
    } else {
      const int ws = __ffs(__ballot_sync(0xffffffffu, got.x >= 0)) - 1;
      const int pv = __shfl_sync(0xffffffffu, got.x, ws);
      a = ps.ca[buf][ws][lane];
      p = pv & 0xffff;
      val = pv >> 16;
      if constexpr (D == 2) {
        const int w = lane < nw ? ps.ct[buf][lane] : 0;
        tp = __popc(__ballot_sync(0xffffffffu, w & 1)) & 1;
        kpar = __popc(__ballot_sync(0xffffffffu, w & 2)) & 1;
      }
    }
    const int e = inverse<D>(val), pe = p / L, pl = p % L;
    const int kj = __shfl_sync(0xffffffffu, kb, jn);
    const int nv = D == 2 ? ((kj + 2 * kpar + tp) >> 1) & 1 : kj;
    const int om = lane == 31 ? nv : ps.om[jn][lane];
    const bool act = lane > jn && (lane < cnt || lane == 31);
    const int c = !act ? 0 : D == 2 ? a : small_mod<D>((D - e) * a);
    const int ta = D == 2 ? a : small_mod<D>(e * a);
    if (D == 2 && c) kb += tp + 2 * om;
#pragma unroll
    for (int i = 0; i < CE; ++i) {
      const T fs = E_::shfl(s[i], jn), ft = E_::shfl(t[i], jn);
      T ns = E_::muladd(s[i], fs, c), nt = E_::muladd(t[i], ft, c);
      const uint32_t at = e0 + i == pe ? 1u << pl : 0u;  // the pivot's lane
      if constexpr (D == 2) kacc ^= ns & ft & ~at & (0u - (uint32_t)c);
      s[i] = E_::put_at(ns, act ? at : 0u, om);
      t[i] = E_::put_at(nt, act ? at : 0u, ta);
    }
    if (warp == 0 && lane == 0) {
      ps.pv[jn] = p | (val << 16);
      ps.orow[__popc(randm)] = jn;
      if constexpr (D == 2) ps.tp[jn] = tp;
    }
    randm |= 1u << jn;
    j = jn;
    buf ^= 1;
  }
#pragma unroll
  for (int i = 0; i < CE; ++i) {
    const int e = e0 + i;
    if (e < E && lane < cnt) {
      P[(size_t)lane * (2 * E + 1) + e] = s[i];
      P[(size_t)lane * (2 * E + 1) + E + e] = t[i];
    }
    if (e < E && lane == 31) V[e] = s[i];
  }
  if constexpr (D == 2) {
    if (__popc(kacc) & 1) atomicAdd(&ps.kq[lane], 1);
  }
  if (warp == 0) {
    if (lane < cnt) ps.kk[lane] = kb;
    if (lane == 0) ps.rand = randm;
  }
}

// The rest of a trace row after E elements.
template <int D>
__device__ __forceinline__ void trace_pad(uint8_t* row, int E, int rowb, int lane) {
  for (int b = E * row_elem_bytes(D) + 4 * lane; b < rowb; b += 128) *reinterpret_cast<uint32_t*>(row + b) = 0u;
}

// Eliminates panel k (its rows in P, up to date) and writes its trace records
// and the updates that its random rows are to later rows.
template <int D, int CE, bool kSolo>
__device__ void factor_panel(const RowDesc& rd, int k, typename El<D>::T* P, typename El<D>::T* V, PanelState& ps,
                             int& nopsum) {
  const int nwp = (int)(blockDim.x >> 5);
  using E_ = El<D>;
  using T = typename E_::T;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int E = rd.E, m0 = k * kRowPanel, cnt = min(kRowPanel, rd.nm - m0);
  eliminate<D, CE, kSolo>(rd, cnt, P, V, ps);
  __syncthreads();
  const uint32_t randm = ps.rand;
  const int nops = __popc(randm);
  if constexpr (D != 2) {
    if (threadIdx.x < 32) {  // ops with one pivot; idle lanes have one of their own
      const int o = threadIdx.x;
      const uint32_t same = __match_any_sync(0xffffffffu, o < nops ? ps.pv[ps.orow[o]] & 0xffff : -1 - o);
      ps.dup[o] = 31 - __clz((int)(same & ((1u << o) - 1u)));
      ps.last[o] = (same >> o) == 1u;
    }
    __syncthreads();
    // G[h][o] = -e_h times op h's entry at op o's pivot, nothing where an op
    // from h on has replaced it before o
    for (int i = threadIdx.x; i < 1024; i += (int)blockDim.x) {
      const int o = i >> 5, h = i & 31;
      int g = 0;
      if (h < o && o < nops && h > ps.dup[o]) {
        const int ro = ps.orow[o], rh = ps.orow[h];
        const int p = ps.pv[ro] & 0xffff;
        g = small_mod<D>((D - inverse<D>(ps.pv[rh] >> 16)) * E_::get(P[(size_t)rh * (2 * E + 1) + p / L], p % L));
      }
      reinterpret_cast<uint8_t*>(ps.Gt[o])[h] = (uint8_t)g;
    }
    __syncthreads();
    // W = (1 - G)^-1 by columns, in the last warp: W[i][o] = sum_h W[i][h] G[h][o]
    if (warp == nwp - 1) {
      uint32_t wr[8] = {};
      for (int o = 0; o < nops; ++o) {
        const uint4 g0 = *reinterpret_cast<const uint4*>(ps.Gt[o]), g1 = *reinterpret_cast<const uint4*>(ps.Gt[o] + 4);
        uint32_t a = __dp4a(wr[0], g0.x, 0u), b = __dp4a(wr[4], g1.x, 0u);
        a = __dp4a(wr[1], g0.y, a);
        b = __dp4a(wr[5], g1.y, b);
        a = __dp4a(wr[2], g0.z, a);
        b = __dp4a(wr[6], g1.z, b);
        a = __dp4a(wr[3], g0.w, a);
        b = __dp4a(wr[7], g1.w, b);
        const int v = lane == o ? 1 : lane < o ? small_mod<D>((int)(a + b)) : 0;
        const uint32_t vb = (uint32_t)v << (8 * (o & 3));
#pragma unroll
        for (int q = 0; q < 8; ++q) wr[q] |= q == o >> 2 ? vb : 0u;
        reinterpret_cast<uint8_t*>(ps.Wt[o])[lane] = (uint8_t)v;
      }
      __syncwarp();
      uint32_t* w = rd.opw + (size_t)k * 256;
      for (int i = lane; i < 8 * nops; i += 32) stc(w + i, (&ps.Wt[0][0])[i]);
    }
  }
  // the panel's trace records and updates
  const int writers = D == 2 ? nwp : nwp - 1;
  for (int i = warp; i < cnt && warp < writers; i += writers) {
    const int m = m0 + i;
    const T* row = P + (size_t)i * (2 * E + 1);
    uint8_t* out = rd.mrow + (size_t)m * 2 * rd.rowb;
    const uint32_t info = ps.info[i];
    const uint32_t nord = info & 0x7fffffffu, reset = info >> 31;
    if ((randm >> i) & 1u) {
      const int p = ps.pv[i] & 0xffff, e = inverse<D>(ps.pv[i] >> 16), pe = p / L, pl = p % L;
      const int h = nopsum + __popc(randm & ((1u << i) - 1u));
      T* f = reinterpret_cast<T*>(rd.opf) + (size_t)h * 2 * E;
      for (int w = lane; w < 2 * E; w += 32) {
        T v = row[w];
        if (w == pe || w == E + pe) v = E_::set(v, pl, 0);
        v = E_::mulc(v, D == 2 ? 1 : D - e);
        stc(f + w, v);
        if (w < E) reinterpret_cast<T*>(out)[w] = v;
      }
      if (lane == 0) {
        const int o = h - nopsum;
        __stcg(rd.opm + h, make_int4(p, D == 2 ? 1 | (ps.tp[i] << 8) : e, m,
                                         D == 2 ? 0 : (ps.dup[o] + 1) | (ps.last[o] << 6)));
        rd.mhdr[m] = make_uint4(2u * reset, (uint32_t)p, nord, 0u);
      }
    } else {
      for (int w = lane; w < E; w += 32) reinterpret_cast<T*>(out)[w] = row[E + w];
      const int det = D == 2 ? 2 * (((ps.kk[i] + 2 * ps.kq[i]) >> 1) + ps.dsum[i] & 1)
                             : (ps.dsum[i] - ps.kk[i] + D) % D;
      if (lane == 0) rd.mhdr[m] = make_uint4(2u * reset | 1u, 0u, nord, (uint32_t)det);
    }
    trace_pad<D>(out, E, rd.rowb, lane);
  }
  if (threadIdx.x == 0) {
    if (k == 0) __stcg(rd.pop, 0);
    __stcg(rd.pop + k + 1, nopsum + __popc(randm));
  }
  nopsum += __popc(randm);
  __syncthreads();
}

// The first row from m on that may be random (its flag is set), nm for none.
__device__ __forceinline__ int next_random(const RowDesc& rd, int m) {
  const int lane = threadIdx.x & 31;
  for (; m < rd.nm; m += 256) {
    uint8_t f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = m + 32 * j + lane;
      f[j] = i < rd.nm ? __ldcg(rd.nz + i) : (uint8_t)0;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t b = __ballot_sync(0xffffffffu, f[j] != 0);
      if (b) return m + 32 * j + __ffs(b) - 1;
    }
  }
  return rd.nm;
}

// Trace record of measurement m, an up-to-date row without S entries, by one
// warp: the outcome is T . V and the row's own constant.
template <int D, class GetV>
__device__ __forceinline__ void det_row(const RowDesc& rd, int m, GetV phase) {
  using E_ = El<D>;
  using T = typename E_::T;
  const int lane = threadIdx.x & 31, E = rd.E;
  const T* src = reinterpret_cast<const T*>(rd.raw) + (size_t)m * (2 * E + rd.EK);
  uint8_t* out = rd.mrow + (size_t)m * 2 * rd.rowb;
  const uint32_t info = __ldg(rd.minfo + m);
  T k0 = E_::zero();
  int kk = 0, d = 0;
  if constexpr (D == 2)
    kk = lane == 31 ? (int)__ldcg(rd.ksign + m) : 0;
  else
    k0 = ldc(src + 2 * E);
  for (int w = lane; w < E; w += 32) {
    const T t = ldc(src + E + w);
    if constexpr (D == 2) kk += (int)__ldcg(rd.kpart + (size_t)m * E + w);
    d += E_::dot(t, phase(w));
    reinterpret_cast<T*>(out)[w] = t;
  }
  d = __reduce_add_sync(0xffffffffu, d);
  int det;
  if constexpr (D == 2) {
    kk = __reduce_add_sync(0xffffffffu, kk) & 3;
    det = 2 * ((kk >> 1) + d & 1);
  } else {
    det = (d - E_::get(k0, 0) + D) % D;
  }
  if (lane == 0)
    rd.mhdr[m] = make_uint4(2u * (info >> 31) | 1u, 0u, info & 0x7fffffffu, (uint32_t)det);
  trace_pad<D>(out, E, rd.rowb, lane);
}

// One program per cluster of C CTAs.  rawt > 0: the raw pass first, 2^lg units
// a CTA on rawt threads.  CTA 0 eliminates panel after panel (31
// rows and V in shared memory); the panel's updates then go to the rows after it:
// with C = 1 by this CTA itself, with more the next panel's rows by CTA 0 (it
// eliminates them next) and the others' by the other CTAs meanwhile, so one
// cluster barrier per panel is all they wait for.  A panel that had no random
// row leaves nothing to update; the rows after it up to the next one with S
// entries are then deterministic and independent, a warp takes each, and their
// panels cost no step (the rounds after the first of an error-correction
// memory).
// Bound by CTA 0's elimination, about 550 cycles a random row in one warp and
// 1,000 to 1,900 across warps, and by the layers in front.  As tableau passes,
// every random measurement updating all generators: 256 qudits of d = 5, 516
// measurements, 2,170 us, 390 so; the L = 7 memory 157 and 65 (102 with every
// deterministic panel a step).
template <int D, int CE, bool kSolo>
__global__ void __launch_bounds__(32 * kRowWarps) k_rows_chain(const RowDesc* __restrict__ descs, int nd, int C, int rawt,
                                                               int lg) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ PanelOps po;
  __shared__ PanelState ps;
  __shared__ RowDesc shared;
  using E_ = El<D>;
  using T = typename E_::T;
  const int r = C > 1 ? (int)cluster_rank() : 0;
  const int pi = (int)blockIdx.x / C;
  if (pi >= nd) return;  // the whole cluster
  // odd d: in shared memory, its fields would take a third of the registers
  // that the elements need (the elimination 28.4k cycles a panel at 256 qudits
  // of d = 5, 23.8k with them there); d = 2 has the registers, and is 5% slower
  // with it in shared memory
  RowDesc own;
  if constexpr (D == 2) {
    own = descs[pi];
  } else {
    for (int i = threadIdx.x; i < (int)(sizeof(RowDesc) / 4); i += blockDim.x)
      reinterpret_cast<uint32_t*>(&shared)[i] = reinterpret_cast<const uint32_t*>(descs + pi)[i];
    __syncthreads();
  }
  const RowDesc& rd = D == 2 ? own : shared;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwp = (int)(blockDim.x >> 5);
  const int E = rd.E, RS = 2 * E + rd.EK;
  T* P = reinterpret_cast<T*>(smem);
  T* Fs = reinterpret_cast<T*>(smem + ChainSmem<D>::rows(E));
  T* V = reinterpret_cast<T*>(smem + ChainSmem<D>::rows(E) + ChainSmem<D>::staged(E));
  int* ab = reinterpret_cast<int*>(smem + round_up(ChainSmem<D>::rows(E) + ChainSmem<D>::staged(E) +
                                                  (size_t)E * sizeof(T), 16)) + 40 * warp;
  T* raw = reinterpret_cast<T*>(rd.raw);
  if (rawt > 0) {
    raw_program<D>(rd, r << lg, lg, rawt, smem);
    __syncthreads();
    if (C > 1) cluster_sync_all();
  }
  const int panels = (rd.nm + kRowPanel - 1) / kRowPanel;
  const int G = row_group(E), gl = lane & (G - 1), gpw = 32 / G;  // d = 2: rows per warp
  int nops = 0;
  const int PS = 2 * E + 1;
  // panel k's rows into P, with their entries in each other's K columns and
  // their constants (odd d) or sign exponents (d = 2)
  auto load_panel = [&](int k) {
    const int m0 = k * kRowPanel, cnt = min(kRowPanel, rd.nm - m0);
    constexpr int R = D == 2 ? 2 : 1;  // rows at a time, all their loads first (two of odd d: too many registers)
    for (int i0 = warp; i0 < 32; i0 += R * nwp) {
      T kw[R], v[R][4], k0[R];
      int kk[R];
      uint32_t info[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int i = i0 + j * nwp;
        const bool in = i < cnt;
        const T* src = raw + (size_t)(m0 + i) * RS;
        const int q = m0 + lane + (D == 2 ? 0 : 1);
        kw[j] = in && m0 + lane < rd.nk && lane < i ? ldc(src + 2 * E + q / L) : E_::zero();
        info[j] = in ? __ldg(rd.minfo + m0 + i) : 0u;
        kk[j] = 0;
        k0[j] = E_::zero();
        if constexpr (D == 2) {
          const uint8_t* kp = rd.kpart + (size_t)(m0 + i) * E;
          if (in && lane < E) kk[j] = (int)__ldcg(kp + lane);
          if (in && lane + 32 < E) kk[j] += (int)__ldcg(kp + lane + 32);
          if (in && lane == 31) kk[j] += (int)__ldcg(rd.ksign + m0 + i);
        } else {
          if (in) k0[j] = ldc(src + 2 * E);
        }
#pragma unroll
        for (int h = 0; h < 4; ++h)  // 2 E <= 128 (n <= 2048)
          if (in && lane + 32 * h < 2 * E) v[j][h] = ldc(src + lane + 32 * h);
      }
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int i = i0 + j * nwp;
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (i < cnt && lane + 32 * h < 2 * E) P[(size_t)i * PS + lane + 32 * h] = v[j][h];
        ps.om[lane][i] = (uint8_t)E_::get(kw[j], (m0 + lane + (D == 2 ? 0 : 1)) % L);
        const int k = D == 2 ? __reduce_add_sync(0xffffffffu, kk[j]) & 3 : E_::get(k0[j], 0);
        if (lane == 0) {
          ps.kk[i] = k;
          ps.kq[i] = ps.dsum[i] = 0;
          ps.info[i] = info[j];
        }
      }
    }
    __syncthreads();
  };
  if (r == 0)
    for (int e = threadIdx.x; e < E; e += blockDim.x) V[e] = E_::zero();
  bool flags = false;  // the flags rd.nz of the rows after the next panel are set
  T* vg = reinterpret_cast<T*>(rd.vg);  // C > 1: V for the other CTAs, by parity of the step
  for (int k = -1, step = 0; k + 1 < panels; ++step) {
    int first = 0, cnt = 0, next = k + 1;
    if (k >= 0) {
      if (C > 1) cluster_sync_all(); else __syncthreads();
      first = __ldcg(rd.pop + k);
      cnt = __ldcg(rd.pop + k + 1) - first;
    }
    if (cnt == 0 && flags) {
      // nothing left to update: on to the next panel with a row that may be
      // random, the rows before it are all deterministic
      const int m = (k + 1) * kRowPanel, e = next_random(rd, m);
      next = e < rd.nm ? e / kRowPanel : panels;
      const T* vp = vg + (step & 1) * E;
      if (C == 1 || r > 0)
        for (int i = m + (C > 1 ? (r - 1) * nwp + warp : warp); i < min(next * kRowPanel, rd.nm);
             i += C > 1 ? (C - 1) * nwp : nwp)
          det_row<D>(rd, i, [&](int w) { return C > 1 ? ldc(vp + w) : V[w]; });
      if (r == 0 && threadIdx.x == 0)
        for (int q = k + 2; q <= next; ++q) __stcg(rd.pop + q, first);
      if (next == panels) break;
    }
    if (next + 1 == panels) follow_ready();  // one panel to go
    const int b1 = next * kRowPanel;
    if (cnt > 0) {
      stage_panel<D, true>(po, Fs, rd, k, first, cnt);
      flags = true;
    }
    if (cnt > 0 && (C == 1 || r > 0)) {
      // rows of the panels after the next (of all later ones with C = 1)
      const int m0 = C > 1 ? b1 + kRowPanel : b1;
      const int w0 = C > 1 ? (r - 1) * nwp + warp : warp, dw = C > 1 ? (C - 1) * nwp : nwp;
      if constexpr (D == 2) {
        for (int i0 = m0 + w0 * gpw; i0 < rd.nm; i0 += dw * gpw) {
          const int i = i0 + lane / G;
          const bool in = i < rd.nm;
          uint32_t S[kRowGroupWords] = {}, Tt[kRowGroupWords] = {};
          T* row = raw + (size_t)i * RS;
#pragma unroll
          for (int h = 0; h < kRowGroupWords; ++h) {
            const int w = gl + h * G;
            if (in && w < E) {
              S[h] = ldc(row + w);
              Tt[h] = ldc(row + E + w);
            }
          }
          const uint32_t kw = in ? k_bits(row + 2 * E, rd.EK, k * kRowPanel) : 0u;
          const int dk = update_row2<true>(po, Fs, S, Tt, kw, k * kRowPanel, E, 2 * E, INT_MAX, gl, G);
#pragma unroll
          for (int h = 0; h < kRowGroupWords; ++h) {
            const int w = gl + h * G;
            if (in && w < E) {
              stc(row + w, S[h]);
              stc(row + E + w, Tt[h]);
            }
          }
          uint32_t any = 0u;
#pragma unroll
          for (int h = 0; h < kRowGroupWords; ++h) any |= S[h];
          const uint32_t nz = __ballot_sync(0xffffffffu, any != 0u) >> (lane & ~(G - 1));
          if (in && gl == 0) {
            __stcg(rd.ksign + i, (uint8_t)((__ldcg(rd.ksign + i) + dk) & 3));
            __stcg(rd.nz + i, (uint8_t)((nz << (32 - G)) != 0u));
          }
        }
      } else {
        T* buf = P + (size_t)warp * PS;
        for (int i = m0 + w0; i < rd.nm; i += dw) {
          T* row = raw + (size_t)i * RS;
          copy_elems(row, 2 * E, lane, 32, [&](int e, T x) { buf[e] = x; });
          __syncwarp();
          update_row<D>(po, Fs, buf, row + 2 * E, E, rd.nk, ab);
          uint32_t any = 0u;
          for (int e = lane; e < 2 * E; e += 32) {
            const T v = buf[e];
            stc(row + e, v);
            if (e < E) any |= E_::nzw(v);
          }
          any = __ballot_sync(0xffffffffu, any != 0u);
          if (lane == 0) __stcg(rd.nz + i, (uint8_t)(any != 0u));
        }
      }
    }
    if (r == 0) {
      if (C == 1) __syncthreads();
      load_panel(next);
      if (C > 1 && cnt > 0) {
        const int rows = min(kRowPanel, rd.nm - b1);
        if constexpr (D == 2) {
          for (int i0 = warp * gpw; i0 < rows; i0 += nwp * gpw) {
            const int i = i0 + lane / G;
            const bool in = i < rows;
            uint32_t S[kRowGroupWords] = {}, Tt[kRowGroupWords] = {};
            T* buf = P + (size_t)i * PS;
#pragma unroll
            for (int h = 0; h < kRowGroupWords; ++h) {
              const int w = gl + h * G;
              if (in && w < E) {
                S[h] = buf[w];
                Tt[h] = buf[E + w];
              }
            }
            const uint32_t kw = in ? k_bits(raw + (size_t)(b1 + i) * RS + 2 * E, rd.EK, k * kRowPanel) : 0u;
            const int dk = update_row2<true>(po, Fs, S, Tt, kw, k * kRowPanel, E, 2 * E, INT_MAX, gl, G);
#pragma unroll
            for (int h = 0; h < kRowGroupWords; ++h) {
              const int w = gl + h * G;
              if (in && w < E) {
                buf[w] = S[h];
                buf[E + w] = Tt[h];
              }
            }
            if (in && gl == 0) ps.kk[i] = (ps.kk[i] + dk) & 3;
          }
        } else {
          for (int i = warp; i < rows; i += nwp)
            update_row<D>(po, Fs, P + (size_t)i * PS, raw + (size_t)(b1 + i) * RS + 2 * E, E, rd.nk, ab);
        }
        __syncthreads();
      }
      const int before = nops;
      factor_panel<D, CE, kSolo>(rd, next, P, V, ps, nops);
      if (C > 1 && nops == before)  // what a skip may follow
        for (int e = threadIdx.x; e < E; e += blockDim.x) stc(vg + (~step & 1) * E + e, V[e]);
    }
    k = next;
  }
}

// ---------------------------------------------------------------- extra pass

// Rows of an extra-pass CTA: d = 2 one per lane group, odd d one per warp.
template <int D>
__host__ __device__ inline int extra_rows(int E) {
  return D == 2 ? kRowWarps * (32 / row_group(E)) : kRowWarps;
}

template <int D>
struct ExtraSmem {
  using T = typename El<D>::T;
  static __host__ __device__ size_t staged(int E) { return (size_t)kRowPanel * E * sizeof(T); }
  static __host__ __device__ size_t total(int E) {
    return staged(E) + (size_t)kRowWarps * E * sizeof(T) + kRowWarps * 40 * sizeof(int) + 64;
  }
};

__device__ __forceinline__ uint8_t* extra_row(const RowDesc& rd, uint32_t who) {
  const uint32_t kind = who >> 30, i = who & 0x3fffffffu;
  if (kind == 0) return rd.mrow + ((size_t)i * 2 + 1) * rd.rowb;
  return rd.nrow + ((size_t)i * 2 + (kind == 2 ? 1 : 0)) * rd.rowb;
}

// Stabilizer halves of the rows that only the phase pass reads, through every
// update that precedes them.  Apart from the chain, since nothing in it waits
// for them: bound by their own updates, 38 us for the 256 RESETs of 256 qudits
// of d = 5, 9 us for the L = 7 memory's rows.
template <int D>
__global__ void __launch_bounds__(32 * kRowWarps) k_rows_extra(const RowDesc* __restrict__ descs, int nd) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ PanelOps po;
  using E_ = El<D>;
  using T = typename E_::T;
  follow_wait();
  follow_ready();
  const RowDesc rd = descs[find_tile(descs, nd, (int)blockIdx.x, true)];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int E = rd.E, XS = E + rd.EK;
  const int G = D == 2 ? row_group(E) : 32, gl = lane & (G - 1);
  const int x0 = ((int)blockIdx.x - rd.x_begin) * extra_rows<D>(E);
  const int i = x0 + warp * (32 / G) + lane / G;
  const bool in = i < rd.nx;
  const uint2 info = in ? __ldg(rd.xinfo + i) : make_uint2(0u, 0u);
  const int after = (int)info.x;
  const T* src = reinterpret_cast<const T*>(rd.xraw) + (size_t)(in ? i : 0) * XS;
  T* Fs = reinterpret_cast<T*>(smem);
  T* buf = reinterpret_cast<T*>(smem + ExtraSmem<D>::staged(E)) + (size_t)warp * E;
  int* ab = reinterpret_cast<int*>(smem + round_up(ExtraSmem<D>::staged(E) + (size_t)kRowWarps * E * sizeof(T), 16)) +
            40 * warp;
  uint32_t S[kRowGroupWords] = {}, none[kRowGroupWords] = {};
  if constexpr (D == 2) {
#pragma unroll
    for (int h = 0; h < kRowGroupWords; ++h)
      if (in && gl + h * G < E) S[h] = src[gl + h * G];
  } else {
    for (int e = lane; e < E; e += 32) buf[e] = in ? src[e] : E_::zero();
    __syncwarp();
  }
  // rows are in program order: the CTA's last row takes the most updates
  const int most = (int)__ldg(&rd.xinfo[min(rd.nx, x0 + extra_rows<D>(E)) - 1].x);
  for (int k = 0; k * kRowPanel < most; ++k) {
    const int first = rd.pop[k], cnt = rd.pop[k + 1] - first;
    if (cnt == 0) continue;
    __syncthreads();
    stage_panel<D, false>(po, Fs, rd, k, first, cnt);
    if constexpr (D == 2) {
      const uint32_t kw = in ? k_bits(src + E, rd.EK, k * kRowPanel) : 0u;
      update_row2<false>(po, Fs, S, none, kw, k * kRowPanel, E, E, after, gl, G);
    } else {
      if (in && after > k * kRowPanel) update_half_row<D>(po, Fs, buf, src + E, E, rd.nk, after, ab);
    }
  }
  if (!in) return;
  uint8_t* out = extra_row(rd, info.y);
  if constexpr (D == 2) {
#pragma unroll
    for (int h = 0; h < kRowGroupWords; ++h)
      if (gl + h * G < E) reinterpret_cast<uint32_t*>(out)[gl + h * G] = S[h];
    for (int w = E + gl; 4 * w < rd.rowb; w += G) reinterpret_cast<uint32_t*>(out)[w] = 0u;
  } else {
    for (int e = lane; e < E; e += 32) reinterpret_cast<T*>(out)[e] = buf[e];
    trace_pad<D>(out, E, rd.rowb, lane);
  }
}

// ---------------------------------------------------------------- phase pass

// Every shot's deltas from the trace (trace_bits.cuh, trace_u8.cuh: the same
// updates with the same streams, over the stabilizer half).  A shot is LG =
// 2^lg lanes, element e in lane e mod LG, and a warp 32 / LG shots; the four
// warps of a CTA share the measurements' headers and rows, staged 32 at a time
// while the 32 before them run, and a window's outcomes are drawn at its start
// with every lane on another draw.  A measurement then needs no barrier: a
// shuffle for the pivot's delta or log LG for a factor sum.
// Bound by a measurement's chain of dependent instructions where the warps are
// few, by their issue (172 a measurement and warp at d = 5) where they are many
// (then WPL elements a lane).  As residue bytes, 32 shots a CTA with barriers a
// measurement, 256 qudits of d = 5 and 4,096 shots took 760 us; 185 us with
// packed rows, 175 with a measurement's reads one ahead.
template <int D, int WPL>
__global__ void __launch_bounds__(128) k_rows_phase(const RowPhaseDesc* __restrict__ descs, int nd) {
  extern __shared__ __align__(16) uint8_t smem[];
  using E_ = El<D>;
  using T = typename E_::T;
  follow_wait();
  int di = 0;
  {
    int hi = nd - 1;
    while (di < hi) {
      const int mid = (di + hi + 1) >> 1;
      if (descs[mid].block_begin <= (int)blockIdx.x) di = mid; else hi = mid - 1;
    }
  }
  const RowPhaseDesc td = descs[di];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int lg = td.lg, LG = 1 << lg, SPW = 32 >> lg, gl = lane & (LG - 1), sl = lane >> lg;
  const int E = td.E, nm = td.nm, nmeas = td.c.nmeas;
  const int first = (((int)blockIdx.x - td.block_begin) * 4 + warp) * SPW;  // this warp's first shot
  const int rel = first + sl;
  const bool live = rel < td.c.nshots;
  const long long shot = td.c.shot0 + rel;
  const unsigned long long seed = td.c.seed;
  constexpr int WIN = 32;
  const int pitch = td.pitch;  // staged bytes of a measurement, a multiple of 16
  const bool resets = pitch > td.rowb;  // with the z_q rows of RESETs
  uint4* hdr = reinterpret_cast<uint4*>(smem);  // [2][WIN]
  uint8_t* rows = smem + 2 * WIN * 16;          // [2][WIN][pitch]
  uint8_t* mo = rows + 2 * (size_t)WIN * pitch + warp * (2 * 32 * 36) + sl * 36;  // this shot's outcomes
  uint8_t* rec0 = mo - sl * 36 + 32 * 36;                                         // the warp's records
  auto stage = [&](int wb, int b) {
    const int cnt = min(WIN, nm - wb);
    if (t < cnt) {
      const unsigned dst = (unsigned)__cvta_generic_to_shared(hdr + b * WIN + t);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(td.mhdr + wb + t) : "memory");
    }
    const int per = pitch >> 4;
    for (int i = t; i < cnt * per; i += 128) {
      const int m = i / per, q = i - m * per;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(rows + ((size_t)b * WIN + m) * pitch + 16 * q);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                   "l"(td.mrow + (size_t)(wb + m) * 2 * td.rowb + 16 * q)
                   : "memory");
    }
  };
  T d[WPL];
#pragma unroll
  for (int i = 0; i < WPL; ++i) d[i] = E_::zero();
  uint32_t nord = 0;
  if (nm > 0) stage(0, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int wb = 0, b = 0; wb < nm; wb += WIN, b ^= 1) {
    const int cnt = min(WIN, nm - wb);
    if (wb + WIN < nm) stage(wb + WIN, b ^ 1);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const uint4* hw = hdr + b * WIN;
    const uint8_t* rw = rows + (size_t)b * WIN * pitch;
    const uint32_t rnd = __ballot_sync(0xffffffffu, lane < cnt && !(hw[lane].x & 1u));
    for (int k = gl; k < cnt; k += LG)
      if ((rnd >> k) & 1u) mo[k] = (uint8_t)mulshift(stream_block(seed, shot, (uint32_t)(wb + k), 0u).x, D);
    __syncwarp();
    // what a measurement reads, one ahead of its use
    uint4 hn = make_uint4(0u, 0u, 0u, 0u);
    T rn[WPL], zn[WPL];
    int mn = 0;
    auto fetch = [&](int k) {
      const T* row = reinterpret_cast<const T*>(rw + (size_t)k * pitch);
      hn = hw[k];
      mn = mo[k];
#pragma unroll
      for (int i = 0; i < WPL; ++i) {
        const int e = gl + i * LG;
        rn[i] = e < E ? row[e] : E_::zero();
        zn[i] = e < E && resets ? reinterpret_cast<const T*>(reinterpret_cast<const uint8_t*>(row) + td.rowb)[e]
                                : E_::zero();
      }
    };
    fetch(0);
    for (int k = 0; k < cnt; ++k) {
      const uint4 h = hn;
      T r[WPL], zr[WPL];
#pragma unroll
      for (int i = 0; i < WPL; ++i) {
        r[i] = rn[i];
        zr[i] = zn[i];
      }
      int m = mn;
      if (k + 1 < cnt) fetch(k + 1);
      if constexpr (D != 2) {
        // N1 before the measurement: four coins a lane at a time; a group
        // applies one fire a turn
        const uint32_t nend = min(h.z, (uint32_t)td.nn1);
        for (; nord < nend; nord = min(nend, (nord / 4u + LG) * 4u)) {
          const uint32_t blk = nord / 4u + gl;
          uint32_t f = 0u;
          if (live && blk * 4u < nend) {
            const uint4 w = stream_block(seed, shot, blk, 1u);
            const uint32_t cw[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint32_t j = 4u * blk + q;
              if (j >= nord && j < nend) {
                const uint2 nh = __ldg(td.nhdr + j);
                if (nh.y != OP_N1OFF && cw[q] >= nh.x) f |= 1u << q;
              }
            }
          }
          while (true) {
            const uint32_t pend = __ballot_sync(0xffffffffu, f != 0u);
            if (!pend) break;
            const uint32_t mine = (pend >> (lane & ~(LG - 1))) & (LG == 32 ? 0xffffffffu : (1u << LG) - 1u);
            const int src = mine ? (lane & ~(LG - 1)) + __ffs(mine) - 1 : lane;
            const uint32_t sf = __shfl_sync(0xffffffffu, f, src);
            const uint32_t j = 4u * (nord / 4u + (uint32_t)(src & (LG - 1))) + (uint32_t)(__ffs(sf | 16u) - 1);
            if (mine) {
              const int2 ab = noise_choice(__ldg(&td.nhdr[j].y), D, seed, shot, j);
              const int cz = ab.x ? D - ab.x : 0, cx = ab.y;  // delta += -a z_q + b x_q
              const T* xr = reinterpret_cast<const T*>(td.nrow + (size_t)j * 2 * td.rowb);
              const T* zr = reinterpret_cast<const T*>(td.nrow + ((size_t)j * 2 + 1) * td.rowb);
#pragma unroll
              for (int i = 0; i < WPL; ++i) {
                const int e = gl + i * LG;
                if (e < E) d[i] = E_::muladd(E_::muladd(d[i], zr[e], cz), xr[e], cx);
              }
              if (src == lane) f &= f - 1u;
            }
          }
        }
      }
      if (!(h.x & 1u)) {
        const int p = (int)h.y, pe = p / L, pl = p % L;
        T x = d[0];
#pragma unroll
        for (int i = 1; i < WPL; ++i) x = E_::pick(lane_mask((pe >> lg) == i), d[i], x);
        const int dp = __shfl_sync(0xffffffffu, E_::get(x, pl), pe & (LG - 1), LG);
        const int nv = D == 2 ? m : m ? D - m : 0;
#pragma unroll
        for (int i = 0; i < WPL; ++i)
          d[i] = E_::put_at(E_::muladd(d[i], r[i], dp), gl + i * LG == pe ? 1u << pl : 0u, nv);
      } else {
        int s = 0;
#pragma unroll
        for (int i = 0; i < WPL; ++i) s += E_::dot(r[i], d[i]);
        for (int o = LG >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        m = D == 2 ? (((((int)h.w + 2 * s) & 3) + 1) >> 1) & 1 : (D - ((int)h.w + s) % D) % D;
      }
      if (h.x & 2u) {
#pragma unroll
        for (int i = 0; i < WPL; ++i) d[i] = E_::muladd(d[i], zr[i], m);
      }
      if (gl == 0) rec0[sl * 36 + k] = (uint8_t)(m | (int)((h.x & 1u) << 7));
    }
    __syncwarp();
    if (lane < cnt)
      for (int q = 0; q < SPW && first + q < td.c.nshots; ++q)
        td.c.out[(size_t)(first + q) * nmeas + wb + lane] = rec0[q * 36 + lane];
    __syncthreads();  // the window's buffers and outcomes are free
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------- frame pass

// Pauli frames (k_frame.cu: the rules) of 32 shots a warp, as bit planes: the
// frame of a shot is one more column under the gates, so the words X[q], Z[q]
// of 32 shots walk the row program's layers, a lane to an op.  Frame draws are
// made by lanes as shots and turned into words by ballots; N1 samples likewise,
// for d = 2 from the coin pass's masks (the few ordinals that any of the 32
// shots fires, behind a bitmap), else by atomics into a word per ordinal.  The
// record words stay in shared memory to the end; the output pass
// (k_rows_frame_out) adds the reference shot.
// Bound by its instructions, 22k a warp for the L = 7 memory: the draws' Philox
// blocks and the ops about equally.  A byte per shot and qudit, a lane per shot:
// 100,000 shots 1,500 us; on bit planes 130, 115 with four blocks of draws side
// by side.  10,000 shots of 48 qutrits: 78 and 46 us.
constexpr int kFrameOps = 768;  // ops of a window

template <int D>
struct FrameSmem {
  using T = typename El<D>::T;
  int fb, cb;  // Philox blocks of the frame draws, of the coins (odd d, whole 32 ordinals)
  size_t ordf, ordc, thr, warp0, x, z, rec, fire, warp;
  __host__ __device__ FrameSmem(int n, int nm, int nused, int nchunk, int cap) {
    auto up = [](size_t b) { return (b + 15) & ~(size_t)15; };
    fb = (n + nm + 3) / 4;
    cb = D == 2 ? 0 : (nused + 31) / 32 * 8;
    ordf = kFrameOps * 16 + up(4 * (kRawLayers + 1));  // a window of ops, one of layers
    ordc = ordf + (size_t)fb * sizeof(CoinOrdinal);
    thr = ordc + (size_t)cb * sizeof(CoinOrdinal);
    warp0 = thr + (size_t)cb * 16;
    x = 0;
    z = x + up((size_t)n * sizeof(T));
    rec = z + up((size_t)n * sizeof(T));
    fire = rec + up((size_t)nm * sizeof(T));
    warp = fire + up(D == 2 ? (size_t)nchunk * 8 + (size_t)cap * 8 : (size_t)nused * 2 * sizeof(T));
  }
};

template <int D>
__global__ void __launch_bounds__(128) k_rows_frame(const RowFrameDesc fd) {
  extern __shared__ __align__(16) uint8_t smem[];
  using E_ = El<D>;
  using T = typename E_::T;
  const FrameSmem<D> L_(fd.n, fd.nm, fd.nused, fd.nchunk, fd.cap);
  const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, warp = t >> 5;
  const int n = fd.n, nm = fd.nm;
  uint4* wops = reinterpret_cast<uint4*>(smem);
  uint32_t* wlay = reinterpret_cast<uint32_t*>(smem + kFrameOps * 16);
  CoinOrdinal* ordf = reinterpret_cast<CoinOrdinal*>(smem + L_.ordf);
  CoinOrdinal* ordc = reinterpret_cast<CoinOrdinal*>(smem + L_.ordc);
  uint32_t* thr = reinterpret_cast<uint32_t*>(smem + L_.thr);
  uint8_t* mem = smem + L_.warp0 + warp * L_.warp;
  T* X = reinterpret_cast<T*>(mem + L_.x);
  T* Z = reinterpret_cast<T*>(mem + L_.z);
  T* rec = reinterpret_cast<T*>(mem + L_.rec);  // the z drawn after a measurement, then its record word
  uint32_t* bm = reinterpret_cast<uint32_t*>(mem + L_.fire);  // d = 2: fired ordinals, entries before the chunk, entries
  uint2* ent = reinterpret_cast<uint2*>(bm + 2 * fd.nchunk);
  T* fire = reinterpret_cast<T*>(mem + L_.fire);  // odd d: x and z words of every ordinal
  const PhiloxKeys K(fd.seed);
  for (int i = t; i < L_.fb; i += nt) ordf[i] = coin_ordinal(K, (uint32_t)i, 0u, 3u);
  for (int i = t; i < L_.cb; i += nt) ordc[i] = coin_ordinal(K, (uint32_t)i, 0u, 1u);
  for (int i = t; i < 4 * L_.cb; i += nt) thr[i] = i < fd.nused ? __ldg(&fd.nhdr[i].x) : 0xffffffffu;
  __syncthreads();
  const long long first = ((long long)blockIdx.x * (nt >> 5) + warp) * 32;  // of the launch's shots
  const long long rel = first + lane;
  const bool live = rel < fd.nshots;
  const uint32_t shot = (uint32_t)(fd.shot0 + rel);  // shots are below 2^32: shot_hi 0
  const uint2 sh = coin_shot(K, shot, 0u);
  // frame draws: z of qudit e at the start (e < n), after measurement e - n;
  // four blocks' chains side by side
#pragma unroll 4
  for (int b = 0; b < L_.fb; ++b) {
    const uint4 w = coin_block(K, ordf[b], sh);
    const uint32_t v[4] = {w.x, w.y, w.z, w.w};
    T mine = E_::zero();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = mulshift(v[q], D);
      T word;
      if constexpr (D == 2) {
        word = __ballot_sync(0xffffffffu, r);
      } else if constexpr (D == 3) {
        word = make_uint2(__ballot_sync(0xffffffffu, r == 1), __ballot_sync(0xffffffffu, r == 2));
      } else {
        word = make_uint4(__ballot_sync(0xffffffffu, r & 1), __ballot_sync(0xffffffffu, r & 2),
                          __ballot_sync(0xffffffffu, r & 4), 0u);
      }
      if (lane == q) mine = word;
    }
    const int e = 4 * b + lane;
    if (lane < 4 && e < n + nm) {
      if (e < n) Z[e] = mine; else rec[e - n] = mine;
    }
  }
  for (int q = lane; q < n; q += 32) X[q] = E_::zero();
  // N1 samples
  if constexpr (D == 2) {
    int total = 0;
    for (int c0 = 0; c0 < fd.nchunk; c0 += 8) {  // eight loads in flight
      uint2 mq[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        mq[q] = make_uint2(0u, 0u);
        if (live && c0 + q < fd.nchunk) mq[q] = __ldcs(fd.masks + (size_t)(c0 + q) * fd.mshots + fd.mrel + rel);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint2 m = mq[q];
        const uint32_t any = __reduce_or_sync(0xffffffffu, m.x | m.y);
        if (lane == 0 && c0 + q < fd.nchunk) {
          bm[c0 + q] = any;
          bm[fd.nchunk + c0 + q] = (uint32_t)total;
        }
        for (uint32_t a = any; a; a &= a - 1u, ++total) {
          const int i = __ffs(a) - 1;
          const uint32_t fx = __ballot_sync(0xffffffffu, (m.x >> i) & 1u);
          const uint32_t fz = __ballot_sync(0xffffffffu, (m.y >> i) & 1u);
          if (lane == 0 && total < fd.cap) ent[total] = make_uint2(fx, fz);
        }
      }
    }
  } else {
    for (int i = lane; i < 2 * fd.nused; i += 32) fire[i] = E_::zero();
    __syncwarp();
    for (int b0 = 0; b0 < L_.cb; b0 += 8) {  // 32 ordinals' coins, then their few fires
      uint32_t f = 0u;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const uint4 w = coin_block(K, ordc[b0 + b], sh), th = reinterpret_cast<const uint4*>(thr)[b0 + b];
        f |= ((uint32_t)(w.x >= th.x) | ((uint32_t)(w.y >= th.y) << 1) | ((uint32_t)(w.z >= th.z) << 2) |
              ((uint32_t)(w.w >= th.w) << 3)) << (4 * b);
      }
      while (live && f) {
        const int j = 4 * b0 + __ffs(f) - 1;
        f &= f - 1u;
        // a coin of 0xffffffff meets the threshold of an ordinal that never fires
        const uint32_t op = j < fd.nused ? __ldg(&fd.nhdr[j].y) : (uint32_t)OP_N1OFF;
        if (op == OP_N1OFF) continue;
        const int2 ab = noise_choice(op, D, fd.seed, (long long)shot, (uint32_t)j);
        E_::put(fire + 2 * j, lane, ab.x);
        E_::put(fire + 2 * j + 1, lane, ab.y);
      }
    }
  }
  __syncwarp();
  // words (x, z) of N1 ordinal j
  auto sample = [&](uint32_t j, T& fx, T& fz) {
    if constexpr (D == 2) {
      const uint32_t b = bm[j >> 5], i = j & 31u;
      fx = fz = 0u;
      if (!((b >> i) & 1u)) return;
      const uint32_t k = bm[fd.nchunk + (j >> 5)] + (uint32_t)__popc(b & ((1u << i) - 1u));
      if (k < (uint32_t)fd.cap) {
        fx = ent[k].x;
        fz = ent[k].y;
      } else {  // more fires than entries: gather the word from the masks
        for (int s = 0; s < 32 && first + s < fd.nshots; ++s) {
          const uint2 m = __ldg(fd.masks + (size_t)(j >> 5) * fd.mshots + fd.mrel + first + s);
          fx |= ((m.x >> i) & 1u) << s;
          fz |= ((m.y >> i) & 1u) << s;
        }
      }
    } else {
      fx = fire[2 * j];
      fz = fire[2 * j + 1];
    }
  };
  // the layers; a window's ops are staged for all warps, their N1 riders turned
  // from row numbers into ordinals + 1
  auto ordinal = [&](uint32_t r) { return r ? (__ldg(&fd.xinfo[r - 1u].y) & 0x3fffffffu) + 1u : 0u; };
  auto staged = [&](uint32_t k) {
    uint4 o = __ldg(fd.ops + k);
    if (o.x & kRopN) {
      if (!(o.x & kRopM)) o.z = ordinal(o.z);
      o.w = ordinal(o.w);
    }
    return o;
  };
  auto step = [&](const uint4 o) {
    const uint32_t w = o.x;
    const int i = (int)(w & 0x7ffu), j = (int)((w >> 11) & 0x7ffu);
    const T xa = X[i], za = Z[i], xb = X[j], zb = Z[j];
    const bool mh = w & (kRopH | kRopHInv), mc = w & (kRopC | kRopCInv);
    T nx, nz, nt = xb, zt = zb;
    if constexpr (D == 2) {
      nx = mh ? za : xa;
      nz = mh ? xa : za ^ (mc ? zb : (w & (kRopP | kRopPInv)) ? xa : 0u);
      nt = xb ^ (mc ? xa : 0u);
    } else {
      using U = Unit<D>;
      const uint32_t vh = lane_mask(mh), vc = lane_mask(mc);
      const uint32_t mt = lane_mask(w & (kRopC | kRopCInv | kRopP | kRopPInv)), mn = lane_mask(w & (kRopC | kRopPInv));
      const T t0 = U::pick(vc, zb, xa);
      const T tt = U::mask(U::pick(mn, U::neg(t0), t0), mt);
      const T xn = U::neg(xa), zn = U::neg(za);
      nt = U::add(xb, U::mask(U::pick(lane_mask(w & kRopCInv), xn, xa), vc));
      nz = U::pick(vh, U::pick(lane_mask(w & kRopHInv), xn, xa), U::add(za, tt));
      nx = U::pick(vh, U::pick(lane_mask(w & kRopH), zn, za), xa);
    }
    if (w & kRopM) {
      const bool reset = w & kRopReset;
      nz = rec[o.y];
      rec[o.y] = reset ? E_::zero() : nx;  // RESET records the reference value itself
      if (reset) nx = E_::zero();
    }
    if (w & kRopN) {
      T fx, fz;
      const uint32_t a = (w & kRopM) ? o.w : o.z;
      if (a) {
        sample(a - 1u, fx, fz);
        nx = E_::add(nx, fx);
        nz = E_::add(nz, fz);
      }
      if (mc && o.w) {
        sample(o.w - 1u, fx, fz);
        nt = E_::add(nt, fx);
        zt = E_::add(zb, fz);
      }
    }
    X[i] = nx;
    Z[i] = nz;
    if (mc) {
      X[j] = nt;
      Z[j] = zt;
    }
  };
  int l = 0;
  while (l < fd.nlayers) {
    __syncthreads();
    const int nl = min(kRawLayers, fd.nlayers - l);
    for (int i = t; i <= nl; i += nt) wlay[i] = __ldg(fd.lay + l + i);
    __syncthreads();
    const uint32_t w0 = wlay[0], wend = min(wlay[nl], w0 + (uint32_t)kFrameOps);
    for (uint32_t i = w0 + t; i < wend; i += nt) wops[i - w0] = staged(i);
    __syncthreads();
    int i = 0;
    uint32_t b = w0;
    for (; i < nl; ++i) {
      const uint32_t e = wlay[i + 1];
      const bool in = e <= wend;
      if (!in && i > 0) break;
      for (uint32_t k = b + lane; k < e; k += 32) step(in ? wops[k - w0] : staged(k));
      b = e;
      __syncwarp();
    }
    l += i;
  }
  if (first < fd.nshots) {
    T* out = reinterpret_cast<T*>(fd.words) + (size_t)(first / 32) * nm;
    for (int k = lane; k < nm; k += 32) out[k] = rec[k];
  }
}

// 32 words, one a lane: bit s of lane k becomes bit k of lane s.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, o);
    x = (lane & o) ? (x & ~m) | ((y & ~m) >> o) : (x & m) | ((y & m) << o);
    m ^= m << (o >> 1);
  }
  return x;
}

// Words of a shot's record bits in the shared memory of a frame-output warp
// (odd, one to spare), and the bytes of the warp.
__host__ __device__ inline int frame_out_words(int nm) { return ((nm + 31) / 32 + 1) | 1; }
template <int D>
__host__ __device__ inline size_t frame_out_bytes(int nm) {
  constexpr int planes = D == 2 ? 1 : D == 3 ? 2 : 3;
  return ((size_t)32 * planes + 1) * frame_out_words(nm) * 4;
}
constexpr size_t kFrameOutMost = 12288;  // of a warp: four of them need no opt-in

// Records of 32 shots a warp: the reference shot's value added to the frame
// words as they are, measurement-major; then 32 x 32 bits at a time turned
// round, and out in 16-byte pieces.  A pass of its own, so that the frame pass
// runs beside the reference shot and not behind it.  Rows too long for the
// shared memory leave as bytes, a lane to a measurement.
// Bound by its instructions, and the stores: 100,000 shots of 385 measurements
// of d = 2 19 us (6 us of it the records' bytes); as the end of the frame pass, a
// byte per store, the step 355 us, so 338; 10,000 qutrit shots into host memory 420
// us and 348.
template <int D>
__global__ void __launch_bounds__(128) k_rows_frame_out(const RowFrameDesc fd) {
  extern __shared__ __align__(16) uint8_t smem[];
  using E_ = El<D>;
  using T = typename E_::T;
  constexpr int P = D == 2 ? 1 : D == 3 ? 2 : 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nm = fd.nm;
  const long long group = (long long)blockIdx.x * 4 + warp, first = 32 * group;
  if (first >= fd.nshots) return;
  const int rows = (int)min(32LL, (long long)fd.nshots - first);
  const T* words = reinterpret_cast<const T*>(fd.words) + (size_t)group * nm;
  uint8_t* out = fd.out + first * (long long)nm;
  const bool whole = frame_out_bytes<D>(nm) <= kFrameOutMost;
  const int S = frame_out_words(nm);
  uint32_t* bits = reinterpret_cast<uint32_t*>(smem) + (size_t)warp * (32 * P + 1) * S;
  uint32_t* det = bits + 32 * P * S;
  for (int k0 = 0; k0 < nm; k0 += 32) {
    const int k = k0 + lane, ref = k < nm ? __ldg(fd.ref + k) : 0, v0 = ref & 0x7f;
    T x = k < nm ? words[k] : E_::zero();
    if constexpr (D == 2) {
      x ^= lane_mask(v0);
    } else if constexpr (D == 3) {
      x = E_::add(x, make_uint2(lane_mask(v0 == 1), lane_mask(v0 == 2)));
    } else {
      x = E_::add(x, make_uint4(lane_mask(v0 & 1), lane_mask(v0 & 2), lane_mask(v0 & 4), 0u));
      if constexpr (D == 7) {  // 0 as 111
        const uint32_t all = x.x & x.y & x.z;
        x = make_uint4(x.x & ~all, x.y & ~all, x.z & ~all, 0u);
      }
    }
    if (whole) {
      uint32_t* b = bits + lane * S + (k0 >> 5);
      if constexpr (D == 2) {
        b[0] = transpose32(x, lane);
      } else {
        b[0] = transpose32(x.x, lane);
        b[32 * S] = transpose32(x.y, lane);
        if constexpr (D != 3) b[64 * S] = transpose32(x.z, lane);
      }
      const uint32_t d = __ballot_sync(0xffffffffu, ref & 0x80);
      if (lane == 0) det[k0 >> 5] = d;
    } else if (k < nm) {
      for (int s = 0; s < rows; ++s) out[(size_t)s * nm + k] = (uint8_t)(E_::get(x, s) | (ref & 0x80));
    }
  }
  if (!whole) return;
  __syncwarp();
  store_records<P>(out, rows, nm, lane, bits, S, det);
}

template <int D>
size_t raw_smem(int n, int lg) {
  return round16(raw_bytes<D>(n, lg));
}

// Chain-pass instances, by row_slice (4 for d = 2 alone, kRowSliceSmall for odd d).
template <int D, class Fn>
cudaError_t for_slice(int slice, Fn fn) {
  using std::integral_constant;
  if constexpr (D == 2) {
    if (slice == 4) return fn(integral_constant<int, 4>(), std::true_type());
  } else {
    if (slice == kRowSliceSmall) return fn(integral_constant<int, 1>(), std::false_type());
  }
  switch (slice) {
    case 1: return fn(integral_constant<int, 1>(), std::true_type());
    case 2: return fn(integral_constant<int, 2>(), std::true_type());
    case kRowSliceMid:
    case 16 + 2: return fn(integral_constant<int, 2>(), std::false_type());
    default: return fn(integral_constant<int, 4>(), std::false_type());
  }
}
constexpr int kSlices[] = {1, 2, 4, kRowSliceSmall, kRowSliceMid, 20};

template <int D>
cudaError_t set_smem(int optin) {
  cudaError_t e = set_dynamic_smem(k_rows_raw<D>, optin);
  for (int sl : kSlices)
    if (e == cudaSuccess)
      e = for_slice<D>(sl, [&](auto c, auto solo) { return set_dynamic_smem(k_rows_chain<D, c.value, solo.value>, optin); });
  if (e == cudaSuccess) e = set_dynamic_smem(k_rows_phase<D, 1>, optin);
  if (e == cudaSuccess) e = set_dynamic_smem(k_rows_phase<D, 2>, optin);
  if (e == cudaSuccess) e = set_dynamic_smem(k_rows_phase<D, 4>, optin);
  if (e == cudaSuccess) e = set_dynamic_smem(k_rows_frame<D>, optin);
  return e != cudaSuccess ? e : set_dynamic_smem(k_rows_extra<D>, optin);
}

template <int D>
cudaError_t chain(int slice, int C, int block, int rawt, int lg, size_t smem, cudaStream_t s, const RowDesc* descs,
                  int nd) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(C * nd));
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeClusterDimension;
  a.val.clusterDim.x = (unsigned)C;
  a.val.clusterDim.y = a.val.clusterDim.z = 1;
  cfg.attrs = &a;
  cfg.numAttrs = C > 1 ? 1 : 0;
  return for_slice<D>(slice, [&](auto c, auto solo) {
    return cudaLaunchKernelEx(&cfg, k_rows_chain<D, c.value, solo.value>, descs, nd, C, rawt, lg);
  });
}

}  // namespace

// The instance of one d, as rows.cuh's launchers see it.
template <int D>
RowOps row_ops() {
  RowOps o;
  o.set_smem = set_smem<D>;
  o.raw_smem = raw_smem<D>;
  o.chain_smem = [](int n, int block) { return (size_t)round16(ChainSmem<D>::total(row_elems(n), block / 32)); };
  o.extra_smem = [](int n) { return (size_t)round16(ExtraSmem<D>::total(row_elems(n))); };
  o.extra_per_cta = [](int n) { return extra_rows<D>(row_elems(n)); };
  o.raw = [](int tiles, int block, int lg, size_t smem, cudaStream_t s, const RowDesc* descs, int nd) {
    k_rows_raw<D><<<tiles, block, smem, s>>>(descs, nd, lg);
  };
  o.chain = chain<D>;
  o.extra = [](bool close, int ctas, size_t smem, cudaStream_t s, const RowDesc* descs, int nd) {
    launch_following(close, k_rows_extra<D>, ctas, 32 * kRowWarps, smem, s, descs, nd);
  };
  o.phase = [](bool close, int wpl, int blocks, size_t smem, cudaStream_t s, const RowPhaseDesc* descs, int nd) {
    launch_following(close, wpl == 1 ? k_rows_phase<D, 1> : wpl == 2 ? k_rows_phase<D, 2> : k_rows_phase<D, 4>, blocks,
                     128, smem, s, descs, nd);
  };
  o.frame_smem = [](const RowFrameDesc& f, int warps) {
    const FrameSmem<D> l(f.n, f.nm, f.nused, f.nchunk, f.cap);
    return l.warp0 + (size_t)warps * l.warp;
  };
  o.frame = [](int blocks, int warps, size_t smem, cudaStream_t s, const RowFrameDesc& f) {
    k_rows_frame<D><<<blocks, 32 * warps, smem, s>>>(f);
  };
  o.frame_out = [](cudaStream_t s, const RowFrameDesc& f) {
    const size_t b = frame_out_bytes<D>(f.nm);
    k_rows_frame_out<D><<<(f.nshots + 127) / 128, 128, b <= kFrameOutMost ? 4 * b : 0, s>>>(f);
  };
  return o;
}

}  // namespace sdim
