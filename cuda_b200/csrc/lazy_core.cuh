// Lazily reduced transforms of up to 16 points with power-of-two roots: the
// register butterflies of the pass kernels (smem_passes.cuh).
//
// Between the general multiplications of a pass nothing needs a residue in
// [0, p).  Here a value inside a butterfly network is a signed 96-bit integer in
// three 32-bit words (W3), congruent to the residue: an addition is one carry
// chain of three instructions and no correction, a multiplication by 2^24, 2^48
// or 2^72 a few shifts with 2^96 = -1 and 2^64 = 2^32 - 1 folded in.  A word is
// brought back below 2^64 once per pass (reduce), congruent but not canonical:
// every consumer is a product or another network, which take any 64-bit word.
//
// Cost of an 8-point transform: 72 instructions of additions, 42 of shifts, 51 of bias and
// reduction, against 273 with canonical additions (ntt_core.cuh).  The kernels are bound by
// integer issue (ALU and multiplier pipes 50-65 % busy, HBM 14 %): at n = 2^23 a squaring took
// 441.2 us with canonical values and takes 363.1 us with these (row_square 210.5 -> 161.5,
// col_fused 240.8 -> 212.2); n = 2048 on one SM 10.15 -> 8.99 us.
//
// Ranges.  Inputs of a network: |x| <= 2^65 (a 64-bit word, or the three words of
// mul3, in (-2^32, 2^65)); a sum of two words is too large.  Then, for 16 points:
// - a first 4-point step leaves at most 2^67 (s0 +- s1), or 1.5 2^66 + 2^33 where one of its
//   terms came from mul_2_48 (which leaves 2^65 + 2^33);
// - times 2^24 that is at most 2^91; the second bound times 2^12, plus a term below 2^66, stays below
//   the 2^79 that mul_2_48 takes; mul_mid<60>, which takes 2^67, sees the second bound only, and
//   mul_mid<36>, mul_2_72 and mul_high<84> take 2^75 and more;
// - at most one term of an output is a multiple of 2^24, so without the bias its magnitude is
//   below 2^92.
// Fewer points leave less.  The bias kBias p (2^28 p, congruent to 0) is added to input 0, which
// reaches every output with coefficient +1 and is never multiplied, so every output is
// non-negative and below 2^93: three words never overflow.
//
// On the host the same formulas run on 128-bit integers and check those ranges
// (tests/native/lazy_selftest.cpp).
#pragma once
#include <stdint.h>

#include "goldilocks.cuh"

namespace lnt {
namespace lazy {

// a0 + a1 2^32 + a2 2^64 with a2 signed
struct W3 {
  uint32_t a0, a1, a2;
};

constexpr uint32_t kBias = 1u << 28;
#if !defined(__CUDA_ARCH__)
constexpr __int128 kInputBound = (__int128)1 << 65;
#endif

GL_HD W3 from_word(uint64_t x) { return {(uint32_t)x, (uint32_t)(x >> 32), 0u}; }

#if !defined(__CUDA_ARCH__)
inline __int128 to_int(const W3& x) {
  return ((__int128)(int32_t)x.a2 << 64) + (__int128)(((uint64_t)x.a1 << 32) | x.a0);
}
// a value outside 96 bits is an error of the ranges above; the selftest reads this
inline bool& range_error() {
  static bool bad = false;
  return bad;
}
inline W3 from_int(__int128 v) {
  const __int128 lim = (__int128)1 << 95;
  if (v >= lim || v < -lim) range_error() = true;
  return {(uint32_t)v, (uint32_t)(v >> 32), (uint32_t)(v >> 64)};
}
#endif

GL_HD W3 add(const W3& x, const W3& y) {
#if defined(__CUDA_ARCH__)
  W3 r;
  asm("add.cc.u32 %0, %3, %6;\n\t"
      "addc.cc.u32 %1, %4, %7;\n\t"
      "addc.u32 %2, %5, %8;"
      : "=r"(r.a0), "=r"(r.a1), "=r"(r.a2)
      : "r"(x.a0), "r"(x.a1), "r"(x.a2), "r"(y.a0), "r"(y.a1), "r"(y.a2));
  return r;
#else
  return from_int(to_int(x) + to_int(y));
#endif
}

GL_HD W3 sub(const W3& x, const W3& y) {
#if defined(__CUDA_ARCH__)
  W3 r;
  asm("sub.cc.u32 %0, %3, %6;\n\t"
      "subc.cc.u32 %1, %4, %7;\n\t"
      "subc.u32 %2, %5, %8;"
      : "=r"(r.a0), "=r"(r.a1), "=r"(r.a2)
      : "r"(x.a0), "r"(x.a1), "r"(x.a2), "r"(y.a0), "r"(y.a1), "r"(y.a2));
  return r;
#else
  return from_int(to_int(x) - to_int(y));
#endif
}

// x + kBias p
GL_HD W3 add_bias(const W3& x) {
  return add(x, W3{kBias, 0u - kBias, kBias - 1u});
}

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ uint32_t sign_word(uint32_t a2) { return (uint32_t)((int32_t)a2 >> 31); }
#endif

// x 2^S for S < 32, |x| < 2^(95 - S)
template <int S>
GL_HD W3 mul_low(const W3& x) {
  static_assert(S > 0 && S < 32, "shift range");
#if defined(__CUDA_ARCH__)
  return {x.a0 << S, __funnelshift_l(x.a0, x.a1, S), __funnelshift_l(x.a1, x.a2, S)};
#else
  return from_int(to_int(x) * ((__int128)1 << S));
#endif
}
GL_HD W3 mul_2_24(const W3& x) { return mul_low<24>(x); }

// x 2^S for 32 < S < 64, |x| < 2^(127 - S); the result is below 2^65 + 2^33 in magnitude.  With
// (l2 : l1 : l0) = x 2^(S - 32) it is l0 2^32 + l1 2^64 + l2 2^96 = l0 2^32 + l1 (2^32 - 1) - l2.
template <int S>
GL_HD W3 mul_mid(const W3& x) {
  static_assert(S > 32 && S < 64, "shift range");
#if defined(__CUDA_ARCH__)
  const uint32_t l0 = x.a0 << (S - 32), l1 = __funnelshift_l(x.a0, x.a1, S - 32),
                 l2 = __funnelshift_l(x.a1, x.a2, S - 32);
  const uint32_t sg = sign_word(x.a2);
  W3 r;
  asm("mad.lo.cc.u32  %0, %4, 0xFFFFFFFF, 0;\n\t"
      "madc.hi.cc.u32 %1, %4, 0xFFFFFFFF, %3;\n\t"
      "addc.u32       %2, 0, 0;\n\t"
      "sub.cc.u32     %0, %0, %5;\n\t"
      "subc.cc.u32    %1, %1, %6;\n\t"
      "subc.u32       %2, %2, %6;"
      : "=&r"(r.a0), "=&r"(r.a1), "=&r"(r.a2)
      : "r"(l0), "r"(l1), "r"(l2), "r"(sg));
  return r;
#else
  const __int128 l = to_int(x) * ((__int128)1 << (S - 32));
  from_int(l);
  const __int128 l0 = (uint32_t)l, l1 = (uint32_t)(l >> 32), l2 = l >> 64;
  return from_int((l0 << 32) + l1 * 0xFFFFFFFFll - l2);
#endif
}
GL_HD W3 mul_2_48(const W3& x) { return mul_mid<48>(x); }

// x 2^S for 64 < S < 96, |x| < 2^(159 - S); the result is below 2^65 in magnitude.  With
// (e2 : e1 : e0) = x 2^(S - 64) it is e0 2^64 + e1 2^96 + e2 2^128 = (e0 - e2) 2^32 - e0 - e1.
template <int S>
GL_HD W3 mul_high(const W3& x) {
  static_assert(S > 64 && S < 96, "shift range");
#if defined(__CUDA_ARCH__)
  const uint32_t e0 = x.a0 << (S - 64), e1 = __funnelshift_l(x.a0, x.a1, S - 64),
                 e2 = __funnelshift_l(x.a1, x.a2, S - 64);
  const uint32_t sg = sign_word(x.a2);
  W3 r;
  asm("sub.cc.u32  %0, 0, %3;\n\t"
      "subc.cc.u32 %1, %3, %5;\n\t"
      "subc.u32    %2, 0, %6;\n\t"
      "sub.cc.u32  %0, %0, %4;\n\t"
      "subc.cc.u32 %1, %1, 0;\n\t"
      "subc.u32    %2, %2, 0;"
      : "=&r"(r.a0), "=&r"(r.a1), "=&r"(r.a2)
      : "r"(e0), "r"(e1), "r"(e2), "r"(sg));
  return r;
#else
  const __int128 e = to_int(x) * ((__int128)1 << (S - 64));
  from_int(e);
  const __int128 e0 = (uint32_t)e, e1 = (uint32_t)(e >> 32), e2 = e >> 64;
  return from_int((e0 - e2) * ((__int128)1 << 32) - e0 - e1);
#endif
}
GL_HD W3 mul_2_72(const W3& x) { return mul_high<72>(x); }

// 0 <= x < 2^95 to a congruent 64-bit word: (a1 : a0) + a2 (2^32 - 1), whose carry c
// comes back as c (2^32 - 1): with c = 1 the wrapped sum is below 2^63, so that cannot wrap.
GL_HD uint64_t reduce(const W3& x) {
#if defined(__CUDA_ARCH__)
  uint32_t t0, t1;
  asm("{\n\t"
      ".reg .u32 c;\n\t"
      "mad.lo.cc.u32  %0, %4, 0xFFFFFFFF, %2;\n\t"
      "madc.hi.cc.u32 %1, %4, 0xFFFFFFFF, %3;\n\t"
      "addc.u32       c, 0, 0;\n\t"
      "add.u32        %1, %1, c;\n\t"
      "sub.cc.u32     %0, %0, c;\n\t"
      "subc.u32       %1, %1, 0;\n\t"
      "}"
      : "=&r"(t0), "=&r"(t1)
      : "r"(x.a0), "r"(x.a1), "r"(x.a2));
  return ((uint64_t)t1 << 32) | t0;
#else
  const __int128 v = to_int(x);
  if (v < 0) range_error() = true;
  const __int128 s = (v & (((__int128)1 << 64) - 1)) + (v >> 64) * 0xFFFFFFFFll;
  const __int128 r = (s & (((__int128)1 << 64) - 1)) + (s >> 64) * 0xFFFFFFFFll;
  if (r >> 64) range_error() = true;
  return (uint64_t)r;
#endif
}

// x in (-p, 2^65 - 2^33] (a2 = -1, 0 or 1) to a congruent 64-bit word:
// (a1 : a0) + a2 (2^32 - 1), which can neither carry nor borrow again.
GL_HD uint64_t fold(const W3& x) {
#if defined(__CUDA_ARCH__)
  const uint32_t sg = sign_word(x.a2);
  uint32_t t0, t1;
  asm("{\n\t"
      "add.u32     %1, %3, %4;\n\t"
      "sub.cc.u32  %0, %2, %4;\n\t"
      "subc.u32    %1, %1, %5;\n\t"
      "}"
      : "=&r"(t0), "=&r"(t1)
      : "r"(x.a0), "r"(x.a1), "r"(x.a2), "r"(sg));
  return ((uint64_t)t1 << 32) | t0;
#else
  const __int128 v = to_int(x);
  const __int128 r = (v & (((__int128)1 << 64) - 1)) + (v >> 64) * 0xFFFFFFFFll;
  if (r < 0 || (r >> 64)) range_error() = true;
  return (uint64_t)r;
#endif
}

// a b for any 64-bit words, in (-2^32, 2^65 - 2^33]: with the product's 32-bit words r0..r3,
// (r1 : r0) + r2 (2^32 - 1) - r3.  The outer products are plain wide ones and the cross
// products one chain with a carry, added in on the integer ALU: 17 instructions with the fold of
// mul, against 22 when every partial product is a multiply-add of the one before (the
// multiplier pipe is the fuller one there); at n = 2^23 363.1 against 375.4 us a squaring.
GL_HD W3 mul3(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  W3 t;
  asm("{\n\t"
      ".reg .u32 r0, r1, r2, r3, u0, u1;\n\t"
      ".reg .u64 q0, q3;\n\t"
      "mul.wide.u32   q0, %3, %5;\n\t"
      "mul.wide.u32   q3, %4, %6;\n\t"
      "mul.lo.u32     u0, %3, %6;\n\t"
      "mul.hi.u32     u1, %3, %6;\n\t"
      "mov.b64        {r0, r1}, q0;\n\t"
      "mov.b64        {r2, r3}, q3;\n\t"
      "mad.lo.cc.u32  u0, %4, %5, u0;\n\t"
      "madc.hi.cc.u32 u1, %4, %5, u1;\n\t"
      "addc.u32       r3, r3, 0;\n\t"
      "add.cc.u32     r1, r1, u0;\n\t"
      "addc.cc.u32    r2, r2, u1;\n\t"
      "addc.u32       r3, r3, 0;\n\t"
      "mad.lo.cc.u32  %0, r2, 0xFFFFFFFF, r0;\n\t"
      "madc.hi.cc.u32 %1, r2, 0xFFFFFFFF, r1;\n\t"
      "addc.u32       %2, 0, 0;\n\t"
      "sub.cc.u32     %0, %0, r3;\n\t"
      "subc.cc.u32    %1, %1, 0;\n\t"
      "subc.u32       %2, %2, 0;\n\t"
      "}"
      : "=&r"(t.a0), "=&r"(t.a1), "=&r"(t.a2)
      : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"((uint32_t)b), "r"((uint32_t)(b >> 32)));
  return t;
#else
  const unsigned __int128 q = (unsigned __int128)a * b;
  const __int128 lo = (uint64_t)q, r2 = (uint32_t)(uint64_t)(q >> 64), r3 = (uint64_t)(q >> 96);
  return from_int(lo + r2 * 0xFFFFFFFFll - r3);
#endif
}

// a b as a 64-bit word (congruent, not canonical)
GL_HD uint64_t mul(uint64_t a, uint64_t b) { return fold(mul3(a, b)); }

// d w for a digit |d| < 2^32 and w in [1, p], as a 64-bit word: a 32 x 64-bit product (three
// words), of w or of p - w for a negative digit
GL_HD uint64_t mul_digit(int64_t d, uint64_t w) {
#if defined(__CUDA_ARCH__)
  const uint32_t a = (uint32_t)(d < 0 ? -d : d);
  const uint64_t s = d < 0 ? gl::P - w : w;
  W3 t;
  asm("mul.lo.u32    %0, %3, %4;\n\t"
      "mul.hi.u32    %1, %3, %4;\n\t"
      "mad.lo.cc.u32 %1, %3, %5, %1;\n\t"
      "madc.hi.u32   %2, %3, %5, 0;"
      : "=&r"(t.a0), "=&r"(t.a1), "=&r"(t.a2)
      : "r"(a), "r"((uint32_t)s), "r"((uint32_t)(s >> 32)));
  return reduce(t);  // whose sum also holds for a2 up to 2^32 - 1: wrapped it is below 2^64 - 2^33
#else
  return gl::mul_digit(d, w == gl::P ? 0 : w);
#endif
}

// ---- transforms: x (natural order, overwritten) -> out (bit-reversed order), and back ----

// natural in, bit-reversed out, root 2^(192/R)
template <int R>
GL_HD void dif(W3 (&x)[R], uint64_t (&out)[R]) {
  static_assert(R == 2 || R == 4 || R == 8 || R == 16, "register transform size");
  if constexpr (R == 2) {
    const W3 a = add_bias(x[0]);
    out[0] = reduce(add(a, x[1]));
    out[1] = reduce(sub(a, x[1]));
  } else if constexpr (R == 4) {
    const W3 a = add_bias(x[0]);
    const W3 s0 = add(a, x[2]), d0 = sub(a, x[2]), s1 = add(x[1], x[3]);
    const W3 d1 = mul_2_48(sub(x[1], x[3]));
    out[0] = reduce(add(s0, s1));
    out[1] = reduce(sub(s0, s1));
    out[2] = reduce(add(d0, d1));
    out[3] = reduce(sub(d0, d1));
  } else if constexpr (R == 8) {
    const W3 a = add_bias(x[0]);
    const W3 s0 = add(a, x[4]), d0 = sub(a, x[4]);
    const W3 s2 = add(x[2], x[6]), d2 = mul_2_48(sub(x[2], x[6]));
    const W3 s1 = add(x[1], x[5]), d1 = sub(x[1], x[5]);
    const W3 s3 = add(x[3], x[7]), d3 = sub(x[3], x[7]);
    {
      const W3 e0 = add(s0, s2), e1 = add(s1, s3);
      out[0] = reduce(add(e0, e1));
      out[1] = reduce(sub(e0, e1));
      const W3 e2 = sub(s0, s2), e3 = mul_2_48(sub(s1, s3));
      out[2] = reduce(add(e2, e3));
      out[3] = reduce(sub(e2, e3));
    }
    // frequencies 1, 5: 2^24 (d1 + 2^48 d3); 3, 7: 2^72 (d1 - 2^48 d3) = 2^72 d1 + 2^24 d3
    {
      const W3 f = add(d0, d2), y = add(mul_2_24(d1), mul_2_72(d3));
      out[4] = reduce(add(f, y));
      out[5] = reduce(sub(f, y));
    }
    {
      const W3 f = sub(d0, d2), y = add(mul_2_72(d1), mul_2_24(d3));
      out[6] = reduce(add(f, y));
      out[7] = reduce(sub(f, y));
    }
  } else {
    // 4 x 4: 4-point transforms at stride 4, twiddles 2^(12 k1 n2), 4-point transforms.  A twiddle
    // of 2^24 leaves 2^91, which 2^48 may not be applied to: the k1 = 2 column takes 2^72 and 2^24 of
    // the untwiddled values instead, as the 8-point transform does.
    W3 a[4][4];  // [k1][n2]
    x[0] = add_bias(x[0]);
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
      const W3 s0 = add(x[n2], x[n2 + 8]), d0 = sub(x[n2], x[n2 + 8]), s1 = add(x[n2 + 4], x[n2 + 12]);
      const W3 d1 = mul_2_48(sub(x[n2 + 4], x[n2 + 12]));
      a[0][n2] = add(s0, s1);
      a[2][n2] = sub(s0, s1);
      a[1][n2] = add(d0, d1);
      a[3][n2] = sub(d0, d1);
    }
    auto last = [&](const W3& b0, const W3& b2, const W3& sum13, const W3& diff13, int o) {
      const W3 s = add(b0, b2), d = sub(b0, b2);
      out[o] = reduce(add(s, sum13));
      out[o + 1] = reduce(sub(s, sum13));
      out[o + 2] = reduce(add(d, diff13));
      out[o + 3] = reduce(sub(d, diff13));
    };
    last(a[0][0], a[0][2], add(a[0][1], a[0][3]), mul_2_48(sub(a[0][1], a[0][3])), 0);
    last(a[2][0], mul_2_48(a[2][2]), add(mul_2_24(a[2][1]), mul_2_72(a[2][3])),
         add(mul_2_72(a[2][1]), mul_2_24(a[2][3])), 4);
    {
      const W3 b1 = mul_low<12>(a[1][1]), b3 = mul_mid<36>(a[1][3]);
      last(a[1][0], mul_2_24(a[1][2]), add(b1, b3), mul_2_48(sub(b1, b3)), 8);
    }
    {
      const W3 b1 = mul_mid<36>(a[3][1]), b3 = mul_low<12>(a[3][3]);  // 2^108 = -2^12
      last(a[3][0], mul_2_72(a[3][2]), sub(b1, b3), mul_2_48(add(b1, b3)), 12);
    }
  }
}

// bit-reversed in, natural out, inverse root, unscaled
template <int R>
GL_HD void dit_inv(W3 (&x)[R], uint64_t (&out)[R]) {
  static_assert(R == 2 || R == 4 || R == 8 || R == 16, "register transform size");
  if constexpr (R == 2) {
    dif<2>(x, out);
  } else if constexpr (R == 4) {
    const W3 a = add_bias(x[0]);
    const W3 p0 = add(a, x[1]), p1 = sub(a, x[1]), p2 = add(x[2], x[3]);
    const W3 p3 = mul_2_48(sub(x[2], x[3]));
    out[0] = reduce(add(p0, p2));
    out[2] = reduce(sub(p0, p2));
    out[1] = reduce(sub(p1, p3));
    out[3] = reduce(add(p1, p3));
  } else if constexpr (R == 8) {
    const W3 a = add_bias(x[0]);
    const W3 p0 = add(a, x[1]), p1 = sub(a, x[1]);
    const W3 p2 = add(x[2], x[3]), p3 = mul_2_48(sub(x[2], x[3]));
    const W3 q0 = add(x[4], x[5]), q1 = sub(x[4], x[5]);
    const W3 q2 = add(x[6], x[7]), q3 = sub(x[6], x[7]);
    {
      const W3 e = add(p0, p2), f = add(q0, q2);
      out[0] = reduce(add(e, f));
      out[4] = reduce(sub(e, f));
      const W3 g = sub(p0, p2), h = mul_2_48(sub(q0, q2));  // inverse twiddle 2^-48 = -2^48
      out[2] = reduce(sub(g, h));
      out[6] = reduce(add(g, h));
    }
    {
      // 2^-24 (q1 - 2^48 q3) = -2^72 (q1 - 2^48 q3) = -(2^72 q1 + 2^24 q3)
      const W3 e = sub(p1, p3), z = add(mul_2_72(q1), mul_2_24(q3));
      out[1] = reduce(sub(e, z));
      out[5] = reduce(add(e, z));
    }
    {
      // 2^-72 (q1 + 2^48 q3) = -2^24 (q1 + 2^48 q3) = -(2^24 q1 + 2^72 q3)
      const W3 e = add(p1, p3), z = add(mul_2_24(q1), mul_2_72(q3));
      out[3] = reduce(sub(e, z));
      out[7] = reduce(add(e, z));
    }
  } else {
    // the steps of dif<16> backwards; inverse twiddles 2^-e = -2^(96 - e), 2^-108 = 2^84
    W3 c[4][4];  // [k1][n2]
    x[0] = add_bias(x[0]);
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      const int k1 = (o >> 1) | ((o & 1) << 1);
      const W3 p0 = add(x[4 * o], x[4 * o + 1]), p1 = sub(x[4 * o], x[4 * o + 1]);
      const W3 p2 = add(x[4 * o + 2], x[4 * o + 3]), p3 = mul_2_48(sub(x[4 * o + 2], x[4 * o + 3]));
      c[k1][0] = add(p0, p2);
      c[k1][2] = sub(p0, p2);
      c[k1][1] = sub(p1, p3);
      c[k1][3] = add(p1, p3);
    }
    // s, d: terms 0 +- 2; sum13: terms 1 + 3; diff13: 2^48 (term 1 - term 3)
    auto last = [&](const W3& s, const W3& d, const W3& sum13, const W3& diff13, int o) {
      out[o] = reduce(add(s, sum13));
      out[o + 8] = reduce(sub(s, sum13));
      out[o + 4] = reduce(sub(d, diff13));
      out[o + 12] = reduce(add(d, diff13));
    };
    // the same with sum13 and diff13 negated
    auto last_neg = [&](const W3& s, const W3& d, const W3& sum13, const W3& diff13, int o) {
      out[o] = reduce(sub(s, sum13));
      out[o + 8] = reduce(add(s, sum13));
      out[o + 4] = reduce(add(d, diff13));
      out[o + 12] = reduce(sub(d, diff13));
    };
    last(add(c[0][0], c[2][0]), sub(c[0][0], c[2][0]), add(c[1][0], c[3][0]), mul_2_48(sub(c[1][0], c[3][0])), 0);
    {
      const W3 t2 = mul_2_72(c[2][1]), t1 = mul_high<84>(c[1][1]), t3 = mul_mid<60>(c[3][1]);
      last_neg(sub(c[0][1], t2), add(c[0][1], t2), add(t1, t3), mul_2_48(sub(t1, t3)), 1);
    }
    {
      // terms 1 + 3: -(2^72 c1 + 2^24 c3); 2^48 (term 1 - term 3): 2^24 c1 + 2^72 c3
      const W3 t2 = mul_2_48(c[2][2]), s = sub(c[0][2], t2), d = add(c[0][2], t2);
      const W3 f = add(mul_2_72(c[1][2]), mul_2_24(c[3][2])), g = add(mul_2_24(c[1][2]), mul_2_72(c[3][2]));
      out[2] = reduce(sub(s, f));
      out[10] = reduce(add(s, f));
      out[6] = reduce(sub(d, g));
      out[14] = reduce(add(d, g));
    }
    {
      const W3 t2 = mul_2_24(c[2][3]), t1 = mul_mid<60>(c[1][3]), t3 = mul_high<84>(c[3][3]);
      last_neg(sub(c[0][3], t2), add(c[0][3], t2), sub(t1, t3), mul_2_48(add(t1, t3)), 3);
    }
  }
}

// x 4, |x| < 2^93
GL_HD W3 mul_4(const W3& x) {
#if defined(__CUDA_ARCH__)
  return {x.a0 << 2, __funnelshift_l(x.a0, x.a1, 2), __funnelshift_l(x.a1, x.a2, 2)};
#else
  return from_int(to_int(x) * 4);
#endif
}

// Constants of dft5 from w = omega_5, with C1 = (w + w^4)/2, C2 = (w^2 + w^3)/2, S1 = (w - w^4)/2,
// S2 = (w^2 - w^3)/2: {2 (C1 - C2), 4 S2, 4 (S1 - S2), 4 (S1 + S2)}.
inline void dft5_constants(uint64_t w, uint64_t c[4]) {
  const uint64_t half = gl::inv(2), w2 = gl::mul(w, w), w3 = gl::mul(w2, w), w4 = gl::mul(w3, w);
  const uint64_t c1 = gl::mul(gl::add(w, w4), half), c2 = gl::mul(gl::add(w2, w3), half);
  const uint64_t s1 = gl::mul(gl::sub(w, w4), half), s2 = gl::mul(gl::sub(w2, w3), half);
  c[0] = gl::mul(2, gl::sub(c1, c2));
  c[1] = gl::mul(4, s2);
  c[2] = gl::mul(4, gl::sub(s1, s2));
  c[3] = gl::mul(4, gl::add(s1, s2));
}

// Four times the 5-point transform, |u| <= 2^65, in four general products.  With a1, b1 = u1 +- u4
// and a2, b2 = u2 +- u3 the outputs are u0 + a1 + a2 and u0 + t +- s for (t, s) = (a1 C1 + a2 C2,
// b1 S1 + b2 S2) and (a1 C2 + a2 C1, b1 S2 - b2 S1).  C1 + C2 = -1/2 leaves one product for both t
// (4 t = -(a1 + a2) +- 2 (a1 - a2)(C1 - C2)), three make both s.  The inverse transform is the same
// with outputs 1, 4 and 2, 3 exchanged; the factor 4 of each goes into the unweights.
GL_HD void dft5(const W3 (&u)[5], const uint64_t* c, uint64_t (&out)[5]) {
  const W3 a1 = add(u[1], u[4]), b1 = sub(u[1], u[4]);
  const W3 a2 = add(u[2], u[3]), b2 = sub(u[2], u[3]);
  const W3 a = add(a1, a2);
  const W3 e = mul3(reduce(add_bias(sub(a1, a2))), c[0]);
  const W3 m = mul3(reduce(add_bias(add(b1, b2))), c[1]);
  const W3 s1 = add(m, mul3(reduce(add_bias(b1)), c[2]));
  const W3 s2 = sub(m, mul3(reduce(add_bias(b2)), c[3]));
  const W3 q = add_bias(mul_4(u[0])), p = sub(q, a);
  out[0] = reduce(add(q, mul_4(a)));
  const W3 p1 = add(p, e), p2 = sub(p, e);
  out[1] = reduce(add(p1, s1));
  out[4] = reduce(sub(p1, s1));
  out[2] = reduce(add(p2, s2));
  out[3] = reduce(sub(p2, s2));
}
constexpr uint64_t kDft5Scale = 64;  // forward 4, squared 16, inverse 4

}  // namespace lazy
}  // namespace lnt
