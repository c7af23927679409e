// Goldilocks field arithmetic, p = 2^64 - 2^32 + 1, for sm_103a device code.
// The same source compiles for the host (portable C++ branches) so that the
// arithmetic and the generated codelets can be checked on a CPU; the device
// branches are hand-written PTX carry chains on 32-bit halves, because the
// integer pipes bound these kernels (IADD3/SEL/SHF/ISETP on the ALU pipe, the
// products' multiply-adds on the FMA pipe).
//
// Values at rest are canonical u64 in [0, p).  The reference keeps the
// Montgomery form x*2^64 mod p (ntt/src/field/mod.rs:12); every operation on the
// transform path is F_p-linear, so the kernels work on either representation
// unchanged.  Within a codelet values are three unreduced limbs ("lazy values").
//
// Multiplication is the 64x64->128 product followed by the reduction
// 2^64 = 2^32 - 1, 2^96 = -1 (mod p), restating reduce_159 of
// ntt/src/field/algo/generic.rs:77-108, or a Montgomery product by a table's
// word.  Multiplications by powers of two -- the twiddles of order dividing 192
// (generic.rs:171-193) -- shift the three limbs (gl_lshl).
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define GL_HD __host__ __device__ __forceinline__
#else
#define GL_HD inline
#endif

#define GL_P 0xffffffff00000001ull
#define GL_EPS 0x00000000ffffffffull  // 2^64 mod p

#if defined(__CUDA_ARCH__)
#define GL_DEV_PTX 1
__device__ __forceinline__ uint64_t gl_pack(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void gl_unpack(uint64_t x, uint32_t &lo, uint32_t &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(x));
}
// x >= p  <=>  hi == 0xffffffff and lo != 0; then x - p = lo - 1.
__device__ __forceinline__ uint64_t gl_canon32(uint32_t lo, uint32_t hi) {
  uint32_t r0, r1;
  asm("{\n\t.reg .pred q;\n\t"
      "setp.eq.u32 q, %3, 0xffffffff;\n\t"
      "setp.ne.and.u32 q, %2, 0, q;\n\t"
      "selp.u32 %1, 0, %3, q;\n\t"
      "sub.u32 %0, %2, 1;\n\t"
      "selp.u32 %0, %0, %2, q;\n\t}"
      : "=&r"(r0), "=&r"(r1) : "r"(lo), "r"(hi));
  return gl_pack(r0, r1);
}
#endif

GL_HD uint64_t gl_umulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// Any u64 -> canonical (one conditional subtraction of p).
GL_HD uint64_t gl_canon(uint64_t x) {
#ifdef GL_DEV_PTX
  uint32_t lo, hi;
  gl_unpack(x, lo, hi);
  return gl_canon32(lo, hi);
#else
  return x >= GL_P ? x - GL_P : x;
#endif
}

// a - b mod p for canonical a, b: on borrow add p, i.e. subtract EPS.
GL_HD uint64_t gl_sub(uint64_t a, uint64_t b) {
#ifdef GL_DEV_PTX
  uint32_t a0, a1, b0, b1, r0, r1, m;
  gl_unpack(a, a0, a1);
  gl_unpack(b, b0, b1);
  asm("sub.cc.u32 %0, %3, %5;\n\t"
      "subc.cc.u32 %1, %4, %6;\n\t"
      "subc.u32 %2, 0, 0;\n\t"      // m = borrow ? 0xffffffff : 0  (= borrow * EPS)
      "sub.cc.u32 %0, %0, %2;\n\t"
      "subc.u32 %1, %1, 0;"
      : "=&r"(r0), "=&r"(r1), "=&r"(m) : "r"(a0), "r"(a1), "r"(b0), "r"(b1));
  return gl_pack(r0, r1);
#else
  uint64_t d = a - b;
  return (a < b) ? d - GL_EPS : d;
#endif
}

// a + b mod p for canonical a, b, as a - (p - b) (generic.rs:19-26); p - b is
// exact in 64 bits (b = 0 gives p, which the borrow path handles).
GL_HD uint64_t gl_add(uint64_t a, uint64_t b) {
#ifdef GL_DEV_PTX
  uint32_t a0, a1, b0, b1, n0, n1, r0, r1, m;
  gl_unpack(a, a0, a1);
  gl_unpack(b, b0, b1);
  asm("sub.cc.u32 %2, 1, %7;\n\t"
      "subc.u32 %3, 0xffffffff, %8;\n\t"   // n = p - b
      "sub.cc.u32 %0, %5, %2;\n\t"
      "subc.cc.u32 %1, %6, %3;\n\t"
      "subc.u32 %4, 0, 0;\n\t"
      "sub.cc.u32 %0, %0, %4;\n\t"
      "subc.u32 %1, %1, 0;"
      : "=&r"(r0), "=&r"(r1), "=&r"(n0), "=&r"(n1), "=&r"(m)
      : "r"(a0), "r"(a1), "r"(b0), "r"(b1));
  return gl_pack(r0, r1);
#else
  uint64_t nb = GL_P - b;
  uint64_t r = a - nb;
  return (a < nb) ? r - GL_EPS : r;
#endif
}

GL_HD uint64_t gl_neg(uint64_t a) { return a ? GL_P - a : 0; }

// low + mid*2^64 + high*2^96 (mid < 2^32, high < 2^63) reduced to [0, p):
// low - high + mid*(2^32 - 1).  Restates generic.rs:77-108.
GL_HD uint64_t gl_reduce159(uint64_t low, uint64_t mid, uint64_t high) {
  uint64_t t = low - high;
  if (low < high) t -= GL_EPS;          // + p; cannot wrap again (high < 2^63)
  uint64_t u = (mid << 32) - mid;       // mid * EPS < 2^64
  uint64_t r = t + u;
  if (r < u) r += GL_EPS;               // + 2^64 = + EPS; cannot wrap again
  if (r >= GL_P) r -= GL_P;
  return r;
}

#ifdef GL_DEV_PTX
// value = (l1:l0) + h0*2^64 + h1*2^96 = (l1:l0) - h1 + h0*EPS (mod p), with
// h0, h1 < 2^32; canonical result.
__device__ __forceinline__ uint64_t gl_reduce_words(uint32_t l0, uint32_t l1, uint32_t h0,
                                                    uint32_t h1) {
  uint32_t t0, t1, m, u0, u1, c;
  asm("sub.cc.u32 %0, %6, %9;\n\t"       // t = l - h1
      "subc.cc.u32 %1, %7, 0;\n\t"
      "subc.u32 %2, 0, 0;\n\t"
      "sub.cc.u32 %0, %0, %2;\n\t"       // borrow: + p (t stays >= 0: l - h1 + 2^64 > EPS)
      "subc.u32 %1, %1, 0;\n\t"
      "sub.cc.u32 %3, 0, %8;\n\t"        // u = h0 * EPS = h0*2^32 - h0
      "subc.u32 %4, %8, 0;\n\t"
      "add.cc.u32 %0, %0, %3;\n\t"       // t += u
      "addc.cc.u32 %1, %1, %4;\n\t"
      "addc.u32 %5, 0, 0;\n\t"
      "sub.u32 %2, 0, %5;\n\t"           // carry: + EPS (cannot wrap again)
      "add.cc.u32 %0, %0, %2;\n\t"
      "addc.u32 %1, %1, 0;"
      : "=&r"(t0), "=&r"(t1), "=&r"(m), "=&r"(u0), "=&r"(u1), "=&r"(c)
      : "r"(l0), "r"(l1), "r"(h0), "r"(h1));
  return gl_canon32(t0, t1);
}
#endif

// (hi*2^64 + lo) mod p.
GL_HD uint64_t gl_reduce128(uint64_t lo, uint64_t hi) {
#ifdef GL_DEV_PTX
  uint32_t l0, l1, h0, h1;
  gl_unpack(lo, l0, l1);
  gl_unpack(hi, h0, h1);
  return gl_reduce_words(l0, l1, h0, h1);
#else
  return gl_reduce159(lo, hi & 0xffffffffull, hi >> 32);
#endif
}

GL_HD uint64_t gl_mul(uint64_t a, uint64_t b) {
#ifdef GL_DEV_PTX
  uint32_t a0, a1, b0, b1, l0, l1, h0, h1;
  gl_unpack(a, a0, a1);
  gl_unpack(b, b0, b1);
  asm("mul.lo.u32 %0, %4, %6;\n\t"
      "mul.hi.u32 %1, %4, %6;\n\t"
      "mul.lo.u32 %2, %5, %7;\n\t"
      "mul.hi.u32 %3, %5, %7;\n\t"
      "mad.lo.cc.u32 %1, %4, %7, %1;\n\t"
      "madc.hi.cc.u32 %2, %4, %7, %2;\n\t"
      "addc.u32 %3, %3, 0;\n\t"
      "mad.lo.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.hi.cc.u32 %2, %5, %6, %2;\n\t"
      "addc.u32 %3, %3, 0;"
      : "=&r"(l0), "=&r"(l1), "=&r"(h0), "=&r"(h1) : "r"(a0), "r"(a1), "r"(b0), "r"(b1));
  return gl_reduce_words(l0, l1, h0, h1);
#else
  return gl_reduce128(a * b, gl_umulhi(a, b));
#endif
}

// Montgomery product a*w*2^-64 mod p, for twiddles and constants stored in
// Montgomery form (w = t*2^64 mod p): then gl_mont_mul(a, w) = a*t mod p for
// any word a, whatever representation a is in.  The reduction follows
// mont_reduce_128 of ntt/src/field/algo/generic.rs:114-124: with the product
// x = x1*2^64 + x0, a = x0 + (x0 << 32) (carry e), b = a - (a >> 32) - e,
// result x1 - b (+ p on borrow).  b <= p - 1 for every x0, and x1 < p when
// w < p, so the result is canonical without a final correction: 9 ALU
// operations after the product against 18 for the canonical reduction.
GL_HD uint64_t gl_mont_mul(uint64_t a, uint64_t w) {
#ifdef GL_DEV_PTX
  uint32_t a0, a1, b0, b1, l0, l1, h0, h1;
  gl_unpack(a, a0, a1);
  gl_unpack(w, b0, b1);
  asm("mul.lo.u32 %0, %4, %6;\n\t"
      "mul.hi.u32 %1, %4, %6;\n\t"
      "mul.lo.u32 %2, %5, %7;\n\t"
      "mul.hi.u32 %3, %5, %7;\n\t"
      "mad.lo.cc.u32 %1, %4, %7, %1;\n\t"
      "madc.hi.cc.u32 %2, %4, %7, %2;\n\t"
      "addc.u32 %3, %3, 0;\n\t"
      "mad.lo.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.hi.cc.u32 %2, %5, %6, %2;\n\t"
      "addc.u32 %3, %3, 0;"
      : "=&r"(l0), "=&r"(l1), "=&r"(h0), "=&r"(h1) : "r"(a0), "r"(a1), "r"(b0), "r"(b1));
  // The carry of an add chain is not a borrow-in of a subtract chain, so e
  // is taken into s = a_hi + e first (no overflow: a_hi <= 2^32 - 2 when e = 1).
  uint32_t ah, sh, c0, c1, r0, r1, m;
  asm("add.cc.u32 %2, %8, %7;\n\t"       // a_hi = l1 + l0, carry e
      "addc.u32 %3, %2, 0;\n\t"          // s = a_hi + e
      "sub.cc.u32 %4, %7, %3;\n\t"       // b = (a_hi : l0) - s
      "subc.u32 %5, %2, 0;\n\t"
      "sub.cc.u32 %0, %9, %4;\n\t"       // r = x1 - b
      "subc.cc.u32 %1, %10, %5;\n\t"
      "subc.u32 %6, 0, 0;\n\t"           // borrow: + p = - EPS (mod 2^64)
      "sub.cc.u32 %0, %0, %6;\n\t"
      "subc.u32 %1, %1, 0;"
      : "=&r"(r0), "=&r"(r1), "=&r"(ah), "=&r"(sh), "=&r"(c0), "=&r"(c1), "=&r"(m)
      : "r"(l0), "r"(l1), "r"(h0), "r"(h1));
  return gl_pack(r0, r1);
#else
  const unsigned __int128 x = (unsigned __int128)a * w;
  const uint64_t x0 = (uint64_t)x, x1 = (uint64_t)(x >> 64);
  const uint64_t s = x0 + (x0 << 32);
  const uint64_t e = s < x0;
  const uint64_t b = s - (s >> 32) - e;
  const uint64_t r = x1 - b;
  return x1 < b ? r - GL_EPS : r;
#endif
}

// t*2^64 mod p: the Montgomery form of t (tables of gl_mont_mul factors).
GL_HD uint64_t gl_to_mont(uint64_t t) { return gl_mul(t, GL_EPS); }

// 2^(k + 64) mod p, the Montgomery form of 2^k, at compile time.
GL_HD constexpr uint64_t gl_pow2_mont(int k) {
  uint64_t x = GL_EPS;  // 2^64 mod p
  for (int i = 0; i < k; i++) {
    const uint64_t d = x << 1;
    x = (x >> 63) ? d + GL_EPS : d;   // 2^64 = EPS (mod p); no second wrap: d <= 2^64 - 2^33
    if (x >= GL_P) x -= GL_P;
  }
  return x;
}

// x * 2^K mod p for a compile-time K in [0, 192), canonical: on the device a
// Montgomery product by the constant 2^(K+64) mod p.  (The codelets' shifts are
// gl_lshl.)
template <int K>
GL_HD uint64_t gl_shl(uint64_t x) {
  static_assert(K >= 0 && K < 192, "shift out of range");
  if constexpr (K == 0) {
    return x;
  } else if constexpr (K == 96) {
    return gl_neg(x);                     // 2^96 = -1
  } else {
#ifdef GL_DEV_PTX
    constexpr uint64_t c = gl_pow2_mont(K);
    return gl_mont_mul(x, c);
#else
    if constexpr (K > 96) {
      return gl_neg(gl_shl<K - 96>(x));   // 2^96 = -1
    } else if constexpr (K < 64) {
      uint64_t hi = x >> (64 - K);
      return gl_reduce159(x << K, hi & 0xffffffffull, hi >> 32);
    } else {
      constexpr int s = K - 64;
      uint64_t a = (x << s) & 0xffffffffull;
      uint64_t b = x >> (32 - s);
      return gl_reduce159(0, a, b);
    }
#endif
  }
}

// ------------------------------------------------------------- lazy values
//
// The codelets add and subtract in three 32-bit limbs, x0 + x1*2^32 +
// x2*2^64 with x2 signed, and reduce only where a value leaves the codelet or
// meets a general product: an addition is one carry chain of three
// instructions, where the canonical one is eight (8 ALU/FMA instructions for
// gl_add, 5 for gl_sub), and a product by 2^k is a word shift and one or two
// carry chains instead of a Montgomery product (9 ALU + 9 FMA).  The
// generator (codegen.py) tracks the exact interval of every value, so x2
// never overflows.  Measured on GB300 (issue cycles per warp and element in
// a register loop, 64 registers): 16-point DFT 74.6 -> 40.0, 8-point 50.2 ->
// 31.3, 15-point 109 -> 77, 17-point 167 -> 111; the ALU pipe is 93 % busy.
struct gl_l3 {
  uint32_t x0, x1, x2;
};

#if defined(__CUDACC__)
// 2^32 - 1 from constant memory: as a literal the compiler turns the
// multiply-adds below into shifts and subtractions (which measured 14 %
// slower in the 16-point DFT: the ALU pipe is the busier one).
static __device__ __constant__ uint32_t gl_c_eps = 0xffffffffu;
#endif
#ifndef GL_DEV_PTX
inline gl_l3 gl_l_pack(unsigned __int128 v) {
  return {(uint32_t)v, (uint32_t)(v >> 32), (uint32_t)(v >> 64)};
}
inline unsigned __int128 gl_l_value(const gl_l3 &a) {  // two's complement, sign-extended
  return (unsigned __int128)(((__int128)(int32_t)a.x2 << 64)) + (((uint64_t)a.x1 << 32) | a.x0);
}
inline unsigned __int128 gl_l_value(uint64_t a) { return a; }
#endif

GL_HD gl_l3 gl_l3_of(const gl_l3 &a) { return a; }
GL_HD gl_l3 gl_l3_of(uint64_t a) { return {(uint32_t)a, (uint32_t)(a >> 32), 0u}; }

// a + b and a - b; either operand a 64-bit word (any value) or three limbs.
template <class A, class B>
GL_HD gl_l3 gl_ladd(const A &av, const B &bv) {
#ifdef GL_DEV_PTX
  const gl_l3 a = gl_l3_of(av), b = gl_l3_of(bv);
  gl_l3 r;
  asm("add.cc.u32 %0, %3, %6;\n\t"
      "addc.cc.u32 %1, %4, %7;\n\t"
      "addc.u32 %2, %5, %8;"
      : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
      : "r"(a.x0), "r"(a.x1), "r"(a.x2), "r"(b.x0), "r"(b.x1), "r"(b.x2));
  return r;
#else
  return gl_l_pack(gl_l_value(av) + gl_l_value(bv));
#endif
}
template <class A, class B>
GL_HD gl_l3 gl_lsub(const A &av, const B &bv) {
#ifdef GL_DEV_PTX
  const gl_l3 a = gl_l3_of(av), b = gl_l3_of(bv);
  gl_l3 r;
  asm("sub.cc.u32 %0, %3, %6;\n\t"
      "subc.cc.u32 %1, %4, %7;\n\t"
      "subc.u32 %2, %5, %8;"
      : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
      : "r"(a.x0), "r"(a.x1), "r"(a.x2), "r"(b.x0), "r"(b.x1), "r"(b.x2));
  return r;
#else
  return gl_l_pack(gl_l_value(av) - gl_l_value(bv));
#endif
}

// a + M*p = a + M*2^64 - M*2^32 + M, 0 < M < 2^31: raises a value above zero.
template <uint64_t M, class A>
GL_HD gl_l3 gl_lbias(const A &av) {
  static_assert(M > 0 && M < (1ull << 31), "bias out of range");
  const gl_l3 k = {(uint32_t)M, 0u - (uint32_t)M, (uint32_t)M - 1};
  return gl_ladd(av, k);
}
// M*p - a.
template <uint64_t M, class A>
GL_HD gl_l3 gl_lnegb(const A &av) {
  static_assert(M < (1ull << 31), "bias out of range");
  const gl_l3 k = {(uint32_t)M, 0u - (uint32_t)M, (uint32_t)M - (M > 0)};
  return gl_lsub(k, av);
}

// A non-negative value (x2 < 2^31) to a 64-bit word congruent to it, not
// necessarily below p: X + x2*(2^32 - 1), and a carry out of it is another
// 2^32 - 1 (which cannot carry again: the wrapped sum is below 2^63).
GL_HD uint64_t gl_lfold(const gl_l3 &a) {
#ifdef GL_DEV_PTX
  uint32_t r0, r1, c;
  asm("mad.lo.cc.u32 %0, %5, %6, %3;\n\t"
      "madc.hi.cc.u32 %1, %5, %6, %4;\n\t"
      "addc.u32 %2, 0, 0;\n\t"
      "sub.u32 %2, 0, %2;\n\t"
      "add.cc.u32 %0, %0, %2;\n\t"
      "addc.u32 %1, %1, 0;"
      : "=&r"(r0), "=&r"(r1), "=&r"(c)
      : "r"(a.x0), "r"(a.x1), "r"(a.x2), "r"(gl_c_eps));
  return gl_pack(r0, r1);
#else
  const uint64_t x = ((uint64_t)a.x1 << 32) | a.x0, u = (uint64_t)a.x2 * GL_EPS, r = x + u;
  return r < u ? r + GL_EPS : r;
#endif
}

// The same for a signed x2, in three limbs (the new x2 is -1, 0 or 1): makes
// room for a following shift.
GL_HD gl_l3 gl_lnorm(const gl_l3 &a) {
#ifdef GL_DEV_PTX
  const uint32_t sg = (uint32_t)((int32_t)a.x2 >> 31);
  gl_l3 r;
  asm("sub.cc.u32 %0, %3, %5;\n\t"
      "subc.cc.u32 %1, %4, %6;\n\t"
      "subc.u32 %2, 0, %6;\n\t"
      "add.cc.u32 %1, %1, %5;\n\t"
      "addc.u32 %2, %2, %6;"
      : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2)
      : "r"(a.x0), "r"(a.x1), "r"(a.x2), "r"(sg));
  return r;
#else
  const __int128 u = (__int128)(int32_t)a.x2 * (__int128)GL_EPS;
  return gl_l_pack((((uint64_t)a.x1 << 32) | a.x0) + (unsigned __int128)u);
#endif
}

// a * 2^K for 0 < K < 96, where a shifted by K mod 32 bits fits three limbs
// (y0, y1, y2), y2 signed.  With 2^64 = 2^32 - 1 and 2^96 = -1:
//   K < 32   the shifted limbs as they are;
//   K < 64   y0*2^32 + y1*(2^32 - 1) - y2;
//   K < 96   y0*(2^32 - 1) - y1 - y2*2^32.
template <int K, class A>
GL_HD gl_l3 gl_lshl(const A &av) {
  static_assert(K > 0 && K < 96, "shift out of range");
  constexpr int s = K % 32, q = K / 32;
#ifdef GL_DEV_PTX
  const gl_l3 x = gl_l3_of(av);
  uint32_t y0 = x.x0, y1 = x.x1, y2 = x.x2;
  if constexpr (s != 0) {
    y0 = x.x0 << s;
    y1 = __funnelshift_l(x.x0, x.x1, s);
    y2 = __funnelshift_l(x.x1, x.x2, s);
  }
  gl_l3 r;
  if constexpr (q == 0) {
    r = {y0, y1, y2};
  } else if constexpr (q == 1) {
    const uint32_t sg = (uint32_t)((int32_t)y2 >> 31);
    asm("mul.lo.u32 %0, %3, %4;\n\t"          // y1*EPS + y0*2^32, carry to x2
        "mad.hi.cc.u32 %1, %3, %4, %5;\n\t"
        "addc.u32 %2, 0, 0;\n\t"
        "sub.cc.u32 %0, %0, %6;\n\t"
        "subc.cc.u32 %1, %1, %7;\n\t"
        "subc.u32 %2, %2, %7;"
        : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2)
        : "r"(y1), "r"(gl_c_eps), "r"(y0), "r"(y2), "r"(sg));
  } else {
    const uint32_t sg = (uint32_t)((int32_t)y2 >> 31);
    asm("sub.cc.u32 %0, 0, %3;\n\t"           // y0*EPS >= 0
        "subc.u32 %1, %3, 0;\n\t"
        "sub.cc.u32 %0, %0, %4;\n\t"
        "subc.cc.u32 %1, %1, %5;\n\t"
        "subc.u32 %2, 0, %6;"
        : "=&r"(r.x0), "=&r"(r.x1), "=&r"(r.x2)
        : "r"(y0), "r"(y1), "r"(y2), "r"(sg));
  }
  return r;
#else
  const unsigned __int128 y = gl_l_value(av) << s;
  const unsigned __int128 y0 = (uint32_t)y, y1 = (uint32_t)(y >> 32);
  const unsigned __int128 y2 = (unsigned __int128)(__int128)(int32_t)(uint32_t)(y >> 64);
  if (q == 0) return gl_l_pack(y);
  if (q == 1) return gl_l_pack((y0 << 32) + y1 * GL_EPS - y2);
  return gl_l_pack(y0 * GL_EPS - y1 - (y2 << 32));
#endif
}

// x * 2^k mod p for a run-time k (any value; 2^192 = 1).
GL_HD uint64_t gl_shl_rt(uint64_t x, uint32_t k) {
  k %= 192;
  if (k >= 96) { x = gl_neg(x); k -= 96; }
  if (k == 0) return x;
  if (k < 64) {
    uint64_t hi = x >> (64 - k);
    return gl_reduce159(x << k, hi & 0xffffffffull, hi >> 32);
  }
  uint32_t s = k - 64;
  uint64_t a = (x << s) & 0xffffffffull;
  uint64_t b = s ? (x >> (32 - s)) : (x >> 32);
  return gl_reduce159(0, a, b);
}

GL_HD uint64_t gl_pow(uint64_t a, uint64_t e) {
  uint64_t r = 1;
  while (e) {
    if (e & 1) r = gl_mul(r, a);
    a = gl_mul(a, a);
    e >>= 1;
  }
  return r;
}

GL_HD uint64_t gl_inv(uint64_t a) { return gl_pow(a, GL_P - 2); }
