// Correctly rounded FP64 products on the integer pipes.
//
// What bounds the gate kernels is DFMA issue: a warp's FP64 instruction holds
// the SM's FP64 unit for 16 cycles (2 lanes per cycle), while mad.wide.u32
// takes 1.3 and a 32-bit logic, shift or add 0.5, and the two run side by side
// (measured: 1 DFMA + 8 mad.wide in one thread 17.0 cycles, 1 DFMA + 32 lop3
// 17.5).  A product by a gate coefficient, formed here from four 32 x 32-bit
// multiplies and one rounding step (about 25 integer instructions), therefore
// takes the place of a DFMA at roughly half its cost, on pipes that the
// remaining adds and FMAs leave idle.  The result is the IEEE round-to-nearest-
// even product, bit for bit, whenever amplitude, coefficient and product are
// normal numbers well inside the exponent range; mul_ok() says when, and the
// callers use dmul() otherwise (zeros, subnormals, infinities, NaN, products
// near under- or overflow).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define SPZ_HD __host__ __device__ __forceinline__
#else
#define SPZ_HD inline
#endif

namespace spz {

// A coefficient prepared for mul_int: its significand scaled to [2^62, 2^63),
// and what its sign and exponent add to the upper word of a product.
struct MulCoef {
  uint32_t ch, cl;
  uint32_t kexp;
};

// Amplitudes whose upper word without the sign, minus lo, is below span have
// normal products with every coefficient that the range was narrowed by.
struct MulRange {
  uint32_t lo, span;
};

SPZ_HD MulRange mul_range_all() { return MulRange{0x00100000u, 0x7FE00000u}; }

// Prepare the coefficient with bits `c` and narrow r by it (to nothing when c
// is zero, subnormal, 2^1023 or more, infinite or NaN).
SPZ_HD MulCoef mul_prepare(uint64_t c, MulRange& r) {
  const uint32_t hi = (uint32_t)(c >> 32), lo = (uint32_t)c;
  const uint32_t ec = (hi >> 20) & 0x7FFu;
  MulCoef m;
  // 53-bit significand << 10
  m.ch = (((hi & 0x000FFFFFu) | 0x00100000u) << 10) | (lo >> 22);
  m.cl = lo << 10;
  // upper word of the product = significand (bit 20 set) + (y's sign and
  // exponent) + kexp - (s << 20), s = 1 or 2: the normalising shift
  // (bits 31 and 30 of the exponent's part agree, so that where kexp's differ the
  // coefficient is negative)
  m.kexp = ((ec - 1023u + 1u) << 20) + (hi & 0x80000000u);
  // exponents e_y with 1 <= e_y <= 2046 and 2 <= e_y + ec - 1023 <= 2044
  const int shift = (int)ec - 1023;
  int a = 2 - shift, b = 2044 - shift;
  if (a < 1) a = 1;
  if (b > 2046) b = 2046;
  const int ra = (int)(r.lo >> 20), rb = ra + (int)(r.span >> 20) - 1;
  if (a < ra) a = ra;
  if (b > rb) b = rb;
  if (ec == 0u || ec >= 0x7FEu || b < a) {
    r.lo = 0u;
    r.span = 0u;
  } else {
    r.lo = (uint32_t)a << 20;
    r.span = (uint32_t)(b - a + 1) << 20;
  }
  return m;
}

// The diagonal entry (re1, im1) of P on its 1 half, or of RZ on 1, prepared.
struct alignas(16) DiagCoef {
  MulRange range;
  MulCoef mre, mim;
  double re1, im1;
};

SPZ_HD DiagCoef diag_prepare(double re1, double im1, uint64_t re1_bits, uint64_t im1_bits) {
  DiagCoef d;
  d.range = mul_range_all();
  d.mre = mul_prepare(re1_bits, d.range);
  d.mim = mul_prepare(im1_bits, d.range);
  d.re1 = re1;
  d.im1 = im1;
  return d;
}

SPZ_HD bool mul_ok(uint64_t y, const MulRange& r) {
  return (((uint32_t)(y >> 32) & 0x7FFFFFFFu) - r.lo) < r.span;
}

// y * c rounded to nearest even, as bits.  With y's significand (53 bits) times
// the coefficient's (63 bits) = P in [2^114, 2^116), the product's significand
// is P >> (64 - s) with s = 1 when P >= 2^115, else 2, rounded by the bits below.
SPZ_HD uint64_t mul_int(uint64_t y, const MulCoef& c) {
  const uint32_t hi = (uint32_t)(y >> 32), yl = (uint32_t)y;
  const uint32_t yh = (hi & 0x000FFFFFu) | 0x00100000u;
  const uint64_t p0 = (uint64_t)yl * c.cl;
  const uint64_t t = (uint64_t)yl * c.ch + (uint32_t)(p0 >> 32);
  const uint64_t u = (uint64_t)yh * c.cl + t;  // < 2^63 + 2^53
  const uint64_t v = (uint64_t)yh * c.ch + (uint32_t)(u >> 32);
  const uint32_t vh = (uint32_t)(v >> 32), vl = (uint32_t)v, ul = (uint32_t)u, pl = (uint32_t)p0;
  const uint32_t s = 2u - (vh >> 19);
  const uint32_t e = (hi & 0xFFF00000u) + c.kexp - (s << 20);
#ifdef __CUDA_ARCH__
  const uint32_t mh = __funnelshift_l(vl, vh, s), ml = __funnelshift_l(ul, vl, s);
  uint32_t w = __funnelshift_l(pl, ul, s);
#else
  const uint32_t mh = (vh << s) | (vl >> (32 - s)), ml = (vl << s) | (ul >> (32 - s));
  uint32_t w = (ul << s) | (pl >> (32 - s));
#endif
  // Bits below w only break ties.  (Those of pl already shifted into w are
  // zero when w could be a tie, so pl itself tells whether any are set.)
  w |= pl != 0u ? 1u : 0u;
  const uint32_t half = 0x7FFFFFFFu + (ml & 1u);  // carries out of w + half: above half, or at half and odd
#ifdef __CUDA_ARCH__
  uint32_t rl, rh;
  asm("{\n\t.reg .u32 x;\n\tadd.cc.u32 x, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
      : "=r"(rl), "=r"(rh)
      : "r"(w), "r"(half), "r"(ml), "r"(mh), "r"(e));
  return ((uint64_t)rh << 32) | rl;
#else
  const uint64_t up = ((uint64_t)w + half) >> 32;
  return (((uint64_t)mh << 32) | ml) + up + ((uint64_t)e << 32);
#endif
}

// The same with zeros taken too: for gates with integer instructions to spare
// (diagonal ones), so that real-valued and part-empty states stay on this path.
SPZ_HD bool mul_zero(uint64_t y) {
#ifdef __CUDA_ARCH__
  uint32_t m;  // (upper word & 0x7FFFFFFF) | lower word; in asm, or the compiler makes it an FP64 comparison
  asm("lop3.b32 %0, %1, 0x7FFFFFFF, %2, 0xEA;" : "=r"(m) : "r"((uint32_t)(y >> 32)), "r"((uint32_t)y));
  return m == 0u;
#else
  return (y << 1) == 0u;
#endif
}
SPZ_HD bool mul_ok_or_zero(uint64_t y, const MulRange& r) { return mul_ok(y, r) | (mul_zero(y) & (r.span != 0u)); }
SPZ_HD uint64_t mul_int_or_zero(uint64_t y, const MulCoef& c) {
  const uint64_t p = mul_int(y, c);
  const uint32_t sign = ((uint32_t)(y >> 32) ^ c.kexp ^ (c.kexp << 1)) & 0x80000000u;  // the coefficient's: see mul_prepare
  return mul_zero(y) ? (uint64_t)sign << 32 : p;
}
// The coefficient with its sign flipped when `flip`.
SPZ_HD MulCoef mul_flip(MulCoef c, bool flip) {
  c.kexp ^= flip ? 0x80000000u : 0u;
  return c;
}

// |y| * |y| rounded, as bits, for sqr_ok(y): mul_int with the coefficient made
// from y itself.
SPZ_HD bool sqr_ok(uint64_t y) {
  // exponents e with 2 <= 2 e - 1023 <= 2044
  return (((uint32_t)(y >> 32) & 0x7FFFFFFFu) - (513u << 20)) < ((1533u - 513u) << 20);
}

SPZ_HD uint64_t sqr_int(uint64_t y) {
  y &= 0x7FFFFFFFFFFFFFFFull;
  const uint32_t hi = (uint32_t)(y >> 32), lo = (uint32_t)y;
  MulCoef m;
  m.ch = (((hi & 0x000FFFFFu) | 0x00100000u) << 10) | (lo >> 22);
  m.cl = lo << 10;
  m.kexp = (hi & 0x7FF00000u) - (1022u << 20);
  return mul_int(y, m);
}

}  // namespace spz
