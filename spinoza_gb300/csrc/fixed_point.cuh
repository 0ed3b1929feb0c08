// Fast mode's arithmetic on the integer pipes: amplitudes in 64-bit fixed
// point, each with an exponent of its own.
//
// What bounds the fast mode is DFMA issue (a warp's FP64 instruction holds the
// SM's FP64 unit for 16 cycles), and its ops may round differently, so they
// need no IEEE operation each.  For the length of a tile pass an amplitude is
// (re, im) x 2^(exp - 1084): two 64-bit integers on one exponent, the larger of
// them with its top bit at 61 (fx_settle).  An op brings the amplitudes that it
// mixes to the largest of their exponents, a few bits lower to leave it room;
// a multiply-add by a coefficient of magnitude <= 1 is then three 32 x 32-bit
// multiplies (1.0-1.3 cycles each), with no rounding or packing between the
// ops of a pass.
//
// Precision: an op leaves an error of about 2^-58 of the largest amplitude that
// it mixes, where FP64 rounds every operation to 2^-53 of its result.  So an
// amplitude that comes out 2^-5 of the largest or more (what a rotation by
// t >= 2^-5 makes of it, kFxMinT) is as accurate as in FP64; rotations by less
// have an exponent for each result (fx_lazy_small).  The error is one of the
// amplitude, shared by its real and imaginary part; a component that is zero
// stays zero where the op adds nothing to it.  The amplitudes become FP64 again,
// rounded to nearest, when the pass stores them.  Tiles with a component that is
// not finite or a nonzero amplitude outside [2^-895, 2^600) are worked on in FP64
// (fx_in_range).  (29-qubit brickwork, 10 layers: 662 ms; 637 without kFxMinT's
// rules, 617 with the amplitudes of an op left on one exponent.)
//
// Bounds.  The limbs need inputs below 2^61 - 2^29 (the upper one is rounded up),
// an op's results have to stay below 2^62, and a phase times a component below B
// gives one below sqrt(2) B, a rotation after it below 2 sqrt(2) B, a second one
// below 4 sqrt(2) B.  So two rotations start from components below 2^59 (kFxRoom2),
// one rotation or a phase from below 2^60 (kFxRoom1).
#pragma once

#include <math.h>
#include <stdint.h>

#ifdef __CUDACC__
#define SPZ_HD __host__ __device__ __forceinline__
#else
#define SPZ_HD inline
#endif

namespace spz {

constexpr uint32_t kFxMinHi = 0x08000000u;  // upper words of an amplitude's larger component: at least this ...
// ... and below this.  The lazy ops of a circuit grow a tile's norm by 2^401 at
// most before the carried scale is folded in, so that an amplitude stays finite
// where an exact gate takes it through FP64.
constexpr uint32_t kFxMaxHi = 0x65700000u;
constexpr int kFxZeroExp = -(1 << 28);      // exponent of a zero amplitude

struct FxAmp {
  int64_t r, i;
  int32_t e;
};

constexpr int kFxRoom2 = 3, kFxRoom1 = 2;  // bits below 2^62 that an op's inputs leave free
constexpr double kFxMinT = 0x1p-5;

// A coefficient c, |c| <= 1 (and a rounding more), as (h 2^32 + l) / 2^62.
struct FxCoef {
  int32_t h, l;
};

inline FxCoef fx_coef(double c) {
  const long long v = llrint(ldexp(c, 62));
  const int32_t l = (int32_t)(uint32_t)(uint64_t)v;
  return FxCoef{(int32_t)((v - l) >> 32), l};
}

// 4 y = h 2^32 + l, |y| < 2^61 - 2^29
struct FxLimb {
  int32_t h, l;
};

SPZ_HD FxLimb fx_split(int64_t y) {
  const int32_t l = (int32_t)((uint32_t)y << 2);
  return FxLimb{(int32_t)(y >> 30) + (int32_t)((uint32_t)l >> 31), l};
}

SPZ_HD int32_t fx_mulhi(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
SPZ_HD int64_t fx_mad(int32_t a, int32_t b, int64_t c) { return (int64_t)a * b + c; }

// x + c y = x + 4 y c 2^62 / 2^64: of the cross products only the upper words are
// formed, the product of the two low limbs (below the last bit) is left out; a zero
// stays one.  (Unsigned low limbs, two instructions to split instead of four,
// measured 10% slower; 64-bit cross products 2% slower.)
SPZ_HD int64_t fx_mac(int64_t x, const FxLimb& y, const FxCoef& c) {
  return fx_mad(y.h, c.h, x) + (fx_mulhi(y.l, c.h) + fx_mulhi(y.h, c.l));
}

// x - c y
SPZ_HD int64_t fx_msub(int64_t x, const FxLimb& y, const FxCoef& c) {
  return fx_mad(y.h, -c.h, x) - (fx_mulhi(y.l, c.h) + fx_mulhi(y.h, c.l));
}

// (r, i) *= (x, y)
SPZ_HD void fx_cmul(int64_t& r, int64_t& i, const FxCoef& x, const FxCoef& y) {
  const FxLimb R = fx_split(r), I = fx_split(i);
  const int32_t tr = fx_mulhi(R.l, x.h) + fx_mulhi(R.h, x.l) - fx_mulhi(I.l, y.h) - fx_mulhi(I.h, y.l);
  const int32_t ti = fx_mulhi(R.l, y.h) + fx_mulhi(R.h, y.l) + fx_mulhi(I.l, x.h) + fx_mulhi(I.h, x.l);
  r = fx_mad(I.h, -y.h, fx_mad(R.h, x.h, tr));
  i = fx_mad(I.h, x.h, fx_mad(R.h, y.h, ti));
}

SPZ_HD int64_t fx_shr(int64_t v, int32_t d) {  // d >= 0, any size
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(d));
  return r;
#else
  return v >> (d < 63 ? d : 63);
#endif
}

// The lazy rotation [[1, -t], [t, 1]] on s0, s1 with one exponent, 0 <= t <= 1.
SPZ_HD void fx_rotate(FxAmp& s0, FxAmp& s1, const FxCoef& t) {
  const FxLimb a = fx_split(s0.r), b = fx_split(s0.i), c = fx_split(s1.r), d = fx_split(s1.i);
  s0.r = fx_msub(s0.r, c, t);
  s0.i = fx_msub(s0.i, d, t);
  s1.r = fx_mac(s1.r, a, t);
  s1.i = fx_mac(s1.i, b, t);
}

// a *= i^p
SPZ_HD void fx_quarter(FxAmp& a, uint32_t p) {
  if (p & 2u) {
    a.r = -a.r;
    a.i = -a.i;
  }
  if (p & 1u) {
    const int64_t r = a.r;
    a.r = -a.i;
    a.i = r;
  }
}

SPZ_HD void fx_swap(FxAmp& a, FxAmp& b) {
  const FxAmp t = a;
  a = b;
  b = t;
}

// Bring a[0 .. N-1] to the largest of their exponents and ROOM bits down; returns
// the exponent that they are on then.
template <int N, int ROOM>
SPZ_HD int32_t fx_align(FxAmp* a) {
  int32_t E = a[0].e;
#pragma unroll
  for (int j = 1; j < N; ++j) E = a[j].e > E ? a[j].e : E;
  E += ROOM;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    a[j].r = fx_shr(a[j].r, E - a[j].e);
    a[j].i = fx_shr(a[j].i, E - a[j].e);
    if constexpr (N == 1) a[j].e = E;
  }
  return E;
}

SPZ_HD int32_t fx_clz(uint32_t v) {
#ifdef __CUDA_ARCH__
  return __clz((int)v);
#else
  return v ? __builtin_clz(v) : 32;
#endif
}

// The larger of an amplitude's upper words without their signs, and the shift that
// brings its top bit to 29 (the component's to 61; one bit less at some negative
// powers of two).
SPZ_HD uint32_t fx_top(const FxAmp& a) {
  const int32_t r = (int32_t)(a.r >> 32), i = (int32_t)(a.i >> 32);
  return (uint32_t)(r < 0 ? -r : r) | (uint32_t)(i < 0 ? -i : i);
}
SPZ_HD void fx_shift_up(FxAmp& a, int32_t E, uint32_t top) {
  const int32_t d = fx_clz(top) - 2;
  a.r <<= d;
  a.i <<= d;
  a.e = E - d;
}

// a[0 .. N-1], below 2^62 on exponent E, shifted up so that the larger component of
// each has its top bit at 61 (a zero amplitude: on kFxZeroExp).  The upper words say
// by how much; where they are zero (zeros, cancellations) the lower ones are
// shifted in first.
template <int N>
SPZ_HD void fx_settle(FxAmp* a, int32_t E) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    uint32_t top = fx_top(a[j]);
    int32_t e = E;
    if (top == 0u) {
      a[j].r <<= 29;
      a[j].i <<= 29;
      e = (a[j].r | a[j].i) == 0 ? kFxZeroExp : E - 29;
      top = fx_top(a[j]) | 1u;
    }
    fx_shift_up(a[j], e, top);
  }
}

// The bits of an amplitude's components as FxAmp (any finite normal numbers; a
// component far below the other, or subnormal, loses its low bits).
SPZ_HD FxAmp fx_from(uint64_t re, uint64_t im) {
  const uint32_t hr = (uint32_t)(re >> 32) & 0x7FFFFFFFu, hi = (uint32_t)(im >> 32) & 0x7FFFFFFFu;
  const int32_t e = (int32_t)((hr > hi ? hr : hi) >> 20);
  int64_t v[2];
  const uint64_t b[2] = {re, im};
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint32_t h = (uint32_t)(b[j] >> 32);
    const uint64_t m = (((uint64_t)((h & 0x000FFFFFu) | 0x00100000u) << 32) | (uint32_t)b[j]) << 9;
    const int32_t f = (int32_t)((h >> 20) & 0x7FFu);
    const int64_t s = (int64_t)((int32_t)h >> 31);
    v[j] = f == 0 ? 0 : ((fx_shr((int64_t)m, e - f) ^ s) - s);
  }
  return FxAmp{v[0], v[1], e == 0 ? kFxZeroExp : e};
}

// Whether fx_from keeps the amplitude (zero, or its larger component in range).
SPZ_HD bool fx_in_range(uint64_t re, uint64_t im) {
  const uint32_t hr = (uint32_t)(re >> 32) & 0x7FFFFFFFu, hi = (uint32_t)(im >> 32) & 0x7FFFFFFFu;
  const uint32_t big = hr > hi ? hr : hi;
  return big - kFxMinHi < kFxMaxHi - kFxMinHi || ((re | im) << 1) == 0;
}

// v 2^(E - 1084) as FP64 bits, rounded to nearest, for 64 <= E < 1980.
SPZ_HD uint64_t fx_bits(int64_t v, int32_t E) {
  const int64_t s = v >> 63;
  const uint64_t a = (uint64_t)((v ^ s) - s);
#ifdef __CUDA_ARCH__
  // the exponent of a: its upper and lower half rounded toward zero to FP32
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
  const uint32_t q = __float_as_uint(__fmaf_rz(__uint2float_rz(ah), 4294967296.0f, __uint2float_rz(al))) >> 23;
  uint64_t n;
  asm("shl.b64 %0, %1, %2;" : "=l"(n) : "l"(a), "r"(189u - q));  // leading one to bit 62 (0 for a = 0)
#else
  const uint32_t q = a ? 127u + 63u - (uint32_t)__builtin_clzll(a) : 0u;
  const uint64_t n = a ? a << (189u - q) : 0;
#endif
  const uint64_t m = (n + 0x200u) >> 10;
  uint32_t hi = (uint32_t)(m >> 32) + ((q + (uint32_t)(E - 189)) << 20);  // E + (q - 127 - 61) - 1
  hi |= (uint32_t)s & 0x80000000u;
  hi = a ? hi : 0u;
  return ((uint64_t)hi << 32) | (uint32_t)m;
}

}  // namespace spz
