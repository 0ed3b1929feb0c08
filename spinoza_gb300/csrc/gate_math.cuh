// Per-pair and per-element gate arithmetic, shared by the plain per-gate
// kernels and the fused tile executor.  Each function performs the reference's
// floating-point operations in the reference's order (no contraction, FMA only
// where the reference calls mul_add), so results are bit-identical to
// spinoza's CPU path; the cited lines are in spinoza/src/gates.rs.
//
// (a, b) = (re, im) of s0 (target bit 0); (c, d) = (re, im) of s1.
#pragma once

#include "common.cuh"
#include "exact_mul.cuh"

namespace spz {

constexpr double kSqrtOneHalf = 0.70710678118654752440;  // math.rs:5

__device__ __forceinline__ uint64_t dbits(double a) { return (uint64_t)__double_as_longlong(a); }

// Fast-mode lazy ops (the gate divided by a scalar carried elsewhere): four
// FP64 instructions per pair.  Coefficient in g.cs (t or u).
template <int FK>
__device__ __forceinline__ void fast_pair_t(const double t, double& a, double& b, double& c, double& d) {
  double na, nb, nc, nd;
  if constexpr (FK == FK_LAZY_H) {
    na = dadd(a, c); nb = dadd(b, d); nc = dsub(a, c); nd = dsub(b, d);
  } else if constexpr (FK == FK_LAZY_RX_A) {  // s0 - i t s1, -i t s0 + s1
    na = dfma(t, d, a); nb = dfma(dneg(t), c, b); nc = dfma(t, b, c); nd = dfma(dneg(t), a, d);
  } else if constexpr (FK == FK_LAZY_RX_B) {  // u s0 - i s1, -i s0 + u s1
    na = dfma(t, a, d); nb = dfma(t, b, dneg(c)); nc = dfma(t, c, b); nd = dfma(t, d, dneg(a));
  } else if constexpr (FK == FK_LAZY_RY_A) {  // s0 - t s1, t s0 + s1
    na = dfma(dneg(t), c, a); nb = dfma(dneg(t), d, b); nc = dfma(t, a, c); nd = dfma(t, b, d);
  } else {  // FK_LAZY_RY_B: u s0 - s1, s0 + u s1
    na = dfma(t, a, dneg(c)); nb = dfma(t, b, dneg(d)); nc = dfma(t, c, a); nd = dfma(t, d, b);
  }
  a = na; b = nb; c = nc; d = nd;
}

template <int FK>
__device__ __forceinline__ void fast_pair(const Coef& g, double& a, double& b, double& c, double& d) {
  fast_pair_t<FK>(g.cs, a, b, c, d);
}

// A lazy op whose kind is known only at run time (uniform over the block).
__device__ __forceinline__ void fast_pair_kind(int kind, double t, double& a, double& b, double& c, double& d) {
  switch (kind) {
    case FK_LAZY_H: fast_pair_t<FK_LAZY_H>(t, a, b, c, d); break;
    case FK_LAZY_RX_A: fast_pair_t<FK_LAZY_RX_A>(t, a, b, c, d); break;
    case FK_LAZY_RX_B: fast_pair_t<FK_LAZY_RX_B>(t, a, b, c, d); break;
    case FK_LAZY_RY_A: fast_pair_t<FK_LAZY_RY_A>(t, a, b, c, d); break;
    default: fast_pair_t<FK_LAZY_RY_B>(t, a, b, c, d); break;
  }
}

// Products by a gate's coefficients come from the integer pipes (mul_int, see
// exact_mul.cuh), adds and FMAs stay DFMA: 4 DFMA instead of 8 per H pair, 4
// instead of 12 for RX / RY, 10 instead of 14 for U, 4 instead of 8 for RZ.
// All eight products of a rotation on the integer pipes measured best (27
// qubits, H + RX + RZ + U + CX + 3-control X on every target: 159.1 ms with
// DFMA products, 109.7 with six of a rotation's eight moved, 107.5 with eight,
// 100.8 with RZ's signs on the integer pipe; 26-qubit exact brickwork 226.4 ->
// 177.5 ms).
__device__ __forceinline__ double imul(double y, const MulCoef& c) {
  return __longlong_as_double((long long)mul_int(dbits(y), c));
}

__device__ __forceinline__ double imul_or_zero(double y, const MulCoef& c) {
  return __longlong_as_double((long long)mul_int_or_zero(dbits(y), c));
}

// x with its sign flipped when `flip`, on the integer pipe (a negation that no FP64
// instruction takes in as an operand's sign is an FP64 instruction itself).
__device__ __forceinline__ double flip_sign(double x, bool flip) {
  return __hiloint2double(__double2hiint(x) ^ (flip ? (int)0x80000000 : 0), __double2loint(x));
}

// Whether p holds in every lane that is here.  The two ways of a gate are chosen
// by the warp, not by the lane: a warp with zeros in some lanes would otherwise
// go both ways, one after the other, and cost more than DFMA products alone (25
// qubits, real-valued state with a qubit in |0>: RY 657 us by lane, 403 by warp; H
// 404 and 276).
__device__ __forceinline__ bool warp_all(bool p) { return __all_sync(__activemask(), p) != 0; }

// One gate on one pair, its coefficients prepared once (before a kernel's
// loop).  Products by a coefficient come from the integer pipes when every
// amplitude of the warp's pairs is in the prepared range, from dmul() otherwise;
// both give the reference's bits.
template <int KIND>
struct PairGate {
  MulRange range = mul_range_all();
  MulCoef m0{}, m1{}, m2{}, m3{};
  Coef g;

  __device__ __forceinline__ explicit PairGate(const Coef& c) : g(c) {
    if constexpr (KIND == SPZ_GATE_H) {
      m0 = mul_prepare(dbits(kSqrtOneHalf), range);
    } else if constexpr (KIND == SPZ_GATE_RX) {
      m0 = mul_prepare(dbits(g.cs), range);
      m1 = mul_prepare(dbits(g.nsn), range);
    } else if constexpr (KIND == SPZ_GATE_RY) {
      m0 = mul_prepare(dbits(g.cs), range);
      m1 = mul_prepare(dbits(g.sn), range);
    } else if constexpr (KIND == SPZ_GATE_U) {
      m0 = mul_prepare(dbits(dneg(g.l)), range);
      m1 = mul_prepare(dbits(g.l), range);
      m2 = mul_prepare(dbits(dneg(g.t)), range);
      m3 = mul_prepare(dbits(g.t), range);
    }
  }

  __device__ __forceinline__ bool ok(double x) const { return mul_ok(dbits(x), range); }

  __device__ __forceinline__ void operator()(double& a, double& b, double& c, double& d) const {
    if constexpr (KIND == SPZ_GATE_H) {  // h_apply_strat2, gates.rs:547-562
      double a1, b1, c1, d1;
      if (warp_all(ok(a) & ok(b) & ok(c) & ok(d))) {
        a1 = imul(a, m0); b1 = imul(b, m0); c1 = imul(c, m0); d1 = imul(d, m0);
      } else {
        a1 = dmul(kSqrtOneHalf, a); b1 = dmul(kSqrtOneHalf, b);
        c1 = dmul(kSqrtOneHalf, c); d1 = dmul(kSqrtOneHalf, d);
      }
      a = dadd(a1, c1);
      b = dadd(b1, d1);
      c = dsub(a1, c1);
      d = dsub(b1, d1);
    } else if constexpr (KIND == SPZ_GATE_X) {  // x_apply_target, gates.rs:329-334
      double t = a; a = c; c = t;
      t = b; b = d; d = t;
    } else if constexpr (KIND == SPZ_GATE_Y) {  // y_proc_chunk, gates.rs:455-463
      const double na = d, nb = dneg(c), nc = dneg(b), nd = a;
      a = na; b = nb; c = nc; d = nd;
    } else if constexpr (KIND == SPZ_GATE_RX) {  // rx_apply_target, gates.rs:713-725
      double ac, bc, cc, dc, an, bn, cn, dn;  // times cos, times neg_sin
      if (warp_all(ok(a) & ok(b) & ok(c) & ok(d))) {
        ac = imul(a, m0); an = imul(a, m1); bc = imul(b, m0); bn = imul(b, m1);
        cc = imul(c, m0); cn = imul(c, m1); dc = imul(d, m0); dn = imul(d, m1);
      } else {
        ac = dmul(a, g.cs); an = dmul(a, g.nsn); bc = dmul(b, g.cs); bn = dmul(b, g.nsn);
        cc = dmul(c, g.cs); cn = dmul(c, g.nsn); dc = dmul(d, g.cs); dn = dmul(d, g.nsn);
      }
      a = dsub(ac, dn);
      b = dadd(bc, cn);
      c = dsub(cc, bn);  // b * -neg_sin + c * cos (rounding is sign-symmetric)
      d = dadd(dc, an);
    } else if constexpr (KIND == SPZ_GATE_RY) {  // ry_apply_strategy2, gates.rs:1116-1119
      double ac, bc, cc, dc, as, bs, cs, ds;  // times cos, times sin
      if (warp_all(ok(a) & ok(b) & ok(c) & ok(d))) {
        ac = imul(a, m0); as = imul(a, m1); bc = imul(b, m0); bs = imul(b, m1);
        cc = imul(c, m0); cs = imul(c, m1); dc = imul(d, m0); ds = imul(d, m1);
      } else {
        ac = dmul(a, g.cs); as = dmul(a, g.sn); bc = dmul(b, g.cs); bs = dmul(b, g.sn);
        cc = dmul(c, g.cs); cs = dmul(c, g.sn); dc = dmul(d, g.cs); ds = dmul(d, g.sn);
      }
      a = dsub(ac, cs);
      b = dsub(bc, ds);
      c = dadd(as, cc);
      d = dadd(bs, dc);
    } else if constexpr (KIND == SPZ_GATE_U) {  // u_apply_target, gates.rs:1256-1259
      const double p = a, q = b, m = c, n = d;
      double ln, lm, tn, tm;  // -l n, l m, -t n, t m
      if (warp_all(ok(m) & ok(n))) {
        ln = imul(n, m0); lm = imul(m, m1); tn = imul(n, m2); tm = imul(m, m3);
      } else {
        ln = dmul(dneg(g.l), n); lm = dmul(g.l, m); tn = dmul(dneg(g.t), n); tm = dmul(g.t, m);
      }
      a = dfma(g.a, p, dfma(g.k, m, ln));
      b = dfma(g.a, q, dfma(g.k, n, lm));
      c = dfma(g.q, p, dfma(dneg(g.r), q, dfma(g.s, m, tn)));
      d = dfma(g.q, q, dfma(g.r, p, dfma(g.s, n, tm)));
    } else if constexpr (KIND >= FK_LAZY_H) {
      fast_pair<KIND>(g, a, b, c, d);
    }
  }
};

// Diagonal gates on one amplitude; `one` is the amplitude's target bit.  RZ's
// entries are (re, im) = (cos, -sin) on 0 and (cos, sin) on 1.
// ZEROS: warps with amplitudes that are zero have an integer path too (the
// per-gate kernels, which HBM bounds; 25 qubits, real-valued state: RZ 366 us
// without, 178 with, P 147 and 98).  In tile passes, where the integer pipes are
// the busier ones, it costs more than it gives (20-qubit QFT 632 us without, 674
// with it for every warp).
template <int KIND, bool ZEROS = false>
struct DiagGate : DiagCoef {
  __device__ __forceinline__ explicit DiagGate(const DiagCoef& d) : DiagCoef(d) {}
  __device__ __forceinline__ explicit DiagGate(const Coef& c) : DiagCoef{} {
    if constexpr (KIND != SPZ_GATE_Z) {
      const double r = KIND == SPZ_GATE_P ? c.cs : c.d1re, i = KIND == SPZ_GATE_P ? c.sn : c.d1im;
      *static_cast<DiagCoef*>(this) = diag_prepare(r, i, dbits(r), dbits(i));
    }
  }

  // The products' ways: FP64, integer, integer with zeros.
  enum Way { FP = 0, INT = 1, INT_ZERO = 2 };

  // Whether the amplitude's products may take the way W.
  template <Way W>
  __device__ __forceinline__ bool fits(double re, double im) const {
    const auto ok = [this](double y) {
      return W == INT_ZERO ? mul_ok_or_zero(dbits(y), range) : mul_ok(dbits(y), range);
    };
    if constexpr (KIND == SPZ_GATE_P) return ok(re) & ok(im);
    else if constexpr (KIND == SPZ_GATE_RZ) return ok(im);
    else return true;
  }

  template <Way W>
  __device__ __forceinline__ void apply(bool one, double& re, double& im) const {
    if constexpr (KIND == SPZ_GATE_Z) {  // z_proc_chunk, gates.rs:1054-1056
      if (one) { re = dneg(re); im = dneg(im); }
    } else if constexpr (KIND == SPZ_GATE_P) {  // p_proc_chunk, gates.rs:837-838
      if (one) {
        const double zr = re, zi = im;
        double is, rs;  // -im * sin, re * sin
        if constexpr (W == FP) { is = dmul(dneg(zi), im1); rs = dmul(zr, im1); }
        else if constexpr (W == INT_ZERO) { is = imul_or_zero(zi, mul_flip(mim, true)); rs = imul_or_zero(zr, mim); }
        else { is = dneg(imul(zi, mim)); rs = imul(zr, mim); }
        re = dfma(zr, re1, is);
        im = dfma(zi, re1, rs);
      }
    } else if constexpr (KIND == SPZ_GATE_RZ) {  // rz_apply_strategy1, gates.rs:939-946
      const double cr = re, ci = im, s = flip_sign(im1, !one);
      double is, ic;  // -im * the entry's sin, im * cos
      if constexpr (W == FP) { is = dmul(dneg(ci), s); ic = dmul(ci, re1); }
      else if constexpr (W == INT_ZERO) { is = imul_or_zero(ci, mul_flip(mim, one)); ic = imul_or_zero(ci, mre); }
      else { is = flip_sign(imul(ci, mim), one); ic = imul(ci, mre); }
      re = dfma(cr, re1, is);
      im = dfma(cr, s, ic);
    }
  }

  __device__ __forceinline__ void operator()(bool one, double& re, double& im) const {
    if (warp_all(fits<INT>(re, im))) apply<INT>(one, re, im);
    else if (ZEROS && warp_all(fits<INT_ZERO>(re, im))) apply<INT_ZERO>(one, re, im);
    else apply<FP>(one, re, im);
  }

  // Two amplitudes of a thread, their instructions side by side.
  __device__ __forceinline__ void operator()(bool one0, double& re0, double& im0, bool one1, double& re1, double& im1) const {
    if (warp_all(fits<INT>(re0, im0) & fits<INT>(re1, im1))) {
      apply<INT>(one0, re0, im0);
      apply<INT>(one1, re1, im1);
    } else if (ZEROS && warp_all(fits<INT_ZERO>(re0, im0) & fits<INT_ZERO>(re1, im1))) {
      apply<INT_ZERO>(one0, re0, im0);
      apply<INT_ZERO>(one1, re1, im1);
    } else {
      apply<FP>(one0, re0, im0);
      apply<FP>(one1, re1, im1);
    }
  }
};

}  // namespace spz
