// Fast-mode gate ops on a tile held in shared memory in fixed point
// (fixed_point.cuh): two 64-bit integers and an exponent per amplitude.
//
// Every lazy op runs as one rotation [[1, -t], [t, 1]] with 0 <= t <= 1 between
// quarter turns, swaps and signs that the descriptor holds (FxLazy), so one
// piece of code serves all kinds: with a copy per kind and per number of phase
// masks the passes were bound by instruction fetch (ncu: no-instruction stalls
// 2.5 of 9.2 cycles per instruction).
#pragma once

#include "executor.cuh"
#include "fixed_point.cuh"
#include "gate_math.cuh"
#include "tile_map.cuh"

namespace spz {

struct FxTile {
  int64_t* r;
  int64_t* i;
  int32_t* e;
  __device__ __forceinline__ FxAmp load(uint32_t k) const { return FxAmp{r[k], i[k], e[k]}; }
  __device__ __forceinline__ void store(uint32_t k, const FxAmp& a) const {
    r[k] = a.r;
    i[k] = a.i;
    e[k] = a.e;
  }
};

// An amplitude as FP64, and back.
__device__ __forceinline__ double2 fx_to_double(const FxAmp& a) {
  if ((uint32_t)(a.e - 64) < 1916u)
    return make_double2(__longlong_as_double((long long)fx_bits(a.r, a.e)),
                        __longlong_as_double((long long)fx_bits(a.i, a.e)));
  if (a.e <= kFxZeroExp + (1 << 20)) return make_double2(0.0, 0.0);
  const int32_t x = a.e < -2000 ? -2000 : a.e > 4000 ? 4000 : a.e;  // near or past the ends of the range
  return make_double2(scalbn(__longlong_as_double((long long)fx_bits(a.r, 1023)), x - 1023),
                      scalbn(__longlong_as_double((long long)fx_bits(a.i, 1023)), x - 1023));
}

__device__ __forceinline__ FxAmp fx_from_double(double re, double im) {
  return fx_from(dbits(re), dbits(im));
}

// parities of the tile's base index under the op's masks
__device__ __forceinline__ uint32_t fx_base_index(const TileGate& g, uint64_t base) {
  uint32_t idx = 0;
  for (int j = 0; j < g.pm; ++j) idx |= (uint32_t)(__popcll(base & g.pmask[j]) & 1) << j;
  return idx;
}

// One lazy op on a pair; w: its phase entry (with has_w), fx* from the descriptor.
__device__ __forceinline__ void fx_lazy_pair(FxAmp* a, const FxCoef& t, bool has_w, const int4& w, uint32_t swaps,
                                             uint32_t turns) {
  const int32_t E = fx_align<2, kFxRoom1>(a);
  if (has_w) fx_cmul(a[1].r, a[1].i, FxCoef{w.x, w.y}, FxCoef{w.z, w.w});
  else fx_quarter(a[1], turns >> 8);
  if (swaps & 1u) fx_swap(a[0], a[1]);
  fx_rotate(a[0], a[1], t);
  if (turns & 0xFFu) {
    fx_quarter(a[0], turns);
    fx_quarter(a[1], turns >> 2);
  }
  fx_settle<2>(a, E);
}

// The same for a rotation by t 2^-k below kFxMinT, 1/2 <= t < 1 or t = 0 (k above
// FX_SMALL's shift in `swaps`): what it adds to an amplitude may lie far below the
// other one, so each result has a common exponent of its own for its two terms.
__device__ __forceinline__ void fx_lazy_small(FxAmp* a, const FxCoef& t, bool has_w, const int4& w, uint32_t swaps,
                                              uint32_t turns) {
  const int32_t k = (int32_t)(swaps >> kFxSmallShift);
  fx_align<1, kFxRoom1>(a);
  fx_align<1, kFxRoom1>(a + 1);
  if (has_w) fx_cmul(a[1].r, a[1].i, FxCoef{w.x, w.y}, FxCoef{w.z, w.w});
  else fx_quarter(a[1], turns >> 8);
  if (swaps & 1u) fx_swap(a[0], a[1]);
  const int32_t e0 = a[0].e, e1 = a[1].e, E0 = max(e0, e1 - k), E1 = max(e1, e0 - k);
  const FxLimb c = fx_split(fx_shr(a[1].r, E0 + k - e1)), d = fx_split(fx_shr(a[1].i, E0 + k - e1));
  const FxLimb p = fx_split(fx_shr(a[0].r, E1 + k - e0)), q = fx_split(fx_shr(a[0].i, E1 + k - e0));
  a[0].r = fx_msub(fx_shr(a[0].r, E0 - e0), c, t);
  a[0].i = fx_msub(fx_shr(a[0].i, E0 - e0), d, t);
  a[1].r = fx_mac(fx_shr(a[1].r, E1 - e1), p, t);
  a[1].i = fx_mac(fx_shr(a[1].i, E1 - e1), q, t);
  fx_quarter(a[0], turns);
  fx_quarter(a[1], turns >> 2);
  fx_settle<1>(a, E0);
  fx_settle<1>(a + 1, E1);
}

// A phase entry times one amplitude (2^fexp: the table's scale).
__device__ __forceinline__ void fx_phase(FxAmp& a, const int4& w, int32_t fexp) {
  const int32_t E = fx_align<1, kFxRoom1>(&a);
  fx_cmul(a.r, a.i, FxCoef{w.x, w.y}, FxCoef{w.z, w.w});
  fx_settle<1>(&a, E + fexp);
}

template <bool SMALL>
static __device__ void fx_tile_lazy(const TileGate& g, const int4* __restrict__ tables, Walk W,
                                    const FxTile& S, uint32_t npairs) {
  const uint32_t tmask = g.tmask, swaps = g.fxswaps, turns = g.fxturns;
  const bool has_w = g.pm > 0;
  const int4* tab = tables + g.ptab;
  const FxCoef t = g.fx1;
  for (uint32_t m = threadIdx.x, it = 0; m < npairs; m += blockDim.x, ++it) {
    const uint32_t word = W.word(it), s0 = word & 0xFFFFu, s1 = s0 ^ tmask;
    FxAmp a[2] = {S.load(s0), S.load(s1)};
    int4 w = make_int4(0, 0, 0, 0);
    if (has_w) w = __ldg(tab + (word >> 16));
    if constexpr (SMALL) fx_lazy_small(a, t, has_w, w, swaps, turns);
    else fx_lazy_pair(a, t, has_w, w, swaps, turns);
    S.store(s0, a[0]);
    S.store(s1, a[1]);
  }
}

// Two lazy rotations on blocks of four amplitudes, as tile_lazy2_op (circuit.cu):
// three phases, the first rotation along b1, the second along b2.
static __device__ void fx_tile_lazy2(const TileGate& g, const int4* __restrict__ tables, Walk W,
                                     const FxTile& S, uint32_t nblocks) {
  const uint32_t b1 = g.tmask, b2 = g.tmask2, swaps = g.fxswaps, turns = g.fxturns;
  const int4* tab = tables + g.ptab;
  const FxCoef t1 = g.fx1, t2 = g.fx2;
  for (uint32_t m = threadIdx.x, it = 0; m < nblocks; m += blockDim.x, ++it) {
    const uint32_t word = W.word(it), e = word & 0xFFFFu;
    const int4* row = tab + 3 * (word >> 16);
    FxAmp a[4] = {S.load(e), S.load(e ^ b1), S.load(e ^ b2), S.load(e ^ b1 ^ b2)};
    const int32_t X = fx_align<4, kFxRoom2>(a);
#pragma unroll
    for (int j = 1; j < 4; ++j) {
      const int4 w = __ldg(row + j - 1);
      fx_cmul(a[j].r, a[j].i, FxCoef{w.x, w.y}, FxCoef{w.z, w.w});
    }
    if (swaps & 1u) {
      fx_swap(a[0], a[1]);
      fx_swap(a[2], a[3]);
    }
    fx_rotate(a[0], a[1], t1);
    fx_rotate(a[2], a[3], t1);
    if (swaps & 2u) {
      fx_swap(a[0], a[2]);
      fx_swap(a[1], a[3]);
    }
    fx_rotate(a[0], a[2], t2);
    fx_rotate(a[1], a[3], t2);
    if (turns) {
#pragma unroll
      for (int j = 0; j < 4; ++j) fx_quarter(a[j], turns >> (2 * j));
    }
    fx_settle<4>(a, X);
    S.store(e, a[0]);
    S.store(e ^ b1, a[1]);
    S.store(e ^ b2, a[2]);
    S.store(e ^ b1 ^ b2, a[3]);
  }
}

static __device__ void fx_tile_phase(const TileGate& g, const int4* __restrict__ tables, Walk W,
                                     const FxTile& S, uint32_t nelem) {
  const int4* tab = tables + g.ptab;
  const int32_t fexp = g.fexp;
  for (uint32_t m = threadIdx.x, it = 0; m < nelem; m += blockDim.x, ++it) {
    const uint32_t word = W.word(it), e = word & 0xFFFFu;
    FxAmp a = S.load(e);
    fx_phase(a, __ldg(tab + (word >> 16)), fexp);
    S.store(e, a);
  }
}

// Gates that the fast mode leaves as they are: moves and signs on the integers,
// the others (controlled, or conditioned on an outcome) through FP64.
__device__ __forceinline__ void fx_exact_pair(const TileGate& g, FxAmp& a, FxAmp& b) {
  if (g.kind == SPZ_GATE_X || g.kind == SPZ_GATE_Y) {
    fx_swap(a, b);
    if (g.kind == SPZ_GATE_Y) {  // s0 <- -i s1, s1 <- i s0
      fx_quarter(a, 3u);
      fx_quarter(b, 1u);
    }
    return;
  }
  double2 x = fx_to_double(a), y = fx_to_double(b);
  switch (g.kind) {
    case SPZ_GATE_H: PairGate<SPZ_GATE_H>(g.c)(x.x, x.y, y.x, y.y); break;
    case SPZ_GATE_RX: PairGate<SPZ_GATE_RX>(g.c)(x.x, x.y, y.x, y.y); break;
    case SPZ_GATE_RY: PairGate<SPZ_GATE_RY>(g.c)(x.x, x.y, y.x, y.y); break;
    default: PairGate<SPZ_GATE_U>(g.c)(x.x, x.y, y.x, y.y); break;
  }
  a = fx_from_double(x.x, x.y);
  b = fx_from_double(y.x, y.y);
}

__device__ __forceinline__ void fx_exact_diag(const TileGate& g, bool one, FxAmp& a) {
  if (g.kind == SPZ_GATE_Z) {
    if (one) fx_quarter(a, 2u);
    return;
  }
  if (!one && g.kind == SPZ_GATE_P) return;
  double2 x = fx_to_double(a);
  if (g.kind == SPZ_GATE_P) DiagGate<SPZ_GATE_P>(g.d)(one, x.x, x.y);
  else DiagGate<SPZ_GATE_RZ>(g.d)(one, x.x, x.y);
  a = fx_from_double(x.x, x.y);
}

static __device__ void fx_tile_exact(const TileGate& g, uint64_t base, Walk W, const FxTile& S, uint32_t nw) {
  const uint32_t tmask = g.tmask, tmask2 = g.tmask2;
  const int mode = g.mode;
  const bool gone = mode == TM_DIAG_GLOBAL && (base & g.g_tbit) != 0;
  for (uint32_t m = threadIdx.x, it = 0; m < nw; m += blockDim.x, ++it) {
    const uint32_t word = W.word(it), e = word & 0xFFFFu;
    if (mode == TM_SWAP) {
      const FxAmp a = S.load(e ^ tmask2), b = S.load(e ^ tmask);
      S.store(e ^ tmask2, b);
      S.store(e ^ tmask, a);
    } else if (mode == TM_PAIR) {
      FxAmp a = S.load(e), b = S.load(e ^ tmask);
      fx_exact_pair(g, a, b);
      S.store(e, a);
      S.store(e ^ tmask, b);
    } else {
      FxAmp a = S.load(e);
      fx_exact_diag(g, mode == TM_DIAG_GLOBAL ? gone : (word >> 16) != 0, a);
      S.store(e, a);
    }
  }
}

// Op g on the tile; x: the tile's (tile_map.cuh).
static __device__ __forceinline__ void fx_tile_gate(const TileGate& g, const int4* __restrict__ tables, uint64_t base,
                                                    uint32_t x, const FxTile& S, uint32_t T) {
  const uint32_t nw = T >> g.npos;
  Walk W(g, x, fx_base_index(g, base));
  if (g.mode == TM_LAZY2) fx_tile_lazy2(g, tables, W, S, nw);
  else if (g.mode == TM_PHASE) fx_tile_phase(g, tables, W, S, nw);
  else if (g.mode == TM_PAIR && (g.fxswaps & FX_SMALL)) fx_tile_lazy<true>(g, tables, W, S, nw);
  else if (g.mode == TM_PAIR && g.kind >= FK_LAZY_H) fx_tile_lazy<false>(g, tables, W, S, nw);
  else fx_tile_exact(g, base, W, S, nw);
}

// One gate of a run inside rows of 32 amplitudes (SPZ_EXEC_SHUFFLE, see
// tile_run_shfl in circuit.cu), on R rows: lane l holds amplitude 32 r + l of a
// row, both lanes of a pair form it whole and keep their own member.  The tile's
// part of a phase index is formed once for the R rows (row by row, a fast QFT of
// 24 qubits took 8.9 ms; in FP64 7.3).
template <int R>
__device__ __forceinline__ void fx_run_gate(const TileGate& g, const int4* __restrict__ tables, uint64_t base,
                                            const uint32_t* e, FxAmp* x) {
  uint32_t idx[R];
  const uint32_t tb = g.mode == TM_PAIR ? g.tbit : 0u;
  if (g.pm > 0) {
    const uint32_t b = fx_base_index(g, base);
#pragma unroll
    for (int u = 0; u < R; ++u) idx[u] = b;
    for (int j = 0; j < g.pm; ++j) {
      const uint32_t m = g.pemask[j] & ~tb;
#pragma unroll
      for (int u = 0; u < R; ++u) idx[u] ^= (uint32_t)(__popc(e[u] & m) & 1) << j;
    }
  } else {
#pragma unroll
    for (int u = 0; u < R; ++u) idx[u] = 0;
  }
  const int4* tab = tables + g.ptab;
  if (g.mode == TM_PAIR) {
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const bool hi = (e[u] & tb) != 0;
      FxAmp p;
      p.r = (int64_t)__shfl_xor_sync(0xffffffffu, (long long)x[u].r, tb);
      p.i = (int64_t)__shfl_xor_sync(0xffffffffu, (long long)x[u].i, tb);
      p.e = __shfl_xor_sync(0xffffffffu, x[u].e, tb);
      FxAmp a[2] = {hi ? p : x[u], hi ? x[u] : p};
      if (g.kind >= FK_LAZY_H) {
        int4 w = make_int4(0, 0, 0, 0);
        if (g.pm > 0) w = __ldg(tab + idx[u]);
        if (g.fxswaps & FX_SMALL) fx_lazy_small(a, g.fx1, g.pm > 0, w, g.fxswaps, g.fxturns);
        else fx_lazy_pair(a, g.fx1, g.pm > 0, w, g.fxswaps, g.fxturns);
      } else if ((e[u] & ~tb & g.e_mask) == g.l_ones) {
        fx_exact_pair(g, a[0], a[1]);
      }
      x[u] = hi ? a[1] : a[0];
    }
  } else if (g.mode == TM_PHASE) {
#pragma unroll
    for (int u = 0; u < R; ++u)
      if ((e[u] & g.e_mask) == g.l_ones) fx_phase(x[u], __ldg(tab + idx[u]), g.fexp);
  } else {
    const bool global = g.mode == TM_DIAG_GLOBAL, gone = global && (base & g.g_tbit) != 0;
    if (global && !gone && g.kind != SPZ_GATE_RZ) return;
#pragma unroll
    for (int u = 0; u < R; ++u)
      if ((e[u] & g.e_mask) == g.l_ones) fx_exact_diag(g, global ? gone : (e[u] & g.tbit) != 0, x[u]);
  }
}

}  // namespace spz
