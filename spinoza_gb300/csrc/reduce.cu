// Measurement, probability and expectation reductions, and sampling.
// Replaces spinoza/src/measurement.rs:12-92 (measure_qubit) and the
// reductions of spinoza/src/core.rs:65-264 (reservoir sampling,
// qubit_expectation_value, xyz_expectation_value).
//
// All sums are deterministic: a fixed grid (a function of the size only),
// each thread folding its strided elements in a fixed order, a fixed warp-
// shuffle + shared-memory tree per block, then one block folding the block
// partials in a fixed tree.  Results are identical from run to run.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "exact_mul.cuh"

namespace spz {

constexpr int kRedThreads = 256;
constexpr int kMaxRedBlocks = kNumSMs * 8;  // 1216 partials per quantity

__device__ __forceinline__ double block_sum(double v, double* smem) {
  for (int off = 16; off > 0; off >>= 1) v = dadd(v, __shfl_down_sync(0xffffffffu, v, off));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  double r = 0.0;
  if (warp == 0) {
    r = lane < (int)(blockDim.x >> 5) ? smem[lane] : 0.0;
    for (int off = 16; off > 0; off >>= 1) r = dadd(r, __shfl_down_sync(0xffffffffu, r, off));
  }
  __syncthreads();
  return r;  // valid in thread 0
}

// Fold nq rows of `nblocks` partials each: out[q] = sum of partials[q][*].
__global__ void finalize_kernel(const double* __restrict__ partials, int nblocks, int nq, double* __restrict__ out) {
  __shared__ double smem[32];
  for (int q = 0; q < nq; ++q) {
    double v = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) v = dadd(v, partials[(size_t)q * nblocks + b]);
    v = block_sum(v, smem);
    if (threadIdx.x == 0) out[q] = v;
  }
}

enum RedMode { RED_PROB0 = 0, RED_X = 1, RED_Y = 2, RED_Z = 3, RED_NORM = 4 };

// Per-pair functionals over the pairs (s0, s1 = s0 | tbit) with s0 enumerated
// by inserting a zero at the target bit.  With tbit == 0 (RED_NORM) every
// amplitude is one "pair" element s0.
template <int MODE>
__global__ void __launch_bounds__(kRedThreads) pair_reduce_kernel(const double* __restrict__ re,
                                                                  const double* __restrict__ im, uint64_t nwork,
                                                                  int t, double* __restrict__ partials) {
  __shared__ double smem[32];
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tbit = 1ull << t, lowmask = tbit - 1;
  double acc = 0.0;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwork; w += stride) {
    if constexpr (MODE == RED_NORM) {
      const double a = re[w], b = im[w];
      acc = dadd(acc, dfma(a, a, dmul(b, b)));
    } else {
      const uint64_t s0 = ((w & ~lowmask) << 1) | (w & lowmask);
      const double a = re[s0], b = im[s0];
      if constexpr (MODE == RED_PROB0) {
        acc = dadd(acc, dfma(a, a, dmul(b, b)));
      } else {
        const uint64_t s1 = s0 | tbit;
        const double c = re[s1], d = im[s1];
        if constexpr (MODE == RED_X) {  // Re<psi|X psi> per pair: 2 (a c + b d)
          acc = dadd(acc, dmul(2.0, dfma(a, c, dmul(b, d))));
        } else if constexpr (MODE == RED_Y) {  // 2 (a d - b c)
          acc = dadd(acc, dmul(2.0, dfma(a, d, dmul(dneg(b), c))));
        } else {  // Z: |s0|^2 - |s1|^2
          acc = dadd(acc, dsub(dfma(a, a, dmul(b, b)), dfma(c, c, dmul(d, d))));
        }
      }
    }
  }
  const double s = block_sum(acc, smem);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// Launch a pair reduction, fold the partials into d_out[0] (device).
template <int MODE>
static int pair_reduce_to_device(spz_state_t h, int t, double* d_partials, double* d_out) {
  const uint64_t nwork = MODE == RED_NORM ? h->N : h->N / 2;
  const int blocks = std::min<int>(grid_for(nwork, kRedThreads, 8), kMaxRedBlocks);
  pair_reduce_kernel<MODE><<<blocks, kRedThreads, 0, h->stream>>>(h->re, h->im, nwork, t, d_partials);
  finalize_kernel<<<1, 1024, 0, h->stream>>>(d_partials, blocks, 1, d_out);
  SPZ_CHECK_LAUNCH("pair_reduce_kernel");
  return SPZ_OK;
}

// Read `count` doubles from the device into host memory (synchronises).
static int read_back(spz_state_t h, const double* d_src, double* host, size_t count) {
  void* pinned;
  int rc = ensure_host_scratch(h, count * sizeof(double), &pinned);
  if (rc) return rc;
  SPZ_CUDA(cudaMemcpyAsync(pinned, d_src, count * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  SPZ_CUDA(cudaStreamSynchronize(h->stream));
  std::copy((double*)pinned, (double*)pinned + count, host);
  return SPZ_OK;
}

static int reduce_scalar(spz_state_t h, int mode, int t, double* out) {
  void* scratch;
  int rc = ensure_dev_scratch(h, (kMaxRedBlocks + 8) * sizeof(double), &scratch);
  if (rc) return rc;
  double* partials = (double*)scratch;
  double* slot = partials + kMaxRedBlocks;
  switch (mode) {
    case RED_PROB0: rc = pair_reduce_to_device<RED_PROB0>(h, t, partials, slot); break;
    case RED_X: rc = pair_reduce_to_device<RED_X>(h, t, partials, slot); break;
    case RED_Y: rc = pair_reduce_to_device<RED_Y>(h, t, partials, slot); break;
    case RED_Z: rc = pair_reduce_to_device<RED_Z>(h, t, partials, slot); break;
    default: rc = pair_reduce_to_device<RED_NORM>(h, 0, partials, slot); break;
  }
  if (rc) return rc;
  return read_back(h, slot, out, 1);
}

// ------------------------------------------------ several targets at once
// <X>, <Y> or <Z> of many targets took one reduction (a whole read of the
// state, two launches and a read-back) per target.  Small states now take one
// launch with a block per target; larger ones <Z> of every qubit from one read
// (z_all_kernel) and <X> / <Y> of up to 16 targets per read (the Pauli tile
// passes).  26 qubits, energy of an Ising chain (4.3 ms) and <Z> of every
// qubit: 15.0 -> 5.2 ms.
constexpr int kSmallMultiQubits = 13;  // a block reads the state once from L2: 2^13 amplitudes in about 5 us
constexpr int kMaxTargetsArg = 64;

struct TargetList {
  int count;
  uint8_t t[kMaxTargetsArg];
};

template <int MODE>
__global__ void __launch_bounds__(1024) small_multi_kernel(const double* __restrict__ re, const double* __restrict__ im,
                                                           uint32_t pairs, TargetList T, double* __restrict__ out) {
  __shared__ double smem[32];
  const uint32_t tbit = 1u << T.t[blockIdx.x], lowmask = tbit - 1;
  double acc = 0.0;
  for (uint32_t w = threadIdx.x; w < pairs; w += blockDim.x) {
    const uint32_t s0 = ((w & ~lowmask) << 1) | (w & lowmask), s1 = s0 | tbit;
    const double a = re[s0], b = im[s0], c = re[s1], d = im[s1];
    if constexpr (MODE == RED_X) acc = dadd(acc, dmul(2.0, dfma(a, c, dmul(b, d))));
    else if constexpr (MODE == RED_Y) acc = dadd(acc, dmul(2.0, dfma(a, d, dmul(dneg(b), c))));
    else acc = dadd(acc, dsub(dfma(a, a, dmul(b, b)), dfma(c, c, dmul(d, d))));
  }
  const double s = block_sum(acc, smem);
  if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// <Z_q> of every qubit q from one read of the state.  A warp takes tiles of
// 2^10 consecutive amplitudes: lane l holds amplitudes j 64 + 2 l and the next
// one for j = 0 .. 15, so qubit 0 lies inside a load, qubits 1-5 in the lane
// and 6-9 in j.  Sums and differences of the 16 register values (a binary
// tree) give qubits 0 and 6-9 and the lane's total; lane totals, summed over
// the tiles, give 1-5; the tile's total goes to `tiles`, from which
// z_high_kernel forms the higher qubits.  About 5 FP64 instructions per
// amplitude for all qubits (5 per amplitude and qubit before), so DFMA issue
// still bounds it, not HBM.  Row r of `partials` is qubit r of the first 10.
constexpr int kZTileBits = 10;

__global__ void __launch_bounds__(kRedThreads) z_all_kernel(const double* __restrict__ re, const double* __restrict__ im,
                                                            uint64_t ntiles, double* __restrict__ tiles,
                                                            double* __restrict__ partials) {
  __shared__ double smem[32];
  const int lane = threadIdx.x & 31;
  const uint64_t warps = (uint64_t)gridDim.x * (kRedThreads / 32);
  double z0 = 0.0, zj[4] = {0.0, 0.0, 0.0, 0.0}, total = 0.0;
  for (uint64_t t = (uint64_t)blockIdx.x * (kRedThreads / 32) + (threadIdx.x >> 5); t < ntiles; t += warps) {
    const double2* r = reinterpret_cast<const double2*>(re + (t << kZTileBits)) + lane;
    const double2* m = reinterpret_cast<const double2*>(im + (t << kZTileBits)) + lane;
    double s[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const double2 a = __ldg(r + 32 * j), b = __ldg(m + 32 * j);
      const double p0 = dfma(a.x, a.x, dmul(b.x, b.x)), p1 = dfma(a.y, a.y, dmul(b.y, b.y));
      z0 = dadd(z0, dsub(p0, p1));
      s[j] = dadd(p0, p1);
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {  // bit l of j: differences of neighbours, then their sums
      const int n = 8 >> l;
      double d = dsub(s[0], s[1]);
      s[0] = dadd(s[0], s[1]);
#pragma unroll
      for (int i = 1; i < n; ++i) {
        d = dadd(d, dsub(s[2 * i], s[2 * i + 1]));
        s[i] = dadd(s[2 * i], s[2 * i + 1]);
      }
      zj[l] = dadd(zj[l], d);
    }
    total = dadd(total, s[0]);
    double v = s[0];
    for (int off = 16; off > 0; off >>= 1) v = dadd(v, __shfl_down_sync(0xffffffffu, v, off));
    if (lane == 0) tiles[t] = v;
  }
#pragma unroll
  for (int q = 0; q < kZTileBits; ++q) {
    double v;
    if (q == 0) v = z0;
    else if (q < 6) v = ((lane >> (q - 1)) & 1) ? dneg(total) : total;
    else v = zj[q - 6];
    v = block_sum(v, smem);
    if (threadIdx.x == 0) partials[(size_t)q * gridDim.x + blockIdx.x] = v;
  }
}

// Qubits kZTileBits and up from the tile totals: row b is bit b of the tile index.
__global__ void __launch_bounds__(kRedThreads) z_high_kernel(const double* __restrict__ tiles, uint64_t ntiles,
                                                             double* __restrict__ partials) {
  __shared__ double smem[32];
  const int b = (int)blockIdx.y;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, low = (1ull << b) - 1;
  double acc = 0.0;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < ntiles / 2; w += stride) {
    const uint64_t s0 = ((w & ~low) << 1) | (w & low);
    acc = dadd(acc, dsub(tiles[s0], tiles[s0 | (1ull << b)]));
  }
  acc = block_sum(acc, smem);
  if (threadIdx.x == 0) partials[(size_t)b * gridDim.x + blockIdx.x] = acc;
}

int norm_sqr_to_device(spz_state_t h, double* d_out) {
  void* scratch;
  int rc = ensure_dev_scratch(h, 64 * 1024 * sizeof(double), &scratch);
  if (rc) return rc;
  return pair_reduce_to_device<RED_NORM>(h, 0, (double*)scratch, d_out);
}

int prob0_device(spz_state_t h, uint32_t target, double* out) { return reduce_scalar(h, RED_PROB0, (int)target, out); }

// ------------------------------------------------------------ collapse
// measurement.rs:39-86: keep the measured half scaled by 1/sqrt(p), zero the other.
__global__ void collapse_kernel(double* __restrict__ re, double* __restrict__ im, uint64_t nwork, int t,
                                int outcome, double scale) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tbit = 1ull << t, lowmask = tbit - 1;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwork; w += stride) {
    const uint64_t s0 = ((w & ~lowmask) << 1) | (w & lowmask);
    const uint64_t s1 = s0 | tbit;
    const uint64_t keep = outcome ? s1 : s0, drop = outcome ? s0 : s1;
    re[keep] = dmul(re[keep], scale);
    im[keep] = dmul(im[keep], scale);
    re[drop] = 0.0;
    im[drop] = 0.0;
  }
}

int collapse_device(spz_state_t h, uint32_t target, int outcome, double scale) {
  collapse_kernel<<<grid_for(h->N / 2), kThreads, 0, h->stream>>>(h->re, h->im, h->N / 2, (int)target, outcome,
                                                                   scale);
  SPZ_CHECK_LAUNCH("collapse_kernel");
  return SPZ_OK;
}

// measure_qubit (measurement.rs:12-92) with an explicit draw.
// Outcome and scale from prob0 on the device (same arithmetic as measure_qubit).
__global__ void measure_decide_kernel(double* meas, int t, double u) {
  const double prob0 = meas[t];
  const int val = u < 1.0 - prob0 ? 1 : 0;
  meas[64 + t] = val == 0 ? 1.0 / sqrt(prob0) : 1.0 / sqrt(1.0 - prob0);
  reinterpret_cast<int32_t*>(meas + kMeasOutcomeOffset)[t] = val;
}

// Collapse with outcome and scale read from the device; with reset, the kept
// 1 half lands on the 0 half (collapse followed by X, which only moves).
__global__ void collapse_meas_kernel(double* __restrict__ re, double* __restrict__ im, uint64_t nwork, int t,
                                     const double* __restrict__ meas, int reset) {
  const int outcome = reinterpret_cast<const int32_t*>(meas + kMeasOutcomeOffset)[t];
  const double scale = meas[64 + t];
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tbit = 1ull << t, lowmask = tbit - 1;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwork; w += stride) {
    const uint64_t s0 = ((w & ~lowmask) << 1) | (w & lowmask);
    const uint64_t s1 = s0 | tbit;
    const uint64_t keep = outcome ? s1 : s0;
    const double kr = dmul(re[keep], scale), ki = dmul(im[keep], scale);
    const bool to0 = !outcome || reset;
    re[s0] = to0 ? kr : 0.0;
    im[s0] = to0 ? ki : 0.0;
    re[s1] = to0 ? 0.0 : kr;
    im[s1] = to0 ? 0.0 : ki;
  }
}

int measure_on_device(spz_state_t h, uint32_t target, int reset, double u) {
  if (target >= h->n) return fail(SPZ_ERR_INVALID_ARGUMENT, "target qubit out of range");
  if (!h->meas) {
    SPZ_CUDA(dev_alloc(&h->meas, (kMeasOutcomeOffset + 64) * sizeof(double)));
    SPZ_CUDA(cudaMemsetAsync(h->meas, 0, (kMeasOutcomeOffset + 64) * sizeof(double), h->stream));
  }
  void* scratch;
  int rc = ensure_dev_scratch(h, (kMaxRedBlocks + 8) * sizeof(double), &scratch);
  if (rc) return rc;
  rc = pair_reduce_to_device<RED_PROB0>(h, (int)target, (double*)scratch, h->meas + target);
  if (rc) return rc;
  measure_decide_kernel<<<1, 1, 0, h->stream>>>(h->meas, (int)target, u);
  collapse_meas_kernel<<<grid_for(h->N / 2), kThreads, 0, h->stream>>>(h->re, h->im, h->N / 2, (int)target, h->meas,
                                                                       reset);
  SPZ_CHECK_LAUNCH("collapse_meas_kernel");
  return SPZ_OK;
}

int measure_qubit(spz_state_t h, uint32_t target, int reset, int forced, double u, uint8_t* outcome,
                  double* prob0_out) {
  if (target >= h->n) return fail(SPZ_ERR_INVALID_ARGUMENT, "target qubit out of range");
  if (forced < -1 || forced > 1) return fail(SPZ_ERR_INVALID_ARGUMENT, "forced must be -1, 0 or 1");
  double prob0;
  int rc = prob0_device(h, target, &prob0);
  if (rc) return rc;
  const uint8_t val = forced >= 0 ? (uint8_t)forced : (uint8_t)(u < 1.0 - prob0 ? 1 : 0);
  double scale;
  if (val == 0) {
    scale = 1.0 / std::sqrt(prob0);
  } else {
    const double prob1 = 1.0 - prob0;
    scale = 1.0 / std::sqrt(prob1);
  }
  rc = collapse_device(h, target, val, scale);
  if (rc) return rc;
  if (val == 1 && reset) {  // measurement.rs:87-89
    spz_gate x{};
    x.kind = SPZ_GATE_X;
    GateApp a;
    rc = make_gate_app(h->n, x, target, 0, 0, &a);
    if (!rc) rc = launch_gate(h, a);
    if (rc) return rc;
  }
  if (outcome) *outcome = val;
  if (prob0_out) *prob0_out = prob0;
  return SPZ_OK;
}

// ------------------------------------------------------------ Pauli sums
// Diagonal terms (x_mask == 0): sum_x |psi_x|^2 D(x), D(x) = sum_k c_k (-1)^popc(x & z_k).
struct DiagTerms {
  int nterms;
  double coeff[64];
  uint64_t zmask[64];
};

__global__ void __launch_bounds__(kRedThreads) diag_pauli_kernel(const double* __restrict__ re,
                                                                 const double* __restrict__ im, uint64_t N,
                                                                 DiagTerms T, double* __restrict__ partials) {
  __shared__ double smem[32];
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  double acc = 0.0;
  for (uint64_t x = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; x < N; x += stride) {
    const double a = re[x], b = im[x];
    const double p = dfma(a, a, dmul(b, b));
    double dsum = 0.0;
    for (int k = 0; k < T.nterms; ++k) {
      const double ck = (__popcll(x & T.zmask[k]) & 1) ? dneg(T.coeff[k]) : T.coeff[k];
      dsum = dadd(dsum, ck);
    }
    acc = dfma(p, dsum, acc);
  }
  const double s = block_sum(acc, smem);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// Terms sharing one x_mask != 0.  Pairs (x, y = x ^ xmask) with x's lowest
// x_mask bit 0; w = conj(psi_x) psi_y.  For ny = popc(x_mask & z_mask):
// even ny: term = i^ny (s_y + s_x) Re w; odd ny: term = -i^(ny-1) (s_y - s_x) Im w,
// with s_x = (-1)^popc(x & z_mask).
struct XTerms {
  int nterms;
  uint64_t xmask;
  int lowbit;
  double coeff[64];
  uint64_t zmask[64];
  int ny[64];
};

__global__ void __launch_bounds__(kRedThreads) x_pauli_kernel(const double* __restrict__ re,
                                                              const double* __restrict__ im, uint64_t nwork,
                                                              XTerms T, double* __restrict__ partials) {
  __shared__ double smem[32];
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t lowmask = (1ull << T.lowbit) - 1;
  double acc = 0.0;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwork; w += stride) {
    const uint64_t x = ((w & ~lowmask) << 1) | (w & lowmask);
    const uint64_t y = x ^ T.xmask;
    const double a = re[x], b = im[x], c = re[y], d = im[y];
    const double wre = dfma(a, c, dmul(b, d));
    const double wim = dfma(a, d, dmul(dneg(b), c));
    for (int k = 0; k < T.nterms; ++k) {
      const int sx = (__popcll(x & T.zmask[k]) & 1) ? -1 : 1;
      const int sy = (__popcll(y & T.zmask[k]) & 1) ? -1 : 1;
      const int ny = T.ny[k] & 3;
      double v;
      if ((ny & 1) == 0) {
        const int f = (sx + sy) * (ny == 0 ? 1 : -1);  // i^0 = 1, i^2 = -1
        v = f == 0 ? 0.0 : (f > 0 ? (f == 2 ? dmul(2.0, wre) : wre) : (f == -2 ? dmul(-2.0, wre) : dneg(wre)));
      } else {
        const int f = (sy - sx) * (ny == 1 ? -1 : 1);  // Re(i (...)) = -Im, Re(-i (...)) = +Im
        v = f == 0 ? 0.0 : (f > 0 ? dmul(2.0, wim) : dmul(-2.0, wim));
      }
      acc = dfma(T.coeff[k], v, acc);
    }
  }
  const double s = block_sum(acc, smem);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// ------------------------------------------------ fused Pauli-sum tile passes
// One pass loads a tile of 2^k amplitudes (all values of k local qubits) into
// shared memory and accumulates, per thread:
//  * (first pass only) the diagonal terms: with w_k = parity(x & z_k), the
//    diagonal part is D(x) = sum_j T_j[w bits 8j..8j+7], T_j 256-entry tables of
//    the eight terms' signed sums, so a whole Ising-type chain costs a few FP64
//    operations per amplitude; energy += |psi_x|^2 D(x);
//  * every X/Y-type term whose X-mask lies in the tile: per pair (x, x ^ xmask)
//    the pair's contribution to Re<psi|P|psi>, one accumulator per term.
// Each term's accumulators are reduced once at the end (fixed order).
//
// DFMA issue bounds the passes, two per pair and term (26 qubits, <X> of every
// qubit and an Ising chain's energy: 7.9 ms).  A tile as 64-bit integers on one
// exponent took 5.8 ms, but held components 2^6 and more below the tile's largest
// in fewer bits than FP64: a sum that is small against the largest probability
// lost them.
constexpr int kPtMaxTerms = 16;   // X-type terms per pass
constexpr int kPtMaxDiag = 64;    // diagonal terms (8 chunks of 8)
constexpr int kPtK = 12, kPtLow = 3, kPtThreads = 512;

struct PtTerm {
  uint32_t xl;      // X-mask in local bits
  int32_t lowbit;   // lowest bit of xl
  uint64_t z;       // Z-mask (qubits)
  int32_t ny;       // Y count
  int32_t simple;   // 1: pure X string (z = 0, ny = 0): 2 Re w; 2: Y on one qubit: 2 Im w; 0: any
};

struct PtArgs {
  const double* re;
  const double* im;
  uint64_t ntiles;
  int k, c, nhigh;
  uint8_t lpos[kPtK];
  int ndiag;                 // diagonal terms handled in this pass (0 or all)
  uint64_t dz[kPtMaxDiag];   // their Z-masks
  const double* dtab;        // nchunks x 256 table entries
  // The chunk index w(x) = sum_j parity(x & dz_j) << j is linear over GF(2):
  // w(base | e) = w(base) ^ L0[e & 63] ^ L1[e >> 6] for the tile offset e.
  uint8_t lz[kPtMaxDiag / 8][2][64];
  int nt;
  PtTerm t[kPtMaxTerms];
  double* partials;          // (nt + 1) x gridDim.x
};

__global__ void __launch_bounds__(kPtThreads) pauli_tile_kernel(PtArgs A) {
  extern __shared__ double sm[];
  const uint32_t T = 1u << A.k;
  double* sre = sm;
  double* sim = sm + T;
  uint64_t* rowoff = reinterpret_cast<uint64_t*>(sm + 2 * T);
  double* red = sm + 2 * T + (T >> kPtLow) + 1;
  const uint32_t cmask = (1u << A.c) - 1;
  for (uint32_t r = threadIdx.x; r < (1u << A.nhigh); r += blockDim.x) {
    uint64_t off = 0;
    for (int j = 0; j < A.nhigh; ++j)
      if ((r >> j) & 1) off |= 1ull << A.lpos[A.c + j];
    rowoff[r] = off;
  }
  const int nch = (A.ndiag + 7) / 8;
  double* stab = red + 32;                                          // nch x 256 chunk tables
  uint8_t* slz = reinterpret_cast<uint8_t*>(stab + (size_t)nch * 256);  // nch x 2 x 64
  for (int j = threadIdx.x; j < nch * 256; j += blockDim.x) stab[j] = A.dtab[j];
  for (int j = threadIdx.x; j < nch * 128; j += blockDim.x) slz[j] = (&A.lz[0][0][0])[j];
  double acc[kPtMaxTerms + 1];
#pragma unroll
  for (int j = 0; j <= kPtMaxTerms; ++j) acc[j] = 0.0;
  __syncthreads();
  for (uint64_t tile = blockIdx.x; tile < A.ntiles; tile += gridDim.x) {
    const uint64_t base = deposit(tile, A.lpos, A.k);
    for (uint32_t e2 = threadIdx.x; e2 < T / 2; e2 += blockDim.x) {
      const uint32_t e = 2 * e2;
      const uint64_t gi = base | rowoff[e >> A.c] | (e & cmask);
      *reinterpret_cast<double2*>(sre + e) = *reinterpret_cast<const double2*>(A.re + gi);
      *reinterpret_cast<double2*>(sim + e) = *reinterpret_cast<const double2*>(A.im + gi);
    }
    __syncthreads();
    if (A.ndiag) {
      uint32_t wb[kPtMaxDiag / 8];  // the tile base's part of each chunk index
#pragma unroll
      for (int ch = 0; ch < kPtMaxDiag / 8; ++ch) {
        wb[ch] = 0;
        if (ch < nch) {
          const int jn = min(8, A.ndiag - ch * 8);
          for (int j = 0; j < jn; ++j) wb[ch] |= (uint32_t)(__popcll(base & A.dz[ch * 8 + j]) & 1) << j;
        }
      }
      for (uint32_t e = threadIdx.x; e < T; e += blockDim.x) {
        double d = 0.0;
        const uint32_t e0 = e & 63, e1 = (e >> 6) & 63;
#pragma unroll
        for (int ch = 0; ch < kPtMaxDiag / 8; ++ch) {
          if (ch >= nch) break;
          const double v = stab[ch * 256 + (wb[ch] ^ slz[ch * 128 + e0] ^ slz[ch * 128 + 64 + e1])];
          d = ch == 0 ? v : dadd(d, v);
        }
        const double a = sre[e], b = sim[e];
        acc[kPtMaxTerms] = dfma(dfma(a, a, dmul(b, b)), d, acc[kPtMaxTerms]);
      }
    }
#pragma unroll
    for (int t = 0; t < kPtMaxTerms; ++t) {
      if (t >= A.nt) break;
      const PtTerm P = A.t[t];
      const uint32_t lowmask = (1u << P.lowbit) - 1;
      // Re (even) or Im (odd) of conj(psi_x) psi_y; the factor 2 is applied at the end
      if (P.simple != 0) {
        const bool odd = P.simple == 2;
        const double *sc = odd ? sim : sre, *sd = odd ? sre : sim;
        for (uint32_t m = threadIdx.x; m < T / 2; m += blockDim.x) {
          const uint32_t x = ((m & ~lowmask) << 1) | (m & lowmask), y = x ^ P.xl;
          const double a = sre[x], b = sim[x], c = sc[y], d = sd[y];
          acc[t] = dfma(a, c, acc[t]);
          acc[t] = odd ? dfma(dneg(b), d, acc[t]) : dfma(b, d, acc[t]);
        }
        continue;
      }
      // with Z factors: added, subtracted or, where the pair's two halves cancel, left out
      const int ny = P.ny & 3;
      const bool odd = (ny & 1) != 0;
      for (uint32_t m = threadIdx.x; m < T / 2; m += blockDim.x) {
        const uint32_t x = ((m & ~lowmask) << 1) | (m & lowmask), y = x ^ P.xl;
        const uint64_t gx = base | rowoff[x >> A.c] | (x & cmask), gy = base | rowoff[y >> A.c] | (y & cmask);
        const int px = __popcll(gx & P.z) & 1, py = __popcll(gy & P.z) & 1;
        if ((px != py) != odd) continue;
        const bool neg = odd ? (py != 0) != (ny == 1) : (px != 0) != (ny != 0);
        const double a = sre[x], b = sim[x], c = odd ? sim[y] : sre[y], d = odd ? sre[y] : sim[y];
        acc[t] = neg ? dfma(dneg(a), c, acc[t]) : dfma(a, c, acc[t]);
        acc[t] = neg != odd ? dfma(dneg(b), d, acc[t]) : dfma(b, d, acc[t]);
      }
    }
    __syncthreads();
  }
  // one fixed-order block reduction per accumulator; row t < nt: term t, row nt: diagonal
#pragma unroll
  for (int s = 0; s <= kPtMaxTerms; ++s) {
    if (s < kPtMaxTerms && s >= A.nt) continue;
    const int row = s == kPtMaxTerms ? A.nt : s;
    double v = acc[s];
    for (int off = 16; off > 0; off >>= 1) v = dadd(v, __shfl_down_sync(0xffffffffu, v, off));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
      double r = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0;
      for (int off = 16; off > 0; off >>= 1) r = dadd(r, __shfl_down_sync(0xffffffffu, r, off));
      if (lane == 0) A.partials[(size_t)row * gridDim.x + blockIdx.x] = r;
    }
    __syncthreads();
  }
}

// Tile-pass evaluation; returns false (nothing launched) when the terms do not
// fit its limits, so the caller uses the per-group kernels.  With `per_term`
// (X-type terms only) each term's own value goes there, and *out is not set.
static int pauli_tiles(spz_state_t h, const spz_pauli_term* terms, size_t nterms, double* out, bool* done,
                       double* per_term = nullptr) {
  *done = false;
  const uint32_t n = h->n;
  const int k = std::min<int>((int)n, kPtK);
  const int c = std::min<int>(kPtLow, k);
  std::vector<size_t> diag, xt;
  for (size_t i = 0; i < nterms; ++i) (terms[i].x_mask ? xt : diag).push_back(i);
  if (diag.size() > (size_t)kPtMaxDiag) return SPZ_OK;
  for (size_t i : xt)
    if (__builtin_popcountll(terms[i].x_mask) > k - c) return SPZ_OK;
  // passes: greedy local sets covering the X-masks
  struct Pass { std::vector<int> local; std::vector<size_t> terms; bool diag; };
  std::vector<Pass> passes;
  std::vector<int> done_t(xt.size(), 0);
  size_t left = xt.size();
  bool first = true;
  while (left > 0 || first) {
    uint64_t L = (1ull << c) - 1;
    int nl = c;
    Pass P;
    P.diag = first && !diag.empty();
    for (size_t j = 0; j < xt.size() && (int)P.terms.size() < kPtMaxTerms; ++j) {
      if (done_t[j]) continue;
      const uint64_t need = terms[xt[j]].x_mask & ~L;
      const int add = __builtin_popcountll(need);
      if (nl + add <= k) {
        L |= need;
        nl += add;
        P.terms.push_back(xt[j]);
        done_t[j] = 1;
        left--;
      }
    }
    for (int q = 0; q < (int)n && nl < k; ++q)
      if (!((L >> q) & 1)) { L |= 1ull << q; nl++; }
    for (int q = 0; q < (int)n; ++q)
      if ((L >> q) & 1) P.local.push_back(q);
    first = false;
    if (P.diag || !P.terms.empty()) passes.push_back(std::move(P));
    if (left == 0) break;
  }
  // diagonal tables
  const size_t nd = diag.size();
  const size_t nchunks = (nd + 7) / 8;
  std::vector<double> tab(std::max<size_t>(1, nchunks) * 256, 0.0);
  for (size_t ch = 0; ch < nchunks; ++ch) {
    double c[8];
    const int count = (int)std::min<size_t>(8, nd - ch * 8);
    for (int b = 0; b < count; ++b) c[b] = terms[diag[ch * 8 + b]].coeff;
    for (int v = 0; v < (1 << count); ++v) tab[ch * 256 + v] = signed_sum(c, count, v);
  }
  const int blocks = (int)std::min<uint64_t>(1ull << (n - k), (uint64_t)kNumSMs * 3);
  const size_t slots_per_pass = (size_t)(kPtMaxTerms + 1) * blocks;
  const size_t nres = passes.size() * (kPtMaxTerms + 1);
  void* scratch;
  int rc = ensure_dev_scratch(h, (tab.size() + passes.size() * slots_per_pass + nres) * sizeof(double), &scratch);
  if (rc) return rc;
  double* dtab = (double*)scratch;
  double* dpart = dtab + tab.size();
  double* dres = dpart + passes.size() * slots_per_pass;
  SPZ_CUDA(cudaMemcpyAsync(dtab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice, h->stream));
  {  // the shared-memory opt-in, once per device (a per-device kernel attribute)
    static std::mutex attr_mu;
    static bool attr[kMaxDevices] = {};
    if (h->device < 0 || h->device >= kMaxDevices) return fail(SPZ_ERR_INVALID_ARGUMENT, "device index out of range");
    std::lock_guard<std::mutex> lock(attr_mu);
    if (!attr[h->device]) {
      SPZ_CUDA(cudaFuncSetAttribute(pauli_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)((2 << kPtK) + (1 << (kPtK - kPtLow)) + 64 + (kPtMaxDiag / 8) * (256 + 16)) * 8));
      attr[h->device] = true;
    }
  }
  for (size_t p = 0; p < passes.size(); ++p) {
    const Pass& P = passes[p];
    PtArgs A{};
    A.re = h->re;
    A.im = h->im;
    A.k = (int)P.local.size();
    A.c = c;
    A.nhigh = A.k - c;
    for (int j = 0; j < A.k; ++j) A.lpos[j] = (uint8_t)P.local[j];
    A.ntiles = 1ull << (n - A.k);
    int where[64];
    for (int q = 0; q < 64; ++q) where[q] = -1;
    for (size_t j = 0; j < P.local.size(); ++j) where[P.local[j]] = (int)j;
    if (P.diag) {
      A.ndiag = (int)nd;
      for (size_t j = 0; j < nd; ++j) A.dz[j] = terms[diag[j]].z_mask;
      A.dtab = dtab;
      // column of tile-offset bit b in chunk ch: the chunk's terms whose Z-mask
      // holds the local qubit lpos[b]
      for (int ch = 0; ch < (int)((nd + 7) / 8); ++ch) {
        uint32_t col[12] = {};
        const int jn = std::min<int>(8, (int)nd - ch * 8);
        for (int b = 0; b < A.k && b < 12; ++b)
          for (int j = 0; j < jn; ++j) col[b] |= (uint32_t)((A.dz[ch * 8 + j] >> A.lpos[b]) & 1) << j;
        for (int v = 0; v < 64; ++v) {
          uint32_t w0 = 0, w1 = 0;
          for (int b = 0; b < 6; ++b) {
            if ((v >> b) & 1) {
              w0 ^= col[b];
              w1 ^= col[b + 6];
            }
          }
          A.lz[ch][0][v] = (uint8_t)w0;
          A.lz[ch][1][v] = (uint8_t)w1;
        }
      }
    }
    A.nt = (int)P.terms.size();
    for (int t = 0; t < A.nt; ++t) {
      const spz_pauli_term& tm = terms[P.terms[t]];
      PtTerm& pt = A.t[t];
      for (int q = 0; q < 64; ++q)
        if ((tm.x_mask >> q) & 1) pt.xl |= 1u << where[q];
      pt.lowbit = __builtin_ctz(pt.xl);
      pt.z = tm.z_mask;
      pt.ny = __builtin_popcountll(tm.x_mask & tm.z_mask);
      pt.simple = tm.z_mask == 0 ? 1 : (tm.z_mask == tm.x_mask && pt.ny == 1 ? 2 : 0);
    }
    A.partials = dpart + p * slots_per_pass;
    const uint32_t T = 1u << A.k;
    const size_t nch = P.diag ? (nd + 7) / 8 : 0;
    const size_t smem = (2 * T + (T >> kPtLow) + 1 + 32 + nch * 256 + nch * 16) * sizeof(double);
    const int threads = (int)std::min<uint32_t>(kPtThreads, std::max<uint32_t>(32, T / 2));
    const int nb = (int)std::min<uint64_t>(A.ntiles, (uint64_t)blocks);
    pauli_tile_kernel<<<nb, threads, smem, h->stream>>>(A);
    finalize_kernel<<<1, 1024, 0, h->stream>>>(A.partials, nb, A.nt + 1, dres + p * (kPtMaxTerms + 1));
    SPZ_CHECK_LAUNCH("pauli_tile_kernel");
  }
  std::vector<double> res(nres);
  rc = read_back(h, dres, res.data(), nres);
  if (rc) return rc;
  if (per_term) {
    for (size_t p = 0; p < passes.size(); ++p)
      for (size_t t = 0; t < passes[p].terms.size(); ++t) {
        const size_t k = passes[p].terms[t];
        per_term[k] = terms[k].coeff * 2.0 * res[p * (kPtMaxTerms + 1) + t];
      }
    *done = true;
    return SPZ_OK;
  }
  double total = 0.0;
  for (size_t p = 0; p < passes.size(); ++p) {
    const Pass& P = passes[p];
    const double* r = res.data() + p * (kPtMaxTerms + 1);
    for (size_t t = 0; t < P.terms.size(); ++t) total += terms[P.terms[t]].coeff * 2.0 * r[t];
    if (P.diag) total += r[P.terms.size()];
  }
  *out = total;
  *done = true;
  return SPZ_OK;
}

// <X>, <Y> or <Z> of several targets (see small_multi_kernel).  One target keeps
// the pair reduction, which reads what it needs once.
static int xyz_multi(spz_state_t h, int mode, const uint32_t* targets, uint32_t ntargets, double* out) {
  if (h->n <= (uint32_t)kSmallMultiQubits) {
    void* scratch;
    int rc = ensure_dev_scratch(h, ntargets * sizeof(double), &scratch);
    if (rc) return rc;
    double* slots = (double*)scratch;
    const uint32_t pairs = (uint32_t)(h->N / 2);
    const int threads = (int)std::min<uint32_t>(1024, std::max<uint32_t>(32, pairs));
    for (uint32_t i = 0; i < ntargets; i += kMaxTargetsArg) {
      TargetList T{};
      T.count = (int)std::min<uint32_t>(kMaxTargetsArg, ntargets - i);
      for (int j = 0; j < T.count; ++j) T.t[j] = (uint8_t)targets[i + j];
      const unsigned nb = (unsigned)T.count;
      if (mode == RED_X) small_multi_kernel<RED_X><<<nb, threads, 0, h->stream>>>(h->re, h->im, pairs, T, slots + i);
      else if (mode == RED_Y) small_multi_kernel<RED_Y><<<nb, threads, 0, h->stream>>>(h->re, h->im, pairs, T, slots + i);
      else small_multi_kernel<RED_Z><<<nb, threads, 0, h->stream>>>(h->re, h->im, pairs, T, slots + i);
      SPZ_CHECK_LAUNCH("small_multi_kernel");
    }
    return read_back(h, slots, out, ntargets);
  }
  if (mode == RED_Z) {
    const int n = (int)h->n, high = n - kZTileBits;
    const uint64_t ntiles = h->N >> kZTileBits;
    const int blocks = (int)std::min<uint64_t>((ntiles + 7) / 8, (uint64_t)kNumSMs * 4);
    const int hblocks = (int)std::min<uint64_t>((ntiles / 2 + kRedThreads - 1) / kRedThreads, (uint64_t)kNumSMs);
    void* scratch;
    int rc = ensure_dev_scratch(h, (ntiles + (size_t)kZTileBits * blocks + (size_t)high * hblocks + 64) * sizeof(double),
                                &scratch);
    if (rc) return rc;
    double* tiles = (double*)scratch;
    double* low_part = tiles + ntiles;
    double* high_part = low_part + (size_t)kZTileBits * blocks;
    double* slots = high_part + (size_t)high * hblocks;
    z_all_kernel<<<blocks, kRedThreads, 0, h->stream>>>(h->re, h->im, ntiles, tiles, low_part);
    z_high_kernel<<<dim3((unsigned)hblocks, (unsigned)high), kRedThreads, 0, h->stream>>>(tiles, ntiles, high_part);
    finalize_kernel<<<1, 1024, 0, h->stream>>>(low_part, blocks, kZTileBits, slots);
    finalize_kernel<<<1, 1024, 0, h->stream>>>(high_part, hblocks, high, slots + kZTileBits);
    SPZ_CHECK_LAUNCH("z_all_kernel");
    double z[64];
    rc = read_back(h, slots, z, (size_t)n);
    if (rc) return rc;
    for (uint32_t i = 0; i < ntargets; ++i) out[i] = z[targets[i]];
    return SPZ_OK;
  }
  std::vector<spz_pauli_term> terms(ntargets);
  for (uint32_t i = 0; i < ntargets; ++i) {
    terms[i].coeff = 1.0;
    terms[i].x_mask = 1ull << targets[i];
    terms[i].z_mask = mode == RED_Y ? terms[i].x_mask : 0;
  }
  bool done = false;
  double unused;
  return pauli_tiles(h, terms.data(), terms.size(), &unused, &done, out);
}

int pauli_expectation(spz_state_t h, const spz_pauli_term* terms, size_t nterms, double* out) {
  if (nterms && !terms) return fail(SPZ_ERR_NULL, "terms is NULL");
  for (size_t k = 0; k < nterms; ++k)
    if (h->n < 64 && ((terms[k].x_mask | terms[k].z_mask) >> h->n) != 0)
      return fail(SPZ_ERR_INVALID_ARGUMENT, "Pauli term acts on a qubit out of range");
  if (nterms == 0) {
    *out = 0.0;
    return SPZ_OK;
  }
  bool done = false;
  int rc0 = pauli_tiles(h, terms, nterms, out, &done);
  if (rc0 || done) return rc0;
  // Fallback: diagonal terms, then one pass per distinct x_mask (chunks of 64 terms).
  std::vector<std::vector<size_t>> groups;
  std::vector<uint64_t> group_x;
  for (size_t k = 0; k < nterms; ++k) {
    size_t g = 0;
    for (; g < groups.size(); ++g)
      if (group_x[g] == terms[k].x_mask && groups[g].size() < 64) break;
    if (g == groups.size()) {
      groups.emplace_back();
      group_x.push_back(terms[k].x_mask);
    }
    groups[g].push_back(k);
  }
  void* scratch;
  const size_t ng = groups.size();
  int rc = ensure_dev_scratch(h, ((ng + 1) * kMaxRedBlocks + ng + 8) * sizeof(double), &scratch);
  if (rc) return rc;
  double* partials = (double*)scratch;
  double* slots = partials + (ng + 1) * kMaxRedBlocks;
  for (size_t g = 0; g < ng; ++g) {
    double* part = partials + g * kMaxRedBlocks;
    if (group_x[g] == 0) {
      DiagTerms T{};
      T.nterms = (int)groups[g].size();
      for (int j = 0; j < T.nterms; ++j) {
        T.coeff[j] = terms[groups[g][j]].coeff;
        T.zmask[j] = terms[groups[g][j]].z_mask;
      }
      const int blocks = std::min<int>(grid_for(h->N, kRedThreads, 8), kMaxRedBlocks);
      diag_pauli_kernel<<<blocks, kRedThreads, 0, h->stream>>>(h->re, h->im, h->N, T, part);
      finalize_kernel<<<1, 1024, 0, h->stream>>>(part, blocks, 1, slots + g);
    } else {
      XTerms T{};
      T.nterms = (int)groups[g].size();
      T.xmask = group_x[g];
      T.lowbit = __builtin_ctzll(group_x[g]);
      for (int j = 0; j < T.nterms; ++j) {
        const spz_pauli_term& tm = terms[groups[g][j]];
        T.coeff[j] = tm.coeff;
        T.zmask[j] = tm.z_mask;
        T.ny[j] = __builtin_popcountll(tm.x_mask & tm.z_mask);
      }
      const uint64_t nwork = h->N / 2;
      const int blocks = std::min<int>(grid_for(nwork, kRedThreads, 8), kMaxRedBlocks);
      x_pauli_kernel<<<blocks, kRedThreads, 0, h->stream>>>(h->re, h->im, nwork, T, part);
      finalize_kernel<<<1, 1024, 0, h->stream>>>(part, blocks, 1, slots + g);
    }
    SPZ_CHECK_LAUNCH("pauli kernel");
  }
  std::vector<double> vals(ng);
  if (ng) {
    rc = read_back(h, slots, vals.data(), ng);
    if (rc) return rc;
  }
  double total = 0.0;
  for (size_t g = 0; g < ng; ++g) total += vals[g];
  *out = total;
  return SPZ_OK;
}

// ------------------------------------------------------------ sampling
// Fixed blocked cumulative order (bit-identical to the oracle's restatement):
// p_i = re*re + im*im; sub-chunks of 32 amplitudes, chunks of 8 sub-chunks,
// super-chunks of 1024 chunks; every total is a sequential sum of the level
// below; bases are exclusive sequential scans; per shot: target = u * total,
// the first chunk whose end exceeds it, then inside the chunk the first
// sub-chunk whose running end exceeds it, then the first element.  A shot
// walks at most 8 sub-totals and 32 elements (instead of up to 256 elements).
constexpr uint64_t kSub = 32, kChunk = 256, kSuper = 1024;

// re*re + im*im, the squares on the integer pipes (the kernels here are bound
// by DFMA issue; the same bits).
__device__ __forceinline__ double prob_of(double r, double m) {
  const uint64_t a = (uint64_t)__double_as_longlong(r), b = (uint64_t)__double_as_longlong(m);
  double x, y;
  if (sqr_ok(a) && sqr_ok(b)) {
    x = __longlong_as_double((long long)sqr_int(a));
    y = __longlong_as_double((long long)sqr_int(b));
  } else {
    x = dmul(r, r);
    y = dmul(m, m);
  }
  return dadd(x, y);
}

__device__ __forceinline__ double prob_exact(const double* re, const double* im, uint64_t i) {
  return prob_of(re[i], im[i]);
}

// p of 32 sub-chunks of kSub amplitudes, one per row of a warp's tile: row i
// starts at amplitude at(i) (a multiple of 2), for i < rows.  Half a warp reads a
// row with 16-byte loads, eight of them in flight per lane.
template <class At>
__device__ __forceinline__ void stage_rows(const double* __restrict__ re, const double* __restrict__ im, const At& at,
                                           int rows, int lane, double (*tile)[33]) {
  constexpr int kAhead = 4;
  const int half = lane >> 4, j = 2 * (lane & 15);
  for (int i0 = 0; i0 < 32; i0 += 2 * kAhead) {
    double2 r[kAhead], m[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int i = i0 + 2 * u + half;
      if (i < rows) {
        const uint64_t g = at(i) + j;
        r[u] = *reinterpret_cast<const double2*>(re + g);
        m[u] = *reinterpret_cast<const double2*>(im + g);
      }
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int i = i0 + 2 * u + half;
      if (i < rows) {
        tile[i][j] = prob_of(r[u].x, m[u].x);
        tile[i][j + 1] = prob_of(r[u].y, m[u].y);
      }
    }
  }
}

// One warp covers 32 chunks; data is staged through shared memory 32
// amplitudes of each chunk at a time (coalesced loads), so each lane folds one
// sub-chunk per step: its sub-total, then the chunk total from the sub-totals.
__global__ void __launch_bounds__(128) chunk_total_kernel(const double* __restrict__ re,
                                                          const double* __restrict__ im, uint64_t nchunks,
                                                          uint64_t cs, uint64_t ss, double* __restrict__ totals,
                                                          double* __restrict__ subs) {
  __shared__ double tile[4][32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t warps_total = (uint64_t)gridDim.x * 4;
  const uint64_t ns = cs / ss;
  for (uint64_t c0 = ((uint64_t)blockIdx.x * 4 + warp) * 32; c0 < nchunks; c0 += warps_total * 32) {
    double t = 0.0;
    const int rows = (int)(nchunks - c0 < 32 ? nchunks - c0 : 32);
    for (uint64_t j0 = 0; j0 < cs; j0 += ss) {
      if (ss == kSub) {
        stage_rows(re, im, [&](int i) { return (c0 + i) * cs + j0; }, rows, lane, tile[warp]);
      } else {
        for (int i = 0; i < rows; ++i)
          if ((uint64_t)lane < ss) tile[warp][i][lane] = prob_exact(re, im, (c0 + i) * cs + j0 + lane);
      }
      __syncwarp();
      if (lane < rows) {
        double u = 0.0;
        for (uint64_t j = 0; j < ss; ++j) u = dadd(u, tile[warp][lane][j]);
        subs[(c0 + lane) * ns + j0 / ss] = u;
        t = dadd(t, u);
      }
      __syncwarp();
    }
    if (lane < rows) totals[c0 + lane] = t;
  }
}

// Sequential exclusive scan of v[0 .. n - 1] in place by one thread; returns the
// total.  Sixteen values at a time, so that only the adds are a chain.
__device__ __forceinline__ double scan_in_place(double* v, int n, double t) {
  int i = 0;
  for (; i + 16 <= n; i += 16) {
    double x[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = v[i + j];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const double y = x[j];
      x[j] = t;
      t = dadd(t, y);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) v[i + j] = x[j];
  }
  for (; i < n; ++i) {
    const double y = v[i];
    v[i] = t;
    t = dadd(t, y);
  }
  return t;
}

// One block per super-chunk: its chunk totals ct become their exclusive prefixes
// within the super-chunk, its total goes to st.
__global__ void __launch_bounds__(128) super_scan_kernel(double* __restrict__ ct, uint64_t nchunks,
                                                         double* __restrict__ st) {
  __shared__ double v[kSuper];
  const uint64_t c0 = (uint64_t)blockIdx.x * kSuper;
  const int n = (int)(nchunks - c0 < kSuper ? nchunks - c0 : kSuper);
  for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = ct[c0 + i];
  __syncthreads();
  if (threadIdx.x == 0) st[blockIdx.x] = scan_in_place(v, n, 0.0);
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) ct[c0 + i] = v[i];
}

// One block: super totals st become their exclusive prefixes, and the total.
__global__ void __launch_bounds__(128) super_base_kernel(double* __restrict__ st, uint64_t nsuper,
                                                         double* __restrict__ total) {
  __shared__ double v[1024];
  __shared__ double t;
  if (threadIdx.x == 0) t = 0.0;
  for (uint64_t s0 = 0; s0 < nsuper; s0 += 1024) {
    const int n = (int)(nsuper - s0 < 1024 ? nsuper - s0 : 1024);
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = st[s0 + i];
    __syncthreads();
    if (threadIdx.x == 0) t = scan_in_place(v, n, t);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) st[s0 + i] = v[i];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = t;
}

// A shot per lane.  The base of chunk c is sb[c / kSuper] + pre[c]; bases never
// fall with c, so the first chunk whose end exceeds the target is the last one
// whose base does not: found among the super-chunks, then inside one.  The warp
// then stages the 32 sub-chunks that its shots end in (whole rows, many loads in
// flight) and each lane walks its own.  27 qubits, 1e6 shots, the whole call:
// 2378 us with a lane reading its own amplitudes, DFMA squares, and chunk bases
// and ends formed by one thread per super-chunk; 1201 us now.
__global__ void __launch_bounds__(128) sample_kernel(const double* __restrict__ re, const double* __restrict__ im,
                                                     uint64_t nchunks, uint64_t cs, uint64_t ss,
                                                     const double* __restrict__ subs, const double* __restrict__ pre,
                                                     const double* __restrict__ sb, uint64_t nsuper,
                                                     const double* __restrict__ total_p, const double* __restrict__ u,
                                                     uint64_t nshots, uint64_t* __restrict__ out) {
  __shared__ double tile[4][32][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t mine = k < nshots ? k : nshots - 1;  // lanes past the end repeat the last shot
  const double total = __ldg(total_p);
  double target = dmul(u[mine], total);
  if (target >= total) target = nextafter(total, 0.0);
  uint64_t lo = 0, hi = nsuper - 1;
  while (lo < hi) {  // the last super-chunk whose base is at most the target
    const uint64_t mid = lo + (hi - lo + 1) / 2;
    if (__ldg(sb + mid) > target) hi = mid - 1; else lo = mid;
  }
  const uint64_t first = lo * kSuper;
  const double base = __ldg(sb + lo);
  lo = first;
  hi = (first + kSuper < nchunks ? first + kSuper : nchunks) - 1;
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo + 1) / 2;
    if (dadd(base, __ldg(pre + mid)) > target) hi = mid - 1; else lo = mid;
  }
  const uint64_t c = lo, ns = cs / ss;
  double r = dadd(base, __ldg(pre + c));
  uint64_t kk = ns;
  for (uint64_t q = 0; q < ns; ++q) {
    const double rn = dadd(r, __ldg(subs + c * ns + q));
    if (rn > target) {
      kk = q;
      break;
    }
    r = rn;
  }
  const uint64_t i0 = c * cs + (kk < ns ? kk : 0) * ss;
  if (ss == kSub) {
    // (32 rows: the whole warp takes part in every shuffle)
    stage_rows(re, im, [&](int i) { return __shfl_sync(0xffffffffu, i0, i); }, 32, lane, tile[warp]);
  }
  __syncwarp();
  uint64_t outcome = ~0ull;
  if (kk < ns) {
    uint64_t last_pos = ~0ull;
    for (uint64_t j = 0; j < ss; ++j) {
      const double pj = ss == kSub ? tile[warp][lane][j] : prob_exact(re, im, i0 + j);
      if (pj > 0.0) last_pos = i0 + j;
      r = dadd(r, pj);
      if (r > target) {
        outcome = i0 + j;
        break;
      }
    }
    if (outcome == ~0ull) outcome = last_pos;
  }
  if (outcome == ~0ull) {  // the last index of the chunk with p > 0, or its first
    outcome = c * cs;
    for (uint64_t j = cs; j-- > 0;)
      if (prob_exact(re, im, c * cs + j) > 0.0) {
        outcome = c * cs + j;
        break;
      }
  }
  if (k < nshots) out[k] = outcome;
}

int sample(spz_state_t h, const double* u, size_t nshots, uint64_t* out) {
  if (!u || !out) return fail(SPZ_ERR_NULL, "NULL argument");
  if (nshots == 0) return SPZ_OK;
  const uint64_t cs = std::min<uint64_t>(h->N, kChunk);
  const uint64_t ss = std::min<uint64_t>(cs, kSub);
  const uint64_t nchunks = h->N / cs;
  const uint64_t nsuper = (nchunks + kSuper - 1) / kSuper;
  // scratch: subs[N/ss] pre[nchunks] sb[nsuper] total[1] u[nshots] out[nshots]
  const size_t doubles = h->N / ss + nchunks + nsuper + 8 + 2 * nshots;
  void* scratch;
  int rc = ensure_dev_scratch(h, doubles * sizeof(double), &scratch);
  if (rc) return rc;
  double* subs = (double*)scratch;
  double* pre = subs + h->N / ss;
  double* sb = pre + nchunks;
  double* total = sb + nsuper;
  double* du = total + 8;
  uint64_t* dout = (uint64_t*)(du + nshots);
  SPZ_CUDA(cudaMemcpyAsync(du, u, nshots * sizeof(double), copy_kind(u, true), h->stream));
  const int cblocks = (int)std::min<uint64_t>((nchunks + 127) / 128, (uint64_t)kNumSMs * 16);
  chunk_total_kernel<<<cblocks, 128, 0, h->stream>>>(h->re, h->im, nchunks, cs, ss, pre, subs);
  super_scan_kernel<<<(unsigned)nsuper, 128, 0, h->stream>>>(pre, nchunks, sb);
  super_base_kernel<<<1, 128, 0, h->stream>>>(sb, nsuper, total);
  sample_kernel<<<(unsigned)((nshots + 127) / 128), 128, 0, h->stream>>>(h->re, h->im, nchunks, cs, ss, subs, pre, sb,
                                                                         nsuper, total, du, nshots, dout);
  SPZ_CHECK_LAUNCH("sampling kernels");
  double host_total;
  rc = read_back(h, total, &host_total, 1);
  if (rc) return rc;
  if (!(host_total > 0.0)) return fail(SPZ_ERR_INVALID_ARGUMENT, "state has zero norm");
  SPZ_CUDA(cudaMemcpyAsync(out, dout, nshots * sizeof(uint64_t), copy_kind(out, false), h->stream));
  SPZ_CUDA(cudaStreamSynchronize(h->stream));
  return SPZ_OK;
}

}  // namespace spz

using namespace spz;

extern "C" {

int spz_prob0(spz_state_t h, uint32_t target, double* prob0) {
  if (!h || !prob0) return fail(SPZ_ERR_NULL, "NULL argument");
  if (int rc0 = settle(h)) return rc0;
  if (target >= h->n) return fail(SPZ_ERR_INVALID_ARGUMENT, "target qubit out of range");
  return prob0_device(h, target, prob0);
}

int spz_measure_qubit(spz_state_t h, uint32_t target, int reset, int forced, double u, uint8_t* outcome,
                      double* prob0) {
  if (!h || !outcome) return fail(SPZ_ERR_NULL, "NULL argument");
  if (int rc0 = settle(h)) return rc0;
  return measure_qubit(h, target, reset, forced, u, outcome, prob0);
}

int spz_qubit_expectation_value(spz_state_t h, uint32_t target, double* out) {
  if (!h || !out) return fail(SPZ_ERR_NULL, "NULL argument");
  if (int rc0 = settle(h)) return rc0;
  if (target >= h->n) return fail(SPZ_ERR_INVALID_ARGUMENT, "target qubit out of range");
  double p0;
  int rc = prob0_device(h, target, &p0);
  if (rc) return rc;
  *out = 2.0 * p0 - 1.0;  // core.rs:217
  return SPZ_OK;
}

int spz_xyz_expectation_value(spz_state_t h, char observable, const uint32_t* targets, uint32_t ntargets,
                              double* out) {
  if (!h || (ntargets && (!targets || !out))) return fail(SPZ_ERR_NULL, "NULL argument");
  if (int rc0 = settle(h)) return rc0;
  int mode;
  switch (observable) {
    case 'x': mode = RED_X; break;
    case 'y': mode = RED_Y; break;
    case 'z': mode = RED_Z; break;
    default: return fail(SPZ_ERR_INVALID_ARGUMENT, "observable must be 'x', 'y' or 'z' (core.rs:223-225)");
  }
  for (uint32_t i = 0; i < ntargets; ++i)
    if (targets[i] >= h->n) return fail(SPZ_ERR_INVALID_ARGUMENT, "target qubit out of range");
  // One target, or <Z> of two, takes less time by the pair reductions: a read of
  // the state each, against four launches (20 qubits, <Z> of two 60 us against 84,
  // of three 92 against 84) and, up to 24 qubits, more arithmetic (24 qubits 246 and
  // 261 us; 26 qubits 798 and 747).
  const bool one_by_one =
      ntargets == 1 || (mode == RED_Z && ntargets == 2 && h->n > (uint32_t)kSmallMultiQubits && h->n <= 24);
  if (!one_by_one) return ntargets ? xyz_multi(h, mode, targets, ntargets, out) : SPZ_OK;
  for (uint32_t i = 0; i < ntargets; ++i)
    if (int rc = reduce_scalar(h, mode, (int)targets[i], &out[i])) return rc;
  return SPZ_OK;
}

int spz_pauli_expectation(spz_state_t h, const spz_pauli_term* terms, size_t nterms, double* out) {
  if (!h || !out) return fail(SPZ_ERR_NULL, "NULL argument");
  if (int rc0 = settle(h)) return rc0;
  return pauli_expectation(h, terms, nterms, out);
}

int spz_norm_sqr(spz_state_t h, double* out) {
  if (!h || !out) return fail(SPZ_ERR_NULL, "NULL argument");
  if (int rc0 = settle(h)) return rc0;
  return reduce_scalar(h, RED_NORM, 0, out);
}

int spz_sample(spz_state_t h, const double* u, size_t nshots, uint64_t* out) {
  if (!h) return fail(SPZ_ERR_NULL, "handle is NULL");
  if (int rc0 = settle(h)) return rc0;
  return sample(h, u, nshots, out);
}

}  // extern "C"
