// The fused executor's tile geometry and gate descriptor, shared by the
// circuit executor (circuit.cu) and the fused adjoint sweep (adjoint.cu).
#pragma once

#include <vector>

#include "common.cuh"
#include "exact_mul.cuh"
#include "fixed_point.cuh"

namespace spz {

#ifndef SPZ_TILE_K
#define SPZ_TILE_K 10
#endif
constexpr int kTileMaxK = SPZ_TILE_K;  // 2^10 amplitudes x 16 B = 16 KiB of shared memory
constexpr int kTileLowBits = 3;   // qubits 0..2 always local: 64-byte contiguous rows
// Small blocks, many of them: every op in a pass ends with a block barrier, so
// the FP64 pipe stays busier with many independent small blocks per SM than
// with a few large ones.  Measured on the 30-qubit brickwork, fast mode, share
// of the DFMA issue rate: 2^12 tiles x 256 threads x 3 blocks 0.81; 2^11 x 128
// x 6 0.84; 2^10 x 64 x 12 0.86 (exact mode 0.86-0.87 for all three).
#ifndef SPZ_TILE_THREADS
#define SPZ_TILE_THREADS 64
#endif
// A state of few tiles gets blocks of up to kTileMaxThreads, so that every SM
// still has about kTileSmThreads threads to hide latencies with (tile_threads
// in circuit.cu).
#ifndef SPZ_TILE_MAX_THREADS
#define SPZ_TILE_MAX_THREADS 256
#endif
constexpr int kTileMaxThreads = SPZ_TILE_MAX_THREADS;
constexpr int kTileSmThreads = 400;
// Registers a thread: 12 blocks of 64 threads on an SM in the exact mode (26
// qubits, 10 brickwork layers: 171.1 ms; 72 registers and 13 blocks 177.7), 10
// in the fast mode, whose tiles take 21 KiB.
#ifndef SPZ_TILE_REGS
#define SPZ_TILE_REGS 80
#endif
#ifndef SPZ_FAST_REGS
#define SPZ_FAST_REGS 96
#endif
constexpr int kTileThreads = SPZ_TILE_THREADS;

// TM_MOVE: X, CX or SWAP as a step of the tile's index map; TM_END: the walk of
// the tile's store (tile_map.cuh).
enum TileMode {
  TM_PAIR = 0, TM_DIAG_LOCAL = 1, TM_DIAG_GLOBAL = 2, TM_SWAP = 3, TM_PHASE = 4, TM_LAZY2 = 5, TM_MOVE = 6, TM_END = 7
};
enum MoveKind { MV_X = 0, MV_CX1 = 1, MV_CX0 = 2, MV_SWAP = 3 };

constexpr uint32_t FX_SMALL = 0x100u;
constexpr int kFxSmallShift = 16;

struct TileGate {
  int32_t kind;
  int32_t mode;
  uint32_t tbit;    // local bit of the target (SWAP: first qubit)
  uint32_t tbit2;   // SWAP: local bit of the second qubit
  uint32_t l_ones;  // local bits that must be 1 (controls; plus the target for Z/P on s1)
  int32_t npos;     // number of local positions inserted by the enumeration
  uint8_t pos[16];  // sorted local bit positions inserted as zeros
  uint64_t g_ones;  // non-local bits the tile base must have set
  uint64_t g_zeros; // non-local bits the tile base must have clear
  uint64_t g_tbit;  // TM_DIAG_GLOBAL: the non-local target bit
  Coef c;
  // TM_PHASE: amplitude x (with x & half_bit, if half_bit != 0) is multiplied by
  // table[sum_j parity(x & pmask[j]) << j] (complex, ptab .. ptab + 2^pm - 1).
  uint64_t half_bit;
  uint64_t pmask[kPhaseMaxTerms];  // parity masks over the global index
  uint32_t pemask[kPhaseMaxTerms]; // their local part, as bits of the tile offset e
  int32_t pm;
  uint32_t ptab;
  int32_t cond;  // >= 0: applies only if that qubit's device-side measurement read 1
  uint32_t e_mask;  // pos[0 .. npos - 1] as a bit mask of the tile offset
  // TM_LAZY2 (fast mode): two lazy rotations with phase entries, `kind` on
  // tbit (coefficient c.cs) then `kind2` on tbit2 (c.sn), fused over blocks
  // of four amplitudes.  pmask / pemask [0 .. pm1) are the first op's phase
  // masks, [pm1 .. pm) the second's; the table holds three entries per index
  // (w1, w2, w1' w2), w1' being the first op's entry with its masks' tbit2
  // parities flipped.
  int32_t kind2;
  int32_t pm1;
  // SPZ_EXEC_SHUFFLE: > this gate's index, the end of a run of gates that the
  // block applies with warp shuffles (circuit.cu, tile_run_shfl); 0 otherwise.
  int32_t run_end;
  // Fast mode in fixed point (tile_fixed.cuh).  A lazy op: its rotation's t
  // (a TM_LAZY2's in fx1 and fx2), bit 0 / 1 of fxswaps: the two members are
  // swapped before the first / second rotation (FX_SMALL: t is fx1 times 2 to
  // the minus fxswaps >> kFxSmallShift), fxturns bits 2 j, 2 j + 1: the
  // power of i that output j is multiplied by, bits 8, 9: the power of i on s1
  // before the op (of a lazy op without a phase table; a table holds it in its
  // entries).  A phase op: fexp, the power of two of its table.
  FxCoef fx1, fx2;
  uint32_t fxswaps, fxturns;
  int32_t fexp;
  // The op's walk (circuit executor, tile_map.cuh): word(m) = wk0 ^ XOR of
  // wcol[i] over the bits i of item m ^ XOR of wx[q] over the bits q of the
  // tile's x; bits 0-15 the item's slot, 16 and up its phase index (or, for a
  // TM_DIAG_LOCAL, its target bit).  tmask, tmask2: what flips tbit, tbit2.
  // TM_MOVE: tmask, tmask2 are the bit numbers of target and control.
  alignas(16) uint32_t wk0;
  uint32_t tmask, tmask2, wpad;
  uint32_t wcol[12];  // kTileMaxK used: read as three 16-byte words
  uint32_t wx[kTileMaxK];
  DiagCoef d;  // P, RZ: the coefficients prepared for DiagGate
};

// The descriptor of gate g inside a tile pass whose local qubits are `local`
// (sorted); not for fast-mode phase ops.
TileGate make_tile_gate(const GateApp& g, const std::vector<int>& local);

}  // namespace spz
