// Where a tile's amplitudes lie while a pass works on it.
//
// X, CX and SWAP only move amplitudes.  Inside a pass they move nothing: the
// tile keeps its amplitudes in place and the pass keeps an index map, so these
// gates cost no shared-memory traffic and no barrier (they were about half of
// a brickwork pass's ops).  The offset e that an amplitude has in program order
// and its slot p are related by e = B p ^ x over GF(2): B is known on the host
// (CX and SWAP), x is kept by the kernel (X, whose controls may sit on qubits
// outside the tile).  An op enumerates its work items m linearly: slot(m) is an
// XOR of columns over the bits of m, with the parities that select a phase
// entry in the same word.
#pragma once

#include <vector>

#include "executor.cuh"

namespace spz {

// ------------------------------------------------------------ host
struct TileMap {
  int k;
  uint32_t row[kTileMaxK];  // e bit q = parity(p & row[q]) ^ x bit q
  uint32_t col[kTileMaxK];  // slot(e) = XOR of col[q] over the bits q of e ^ x
  explicit TileMap(int k_) : k(k_) {
    for (int q = 0; q < kTileMaxK; ++q) row[q] = col[q] = 1u << q;
  }
  void cx(int c, int t) {
    row[t] ^= row[c];
    col[c] ^= col[t];
  }
  void swap(int a, int b) {
    std::swap(row[a], row[b]);
    std::swap(col[a], col[b]);
  }
};

inline uint32_t parity32(uint32_t v) { return (uint32_t)__builtin_popcount(v) & 1u; }

// The walk of op t under the map: items have the offset bits of t.e_mask fixed
// (set where t.l_ones has them); sel[0 .. nsel) are the offset masks whose parities
// come in bits 16 and up of a word.  (On fixed arrays: an execute forms a walk per
// gate, 0.3 us each with vectors, more than a small circuit's gate takes on the GPU.)
inline void set_walk(TileGate* t, const TileMap& map, const uint32_t* sel, int nsel) {
  struct Fn {
    uint32_t f, xs, v;  // parity(p & f) = v ^ parity(x & xs)
  };
  Fn fn[kTileMaxK];
  int piv[kTileMaxK], nf = 0;
  uint32_t fixed = 0;
  for (uint32_t left = t->e_mask & ((1u << map.k) - 1u); left; left &= left - 1) {
    const int q = __builtin_ctz(left);
    Fn n{map.row[q], 1u << q, (t->l_ones >> q) & 1u};
    for (int i = 0; i < nf; ++i)
      if ((n.f >> piv[i]) & 1) n = Fn{n.f ^ fn[i].f, n.xs ^ fn[i].xs, n.v ^ fn[i].v};
    const int p = 31 - __builtin_clz(n.f);  // highest bit: the low slot bits stay with the low bits of m
    for (int i = 0; i < nf; ++i)
      if ((fn[i].f >> p) & 1) fn[i] = Fn{fn[i].f ^ n.f, fn[i].xs ^ n.xs, fn[i].v ^ n.v};
    fn[nf] = n;
    piv[nf++] = p;
    fixed |= 1u << p;
  }
  uint32_t g[16] = {};  // sel as masks of the slot
  for (int l = 0; l < nsel; ++l)
    for (uint32_t left = sel[l]; left; left &= left - 1) g[l] ^= map.row[__builtin_ctz(left)];
  auto with_sel = [&](uint32_t p, uint32_t e) {  // e: offset bits that x adds beside the slot
    for (int l = 0; l < nsel; ++l) p |= (parity32(p & 0xFFFFu & g[l]) ^ parity32(e & sel[l])) << (16 + l);
    return p;
  };
  int m = 0;
  for (int b = 0; b < map.k; ++b) {
    if ((fixed >> b) & 1) continue;
    uint32_t p = 1u << b;
    for (int j = 0; j < nf; ++j)
      if ((fn[j].f >> b) & 1) p |= 1u << piv[j];
    t->wcol[m++] = with_sel(p, 0);
  }
  for (; m < 12; ++m) t->wcol[m] = 0;
  uint32_t k0 = 0;
  for (int j = 0; j < nf; ++j) k0 |= fn[j].v << piv[j];
  t->wk0 = with_sel(k0, 0);
  for (int q = 0; q < kTileMaxK; ++q) {
    uint32_t p = 0;
    for (int j = 0; j < nf; ++j) p |= ((fn[j].xs >> q) & 1u) << piv[j];
    t->wx[q] = q < map.k ? with_sel(p, 1u << q) : 0;
  }
  auto slot_of = [&](uint32_t bit) { return bit ? map.col[__builtin_ctz(bit)] : 0u; };
  t->tmask = slot_of(t->tbit);
  t->tmask2 = slot_of(t->tbit2);
}

// Give every op of a pass (k local qubits) its walk, turn the moves into steps
// of the map (unless `keep_moves`), and append the walk of the tile's store.
// A step that leaves x as it is (a CX or SWAP while x is 0) needs no op.
inline void map_pass(std::vector<TileGate>* ops, int k, bool keep_moves) {
  TileMap map(k);
  bool x_set = false;  // x may be other than 0
  std::vector<TileGate> out;
  out.reserve(ops->size() + 1);
  for (TileGate& t : *ops) {
    const bool anywhere = t.g_ones == 0 && t.g_zeros == 0 && t.cond < 0;
    const uint32_t local = t.e_mask & ~t.tbit;  // of an X: its controls inside the tile
    if (!keep_moves && t.mode == TM_PAIR && t.kind == SPZ_GATE_X && (local == 0 || (anywhere && !(local & (local - 1))))) {
      t.mode = TM_MOVE;
      t.tmask = (uint32_t)__builtin_ctz(t.tbit);
      if (local) {
        t.kind = (t.l_ones & local) ? MV_CX1 : MV_CX0;
        t.tmask2 = (uint32_t)__builtin_ctz(local);
        map.cx((int)t.tmask2, (int)t.tmask);
      } else {
        t.kind = MV_X;
      }
      x_set = x_set || t.kind != MV_CX1;
      if (x_set) out.push_back(t);
      continue;
    }
    if (!keep_moves && t.mode == TM_SWAP && anywhere && t.e_mask == (t.tbit | t.tbit2)) {
      t.mode = TM_MOVE;
      t.kind = MV_SWAP;
      t.tmask = (uint32_t)__builtin_ctz(t.tbit);
      t.tmask2 = (uint32_t)__builtin_ctz(t.tbit2);
      map.swap((int)t.tmask, (int)t.tmask2);
      if (x_set) out.push_back(t);
      continue;
    }
    if (t.mode == TM_DIAG_LOCAL) set_walk(&t, map, &t.tbit, 1);
    else set_walk(&t, map, t.pemask, t.pm);
    out.push_back(t);
  }
  TileGate end{};  // item m: the slot of offset 2 m; tmask: what offset 2 m + 1 adds
  end.mode = TM_END;
  for (int q = 0; q < k; ++q) {
    if (q) end.wcol[q - 1] = map.col[q];
    end.wx[q] = map.col[q];
  }
  end.tmask = map.col[0];
  out.push_back(end);
  ops->swap(out);
}

// ------------------------------------------------------------ device
// A move's step of x.
__device__ __forceinline__ uint32_t move_step(const TileGate& g, uint32_t x) {
  const uint32_t t = g.tmask, c = g.tmask2;
  switch (g.kind) {
    case MV_X: return x ^ (1u << t);
    case MV_CX1: return x ^ (((x >> c) & 1u) << t);
    case MV_CX0: return x ^ ((((x >> c) & 1u) ^ 1u) << t);
    default: {  // MV_SWAP
      const uint32_t d = ((x >> t) ^ (x >> c)) & 1u;
      return x ^ (d << t) ^ (d << c);
    }
  }
}

// This thread's words of an op: word(it) for item m = it * blockDim.x +
// threadIdx.x, asked for in order from it = 0.
struct Walk {
  uint32_t w;           // the word of the current group of four items
  uint32_t c0, c1;      // columns of the item bits inside the group
  const uint32_t* cols; // the columns above
  __device__ __forceinline__ Walk(const TileGate& g, uint32_t x, uint32_t sel0 = 0u) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(g.wcol)), b = __ldg(reinterpret_cast<const uint4*>(g.wcol) + 1);
    const uint32_t t = threadIdx.x;
    const int lg = 31 - __clz((int)blockDim.x);  // 5 to 9
    c0 = __ldg(g.wcol + lg);
    c1 = __ldg(g.wcol + lg + 1);
    cols = g.wcol + lg + 2;
    w = __ldg(&g.wk0) ^ (sel0 << 16);
    w ^= (t & 1u) ? a.x : 0u;
    w ^= (t & 2u) ? a.y : 0u;
    w ^= (t & 4u) ? a.z : 0u;
    w ^= (t & 8u) ? a.w : 0u;
    w ^= (t & 16u) ? b.x : 0u;
    w ^= (t & 32u) ? b.y : 0u;
    if (lg > 6) {
      w ^= (t & 64u) ? b.z : 0u;
      w ^= (t & 128u) ? b.w : 0u;
      w ^= (t & 256u) ? __ldg(g.wcol + 8) : 0u;
    }
    for (; x; x &= x - 1) w ^= __ldg(&g.wx[__ffs((int)x) - 1]);
  }
  __device__ __forceinline__ uint32_t word(uint32_t it) {
    if (it && !(it & 3u)) {  // the next group: item bits 2 .. z change
      const uint32_t z = __ffs((int)(it >> 2)) - 1u;
      for (uint32_t j = 0; j <= z; ++j) w ^= __ldg(cols + j);
    }
    return w ^ ((it & 1u) ? c0 : 0u) ^ ((it & 2u) ? c1 : 0u);
  }
};

}  // namespace spz
