// The lower-star pairing of a single vertex from its own neighbourhood, with nothing shared
// between vertices.  For the host only: no kernel has this form any more, and the CPU tests
// (tests/lstar_core_host.cpp) check the expansion (lstar_core.cuh) in it against the oracle,
// apart from the tile's keys and byte lattice.
#pragma once
#include "lstar_core.cuh"

namespace msc {

// The (value, then vertex index) order of IsGreater
// (gi_regular_grid_trilinear_function.h:309-314): a comes before (is lower than) b.
// Position order equals global vertex-index order inside a neighbourhood.
inline bool before(float fa, int a, float fb, int b) {
  if (fb > fa) return true;
  if (fa > fb) return false;
  return b > a;
}

inline uint32_t float_bits(float v) {
  uint32_t u;
  __builtin_memcpy(&u, &v, 4);
  return u;
}

// The same order as one integer: the value's order bits (negative zero taken as
// zero, as the float comparison does) above the neighbourhood position, so that
// key(a) < key(b) exactly when before(a, b).  Inputs are NaN-free (checked).
inline uint64_t order_key(float v, int p) {
  if (v == 0.0f) v = 0.0f;
  uint32_t u = float_bits(v);
  u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ((uint64_t)u << 5) | (uint64_t)p;
}

// Per-cell key of the cell's lowest vertex (order_key), indexed by neighbourhood
// position.
struct KeyCol {
  using Key = uint64_t;
  uint64_t* base;
  int stride;
  uint64_t operator()(int p) const { return base[p * stride]; }
  // the key one step along axis a from position p
  uint64_t next(int p, int a, bool up) const {
    const int s = a == 0 ? 1 : (a == 1 ? 3 : 9);
    return base[(up ? p + s : p - s) * stride];
  }
  static uint64_t last() { return ~0ull; }  // after every key
  static bool less(uint64_t a, uint64_t b) { return a < b; }
};

// The pairing kept as bit planes over the neighbourhood's cells.
struct PlaneSink {
  uint32_t K = 0;                   // critical cells
  uint32_t C0 = 0, C1 = 0, C2 = 0;  // pair-direction code bit-planes
  // cell q (bit qb) and cell r (bit rb), one step along `axis` from q (up: in its
  // positive direction); codes 0..5 = +x,-x,+y,-y,+z,-z name each one's partner
  void pair(int, uint32_t qb, uint32_t rb, int axis, bool up) {
    const uint32_t pm = qb | rb;
    C0 |= up ? rb : qb;  // the one whose partner lies in the negative direction
    if (axis == 1) C1 |= pm;
    if (axis == 2) C2 |= pm;
  }
  void critical(int, uint32_t qb, int) { K |= qb; }
};

// First half of one vertex's work: gather its 3^ND neighbourhood through `load(p)`,
// write the cells' lowest-vertex keys to the column `col` (stride `cs`) and return the
// lower-star mask.  `interior`: the vertex is at least one vertex away from every face
// (no bounds checks).  `nan` is set if a NaN was seen.
template <int ND, class Load>
inline uint32_t lower_star_keys(int64_t x, int64_t y, int64_t z, int64_t X, int64_t Y, int64_t Z, bool interior,
                                const Load& load, uint64_t* col, int cs, bool& nan) {
  using N = Nb<ND>;
  constexpr int NPOS = N::NPOS;
  constexpr int C = N::CENTER;
  float fc = 0.f;
  load(C, fc);
  uint64_t k[NPOS];  // vertex keys, folded below into the cells' lowest-vertex keys
  k[C] = order_key(fc, C);
  uint32_t lower = 0;
  nan = (fc != fc);
  if (interior) {
    for (int p = 0; p < NPOS; p++) {
      if (p == C) continue;
      float v = 0.f;
      load(p, v);
      nan |= (v != v);
      k[p] = order_key(v, p);
      if (k[p] < k[C]) lower |= 1u << p;
    }
  } else {
    // out-of-range neighbours are left out of `lower`, so no cell outside the
    // complex enters the lower star
    const uint32_t okx = (x > 0 ? N::axis_mask(0, -1) : 0u) | N::axis_mask(0, 0) | (x < X - 1 ? N::axis_mask(0, 1) : 0u);
    const uint32_t oky = (y > 0 ? N::axis_mask(1, -1) : 0u) | N::axis_mask(1, 0) | (y < Y - 1 ? N::axis_mask(1, 1) : 0u);
    const uint32_t okz = (ND == 2) ? ~0u
                                   : ((z > 0 ? N::axis_mask(2, -1) : 0u) | N::axis_mask(2, 0) |
                                      (z < Z - 1 ? N::axis_mask(2, 1) : 0u));
    const uint32_t ok = okx & oky & okz;
    for (int p = 0; p < NPOS; p++) {
      if (p == C) continue;
      k[p] = ~0ull;
      if (!((ok >> p) & 1u)) continue;
      float v = 0.f;
      load(p, v);
      nan |= (v != v);
      k[p] = order_key(v, p);
      if (k[p] < k[C]) lower |= 1u << p;
    }
  }
  // lowest vertex of every cell: a cell's vertices form the box between the centre
  // and the vertex at its own offset, so three separable min-folds give them all
  for (int a = 0; a < ND; a++) {
    for (int p = 0; p < NPOS; p++) {
      if (N::d(p, a) == 0) continue;
      const int q = p - N::d(p, a) * N::stride(a);
      if (k[q] < k[p]) k[p] = k[q];
    }
  }
  for (int p = 0; p < NPOS; p++) col[p * cs] = k[p];
  return lower_star_mask<ND>(lower);
}

// The bytes of every cell of a processed lower star L (owned by its vertex): assigned |
// flag | pair code (7 if critical) | ldir, where ldir is 2 / 1 / 0 for critical 1- / 2- /
// 3-cells and 3 otherwise (the roots of the ascending-manifold closure).
template <int ND, class State, class Store>
inline void store_cells(const State& st, uint32_t L, uint32_t Bany, uint32_t enc_map, const Store& store) {
  using N = Nb<ND>;
  constexpr uint32_t D0 = N::dim_mask(0), D1 = N::dim_mask(1), D2 = N::dim_mask(2);
  const uint32_t K = st.K;
  uint32_t p0 = st.C0, p1 = st.C1, p2 = st.C2;
  if (enc_map != 0x2C688u) {  // not the identity (0,1,2,3,4,5): remap the non-critical codes
    uint32_t q0 = 0, q1 = 0, q2 = 0;
    uint32_t m = L & ~K;
    while (m) {
      const int p = ffs32(m) - 1;
      m &= m - 1;
      const int lc = (int)(((p0 >> p) & 1u) | (((p1 >> p) & 1u) << 1) | (((p2 >> p) & 1u) << 2));
      const uint32_t e = (enc_map >> (3 * lc)) & 7u;
      q0 |= (e & 1u) << p;
      q1 |= ((e >> 1) & 1u) << p;
      q2 |= ((e >> 2) & 1u) << p;
    }
    p0 = q0; p1 = q1; p2 = q2;
  }
  p0 |= K; p1 |= K; p2 |= K;
  const uint32_t l0 = ~K | (K & (D0 | D2));
  const uint32_t l1 = ~K | (K & (D0 | D1));
  uint32_t m = L;
  while (m) {
    const int p = ffs32(m) - 1;
    m &= m - 1;
    const uint32_t b = 1u | (((Bany >> p) & 1u) << 1) | (((p0 >> p) & 1u) << 2) | (((p1 >> p) & 1u) << 3) |
                       (((p2 >> p) & 1u) << 4) | (((l0 >> p) & 1u) << 5) | (((l1 >> p) & 1u) << 6);
    store(p, (uint8_t)b);
  }
}

// Second half: expand every boundary class of the lower star L (keys in `col`) and
// emit each owned cell's byte through `store(p, byte)`.  bx/by/bz: the vertex lies on
// the first or last plane of that axis (ignored for an interior vertex).
template <int ND, class Store>
inline void expand_and_store(uint32_t L, uint64_t* col, int cs, bool interior, bool bx, bool by, bool bz,
                             uint32_t enc_map, const Store& store) {
  PlaneSink st;
  LowerStarExpand<ND, KeyCol, PlaneSink> ex(KeyCol{col, cs}, st);
  uint32_t Bany = 0;
  if (interior)
    ex.expand(L);
  else
    Bany = run_classes<ND>(ex, L, bx, by, ND == 3 && bz);
  store_cells<ND>(st, L, Bany, enc_map, store);
}

// One vertex of the conforming re-pairing of ondemandaccurate's accurate 3-manifolds
// (ondemandaccurate.cxx:1000-1063): a vertex whose own cell, or a cell of whose lower
// star, carries a restriction label recomputes its lower star split by label; every other
// vertex keeps its pairs.  rlab(p, r): the restriction label of the cell at position p
// (called for positions inside the complex only).  Returns true if the vertex recomputed
// its lower star.  The kernel's form works on a tile (lstar_tile.cuh).
template <int ND, class Load, class Restrict, class Store>
inline bool conform_vertex(int64_t x, int64_t y, int64_t z, int64_t X, int64_t Y, int64_t Z, bool interior,
                           const Load& load, const Restrict& rlab, uint64_t* col, int cs, uint32_t enc_map,
                           const Store& store) {
  using N = Nb<ND>;
  const uint32_t okx = (x > 0 ? N::axis_mask(0, -1) : 0u) | N::axis_mask(0, 0) | (x < X - 1 ? N::axis_mask(0, 1) : 0u);
  const uint32_t oky = (y > 0 ? N::axis_mask(1, -1) : 0u) | N::axis_mask(1, 0) | (y < Y - 1 ? N::axis_mask(1, 1) : 0u);
  const uint32_t okz = (ND == 2) ? ~0u
                                 : ((z > 0 ? N::axis_mask(2, -1) : 0u) | N::axis_mask(2, 0) |
                                    (z < Z - 1 ? N::axis_mask(2, 1) : 0u));
  const uint32_t ok = okx & oky & okz;
  uint32_t r1 = 0, r2 = 0;
  for (int p = 0; p < N::NPOS; p++) {
    uint8_t r = 0;
    if ((ok >> p) & 1u) rlab(p, r);
    r1 |= (uint32_t)(r & 1u) << p;
    r2 |= (uint32_t)((r >> 1) & 1u) << p;
  }
  if (!(r1 | r2)) return false;
  bool nan = false;
  const uint32_t L = lower_star_keys<ND>(x, y, z, X, Y, Z, interior, load, col, cs, nan);
  if (!((r1 | r2) & L)) return false;  // (L holds the vertex itself)
  PlaneSink st;
  LowerStarExpand<ND, KeyCol, PlaneSink> ex(KeyCol{col, cs}, st);
  const uint32_t Bany =
      run_restricted<ND>(ex, L, r1, r2, x == 0 || x == X - 1, y == 0 || y == Y - 1, z == 0 || z == Z - 1);
  store_cells<ND>(st, L, Bany, enc_map, store);
  return true;
}

// One vertex, end to end (both halves).  Returns true if a NaN was seen.
template <int ND, class Load, class Store>
inline bool process_vertex(int64_t x, int64_t y, int64_t z, int64_t X, int64_t Y, int64_t Z, bool interior,
                           const Load& load, uint64_t* col, int cs, uint32_t enc_map, const Store& store) {
  bool nan = false;
  const uint32_t L = lower_star_keys<ND>(x, y, z, X, Y, Z, interior, load, col, cs, nan);
  expand_and_store<ND>(L, col, cs, interior, x == 0 || x == X - 1, y == 0 || y == Y - 1, z == 0 || z == Z - 1,
                       enc_map, store);
  return nan;
}

}  // namespace msc
