// Lower-star pairing on 27-bit (3D) / 9-bit (2D) neighbourhood masks: the expansion of one
// vertex's lower star.  Host+device: the kernels (lstar_kernels.cu) and the CPU tests run it
// on a tile (lstar_tile.cuh); the tests also run it a vertex at a time (lstar_vertex.cuh).
//
// Neighbourhood position p = (dx+1) + 3(dy+1) + 9(dz+1), offsets in {-1,0,1}: the
// order of TopologicalRegularGrid3D::AdjacentCellsIterator
// (gi_topological_regular_grid.h:196-205, 687-790).  The same index names the
// vertex at vertex offset (dx,dy,dz) and the cell at cell offset (dx,dy,dz) around
// the centre vertex; a cell's vertices are the positions whose offsets are 0 or
// equal to the cell's on every axis.
//
// HomotopyExpand (gi_fast_robins_noalloc.h:147-321; gi_modified_robins.h:999-1199)
// restated on sets.  With all lower-dimensional cells processed, a (d+1)-cell c is
// a pairing candidate for its d-facet q exactly when c is in the class S, not yet
// processed, and q is its only unprocessed facet in S (num_missing == 1).  Calling
// those cells "ready" (set R), the reference's restart-from-the-first-cell scan picks
// the first q, in star order, that is the remaining facet of some ready cell -- the
// lowest set bit of Q = facets(R) -- and pairs it with the ready cofacet whose lowest
// vertex comes first (cofacet order +x,-x,+y,-y,+z,-z, first wins ties,
// PickLowestCandidate :130-143).  With no ready cell, the unprocessed d-cell with the
// first lowest vertex becomes critical (:293-310).  Each step costs a few dozen bit
// operations instead of a rescan of the class.
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define MSC_HD __host__ __device__ __forceinline__
#else
#define MSC_HD inline
#endif

namespace msc {

MSC_HD int ffs32(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __ffs((int)x);
#else
  return __builtin_ffs((int)x);
#endif
}

template <int ND>
struct Nb {
  static constexpr int NPOS = (ND == 3) ? 27 : 9;
  static constexpr int CENTER = (ND == 3) ? 13 : 4;
  MSC_HD static constexpr int d(int p, int a) {
    return a == 0 ? p % 3 - 1 : (a == 1 ? (p / 3) % 3 - 1 : p / 9 - 1);
  }
  MSC_HD static constexpr int stride(int a) { return a == 0 ? 1 : (a == 1 ? 3 : 9); }
  MSC_HD static constexpr int dim(int p) {
    int s = 0;
    for (int a = 0; a < ND; a++) s += d(p, a) != 0;
    return s;
  }
  MSC_HD static constexpr uint32_t dim_mask(int k) {
    uint32_t m = 0;
    for (int p = 0; p < NPOS; p++)
      if (dim(p) == k) m |= 1u << p;
    return m;
  }
  MSC_HD static constexpr uint32_t axis_mask(int a, int val) {
    uint32_t m = 0;
    if (a >= ND) return val == 0 ? dim_mask(0) | dim_mask(1) | dim_mask(2) | dim_mask(3) : 0u;
    for (int p = 0; p < NPOS; p++)
      if (d(p, a) == val) m |= 1u << p;
    return m;
  }
  // AND-fold along axis A: keep bit p only if the bit of p with axis A zeroed is set
  template <int A>
  MSC_HD static uint32_t fold(uint32_t m) {
    constexpr int s = stride(A);
    constexpr uint32_t mp = axis_mask(A, 1), mm = axis_mask(A, -1), m0 = axis_mask(A, 0);
    return m & (((m << s) & mp) | ((m >> s) & mm) | m0);
  }
};

template <int ND, class Keys, class Sink>
struct LowerStarExpand {
  using N = Nb<ND>;
  using Key = typename Keys::Key;
  Keys lk;  // lowest-vertex key per cell
  Sink& out;

  MSC_HD LowerStarExpand(Keys k, Sink& s) : lk(k), out(s) {}

  // the cell of U whose lowest vertex comes first (first in star order wins ties)
  MSC_HD int lowest_of(uint32_t U) const {
    int q = ffs32(U) - 1;
    Key kb = lk(q);
    uint32_t W = U & (U - 1);
    while (W) {
      const int o = ffs32(W) - 1;
      W &= W - 1;
      const Key ko = lk(o);
      if (Keys::less(ko, kb)) {
        q = o;
        kb = ko;
      }
    }
    return q;
  }

  // The vertex's own step in its class S; returns the cells of S left to process.
  MSC_HD uint32_t center(uint32_t S) {
    constexpr int C = N::CENTER;
    constexpr uint32_t EDGES = N::dim_mask(1);
    uint32_t A = S;  // unprocessed cells of the class
    if (S & (1u << C)) {
      A &= ~(1u << C);
      // the vertex pairs with the edge to its lowest neighbour (steepest descent; an
      // edge's lowest vertex is its other end, so no two keys are equal)
      if (!(S & EDGES)) {
        out.critical(C, 1u << C, 0);
      } else {
        Key kb = Keys::last();
        uint32_t rb = 0;
        int axis = 0;
        bool up = false;
#pragma unroll
        for (int a = 0; a < ND; a++) {
#pragma unroll
          for (int s = 0; s < 2; s++) {
            const uint32_t eb = 1u << (C + (s == 0 ? N::stride(a) : -N::stride(a)));
            if (!(S & eb)) continue;
            const Key k = lk.next(C, a, s == 0);
            if (Keys::less(k, kb)) {
              kb = k;
              rb = eb;
              axis = a;
              up = s == 0;
            }
          }
        }
        A &= ~rb;
        out.pair(C, 1u << C, rb, axis, up);
      }
    }
    return A;
  }

  // One step of HomotopyExpand on the cells A of a class that are left, always in the
  // lowest dimension that still has unprocessed cells -- the order of the reference's
  // per-dimension loops -- so the loop body is the same straight-line set algebra for
  // every thread of a warp.
  // Within the neighbourhood a cell with offset 0 along an axis has its two cofacets
  // there one stride away on either side, so facets and cofacets along an axis are the
  // set shifted both ways, of the cells (before) or kept on the cells (after) of
  // offset 0.
  MSC_HD void step(uint32_t& A) {
    constexpr uint32_t DM1 = N::dim_mask(1), DM2 = N::dim_mask(2), DM3 = N::dim_mask(3);
    constexpr uint32_t M0 = N::axis_mask(0, 0), M1 = N::axis_mask(1, 0), M2 = N::axis_mask(2, 0);
    constexpr int S1 = N::stride(1), S2 = N::stride(2);
    const uint32_t A1 = A & DM1, A2 = A & DM2;
    const uint32_t D = A1 ? A1 : (A2 ? A2 : A);        // the dimension worked on
    const uint32_t U = A1 ? A2 : (A2 ? A & DM3 : 0u);  // and the next one
    const int dim = A1 ? 1 : (A2 ? 2 : 3);
    const uint32_t Z0 = D & M0, Z1 = D & M1, Z2 = ND == 3 ? D & M2 : 0u;
    const uint32_t F0 = (Z0 << 1) | (Z0 >> 1), F1 = (Z1 << S1) | (Z1 >> S1), F2 = (Z2 << S2) | (Z2 >> S2);
    const uint32_t one = (F0 ^ F1 ^ F2) & ~(F0 & F1 & F2);  // exactly one unprocessed facet
    const uint32_t R = U & one;                             // ready (d+1)-cells
    const uint32_t W0 = R & F0, W1 = R & F1, W2 = R & F2;
    uint32_t Q = (((W0 << 1) | (W0 >> 1)) & M0) | (((W1 << S1) | (W1 >> S1)) & M1);
    if (ND == 3) Q |= ((W2 << S2) | (W2 >> S2)) & M2;
    if (Q) {
      const uint32_t qb = Q & (0u - Q);
      const int q = ffs32(Q) - 1;
      // ready cofacets of q, i.e. its candidates
      const uint32_t q0 = qb & M0, q1 = qb & M1, q2 = ND == 3 ? qb & M2 : 0u;
      const uint32_t u0 = R & (q0 << 1), d0 = R & (q0 >> 1), u1 = R & (q1 << S1), d1 = R & (q1 >> S1);
      const uint32_t u2 = R & (q2 << S2), d2 = R & (q2 >> S2);
      const uint32_t c1 = u1 | d1, c2 = u2 | d2, cm = u0 | d0 | c1 | c2;
      uint32_t rb = cm;
      if (cm & (cm - 1)) {
        // several: the first in cofacet order (+x,-x,+y,-y,+z,-z) whose lowest
        // vertex comes first wins (PickLowestCandidate)
        Key kb = Keys::last();
        rb = 0;
        const uint32_t cand[6] = {u0, d0, u1, d1, u2, d2};
#pragma unroll
        for (int j = 0; j < 2 * ND; j++) {
          if (!cand[j]) continue;
          const Key k = lk.next(q, j >> 1, (j & 1) == 0);
          if (Keys::less(k, kb)) {
            kb = k;
            rb = cand[j];
          }
        }
      }
      A &= ~(qb | rb);
      out.pair(q, qb, rb, (rb & c1) ? 1 : ((rb & c2) ? 2 : 0), rb > qb);
    } else {
      const int q = lowest_of(D);
      A &= ~(1u << q);
      out.critical(q, 1u << q, dim);
    }
  }

  // HomotopyExpand of one boundary class S of the lower star.
  MSC_HD void expand(uint32_t S) {
    uint32_t A = center(S);
    for (int guard = 0; guard < N::NPOS && A; guard++) step(A);
  }

  // HomotopyExpand of every class of the lower star L: two cells are of one class if
  // they agree in all planes of k.  The classes know nothing of one another, so their
  // order is free, and one loop takes them all: the lanes of a warp meet in it, whatever
  // the number of their classes.
  template <int NK>
  MSC_HD void expand_classes(uint32_t L, const uint32_t (&k)[NK]) {
    auto same = [&](int q) {
      uint32_t m = ~0u;
#pragma unroll
      for (int i = 0; i < NK; i++) m &= ((k[i] >> q) & 1u) ? k[i] : ~k[i];
      return m;
    };
    const uint32_t S = L & same(N::CENTER);
    uint32_t rest = L & ~S, A = center(S);
    for (int guard = 0; guard < N::NPOS && (A | rest); guard++) {
      if (!A) {
        A = rest & same(ffs32(rest) - 1);
        rest &= ~A;
      }
      step(A);
    }
  }
};

// Lower star from the mask of neighbours that come before the centre: the cells all
// of whose other vertices are lower (three separable AND-folds).  Out-of-range
// neighbours are never "lower", so cells outside the complex drop out too.
template <int ND>
MSC_HD uint32_t lower_star_mask(uint32_t lower) {
  using N = Nb<ND>;
  uint32_t L = lower | (1u << N::CENTER);
  L = N::template fold<0>(L);
  L = N::template fold<1>(L);
  if (ND == 3) L = N::template fold<2>(L);
  return L;
}

// Runs every boundary class of one vertex's lower star.  bx/by/bz: the vertex lies
// on the first or last plane of that axis.  Class k = cells on the boundary of
// exactly k axes (boundaryValue, gi_topological_regular_grid.h:1291-1297; the split
// is MyRobinsNoalloc::ComputeLowerStar, gi_modified_robins.h:1305-1324).
template <int ND, class State>
MSC_HD uint32_t run_classes(State& st, uint32_t L, bool bx, bool by, bool bz) {
  using N = Nb<ND>;
  constexpr uint32_t A0x = N::axis_mask(0, 0), A0y = N::axis_mask(1, 0), A0z = N::axis_mask(2, 0);
  const uint32_t B0 = bx ? A0x : 0u;
  const uint32_t B1 = by ? A0y : 0u;
  const uint32_t B2 = (ND == 3 && bz) ? A0z : 0u;
  const uint32_t Bany = B0 | B1 | B2;
  if (!Bany) {
    st.expand(L);
  } else {
    const uint32_t all3 = B0 & B1 & B2;
    const uint32_t two = ((B0 & B1) | (B0 & B2) | (B1 & B2)) & ~all3;
    const uint32_t one = (B0 ^ B1 ^ B2) & ~all3;
    uint32_t c;
    if ((c = L & ~Bany)) st.expand(c);
    if ((c = L & one)) st.expand(c);
    if ((c = L & two)) st.expand(c);
    if ((c = L & all3)) st.expand(c);
  }
  return Bany;
}

// The constrained re-pairing of ondemandaccurate's accurate 3-manifolds
// (MyRobinsNoalloc<...,4,6>::ComputeLowerStar with a restriction map,
// gi_modified_robins.h:1281-1343): the lower star L split by class
// restriction_label * maxDim + boundaryValue (maxDim = 3).  A restriction label is 0 to
// 3: bit p of r1 / r2 is the low / high bit of the label of the cell at position p.
// Away from the boundary the label is the class.
template <int ND, class Expand>
MSC_HD uint32_t run_restricted(Expand& ex, uint32_t L, uint32_t r1, uint32_t r2, bool bx, bool by, bool bz) {
  using N = Nb<ND>;
  if (!(bx || by || (ND == 3 && bz))) {
    const uint32_t k[2] = {r1, r2};
    ex.expand_classes(L, k);
    return 0u;
  }
  const uint32_t B0 = bx ? N::axis_mask(0, 0) : 0u;
  const uint32_t B1 = by ? N::axis_mask(1, 0) : 0u;
  const uint32_t B2 = (ND == 3 && bz) ? N::axis_mask(2, 0) : 0u;
  // boundary value 3 with label r is value 0 with label r + 1
  const uint32_t all3 = B0 & B1 & B2, carry = r1 & all3;
  const uint32_t k[5] = {(B0 ^ B1 ^ B2) & ~all3, ((B0 & B1) | (B0 & B2) | (B1 & B2)) & ~all3, r1 ^ all3, r2 ^ carry,
                         r2 & carry};
  ex.expand_classes(L, k);
  return B0 | B1 | B2;
}

}  // namespace msc

#if !defined(__CUDACC__)
#include "lstar_vertex.cuh"
#endif
