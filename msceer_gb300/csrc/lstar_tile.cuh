// The lower-star pass over one tile of vertices, phase by phase.  Host+device: the CUDA
// kernel (lstar_kernels.cu) runs every phase with the threads of a block, the CPU test
// harness (tests/lstar_tile_host.cpp) with one.
//
// A cell's lowest vertex does not depend on the vertex that owns the cell, so the tile
// computes it once per cell (a 2x-1 lattice of cells around the tile's vertices, seven
// comparisons per vertex) instead of once per vertex and neighbouring cell (54), and the
// pairing writes each cell's byte into a byte lattice of the same shape, from which the
// bytes leave the tile row by row.  A cell of the lattice's rim belongs to this tile or
// to a neighbouring one, whichever holds its highest vertex; a byte is written where the
// pairing put one (bit 0 is set in every assigned byte).
#pragma once
#include "lstar_core.cuh"

namespace msc {

// (value, index) of a cell's lowest vertex; the index is the vertex's place in the tile
// (x fastest), whose order is the volume's.
struct alignas(8) LatKey {
  float v;
  int i;
};

template <int ND_>
struct LstarTile {
  static constexpr int ND = ND_;
  static constexpr int BX = 32, BY = ND == 3 ? 4 : 16, BZ = ND == 3 ? 4 : 1;  // vertices
  static constexpr int NV = BX * BY * BZ;
  static constexpr int FX = BX + 2, FY = BY + 2, FZ = ND == 3 ? BZ + 2 : 1;  // with one neighbour around
  static constexpr int NF = FX * FY * FZ;
  static constexpr int LX = 2 * BX + 1, LY = 2 * BY + 1, LZ = ND == 3 ? 2 * BZ + 1 : 1;  // cells
  static constexpr int NL = LX * LY * LZ;
  static constexpr int ROWS = LY * LZ;
  // lattice stride of one step along axis a, and the lattice place of vertex t
  MSC_HD static constexpr int ls(int a) { return a == 0 ? 1 : (a == 1 ? LX : LX * LY); }
  MSC_HD static constexpr int center(int x, int y, int z) {
    return (1 + 2 * x) + (1 + 2 * y) * LX + (ND == 3 ? (1 + 2 * z) * LX * LY : 0);
  }
  // lattice offset of neighbourhood position p
  MSC_HD static constexpr int off(int p) {
    return Nb<ND>::d(p, 0) + Nb<ND>::d(p, 1) * LX + (ND == 3 ? Nb<ND>::d(p, 2) * LX * LY : 0);
  }
  MSC_HD static void vertex(int t, int& x, int& y, int& z) {
    x = t % BX;
    y = (t / BX) % BY;
    z = t / (BX * BY);
  }
};

struct LatKeys {
  using Key = LatKey;
  const LatKey* at;    // lattice at the vertex
  const int16_t* off;  // lattice offsets of the neighbourhood's positions
  int sy, sz;          // lattice strides along y and z
  MSC_HD LatKey operator()(int p) const { return at[off[p]]; }
  MSC_HD LatKey next(int p, int a, bool up) const {
    const int s = a == 0 ? 1 : (a == 1 ? sy : sz);
    return at[off[p] + (up ? s : -s)];
  }
  MSC_HD static LatKey last() { return {__builtin_huge_valf(), 0x7FFFFFFF}; }
  MSC_HD static bool less(LatKey a, LatKey b) { return a.v < b.v || (a.v == b.v && a.i < b.i); }
};

// Writes each cell's byte as it is paired: assigned | flag | pair code (7 if critical) |
// ldir, where ldir is 2 / 1 / 0 for critical 1- / 2- / 3-cells (the roots of the
// ascending-manifold closure) and 3 otherwise.
struct ByteSink {
  uint8_t* at;         // byte lattice at the vertex
  const int16_t* off;
  int sy, sz;
  uint32_t bany;       // positions on the boundary (the flag bit)
  uint32_t enc_map;
  MSC_HD void pair(int q, uint32_t qb, uint32_t rb, int axis, bool up) {
    const int s = axis == 0 ? 1 : (axis == 1 ? sy : sz);
    const int o = off[q], r = up ? o + s : o - s;
    uint32_t cq = 2 * axis + (up ? 0 : 1), cr = cq ^ 1u;
    if (enc_map != 0x2C688u) {  // not the identity: a single-vertex axis
      cq = (enc_map >> (3 * cq)) & 7u;
      cr = (enc_map >> (3 * cr)) & 7u;
    }
    at[o] = (uint8_t)(0x61u | (cq << 2) | ((bany & qb) ? 2u : 0u));
    at[r] = (uint8_t)(0x61u | (cr << 2) | ((bany & rb) ? 2u : 0u));
  }
  MSC_HD void critical(int q, uint32_t qb, int dim) {
    at[off[q]] = (uint8_t)(0x1Du | ((uint32_t)(3 - dim) << 5) | ((bany & qb) ? 2u : 0u));
  }
};

// Negative zero as zero (the order takes them as equal)
MSC_HD float plain_zero(float v) {
#if defined(__CUDA_ARCH__)
  return __fadd_rn(v, 0.0f);
#else
  volatile float z = 0.0f;
  return v + z;
#endif
}

// The keys of the cells whose lowest corner is tile vertex (x, y, z), -1 <= x < BX and so
// on: its edges, quads and hex.  Of two candidates the one listed first has the smaller
// index, so it wins ties.
MSC_HD LatKey lower_key(LatKey a, LatKey b) { return b.v < a.v ? b : a; }
template <int ND>
MSC_HD void tile_cell_keys(const float* sf, LatKey* lat, int x, int y, int z) {
  using T = LstarTile<ND>;
  const int b = (x + 1) + (y + 1) * T::FX + (ND == 3 ? (z + 1) * T::FX * T::FY : 0);
  LatKey* c = lat + T::center(x, y, z);
  auto k = [&](int dx, int dy, int dz) {
    const int i = b + dx + dy * T::FX + dz * T::FX * T::FY;
    return LatKey{sf[i], i};
  };
  // (cells beyond the lattice's last plane do not exist for the rim's bases)
  const LatKey a00 = k(0, 0, 0), a10 = k(1, 0, 0), a01 = k(0, 1, 0), a11 = k(1, 1, 0);
  const LatKey ex = lower_key(a00, a10), ey = lower_key(a00, a01), exy = lower_key(ex, lower_key(a01, a11));
  const bool hx = x >= 0, hy = y >= 0, hz = ND == 2 || z >= 0;  // the base itself lies in the lattice along the axis
  if (hy && hz) c[1] = ex;
  if (hx && hz) c[T::LX] = ey;
  if (hz) c[1 + T::LX] = exy;
  if (ND == 3) {
    const LatKey b00 = k(0, 0, 1), b10 = k(1, 0, 1), b01 = k(0, 1, 1), b11 = k(1, 1, 1);
    const LatKey fx = lower_key(b00, b10), fy = lower_key(b00, b01), fxy = lower_key(fx, lower_key(b01, b11));
    constexpr int SZ = T::LX * T::LY;
    if (hx && hy) c[SZ] = lower_key(a00, b00);
    if (hy) c[1 + SZ] = lower_key(ex, fx);
    if (hx) c[T::LX + SZ] = lower_key(ey, fy);
    c[1 + T::LX + SZ] = lower_key(exy, fxy);
  }
}

// The neighbours of tile vertex (x, y, z) that come before it (value, then index), as
// neighbourhood positions; out-of-range neighbours are the caller's to mask.
template <int ND>
MSC_HD uint32_t tile_lower_mask(const float* sf, int x, int y, int z) {
  using T = LstarTile<ND>;
  using N = Nb<ND>;
  const float* v = sf + (x + 1) + (y + 1) * T::FX + (ND == 3 ? (z + 1) * T::FX * T::FY : 0);
  const float c = *v;
  uint32_t m = 0;
#if defined(__CUDA_ARCH__)
  // the sign of a difference (never of two zeros of different sign, and NaN -- of two
  // equal infinities -- has the sign bit clear) shifted in: one subtraction and one
  // shift per neighbour.  A later neighbour is lower if n - c < 0, an earlier one
  // unless c - n < 0.
#pragma unroll
  for (int p = N::NPOS - 1; p >= 0; p--) {
    if (p == N::CENTER) {
      m <<= 1;
      continue;
    }
    const float n = v[N::d(p, 0) + N::d(p, 1) * T::FX + (ND == 3 ? N::d(p, 2) * T::FX * T::FY : 0)];
    const float d = p > N::CENTER ? __fsub_rn(n, c) : __fsub_rn(c, n);
    m = __funnelshift_l(__float_as_uint(d), m, 1);
  }
  m ^= (1u << N::CENTER) - 1u;
#else
  for (int p = 0; p < N::NPOS; p++) {
    if (p == N::CENTER) continue;
    const float n = v[N::d(p, 0) + N::d(p, 1) * T::FX + (ND == 3 ? N::d(p, 2) * T::FX * T::FY : 0)];
    if (p > N::CENTER ? n < c : n <= c) m |= 1u << p;
  }
#endif
  return m;
}

// The neighbourhood positions inside a volume of extents v around vertex (x, y, z)
template <int ND>
MSC_HD uint32_t inside_mask(int64_t x, int64_t y, int64_t z, const int64_t v[3]) {
  using N = Nb<ND>;
  uint32_t ok = (x > 0 ? N::axis_mask(0, -1) : 0u) | N::axis_mask(0, 0) | (x < v[0] - 1 ? N::axis_mask(0, 1) : 0u);
  ok &= (y > 0 ? N::axis_mask(1, -1) : 0u) | N::axis_mask(1, 0) | (y < v[1] - 1 ? N::axis_mask(1, 1) : 0u);
  if (ND == 3)
    ok &= (z > 0 ? N::axis_mask(2, -1) : 0u) | N::axis_mask(2, 0) | (z < v[2] - 1 ? N::axis_mask(2, 1) : 0u);
  return ok;
}

// The restriction labels of the cells that tile vertex (x, y, z) owns, -1 <= x < BX and so
// on, into the byte lattice: bit s of `word` is the low bit of the label of cell 2v + s
// (s = sx + 2 sy + 4 sz), bit 8 + s the high bit.  They lie there as 2 * label, a value
// that no pairing writes (bit 0 of an assigned byte is set), until the cell is paired:
// only the vertex that owns a cell reads its label.
MSC_HD void tile_restrict(uint32_t word, uint8_t* bytes, int x, int y, int z) {
  using T = LstarTile<3>;
  uint8_t* c = bytes + T::center(x, y, z);
#pragma unroll
  for (int s = 0; s < 8; s++) {
    if ((!(s & 1) && x < 0) || (!(s & 2) && y < 0) || (!(s & 4) && z < 0)) continue;  // not in the lattice
    c[(s & 1) + ((s >> 1) & 1) * T::LX + (s >> 2) * T::LX * T::LY] =
        (uint8_t)((((word >> s) & 1u) << 1) | (((word >> (8 + s)) & 1u) << 2));
  }
}
// The labels of the cells of lower star L of tile vertex t as bit planes; false if all are 0
MSC_HD bool tile_labels(uint32_t L, int t, const uint8_t* bytes, const int16_t* off, uint32_t& r1, uint32_t& r2) {
  using T = LstarTile<3>;
  int x, y, z;
  T::vertex(t, x, y, z);
  const uint8_t* c = bytes + T::center(x, y, z);
  r1 = r2 = 0;
  while (L) {
    const int p = ffs32(L) - 1;
    const uint32_t pb = L & (0u - L), r = c[off[p]];
    L ^= pb;
    if (r & 2u) r1 |= pb;
    if (r & 4u) r2 |= pb;
  }
  return (r1 | r2) != 0;
}

// The pairing of tile vertex t with lower star L (vertex (x, y, z) of the volume; rim:
// the tile touches the volume's boundary)
template <int ND>
MSC_HD void tile_expand(uint32_t L, int t, bool rim, int64_t x, int64_t y, int64_t z, const int64_t v[3],
                        const LatKey* lat, uint8_t* bytes, const int16_t* off, uint32_t enc_map) {
  using T = LstarTile<ND>;
  int lx, ly, lz;
  T::vertex(t, lx, ly, lz);
  const int c = T::center(lx, ly, lz);
  ByteSink out{bytes + c, off, T::LX, T::LX * T::LY, 0u, enc_map};
  LowerStarExpand<ND, LatKeys, ByteSink> ex(LatKeys{lat + c, off, T::LX, T::LX * T::LY}, out);
  if (!rim) {
    ex.expand(L);
    return;
  }
  using N = Nb<ND>;
  const bool bx = x == 0 || x == v[0] - 1, by = y == 0 || y == v[1] - 1, bz = ND == 3 && (z == 0 || z == v[2] - 1);
  out.bany = (bx ? N::axis_mask(0, 0) : 0u) | (by ? N::axis_mask(1, 0) : 0u) | (bz ? N::axis_mask(2, 0) : 0u);
  run_classes<ND>(ex, L, bx, by, bz);
}

// The same with the lower star split by restriction label (r1, r2 of tile_labels) too
MSC_HD void tile_expand_restricted(uint32_t L, uint32_t r1, uint32_t r2, int t, bool rim, int64_t x, int64_t y,
                                   int64_t z, const int64_t v[3], const LatKey* lat, uint8_t* bytes,
                                   const int16_t* off, uint32_t enc_map) {
  using T = LstarTile<3>;
  using N = Nb<3>;
  int lx, ly, lz;
  T::vertex(t, lx, ly, lz);
  const int c = T::center(lx, ly, lz);
  ByteSink out{bytes + c, off, T::LX, T::LX * T::LY, 0u, enc_map};
  LowerStarExpand<3, LatKeys, ByteSink> ex(LatKeys{lat + c, off, T::LX, T::LX * T::LY}, out);
  const bool bx = rim && (x == 0 || x == v[0] - 1), by = rim && (y == 0 || y == v[1] - 1);
  const bool bz = rim && (z == 0 || z == v[2] - 1);
  out.bany = (bx ? N::axis_mask(0, 0) : 0u) | (by ? N::axis_mask(1, 0) : 0u) | (bz ? N::axis_mask(2, 0) : 0u);
  run_restricted<3>(ex, L, r1, r2, bx, by, bz);
}

}  // namespace msc
