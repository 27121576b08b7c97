// Conforming gradient of ondemandaccurate's accurate 3-manifolds (sm_103a).
//
// Replaces, with identical output bytes:
//   VertexLabelingToBoundaryLabeling::ComputeMINBoundary / ComputeMAXBoundary
//     (gi_labeling_to_bounary_labeling.h:48-199): one restriction byte per cell from the
//     final ascending / descending labels
//   the re-pairing loop of ondemandaccurate.cxx:1000-1063 with
//     MyRobinsNoalloc<...,4,6>::ComputeLowerStar (gi_modified_robins.h:1281-1343): the
//     touched vertices' lower stars recomputed, split by restriction label
// The ascending-manifold closure of RecordGrad (:693-699) runs afterwards as the ldir
// stage of the .grad (ldir_kernels.cu) from the roots written here.
//
// The restriction labels of the reference spread from dimension to dimension (a cell is
// restricted if a facet, or a cofacet, is), one pass each.  Spelled out, a cell's low bit
// says that one of its edges joins two different ascending labels, and its high bit that
// around it two hexes that share a quad have different descending labels at their highest
// vertices.  So a vertex finds the labels of the eight cells that it owns from 2 x 2 x 2
// ascending labels and 2 x 2 x 2 hexes, in one pass and 16 bits.  Six passes over the
// cells' bytes, two index divisions a cell, took 2.8 ms at 223 x 187 x 241 (10 M vertices);
// the two kernels here take 0.23 ms, bound by integer issue.  The re-pairing itself runs on
// the lower-star tiles (lstar_kernels.cu, conform_kernel).
#include "msc_device.cuh"

namespace msc {

namespace {

__device__ __forceinline__ void vertex_xyz(const GradDims& D, int64_t id, int64_t& x, int64_t& y, int64_t& z) {
  if ((uint64_t)id <= 0xFFFFFFFFull && D.v[0] * D.v[1] <= 0xFFFFFFFFll) {
    const uint32_t u = (uint32_t)id, X = (uint32_t)D.v[0], Y = (uint32_t)D.v[1];
    const uint32_t q = u / X, r = q / Y;
    x = u - q * X;
    y = q - r * Y;
    z = r;
    return;
  }
  x = id % D.v[0];
  y = (id / D.v[0]) % D.v[1];
  z = id / (D.v[0] * D.v[1]);
}

// IsGreater on vertex indices (gi_regular_grid_trilinear_function.h:309-314)
__device__ __forceinline__ bool vert_greater(float fa, int64_t a, float fb, int64_t b) {
  if (fa > fb) return true;
  if (fb > fa) return false;
  return a > b;
}

// The descending label at the highest vertex (Cell2HighestVertex) of the hex between
// (x, y, z) and (x+1, y+1, z+1), kept at the index of its first vertex.
__global__ void __launch_bounds__(256) hex_label_kernel(const int32_t* __restrict__ dsc, const float* __restrict__ f,
                                                        const GradDims D, int32_t* __restrict__ hex) {
  const int64_t X = D.v[0], XY = X * D.v[1], nv = XY * D.v[2];
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
    int64_t x, y, z;
    vertex_xyz(D, v, x, y, z);
    if (x == X - 1 || y == D.v[1] - 1 || z == D.v[2] - 1) continue;
    int64_t best = v;
    float fb = f[v];
#pragma unroll
    for (int s = 1; s < 8; s++) {
      const int64_t u = v + (s & 1) + ((s >> 1) & 1) * X + (s >> 2) * XY;
      const float fu = f[u];
      if (vert_greater(fu, u, fb, best)) {
        best = u;
        fb = fu;
      }
    }
    hex[v] = dsc[best];
  }
}

// Bit k of `edges` set if the two of l[0..7] (2 x 2 x 2, x fastest) that edge k joins are
// labels that differ: k = 4 a + the edge's place among those along axis a.
__device__ __forceinline__ uint32_t cut_edges(const int32_t (&l)[8]) {
  uint32_t e = 0;
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int lo = a == 0 ? 2 * k : (a == 1 ? (k & 1) + 4 * (k >> 1) : k), hi = lo + (1 << a);
      if (l[lo] != l[hi] && l[lo] != -1 && l[hi] != -1) e |= 1u << (4 * a + k);
    }
  return e;
}
// The edges of the 2 x 2 x 2 corners within the box that spans the axes of `span` (bits)
// and lies at `at` (bits) along the others.
__device__ __forceinline__ constexpr uint32_t box_edges(int span, int at) {
  uint32_t m = 0;
  for (int a = 0; a < 3; a++)
    for (int k = 0; k < 4; k++) {
      const int lo = a == 0 ? 2 * k : (a == 1 ? (k & 1) + 4 * (k >> 1) : k);
      if (((span >> a) & 1) && ((lo ^ at) & ~span & 7 & ~(1 << a)) == 0) m |= 1u << (4 * a + k);
    }
  return m;
}

// The restriction labels of the eight cells that vertex v owns (the cells 2v + s, s in
// {0,1}^3, bit sx + 2 sy + 4 sz): low bits in the low byte of bits[v] (ComputeMINBoundary),
// high bits in its high byte (ComputeMAXBoundary, interior cells only).  `out`, if given,
// takes them as a byte per cell.
__global__ void __launch_bounds__(256) restrict_kernel(const int32_t* __restrict__ asc, const int32_t* __restrict__ hex,
                                                       const GradDims D, uint16_t* __restrict__ bits,
                                                       uint8_t* __restrict__ out) {
  const int64_t X = D.v[0], Y = D.v[1], Z = D.v[2], XY = X * Y, nv = XY * Z;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
    int64_t x, y, z;
    vertex_xyz(D, v, x, y, z);
    // axes along which the cells between v and the next vertex exist, and along which v
    // is not on a face
    const int up = (x < X - 1 ? 1 : 0) | (y < Y - 1 ? 2 : 0) | (z < Z - 1 ? 4 : 0);
    const int in = up & ((x > 0 ? 1 : 0) | (y > 0 ? 2 : 0) | (z > 0 ? 4 : 0));
    uint32_t b = 0;
    if (asc) {
      int32_t l[8];
#pragma unroll
      for (int s = 0; s < 8; s++)
        l[s] = (s & ~up) ? -1 : asc[v + (s & 1) + ((s >> 1) & 1) * X + (s >> 2) * XY];
      const uint32_t e = cut_edges(l);
      if (e)
#pragma unroll
        for (int s = 1; s < 8; s++)
          if (!(s & ~up) && (e & box_edges(s, 0))) b |= 1u << s;
    }
    if (hex) {
      // hexes (x-1..x) x (y-1..y) x (z-1..z)
      const int dn = (x > 0 ? 1 : 0) | (y > 0 ? 2 : 0) | (z > 0 ? 4 : 0);
      int32_t l[8];
#pragma unroll
      for (int s = 0; s < 8; s++)
        l[s] = ((s & ~up) || (~s & 7 & ~dn)) ? -1 : hex[v - (~s & 1) - ((~s >> 1) & 1) * X - ((~s >> 2) & 1) * XY];
      const uint32_t e = cut_edges(l);
      if (e)
#pragma unroll
        for (int s = 0; s < 7; s++)
          if (!(s & ~up) && !(~s & 7 & ~in) && (e & box_edges(~s & 7, 7))) b |= 0x100u << s;
    }
    bits[v] = (uint16_t)b;
    if (out) {
      uint8_t* o = out + 2 * (x + y * D.cs[1] + z * D.cs[2]);
#pragma unroll
      for (int s = 0; s < 8; s++)
        if (!(s & ~up))
          o[(s & 1) + ((s >> 1) & 1) * D.cs[1] + (s >> 2) * D.cs[2]] =
              (uint8_t)(((b >> s) & 1u) | (((b >> (8 + s)) & 1u) << 1));
    }
  }
}

// Every cell's ldir back to the closure roots (critical cells 3 less their dimension, the
// rest 3), so that the ldir stage recomputes the closure of the new pairing.  Four cells
// to a word and four words to a load: a byte and two index divisions a thread took 230 us
// at 223 x 187 x 241; so 91 us.
__device__ __forceinline__ uint32_t root_word(uint32_t w, uint32_t dims) {
  // one per critical byte: its pair code, bits 2-4, is 7
  const uint32_t crit = (~(((w & 0x1C1C1C1Cu) ^ 0x1C1C1C1Cu) + 0x7F7F7F7Fu) >> 7) & 0x01010101u;
  return (w & 0x1F1F1F1Fu) | (0x60606060u - 32u * (dims & (crit * 3u)));
}
__global__ void __launch_bounds__(256) ldir_roots_kernel(uint8_t* __restrict__ g, const GradDims D) {
  const int64_t head = (int64_t)((16 - (reinterpret_cast<uintptr_t>(g) & 15)) & 15);  // cells before the first whole load
  const int64_t chunks = (D.ncells - head + 15) / 16 + 1;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < chunks; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i0 = head + 16 * (k - 1), lo = i0 > 0 ? i0 : 0, hi = i0 + 16 < D.ncells ? i0 + 16 : D.ncells;
    if (lo >= hi) continue;
    int64_t x = lo % D.d[0];
    const int64_t q = lo / D.d[0];
    int yz = (int)((q % D.d[1]) & 1) + (int)((q / D.d[1]) & 1);
    if (hi - lo == 16 && x + 16 <= D.d[0]) {
      uint4* w = reinterpret_cast<uint4*>(g + lo);
      uint4 r = *w;
      const uint32_t dims = 0x01010101u * (uint32_t)yz + ((x & 1) ? 0x00010001u : 0x01000100u);
      r.x = root_word(r.x, dims);
      r.y = root_word(r.y, dims);
      r.z = root_word(r.z, dims);
      r.w = root_word(r.w, dims);
      *w = r;
      continue;
    }
    int64_t row = q;
    for (int64_t i = lo; i < hi; i++) {
      g[i] = (uint8_t)root_word(g[i], (uint32_t)(yz + (int)(x & 1)));
      if (++x == D.d[0]) {
        x = 0;
        row++;
        yz = (int)((row % D.d[1]) & 1) + (int)((row / D.d[1]) & 1);
      }
    }
  }
}

}  // namespace

cudaError_t launch_restriction_labels(const int32_t* asc, const int32_t* dsc, const float* f, const GradDims& D,
                                      int32_t* hex, uint16_t* bits, uint8_t* out, int num_sms, cudaStream_t stream) {
  const int grid = num_sms * 16;
  if (dsc) {
    ::msc::count_launch();
    hex_label_kernel<<<grid, 256, 0, stream>>>(dsc, f, D, hex);
  }
  ::msc::count_launch();
  restrict_kernel<<<grid, 256, 0, stream>>>(asc, dsc ? hex : nullptr, D, bits, out);
  return cudaGetLastError();
}

cudaError_t launch_ldir_roots(uint8_t* g, const GradDims& D, int num_sms, cudaStream_t stream) {
  ::msc::count_launch();
  ldir_roots_kernel<<<num_sms * 16, 256, 0, stream>>>(g, D);
  return cudaGetLastError();
}

}  // namespace msc
