// K1: lower-star discrete gradient, one thread per vertex (sm_103a).
//
// Replaces, with identical output bytes:
//   RegularGridMaxMinVertexLabeling3D::ComputeOutput   gi_max_vertex_labeling.h:1119-1339
//   SlidingWindowRobinsNoalloc::ComputePairing_sliding gi_fast_robins_noalloc.h:1254-1535
//     (interior: ComputeLowerStar :353-428, HomotopyExpand :147-321)
//   MyRobinsNoalloc<...,5,4>::ComputeLowerStar          gi_modified_robins.h:1281-1343
//     (boundary planes, lower star split by cell boundaryValue)
//   2D: RegularGridMaxMinVertexLabeling2D + MyRobinsNoalloc<TopologicalRegularGrid2D,...,4,6>
//       ::ComputePairing (gi_modified_robins.h:1344-1402)
// and the parts of setAscendingManifoldDimensions / outputToFile that are local to a
// cell: the boundary flag and the ldir value of critical cells (the roots of the
// ascending-manifold closure, finished by ldir_kernels.cu).
//
// The max/min vertex labeling is never materialised.  A block takes a tile of 32 x 4 x 4
// vertices (2D: 32 x 16): f with one neighbour around it goes to shared memory, the
// lowest vertex of every cell of the tile is computed there once (lstar_tile.cuh), every
// vertex gets its lower star, and the expansions (lstar_core.cuh) are handed out in order
// of the lower star's size, since their loop runs once per pairing step: the lanes of a
// warp run loops of similar length (one thread per vertex left half the lanes idle).  The
// pairing puts the cells' bytes into shared memory, and they leave it row by row: a
// byte stored from its own thread cost an L2 write of its own.
// What bounds it is integer issue: 52.7 warp instructions per vertex of a 64^3 Gaussian-sum
// field (24 of 32 lanes active), 88.4 with a key per vertex and neighbouring cell; 13.0 ->
// 7.2 ms at 512^3 (k^-3), 2.06 -> 1.35 ms for an 8192^2 image.
#include <cstddef>

#include "lstar_tile.cuh"
#include "msc_device.cuh"

namespace msc {

namespace {
constexpr int kLstarBS = 256;
constexpr int kLstarWarps = kLstarBS / 32;
bool lstar_dims_ok(const GradDims& D) {
  // a z-plane of cells must be addressable with 32-bit offsets
  return !(D.v[0] > (int64_t)1 << 30 || D.v[1] > (int64_t)1 << 30 || D.v[0] * D.v[1] > ((int64_t)1 << 31) - 1 ||
           D.cs[2] > ((int64_t)1 << 31) - 1);
}
template <int ND>
struct LstarSmem {
  using T = LstarTile<ND>;
  LatKey lat[T::NL];
  float f[T::NF];
  uint32_t L[T::NV];
  alignas(16) uint8_t bytes[(T::NL + 15) / 16 * 16];  // cleared 16 bytes at a time
  uint16_t order[T::NV];
  int16_t off[32];
  int hist[32];
};
static_assert(offsetof(LstarSmem<3>, bytes) % 16 == 0 && offsetof(LstarSmem<2>, bytes) % 16 == 0, "uint4 stores");
}  // namespace

// One tile of volume (f, g, D); its first vertex is (x0, y0, z0).  Every thread of the
// block calls this.  RESTRICTED: the vertices with a restricted cell in their lower star
// (`bits`, conform_kernels.cu) are paired again, counted in `touched`, and the others left
// as they are.
template <int ND, bool RESTRICTED = false>
__device__ __forceinline__ bool lstar_tile(const float* __restrict__ f, uint8_t* __restrict__ g, const GradDims& D,
                                           int64_t x0, int64_t y0, int64_t z0, LstarSmem<ND>& S,
                                           const uint16_t* __restrict__ bits = nullptr, int* touched = nullptr) {
  using T = LstarTile<ND>;
  using N = Nb<ND>;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t X = D.v[0], Y = D.v[1], Z = D.v[2];
  const bool rim = x0 == 0 || y0 == 0 || x0 + T::BX >= X || y0 + T::BY >= Y ||
                   (ND == 3 && (z0 == 0 || z0 + T::BZ >= Z));
  if (tid < 32) {
    S.hist[tid] = 0;
    S.off[tid] = (int16_t)(tid < N::NPOS ? T::off(tid) : 0);
  }
  if (!RESTRICTED)
    for (int i = tid; i < (int)sizeof(S.bytes) / 16; i += kLstarBS)
      reinterpret_cast<uint4*>(S.bytes)[i] = make_uint4(0u, 0u, 0u, 0u);
  // f, a warp per row (values outside the volume read as 0: no cell that holds one is in
  // a lower star)
  bool nan = false;
  for (int r = warp; r < T::FY * T::FZ; r += kLstarWarps) {
    const int64_t y = y0 - 1 + r % T::FY, z = ND == 3 ? z0 - 1 + r / T::FY : 0;
    const bool row = y >= 0 && y < Y && z >= 0 && z < Z;
    const float* fr = f + (x0 - 1 + X * (y + Y * z));
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int lx = lane + 32 * h;
      if (lx >= T::FX) break;
      const int64_t x = x0 - 1 + lx;
      float v = 0.f;
      if (row && x >= 0 && x < X) v = __ldg(fr + lx);
      nan |= v != v;
      S.f[r * T::FX + lx] = plain_zero(v);
    }
  }
  __syncthreads();
  // the cells' keys, a thread per base vertex
  constexpr int CX = T::BX + 1, CY = T::BY + 1, CZ = ND == 3 ? T::BZ + 1 : 1;
  for (int i = tid; i < CX * CY * CZ; i += kLstarBS) {
    const int z = i / (CX * CY), r = i - z * (CX * CY), y = r / CX, x = r - y * CX;
    tile_cell_keys<ND>(S.f, S.lat, x - 1, y - 1, ND == 3 ? z - 1 : 0);
    if (RESTRICTED) {
      const int64_t vx = x0 - 1 + x, vy = y0 - 1 + y, vz = z0 - 1 + z;
      const bool in = vx >= 0 && vx < X && vy >= 0 && vy < Y && vz >= 0 && vz < Z;
      tile_restrict(in ? bits[vx + X * (vy + Y * vz)] : 0u, S.bytes, x - 1, y - 1, z - 1);
    }
  }
  if (RESTRICTED) __syncthreads();  // the labels are read next
  // lower stars, and a counting sort of the vertices by their size (28 sizes; 31: no vertex)
  int bin[T::NV / kLstarBS], rank[T::NV / kLstarBS];
#pragma unroll
  for (int h = 0; h < T::NV / kLstarBS; h++) {
    const int t = tid + h * kLstarBS;
    int x, y, z;
    T::vertex(t, x, y, z);
    bin[h] = 31;
    if (x0 + x < X && y0 + y < Y && (ND == 2 || z0 + z < Z)) {
      uint32_t lower = tile_lower_mask<ND>(S.f, x, y, z);
      if (rim) lower &= inside_mask<ND>(x0 + x, y0 + y, z0 + z, D.v);
      const uint32_t L = lower_star_mask<ND>(lower);
      S.L[t] = L;
      bin[h] = __popc(L);
      if (RESTRICTED) {
        uint32_t r1, r2;
        if (tile_labels(L, t, S.bytes, S.off, r1, r2)) (*touched)++;
        else bin[h] = 31;
      }
    }
    rank[h] = atomicAdd(&S.hist[bin[h]], 1);
  }
  __syncthreads();
  if (tid < 32) {
    const int c = S.hist[tid];
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (tid >= o) incl += u;
    }
    S.hist[tid] = incl - c;  // exclusive start of each bin
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < T::NV / kLstarBS; h++)
    S.order[S.hist[bin[h]] + rank[h]] = (uint16_t)(bin[h] == 31 ? 0xFFFF : tid + h * kLstarBS);
  __syncthreads();
  // a warp takes small stars first time and large ones the second, so that all have the
  // same work
#pragma unroll 1
  for (int h = 0; h < T::NV / kLstarBS; h++) {
    const int t = S.order[(h & 1) ? T::NV - 1 - tid - (h - 1) / 2 * kLstarBS : tid + h / 2 * kLstarBS];
    if (t == 0xFFFF) continue;
    int x, y, z;
    T::vertex(t, x, y, z);
    if (RESTRICTED) {
      uint32_t r1, r2;
      tile_labels(S.L[t], t, S.bytes, S.off, r1, r2);
      tile_expand_restricted(S.L[t], r1, r2, t, rim, x0 + x, y0 + y, z0 + z, D.v,
                             reinterpret_cast<const LatKey*>(S.lat), S.bytes, S.off, D.enc_map);
    } else {
      tile_expand<ND>(S.L[t], t, rim, x0 + x, y0 + y, z0 + z, D.v, S.lat, S.bytes, S.off, D.enc_map);
    }
  }
  __syncthreads();
  // the bytes, a warp per lattice row
  uint8_t* g0 = g + (2 * x0 - 1) + (2 * y0 - 1) * D.cs[1] + (ND == 3 ? (2 * z0 - 1) * D.cs[2] : 0);
  for (int r = warp; r < T::ROWS; r += kLstarWarps) {
    const int cy = r % T::LY, cz = r / T::LY;
    uint8_t* gr = g0 + cy * D.cs[1] + cz * D.cs[2];
    const uint8_t* b = S.bytes + r * T::LX;
    const uint8_t b0 = b[lane], b1 = b[lane + 32];
    if (b0 & 1u) gr[lane] = b0;
    if (b1 & 1u) gr[lane + 32] = b1;
    if (lane == 0 && (b[64] & 1u)) gr[64] = b[64];
  }
  return nan;
}

// One volume: grid (x-tiles, y-tiles, z-tiles), looping over z when they exceed the grid.
template <int ND>
__global__ void __launch_bounds__(kLstarBS, 4) lstar_kernel(const float* __restrict__ f, uint8_t* __restrict__ g,
                                                            const GradDims D, int* __restrict__ err) {
  using T = LstarTile<ND>;
  extern __shared__ __align__(16) unsigned char s_tile[];
  LstarSmem<ND>& S = *reinterpret_cast<LstarSmem<ND>*>(s_tile);
  bool nan = false;
  for (int64_t z = blockIdx.z; z * T::BZ < D.v[2]; z += gridDim.z) {
    nan |= lstar_tile<ND>(f, g, D, (int64_t)blockIdx.x * T::BX, (int64_t)blockIdx.y * T::BY, z * T::BZ, S);
    __syncthreads();  // the next tile reuses the shared memory
  }
  if (nan) atomicOr(err, kErrNaN);
}

// Many volumes in one launch: a flat grid over every volume's tiles; a block finds its
// volume by binary search over the volumes' first tiles.
__global__ void __launch_bounds__(kLstarBS, 4) lstar_batch_kernel(const LstarBatch B, int* __restrict__ err) {
  using T = LstarTile<3>;
  extern __shared__ __align__(16) unsigned char s_tile[];
  LstarSmem<3>& S = *reinterpret_cast<LstarSmem<3>*>(s_tile);
  bool nan = false;
  for (int64_t blk = blockIdx.x; blk < B.total_blocks; blk += gridDim.x) {
    int lo = 0, hi = B.n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (B.v[mid].block0 <= blk) lo = mid; else hi = mid - 1;
    }
    const LstarVol& V = B.v[lo];
    const int64_t r = blk - V.block0;
    const int64_t bx = r % V.gx, by = (r / V.gx) % V.gy, bz = r / ((int64_t)V.gx * V.gy);
    nan |= lstar_tile<3>(V.f, V.g, V.D, bx * T::BX, by * T::BY, bz * T::BZ, S);
    __syncthreads();
  }
  if (nan) atomicOr(err, kErrNaN);
}

// The conforming re-pairing of one volume: a flat grid over its tiles.  Between patches of
// labels as small as the labels of noise make them most vertices are touched (8.6 of 10.0 M
// at 223 x 187 x 241), so it is the lower star's pass with classes, bound by integer issue
// like it.  A thread per vertex with its 27 keys in local memory, its classes one after the
// other, took 2.6 ms there, with lists of the touched vertices 2.3 ms (13 of 32 lanes
// active); the tiles and one loop over all classes take 1.07 ms.
__global__ void __launch_bounds__(kLstarBS, 4) conform_kernel(const float* __restrict__ f,
                                                              const uint16_t* __restrict__ bits,
                                                              uint8_t* __restrict__ g, const GradDims D,
                                                              unsigned long long* __restrict__ touched) {
  using T = LstarTile<3>;
  extern __shared__ __align__(16) unsigned char s_tile[];
  LstarSmem<3>& S = *reinterpret_cast<LstarSmem<3>*>(s_tile);
  const int64_t gx = (D.v[0] + T::BX - 1) / T::BX, gy = (D.v[1] + T::BY - 1) / T::BY;
  const int64_t n = gx * gy * ((D.v[2] + T::BZ - 1) / T::BZ);
  int mine = 0;
  for (int64_t b = blockIdx.x; b < n; b += gridDim.x) {
    const int64_t q = b / gx;
    lstar_tile<3, true>(f, g, D, (b - q * gx) * T::BX, (q % gy) * T::BY, (q / gy) * T::BZ, S, bits, &mine);
    __syncthreads();  // the next tile reuses the shared memory
  }
  unsigned long long sum = (unsigned long long)mine;
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(touched, sum);
}

namespace {
template <class K>
cudaError_t allow_smem(K k, size_t bytes) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
template <int ND>
cudaError_t launch_lstar_nd(const float* f, uint8_t* g, const GradDims& D, int* err, cudaStream_t stream) {
  using T = LstarTile<ND>;
  const int64_t gy = (D.v[1] + T::BY - 1) / T::BY, gz = (D.v[2] + T::BZ - 1) / T::BZ;
  // (262,140 rows in either dimension: what a grid of four rows a block along y takes)
  if ((D.v[1] + 3) / 4 > 65535) return cudaErrorInvalidValue;
  const dim3 grid((unsigned)((D.v[0] + T::BX - 1) / T::BX), (unsigned)gy, (unsigned)(gz < 65535 ? gz : 65535));
  if (cudaError_t e = allow_smem(lstar_kernel<ND>, sizeof(LstarSmem<ND>))) return e;
  ::msc::count_launch();
  lstar_kernel<ND><<<grid, kLstarBS, sizeof(LstarSmem<ND>), stream>>>(f, g, D, err);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_lstar(int nd, const float* f, uint8_t* g, const GradDims& D, int* err, int num_sms,
                         cudaStream_t stream) {
  (void)num_sms;
  if (!lstar_dims_ok(D)) return cudaErrorInvalidValue;
  return nd == 3 ? launch_lstar_nd<3>(f, g, D, err, stream) : launch_lstar_nd<2>(f, g, D, err, stream);
}

cudaError_t launch_conform(const float* f, const uint16_t* bits, uint8_t* g, const GradDims& D,
                           unsigned long long* touched, int num_sms, cudaStream_t stream) {
  using T = LstarTile<3>;
  const int64_t n = ((D.v[0] + T::BX - 1) / T::BX) * ((D.v[1] + T::BY - 1) / T::BY) * ((D.v[2] + T::BZ - 1) / T::BZ);
  if (cudaError_t e = allow_smem(conform_kernel, sizeof(LstarSmem<3>))) return e;
  const int64_t grid = (int64_t)num_sms * 64;  // the last tiles even out over the blocks' turns
  ::msc::count_launch();
  conform_kernel<<<(unsigned)(n < grid ? n : grid), kLstarBS, sizeof(LstarSmem<3>), stream>>>(f, bits, g, D, touched);
  return cudaGetLastError();
}

cudaError_t make_lstar_batch(int n, const float* const* f, uint8_t* const* g, const GradDims* D, LstarBatch* B) {
  if (n < 1 || n > kMaxBatch) return cudaErrorInvalidValue;
  B->n = n;
  int64_t off = 0;
  for (int i = 0; i < n; i++) {
    if (!lstar_dims_ok(D[i])) return cudaErrorInvalidValue;
    LstarVol& v = B->v[i];
    v.f = f[i];
    v.g = g[i];
    v.D = D[i];
    using T = LstarTile<3>;
    v.gx = (int)((D[i].v[0] + T::BX - 1) / T::BX);
    v.gy = (int)((D[i].v[1] + T::BY - 1) / T::BY);
    v.block0 = off;
    off += (int64_t)v.gx * v.gy * ((D[i].v[2] + T::BZ - 1) / T::BZ);
  }
  B->total_blocks = off;
  return cudaSuccess;
}

cudaError_t launch_lstar_batch(const LstarBatch& B, int* err, int num_sms, cudaStream_t stream, int blocks_per_sm) {
  const int64_t cap = (int64_t)num_sms * blocks_per_sm;
  const int grid = (int)(B.total_blocks < cap ? B.total_blocks : cap);
  if (grid <= 0) return cudaSuccess;
  if (cudaError_t e = allow_smem(lstar_batch_kernel, sizeof(LstarSmem<3>))) return e;
  ::msc::count_launch();
  lstar_batch_kernel<<<grid, kLstarBS, sizeof(LstarSmem<3>), stream>>>(B, err);
  return cudaGetLastError();
}

}  // namespace msc
