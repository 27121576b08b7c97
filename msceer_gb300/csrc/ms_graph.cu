// The Morse-Smale complex graph of a device-resident .grad: the nodes and arcs
// MorseSmaleComplexBasic::ComputeFromGrad builds without arc geometry
// (gi_morse_smale_complex_basic.h:676-716), as extractmsc uses it after load_from_file
// (extractmsc/extractmsc.cxx:482-504), read from the .grad in HBM instead of a file.
//
//   nodes  every critical cell (pair code 7) in cell-id order (AllCellsIterator):
//          cell id, dimension, boundaryValue, value = f at the cell's highest vertex
//          (createNode, :308-341, with TopologicalMaxVertexMeshFunction::cellValue)
//   arcs   for every node of dimension d >= 1 whose arcs are built (build[d - 1]),
//          the V-paths traced down from it (rec_tdcr_candidates, :550-577): a critical
//          facet ends a path in an arc to that facet's node; a facet whose ldir equals
//          the node's ldir + 1 continues at its pair when the pair is another cell of
//          the traced cell's dimension.  Arcs are listed node by node (the reference's
//          thread-local candidate lists, concatenated in thread order over a static
//          split of the nodes) and, within a node, in depth-first facet order
//          (+x, -x, +y, -y, +z, -z over the cell's odd axes); a path reached twice is
//          an arc twice.  persistence = value(upper) - value(lower) (createArcFromNodeIDs).
//
// GPU form: an ordered compaction of the critical cells (block counts, one scan, an
// ordered write, and a bitmap with the rank of every 32 cells, so that the node of a cell
// is one load and a popcount), one thread per node for the attributes, and one
// depth-first trace per node thread that counts its arcs and keeps them; a scan places
// them and a copy puts them there.  The trace has an explicit task stack: a visited cell
// goes on with its first child in a register and pushes the others (arc ends and cells
// to visit) in reverse facet order, so a path without branches leaves the stack alone.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/msc_gpu.h"
#include "msc_device.cuh"

namespace msc {
namespace {

constexpr int kScanThreads = 1024;
constexpr int kCritThreads = 256;
constexpr int kCritPerThread = 16;
constexpr int64_t kCritChunk = (int64_t)kCritThreads * kCritPerThread;  // cells per block
constexpr int kStack = 64;            // pending tasks of one node's trace
// cells one node's trace may visit: a valid .grad is acyclic, so this only stops the
// endless walk of a .grad with a cycle (a corrupt file, or one read with wrong dims)
constexpr int64_t kMaxVisits = (int64_t)1 << 24;
constexpr int64_t kEmit = (int64_t)1 << 62;  // task tag: an arc to the critical cell

struct MsMesh {
  const uint8_t* g;
  const float* f;
  int64_t d[3], cs[3], v[3];
  int64_t ncells;
  bool i32;  // cell ids fit 32 bits
};

__device__ __forceinline__ bool crit(uint8_t b) { return ((b >> 2) & 7u) == 7u; }
__device__ __forceinline__ int ldir(uint8_t b) { return b >> 5; }

__device__ __forceinline__ void coords(const MsMesh& M, int64_t id, int64_t c[3]) {
  if (M.i32) {
    const uint32_t u = (uint32_t)id, d0 = (uint32_t)M.d[0], d1 = (uint32_t)M.d[1];
    const uint32_t r = u / d0;
    c[0] = u - r * d0;
    c[1] = r % d1;
    c[2] = r / d1;
  } else {
    c[0] = id % M.d[0];
    c[1] = (id / M.d[0]) % M.d[1];
    c[2] = id / (M.d[0] * M.d[1]);
  }
}
__device__ __forceinline__ int dim_of(const int64_t c[3]) { return (int)((c[0] & 1) + (c[1] & 1) + (c[2] & 1)); }

// block-wide exclusive scan of one value per thread (blockDim.x threads, a multiple
// of 32); returns the thread's offset, *total the block's sum
template <class T>
__device__ T block_excl_scan(T v, T* s_warp, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = lane < nw ? s_warp[lane] : (T)0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) s_warp[lane] = w;
  }
  __syncthreads();
  const T before = (warp > 0 ? s_warp[warp - 1] : (T)0) + x - v;
  if (total) *total = s_warp[nw - 1];
  __syncthreads();
  return before;
}

// the critical-cell bits of a thread's 16 cells (one 16-byte load when aligned)
__device__ __forceinline__ uint32_t crit_bits(const uint8_t* g, int64_t ncells, int64_t base) {
  uint32_t m = 0;
  if (base + 16 <= ncells && ((reinterpret_cast<uintptr_t>(g + base) & 15u) == 0)) {
    const uint4 q = *reinterpret_cast<const uint4*>(g + base);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 16; k++) m |= (uint32_t)crit((uint8_t)(w[k >> 2] >> (8 * (k & 3)))) << k;
  } else {
    for (int k = 0; k < 16; k++)
      if (base + k < ncells) m |= (uint32_t)crit(g[base + k]) << k;
  }
  return m;
}

__global__ void __launch_bounds__(kCritThreads) crit_count_kernel(const uint8_t* __restrict__ g, int64_t ncells,
                                                                  int64_t* __restrict__ counts) {
  __shared__ int64_t s_warp[32];
  const int64_t base = (int64_t)blockIdx.x * kCritChunk + (int64_t)threadIdx.x * kCritPerThread;
  int64_t total = 0;
  block_excl_scan<int64_t>(__popc(crit_bits(g, ncells, base)), s_warp, &total);
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

// in place: counts[0, n) -> exclusive offsets; *sum = the total.  One block.
template <class T>
__global__ void __launch_bounds__(kScanThreads) excl_scan_kernel(T* __restrict__ a, int64_t n, T* __restrict__ sum) {
  __shared__ T s_warp[32];
  T carry = 0;
  for (int64_t i0 = 0; i0 < n; i0 += kScanThreads) {
    const int64_t i = i0 + threadIdx.x;
    const T v = i < n ? a[i] : (T)0;
    T tot = 0;
    const T off = block_excl_scan<T>(v, s_warp, &tot);
    if (i < n) a[i] = carry + off;
    carry += tot;
  }
  if (threadIdx.x == 0) *sum = carry;
}

// The same for long arrays, in three launches: the sum of every kScanThreads-element
// chunk, the one-block scan of those sums, then every chunk scanned from its offset.
template <class T>
__global__ void __launch_bounds__(kScanThreads) chunk_sum_kernel(const T* __restrict__ a, int64_t n,
                                                                 T* __restrict__ sums) {
  __shared__ T s_warp[32];
  const int64_t i = (int64_t)blockIdx.x * kScanThreads + threadIdx.x;
  T tot = 0;
  block_excl_scan<T>(i < n ? a[i] : (T)0, s_warp, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}
template <class T>
__global__ void __launch_bounds__(kScanThreads) chunk_scan_kernel(T* __restrict__ a, int64_t n,
                                                                  const T* __restrict__ offs) {
  __shared__ T s_warp[32];
  const int64_t i = (int64_t)blockIdx.x * kScanThreads + threadIdx.x;
  const T v = i < n ? a[i] : (T)0;
  const T off = block_excl_scan<T>(v, s_warp, nullptr);
  if (i < n) a[i] = offs[blockIdx.x] + off;
}

// The nodes in cell order, and for every 32 cells their critical bits and the number of
// critical cells before them.
__global__ void __launch_bounds__(kCritThreads) crit_write_kernel(const uint8_t* __restrict__ g, int64_t ncells,
                                                                  const int64_t* __restrict__ offsets,
                                                                  int64_t* __restrict__ node_cell,
                                                                  uint2* __restrict__ index) {
  __shared__ int64_t s_warp[32];
  const int64_t base = (int64_t)blockIdx.x * kCritChunk + (int64_t)threadIdx.x * kCritPerThread;
  uint32_t m = crit_bits(g, ncells, base);
  int64_t o = offsets[blockIdx.x] + block_excl_scan<int64_t>(__popc(m), s_warp, nullptr);
  // two threads' cells make a word (the index is as long as the blocks' cells)
  const uint32_t hi = __shfl_down_sync(0xffffffffu, m, 1);
  if ((threadIdx.x & 1) == 0) index[base >> 5] = make_uint2(m | (hi << 16), (uint32_t)o);
  while (m) {
    const int k = __ffs(m) - 1;
    m &= m - 1;
    node_cell[o++] = base + k;
  }
}

// createNode: dimension, boundaryValue and the value at the highest vertex ((value,
// then index) order, gi_regular_grid_trilinear_function.h:309-314)
__global__ void node_attr_kernel(const MsMesh M, const int64_t* __restrict__ node_cell, int64_t n,
                                 float* __restrict__ value, uint8_t* __restrict__ dim, uint8_t* __restrict__ bnd) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t c[3];
    coords(M, node_cell[i], c);
    int nb = 0;
    for (int a = 0; a < 3; a++) nb += (c[a] == 0 || c[a] == M.d[a] - 1);
    int64_t best = -1;
    float bv = 0.f;
    const int odd = (int)(c[0] & 1) | (int)((c[1] & 1) << 1) | (int)((c[2] & 1) << 2);
    for (int s = 0; s < 8; s++) {
      if (s & ~odd) continue;  // corners only along the odd axes
      int64_t vi = 0;
      for (int a = 0; a < 3; a++) {
        const int64_t vc = (c[a] & 1) ? ((s >> a) & 1 ? (c[a] + 1) >> 1 : (c[a] - 1) >> 1) : c[a] >> 1;
        vi += vc * M.v[a];
      }
      const float fv = M.f[vi];
      if (best < 0 || fv > bv || (!(bv > fv) && vi > best)) {
        best = vi;
        bv = fv;
      }
    }
    value[i] = bv;
    dim[i] = (uint8_t)dim_of(c);
    bnd[i] = (uint8_t)nb;
  }
}

// the node of a critical cell (fewer than 2^31 nodes)
__device__ __forceinline__ int32_t node_of(const uint2* __restrict__ index, int64_t cell) {
  const uint2 w = __ldg(index + (cell >> 5));
  return (int32_t)(w.y + (uint32_t)__popc(w.x & ((1u << (cell & 31)) - 1u)));
}

// One node's trace (rec_tdcr_candidates): calls emit(critical cell) for every arc in
// order.  Returns 0, kErrLocalQueue if the task stack overflowed, kErrIterLimit past
// kMaxVisits.
template <class Emit>
__device__ __forceinline__ int trace_node(const MsMesh& M, int64_t start, const Emit& emit) {
  const int temp_dim = ldir(M.g[start]) + 1;
  int64_t stack[kStack + 6];  // a visit's children are pushed before they are counted
  int sp = 0;
  int64_t t = start, visits = 0;
  while (true) {
    if (++visits > kMaxVisits) return kErrIterLimit;
    int64_t c[3];
    coords(M, t, c);
    const int dim = dim_of(c);
    // the facets' bytes together
    uint8_t fb[6];
#pragma unroll
    for (int j = 0; j < 6; j++) {
      const int a = j >> 1;
      fb[j] = 0;
      if (c[a] & 1) fb[j] = M.g[(j & 1) ? t - M.cs[a] : t + M.cs[a]];
    }
    // the children, last facet first: the first one stays in `next`
    int64_t next = -1;
    int pending = sp;
#pragma unroll
    for (int j = 5; j >= 0; j--) {
      const int a = j >> 1;
      if (!(c[a] & 1)) continue;
      const int64_t fc = (j & 1) ? t - M.cs[a] : t + M.cs[a];
      const unsigned code = (fb[j] >> 2) & 7u;
      int64_t child = -1;
      if (code == 7u) {
        child = fc | kEmit;
      } else if (code < 6u && ldir(fb[j]) == temp_dim) {
        // the pair: the cell at the code's stride (UncompressByteTo6NeighborOffset;
        // with a single-vertex axis two axes share a stride and the code names the
        // first), inside the array for any byte
        const int64_t st = code < 2u ? M.cs[0] : (code < 4u ? M.cs[1] : M.cs[2]);
        const int64_t p = (code & 1u) ? fc - st : fc + st;
        if (p != t && p >= 0 && p < M.ncells) {
          int64_t pc[3];
          coords(M, p, pc);
          if (dim_of(pc) == dim) child = p;
        }
      }
      if (child < 0) continue;
      pending++;
      if (next >= 0) stack[sp++] = next;
      next = child;
    }
    if (pending > kStack) return kErrLocalQueue;
    // arcs end here; go on at the first cell
    while (true) {
      if (next < 0) {
        if (sp == 0) return 0;
        next = stack[--sp];
      }
      if (!(next & kEmit)) break;
      emit(next & ~kEmit);
      next = -1;
    }
    t = next;
  }
}

// The nodes whose arcs are traced (dimension d >= 1 with build bit d - 1), listed so
// that the tracing threads of a warp all trace, and trace alike: in cell order a warp's
// nodes mix all four dimensions, minima and unbuilt dimensions left most lanes idle, and
// a saddle's two paths waited for a maximum's tree of them.  Maxima go into list[0, n)
// from the back (n_list[1] of them), the others from the front (n_list[0]).
__global__ void traced_list_kernel(const MsMesh M, const int64_t* __restrict__ node_cell, int64_t n, int build,
                                   int32_t* __restrict__ list, unsigned long long* __restrict__ n_list) {
  const int lane = threadIdx.x & 31;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = i0 + threadIdx.x;
    int d = 0;
    if (i < n) {
      int64_t c[3];
      coords(M, node_cell[i], c);
      d = dim_of(c);
      if (d > 0 && !((build >> (d - 1)) & 1)) d = 0;
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const bool want = q == 0 ? d == 1 || d == 2 : d == 3;
      const unsigned m = __ballot_sync(0xffffffffu, want);
      if (!m) continue;
      const int leader = __ffs(m) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(&n_list[q], (unsigned long long)__popc(m));
      base = __shfl_sync(0xffffffffu, base, leader);
      const int64_t at = (int64_t)base + __popc(m & ((1u << lane) - 1u));
      if (want) list[q == 0 ? at : n - 1 - at] = (int32_t)i;
    }
  }
}
// the j-th node to trace: maxima first (their traces are the longest)
__device__ __forceinline__ int64_t traced_node(const int32_t* __restrict__ list, int64_t n, int64_t n_max, int64_t j) {
  return j < n_max ? list[n - 1 - j] : list[j - n_max];
}

// Counts every traced node's arcs; with `store` set, also keeps them (lower node ids):
// the arcs of a warp's nodes in one stretch of store[0, store_cap), place[j] the first of
// list entry j's.  A node with more arcs than its thread keeps, or whose warp found the
// store full, gets place -1 and is traced again by the write.
constexpr int kKeep = 64;  // arcs a thread keeps (16 / 64 / 128: 3.46 / 3.02 / 3.01 ms a 256^3 k^-3 graph)
template <bool STORE>
__global__ void __launch_bounds__(128) arc_trace_kernel(const MsMesh M, const int64_t* __restrict__ node_cell,
                                                        int64_t n, const uint2* __restrict__ index,
                                                        const int32_t* __restrict__ list,
                                                        const unsigned long long* __restrict__ n_list,
                                                        int64_t* __restrict__ counts, int32_t* __restrict__ store,
                                                        unsigned long long* __restrict__ n_store,
                                                        unsigned long long store_cap, int64_t* __restrict__ place,
                                                        int* __restrict__ err) {
  const int64_t n_max = (int64_t)n_list[1], nl = (int64_t)n_list[0] + n_max;
  const int lane = threadIdx.x & 31;
  for (int64_t j0 = blockIdx.x * (int64_t)blockDim.x; j0 < nl; j0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = j0 + threadIdx.x;
    int32_t keep[STORE ? kKeep : 1];
    int k = 0;
    if (j < nl) {
      const int64_t i = traced_node(list, n, n_max, j);
      const int e = trace_node(M, node_cell[i], [&](int64_t cell) {
        if (STORE && k < kKeep) keep[k] = node_of(index, cell);
        k++;
      });
      if (e) {
        atomicOr(err, e);
        k = 0;
      }
      counts[i] = k;
    }
    if (!STORE) continue;
    const int mine = k <= kKeep ? k : 0;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long base = 0;
    if (lane == 31 && total > 0) base = atomicAdd(n_store, (unsigned long long)total);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (j >= nl) continue;
    const bool fits = k <= kKeep && base + (unsigned long long)total <= store_cap;
    const int64_t at = (int64_t)base + incl - mine;
    place[j] = fits ? at : -1;
    if (fits)
      for (int q = 0; q < k; q++) store[at + q] = keep[q];
  }
}

// The kept arcs to their places.
__global__ void __launch_bounds__(128) arc_write_kernel(const MsMesh M, const int64_t* __restrict__ node_cell,
                                                        const uint2* __restrict__ index,
                                                        const int32_t* __restrict__ list,
                                                        const unsigned long long* __restrict__ n_list,
                                                        const int64_t* __restrict__ offsets, int64_t n, int64_t n_arcs,
                                                        const int32_t* __restrict__ store,
                                                        const int64_t* __restrict__ place,
                                                        const float* __restrict__ value, int32_t* __restrict__ lower,
                                                        int32_t* __restrict__ upper, float* __restrict__ pers,
                                                        int* __restrict__ err) {
  const int64_t n_max = (int64_t)n_list[1], nl = (int64_t)n_list[0] + n_max;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nl; j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = traced_node(list, n, n_max, j);
    const int64_t out = offsets[i], at = place[j];
    const float v = value[i];
    auto put = [&](int64_t o, int32_t lo) {
      lower[o] = lo;
      upper[o] = (int32_t)i;
      if (pers) pers[o] = v - value[lo];
    };
    if (at >= 0) {
      const int64_t end = i + 1 < n ? offsets[i + 1] : n_arcs;
      for (int64_t o = out; o < end; o++) put(o, store[at + (o - out)]);
    } else {
      int64_t o = out;
      const int e = trace_node(M, node_cell[i], [&](int64_t cell) { put(o++, node_of(index, cell)); });
      if (e) atomicOr(err, e);
    }
  }
}

int fail(int code, const std::string& m) { return set_last_error(code, m.c_str()); }
#define GCUDA(call, what)                                                                          \
  do {                                                                                             \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess)                                                                         \
      return fail(e_ == cudaErrorMemoryAllocation ? MSC_ERR_OOM : MSC_ERR_CUDA,                   \
                  std::string(what) + ": " + cudaGetErrorString(e_));                              \
  } while (0)

struct Pool {
  std::vector<void*> p;
  cudaStream_t st;
  ~Pool() {
    for (void* q : p) cudaFreeAsync(q, st);
  }
  cudaError_t get(void** out, size_t bytes) {
    cudaError_t e = scratch_alloc(out, bytes ? bytes : 16, st);
    if (e == cudaSuccess) p.push_back(*out);
    return e;
  }
};

int grid_for(int64_t n, int threads) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)sms * 16;
  return (int)(b < 1 ? 1 : (b < cap ? b : cap));
}

// a[0, n) -> exclusive offsets in place, *sum (device) = the total
int scan_in_place(Pool& P, int64_t* a, int64_t n, int64_t* sum, cudaStream_t stream) {
  const int64_t nch = (n + kScanThreads - 1) / kScanThreads;
  int64_t* csum = nullptr;
  GCUDA(P.get((void**)&csum, (size_t)(nch + 1) * sizeof(int64_t)), "scratch alloc(chunk sums)");
  if (nch > 0) {
    count_launch();
    chunk_sum_kernel<int64_t><<<(unsigned)nch, kScanThreads, 0, stream>>>(a, n, csum);
  }
  count_launch();
  excl_scan_kernel<int64_t><<<1, kScanThreads, 0, stream>>>(csum, nch, sum);
  if (nch > 0) {
    count_launch();
    chunk_scan_kernel<int64_t><<<(unsigned)nch, kScanThreads, 0, stream>>>(a, n, csum);
  }
  return MSC_OK;
}

// alloc (when set) supplies every output array once its length is known; the arrays passed
// are then ignored.
int ms_graph_impl(const uint8_t* g, const float* f, const int64_t* dims, const int* build, int64_t node_cap,
                  int64_t* node_cell, float* node_value, uint8_t* node_dim, uint8_t* node_boundary, int64_t arc_cap,
                  int32_t* arc_lower, int32_t* arc_upper, float* arc_pers, int64_t* counts_out, msc_graph_alloc_fn alloc,
                  void* alloc_ctx, cudaStream_t stream) {
  if (!dims || !build || !counts_out) return fail(MSC_ERR_NULL_POINTER, "null argument");
  GradDims D;
  if (!make_grad_dims(3, dims, &D)) return fail(MSC_ERR_BAD_DIMS, "invalid dims");
  if (!g || !f) return fail(MSC_ERR_NULL_POINTER, "null buffer");
  MsMesh M;
  M.g = g;
  M.f = f;
  for (int a = 0; a < 3; a++) {
    M.d[a] = D.d[a];
    M.cs[a] = D.cs[a];
  }
  M.v[0] = 1;
  M.v[1] = D.v[0];
  M.v[2] = D.v[0] * D.v[1];
  M.ncells = D.ncells;
  M.i32 = D.ncells <= (int64_t)0xFFFFFFFF;
  const int bmask = (build[0] ? 1 : 0) | (build[1] ? 2 : 0) | (build[2] ? 4 : 0);

  Pool P{{}, stream};
  const int64_t nblk = (D.ncells + kCritChunk - 1) / kCritChunk;
  int64_t* blk = nullptr;
  int64_t* sums = nullptr;  // [0] nodes [1] arcs
  int* err = nullptr;
  GCUDA(P.get((void**)&blk, (size_t)nblk * sizeof(int64_t)), "scratch alloc(block counts)");
  GCUDA(P.get((void**)&sums, 2 * sizeof(int64_t) + sizeof(int)), "scratch alloc(sums)");
  err = reinterpret_cast<int*>(sums + 2);
  GCUDA(cudaMemsetAsync(err, 0, sizeof(int), stream), "cudaMemsetAsync(status)");
  count_launch();
  crit_count_kernel<<<(unsigned)nblk, kCritThreads, 0, stream>>>(g, D.ncells, blk);
  if (int rc = scan_in_place(P, blk, nblk, sums, stream)) return rc;
  GCUDA(cudaGetLastError(), "critical-cell count launch");
  int64_t h[2] = {0, 0};
  GCUDA(cudaMemcpyAsync(h, sums, sizeof(int64_t), cudaMemcpyDeviceToHost, stream), "read node count");
  GCUDA(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
  const int64_t n = h[0];
  if (n >= ((int64_t)1 << 31)) return fail(MSC_ERR_BAD_DIMS, "more than 2^31 - 1 critical cells");

  if (alloc) {
    node_cell = static_cast<int64_t*>(alloc(alloc_ctx, MSC_GRAPH_NODE_CELL, n));
    node_value = static_cast<float*>(alloc(alloc_ctx, MSC_GRAPH_NODE_VALUE, n));
    node_dim = static_cast<uint8_t*>(alloc(alloc_ctx, MSC_GRAPH_NODE_DIM, n));
    node_boundary = static_cast<uint8_t*>(alloc(alloc_ctx, MSC_GRAPH_NODE_BOUNDARY, n));
    node_cap = n;
    if (n > 0 && !(node_cell && node_value && node_dim && node_boundary))
      return fail(MSC_ERR_OOM, "the node arrays were not allocated");
  }
  const bool nodes_out = node_cell && node_value && node_dim && node_boundary && node_cap >= n;
  int64_t* cells = node_cell;
  float* vals = node_value;
  if (!nodes_out) {
    GCUDA(P.get((void**)&cells, (size_t)n * sizeof(int64_t)), "scratch alloc(node cells)");
    GCUDA(P.get((void**)&vals, (size_t)n * sizeof(float)), "scratch alloc(node values)");
  }
  uint2* index = nullptr;  // (a whole number of words for every block)
  GCUDA(P.get((void**)&index, (size_t)nblk * (kCritChunk / 32) * sizeof(uint2)), "scratch alloc(node index)");
  count_launch();
  crit_write_kernel<<<(unsigned)nblk, kCritThreads, 0, stream>>>(g, D.ncells, blk, cells, index);
  int64_t* acnt = nullptr;
  int32_t* tlist = nullptr;
  unsigned long long* n_tlist = nullptr;
  GCUDA(P.get((void**)&acnt, (size_t)n * sizeof(int64_t)), "scratch alloc(arc counts)");
  GCUDA(P.get((void**)&tlist, (size_t)n * sizeof(int32_t)), "scratch alloc(traced nodes)");
  GCUDA(P.get((void**)&n_tlist, 3 * sizeof(unsigned long long)), "scratch alloc(traced and kept counts)");
  // room for two arcs a node of any dimension (rough fields have 1.5 with extractmsc's
  // flags; what does not fit is traced again)
  const bool want_arcs = alloc || (arc_lower && arc_upper && arc_cap > 0);
  const int64_t store_cap = !want_arcs ? 0 : (alloc ? 2 * n + 4096 : std::min<int64_t>(arc_cap, 2 * n + 4096));
  int32_t* store = nullptr;
  int64_t* place = nullptr;
  if (want_arcs) {
    GCUDA(P.get((void**)&store, (size_t)store_cap * sizeof(int32_t)), "scratch alloc(kept arcs)");
    GCUDA(P.get((void**)&place, (size_t)n * sizeof(int64_t)), "scratch alloc(arc places)");
  }
  GCUDA(cudaMemsetAsync(acnt, 0, (size_t)n * sizeof(int64_t), stream), "cudaMemsetAsync(arc counts)");
  GCUDA(cudaMemsetAsync(n_tlist, 0, 3 * sizeof(unsigned long long), stream), "cudaMemsetAsync(traced count)");
  if (n > 0) {
    count_launch();
    traced_list_kernel<<<grid_for(n, 256), 256, 0, stream>>>(M, cells, n, bmask, tlist, n_tlist);
    count_launch();
    if (want_arcs)
      arc_trace_kernel<true><<<grid_for(n, 128), 128, 0, stream>>>(M, cells, n, index, tlist, n_tlist, acnt, store,
                                                                  n_tlist + 2, (unsigned long long)store_cap, place,
                                                                  err);
    else
      arc_trace_kernel<false><<<grid_for(n, 128), 128, 0, stream>>>(M, cells, n, index, tlist, n_tlist, acnt, nullptr,
                                                                   nullptr, 0ull, nullptr, err);
  }
  if (int rc = scan_in_place(P, acnt, n, sums + 1, stream)) return rc;
  GCUDA(cudaGetLastError(), "arc count launch");
  int st = 0;
  GCUDA(cudaMemcpyAsync(h + 1, sums + 1, sizeof(int64_t), cudaMemcpyDeviceToHost, stream), "read arc count");
  GCUDA(cudaMemcpyAsync(&st, err, sizeof(int), cudaMemcpyDeviceToHost, stream), "read status");
  GCUDA(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
  if (st & kErrIterLimit) return fail(MSC_ERR_ITER_LIMIT, "a V-path trace did not end (is the .grad acyclic?)");
  if (st) return fail(MSC_ERR_QUEUE_OVERFLOW, "a V-path trace branched beyond its task stack");
  const int64_t na = h[1];
  counts_out[0] = n;
  counts_out[1] = na;

  if (alloc) {
    arc_lower = static_cast<int32_t*>(alloc(alloc_ctx, MSC_GRAPH_ARC_LOWER, na));
    arc_upper = static_cast<int32_t*>(alloc(alloc_ctx, MSC_GRAPH_ARC_UPPER, na));
    arc_pers = static_cast<float*>(alloc(alloc_ctx, MSC_GRAPH_ARC_PERSISTENCE, na));
    arc_cap = na;
    if (na > 0 && !(arc_lower && arc_upper && arc_pers)) return fail(MSC_ERR_OOM, "the arc arrays were not allocated");
  }
  const bool arcs_out = arc_lower && arc_upper && arc_cap >= na;
  if (!nodes_out && !arcs_out) return MSC_OK;
  uint8_t* dims_b = node_dim;
  uint8_t* bnd_b = node_boundary;
  if (!nodes_out) {
    GCUDA(P.get((void**)&dims_b, (size_t)n), "scratch alloc(node dims)");
    GCUDA(P.get((void**)&bnd_b, (size_t)n), "scratch alloc(node boundary)");
  }
  if (n > 0) {
    count_launch();
    node_attr_kernel<<<grid_for(n, 256), 256, 0, stream>>>(M, cells, n, vals, dims_b, bnd_b);
  }
  if (arcs_out && na > 0) {
    count_launch();
    arc_write_kernel<<<grid_for(n, 128), 128, 0, stream>>>(M, cells, index, tlist, n_tlist, acnt, n, na, store, place,
                                                           vals, arc_lower, arc_upper, arc_pers, err);
  }
  GCUDA(cudaGetLastError(), "node / arc write launch");
  GCUDA(cudaMemcpyAsync(&st, err, sizeof(int), cudaMemcpyDeviceToHost, stream), "read status");
  GCUDA(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
  if (st & kErrIterLimit) return fail(MSC_ERR_ITER_LIMIT, "a V-path trace did not end (is the .grad acyclic?)");
  if (st) return fail(MSC_ERR_QUEUE_OVERFLOW, "a V-path trace branched beyond its task stack");
  return MSC_OK;
}

}  // namespace
}  // namespace msc

extern "C" {

int msc_ms_graph_3d(const uint8_t* grad, const float* f, const int64_t dims[3], const int build_arcs[3],
                    int64_t node_cap, int64_t* node_cell, float* node_value, uint8_t* node_dim,
                    uint8_t* node_boundary, int64_t arc_cap, int32_t* arc_lower, int32_t* arc_upper,
                    float* arc_persistence, int64_t counts[2], msc_stream_t stream) {
  return msc::ms_graph_impl(grad, f, dims, build_arcs, node_cap, node_cell, node_value, node_dim, node_boundary,
                            arc_cap, arc_lower, arc_upper, arc_persistence, counts, nullptr, nullptr,
                            reinterpret_cast<cudaStream_t>(stream));
}

int msc_ms_graph_alloc_3d(const uint8_t* grad, const float* f, const int64_t dims[3], const int build_arcs[3],
                          msc_graph_alloc_fn alloc, void* ctx, int64_t counts[2], msc_stream_t stream) {
  if (!alloc) return msc::fail(MSC_ERR_NULL_POINTER, "null allocator");
  return msc::ms_graph_impl(grad, f, dims, build_arcs, 0, nullptr, nullptr, nullptr, nullptr, 0, nullptr, nullptr,
                            nullptr, counts, alloc, ctx, reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
