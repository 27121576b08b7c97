// K2: ascending-manifold dimension (the ldir bits of the .grad byte), sm_103a.
//
// Replaces TopologicalGradientUsingAlgorithms::setAscendingManifoldDimensions
// (gi_topological_gradient_using_algorithms.h:430-478) and its per-root queue walk
// rec_man_trace_up_marking (:395-425).  The reference marks, from every critical
// 1-cell, value 2 on everything reachable through "cofacet t, not critical, pair(t)
// != current, continue at pair(t)"; then value 1 from every critical 2-cell; then 0
// on critical 3-cells.  Items of the value-2 walk are edges (and hexes, which end
// it); the cells it marks as cofacets are quads, so the walk is a plain monotone
// reachability closure, independent of visiting order -- the reference's own
// output is thread-count invariant for the same reason.  Likewise for value 1
// (items quads, cofacets hexes).  K1 already wrote the roots (critical 1-cells = 2,
// critical 2-cells = 1, critical 3-cells = 0, everything else 3).
//
// GPU form: a tile kernel.  A CTA stages a tile of .grad bytes plus a 2-cell halo in
// shared memory (every rule reaches at most 2 cells), seeds a shared-memory queue
// with the marked items, runs the value-2 walk to its local fixpoint, then the
// value-1 walk, and writes back the tile.  Marks in the halo stay local.  Two ways
// finish the closure across tile borders:
//   single pass (default)  one tile pass saves the halo cells every tile lowered; a
//       check kernel lowers those cells in global memory where the owner holds them
//       higher and queues the lowered items; a walk kernel finishes their walks in
//       global memory.
//   multi pass (fallback, and the allocation-free entry)  repeated tile passes; later
//       passes revisit only tiles whose halo changed (a neighbour wrote a cell within
//       2 cells of the shared border) and seed only from the halo, because everything
//       reachable from the interior was already walked.  The closure is complete when
//       a pass changes no cell near any tile border.
#include "msc_device.cuh"

namespace msc {

template <int ND, int TX, int TY, int TZ>
struct LdirTile {
  static constexpr int H = 2;
  static constexpr int LX = TX + 2 * H;
  static constexpr int LY = TY + 2 * H;
  static constexpr int LZ = (ND == 3) ? TZ + 2 * H : 1;
  static constexpr int NL = LX * LY * LZ;
  static constexpr int ls(int a) { return a == 0 ? 1 : (a == 1 ? LX : LX * LY); }
  static constexpr int NW = (NL + 31) / 32;
  // dynamic shared memory of the pass kernel: queue (u16) | bytes | visited bits | changed bits
  static constexpr size_t smem_bytes() { return (size_t)NL * 2 + ((NL + 3) / 4) * 4 + (size_t)NW * 8; }
};

// local index -> local coords
template <class T>
__device__ __forceinline__ void lcoords(int i, int& lx, int& ly, int& lz) {
  lx = i % T::LX;
  ly = (i / T::LX) % T::LY;
  lz = i / (T::LX * T::LY);
}

// Queue append for the lanes of a warp that are converged here: one shared-memory
// atomic per warp instead of one per pushed item.
__device__ __forceinline__ void warp_push(uint16_t* sq, int* qtail, int cap, int* err, bool want, int item) {
  const unsigned act = __activemask();
  const unsigned m = __ballot_sync(act, want);
  if (!m) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(qtail, __popc(m));
  base = __shfl_sync(act, base, leader);
  if (want) {
    const int slot = base + __popc(m & ((1u << lane) - 1u));
    if (slot < cap) sq[slot] = (uint16_t)item; else atomicOr(err, kErrLocalQueue);
  }
}

// Walk one item: visit its cofacets (CofacetsIterator order), mark them, follow their
// partners and queue the newly reached items.  All coordinates are local to the
// staged box, whose origin is even on every axis, so local parity is the cell's
// dimension parity.
template <class T, int ND>
struct LdirWalk {
  uint8_t* sg;
  uint16_t* sq;
  uint32_t* vis;
  uint32_t* dirty;
  int* qtail;
  int* err;
  int lmin[3], lmax[3];  // in-complex local range per axis
  uint32_t dec_map;

  __device__ __forceinline__ void touch(int c) {
    if (dirty) atomicOr(&dirty[c >> 5], 1u << (c & 31));
  }

  // returns the item to queue, or -1
  __device__ __forceinline__ int visit(int i, int l[3], int a, int sgn, int phase) {
    const unsigned value = phase == 0 ? 2u : 1u;
    constexpr int LE[3] = {T::LX, T::LY, T::LZ};
    const int la = l[a] + sgn;
    if (la < lmin[a] || la >= lmax[a]) return -1;
    const int t = i + sgn * T::ls(a);
    const uint8_t bt = sg[t];
    const unsigned code = (bt >> 2) & 7u;
    if (!(bt & 1u) || code == 7u) return -1;  // unassigned or critical
    if (phase == 0) {
      if ((bt >> 5) == 3u) { sg[t] = (uint8_t)((bt & 0x1Fu) | (2u << 5)); touch(t); }
    } else {
      if ((bt >> 5) != 1u) { sg[t] = (uint8_t)((bt & 0x1Fu) | (1u << 5)); touch(t); }
    }
    const int pc = map3(dec_map, (int)code);
    const int pa = pc >> 1, psg = (pc & 1) ? -1 : 1;
    int lp[3] = {l[0], l[1], l[2]};
    lp[a] += sgn;
    lp[pa] += psg;
    if (lp[pa] < 0 || lp[pa] >= LE[pa]) return -1;  // partner outside the box
    const int tp = t + psg * T::ls(pa);
    if (tp == i) return -1;
    const uint8_t bp = sg[tp];
    if (phase == 0) {
      if ((bp >> 5) != 3u) return -1;  // already marked: seeded or queued
      const int pdim = (lp[0] & 1) + (lp[1] & 1) + (ND == 3 ? (lp[2] & 1) : 0);
      if (pdim != 1) {  // a hex: the path ends here
        sg[tp] = (uint8_t)((bp & 0x1Fu) | (2u << 5));
        touch(tp);
        return -1;
      }
    } else {
      if ((bp >> 5) == 1u) return -1;
    }
    const uint32_t bit = 1u << (tp & 31);
    if (atomicOr(&vis[tp >> 5], bit) & bit) return -1;
    sg[tp] = (uint8_t)((bp & 0x1Fu) | (value << 5));
    touch(tp);
    return tp;
  }

  __device__ __forceinline__ void step(int i, int phase) {
    int l[3];
    lcoords<T>(i, l[0], l[1], l[2]);
#pragma unroll
    for (int a = 0; a < ND; a++) {
#pragma unroll
      for (int s = 0; s < 2; s++) {
        // cofacets only along even axes, +axis first
        const int nx = (l[a] & 1) ? -1 : visit(i, l, a, s == 0 ? 1 : -1, phase);
        warp_push(sq, qtail, T::NL, err, nx >= 0, nx);
      }
    }
  }
};

template <int ND, int TX, int TY, int TZ, int BS>
__global__ void __launch_bounds__(BS) ldir_pass_kernel(uint8_t* __restrict__ g, const GradDims D,
                                                       const uint8_t* __restrict__ dirty_in,
                                                       uint8_t* __restrict__ dirty_out,
                                                       int* __restrict__ changed, int* __restrict__ err) {
  using T = LdirTile<ND, TX, TY, TZ>;
  constexpr int NL = T::NL;
  static_assert(NL < 65536, "local ids are 16-bit");
  static_assert(TX % 2 == 0 && TY % 2 == 0 && (ND == 2 || TZ % 2 == 0) && T::H % 2 == 0, "box origins must be even");
  extern __shared__ __align__(16) unsigned char s_dyn[];
  uint16_t* sq = reinterpret_cast<uint16_t*>(s_dyn);
  uint8_t* sg = s_dyn + (size_t)NL * 2;
  uint32_t* s_vis = reinterpret_cast<uint32_t*>(s_dyn + (size_t)NL * 2 + ((NL + 3) / 4) * 4);
  uint32_t* s_dirty = s_vis + T::NW;
  __shared__ int s_qtail, s_qseed, s_border;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NWARPS = BS / 32;
  const int64_t dX = D.d[0], dY = D.d[1], dZ = D.d[2];
  const int64_t ntx = (dX + TX - 1) / TX, nty = (dY + TY - 1) / TY;
  const int64_t ntz = (ND == 3) ? (dZ + TZ - 1) / TZ : 1;
  const int64_t ntiles = ntx * nty * ntz;
  const bool first = (dirty_in == nullptr);

  LdirWalk<T, ND> W;
  W.sg = sg;
  W.sq = sq;
  W.vis = s_vis;
  W.dirty = s_dirty;
  W.qtail = &s_qtail;
  W.err = err;
  W.dec_map = D.dec_map;

  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    if (!first && !dirty_in[tile]) continue;
    const int64_t tx = tile % ntx, ty = (tile / ntx) % nty, tz = (ND == 3) ? tile / (ntx * nty) : 0;
    const int64_t o[3] = {tx * TX - T::H, ty * TY - T::H, (ND == 3) ? tz * TZ - T::H : 0};
    const int64_t dd[3] = {dX, dY, dZ};
    constexpr int LE[3] = {T::LX, T::LY, T::LZ};
#pragma unroll
    for (int a = 0; a < 3; a++) {
      W.lmin[a] = (int)(o[a] < 0 ? -o[a] : 0);
      const int64_t hi = dd[a] - o[a];
      W.lmax[a] = (int)(hi < LE[a] ? hi : LE[a]);
    }
    if (tid == 0) {
      s_qtail = 0;
      s_qseed = NL;
      s_border = 0;
    }
    for (int w = tid; w < T::NW; w += BS) {
      s_vis[w] = 0;
      s_dirty[w] = 0;
    }
    __syncthreads();

    // stage the box row by row (cells outside the complex read as 0 = unassigned)
    // and collect the seeds: marked items of both walks (first pass), or of the
    // halo only (later passes: the interior was walked already).  Seeds need no
    // visited bit: being marked already stops a walk from queueing them again.
    constexpr int RPW = 4;  // rows per warp in flight
    for (int row0 = warp * RPW; row0 < T::LY * T::LZ; row0 += NWARPS * RPW) {
      uint8_t b[RPW][(T::LX + 31) / 32];
#pragma unroll
      for (int r = 0; r < RPW; r++) {
        const int row = row0 + r;
        const int ly = row % T::LY, lz = row / T::LY;
        const bool rin = row < T::LY * T::LZ && ly >= W.lmin[1] && ly < W.lmax[1] && lz >= W.lmin[2] && lz < W.lmax[2];
        const uint8_t* grow = g + ((o[1] + ly) * D.cs[1] + (o[2] + lz) * D.cs[2] + o[0]);
#pragma unroll
        for (int c = 0; c < (T::LX + 31) / 32; c++) {
          const int lx = lane + 32 * c;
          b[r][c] = (rin && lx < T::LX && lx >= W.lmin[0] && lx < W.lmax[0]) ? grow[lx] : (uint8_t)0;
        }
      }
#pragma unroll
      for (int r = 0; r < RPW; r++) {
        const int row = row0 + r;
        if (row >= T::LY * T::LZ) break;
        const int ly = row % T::LY, lz = row / T::LY;
        const bool row_halo = ly < T::H || ly >= T::H + TY || (ND == 3 && (lz < T::H || lz >= T::H + TZ));
#pragma unroll
        for (int c = 0; c < (T::LX + 31) / 32; c++) {
          const int lx = lane + 32 * c;
          const int i = lx + T::LX * row;
          const uint8_t v = b[r][c];
          if (lx < T::LX) sg[i] = v;
          const unsigned ld = v >> 5;
          const int dim = (lx & 1) + (ly & 1) + (ND == 3 ? (lz & 1) : 0);
          const bool keep = lx < T::LX && (v & 1u) && (first || row_halo || lx < T::H || lx >= T::H + TX);
          const bool s0 = keep && dim == 1 && ld == 2u;
          const bool s1 = keep && dim == 2 && ld == 1u;
          warp_push(sq, &s_qtail, NL, err, s0, i);
          // value-1 seeds grow down from the top of the queue
          const unsigned m1 = __ballot_sync(0xffffffffu, s1);
          if (m1) {
            int base = 0;
            if (lane == 0) base = atomicSub(&s_qseed, __popc(m1));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (s1) sq[base - 1 - __popc(m1 & ((1u << lane) - 1u))] = (uint16_t)i;
          }
        }
      }
    }
    __syncthreads();

    // value-2 walk, then value-1 walk, level by level
#pragma unroll 1
    for (int phase = 0; phase < 2; phase++) {
      int lo = phase == 0 ? 0 : s_qseed;
      int hi = phase == 0 ? s_qtail : NL;
      if (phase == 1) {
        __syncthreads();
        for (int w = tid; w < T::NW; w += BS) s_vis[w] = 0;
        if (tid == 0) s_qtail = 0;
        __syncthreads();
      }
#pragma unroll 1
      while (lo < hi) {
        for (int k0 = lo; k0 < hi; k0 += BS) {
          const int k = k0 + tid;
          if (k < hi) W.step(sq[k], phase);
        }
        __syncthreads();
        // the first value-1 level came from the seed region; later levels from 0
        const int nlo = (phase == 1 && hi == NL) ? 0 : hi;
        const int nhi = s_qtail;
        __syncthreads();
        lo = nlo;
        hi = nhi;
      }
    }
    __syncthreads();

    // write back the changed interior cells
    for (int w = tid; w < T::NW; w += BS) {
      uint32_t m = s_dirty[w];
      while (m) {
        const int i = w * 32 + __ffs(m) - 1;
        m &= m - 1;
        int lx, ly, lz;
        lcoords<T>(i, lx, ly, lz);
        if (lx < T::H || lx >= T::H + TX || ly < T::H || ly >= T::H + TY) continue;
        if (ND == 3 && (lz < T::H || lz >= T::H + TZ)) continue;
        g[(o[0] + lx) + (o[1] + ly) * D.cs[1] + (o[2] + lz) * D.cs[2]] = sg[i];
        // a change within reach (2 cells) of a neighbour's halo reopens that neighbour
        if (lx < 2 * T::H || lx >= TX || ly < 2 * T::H || ly >= TY || (ND == 3 && (lz < 2 * T::H || lz >= TZ)))
          s_border = 1;
      }
    }
    __syncthreads();
    if (s_border) {
      const int nn = (ND == 3) ? 27 : 9;
      for (int k = tid; k < nn; k += BS) {
        const int64_t nx = tx + (k % 3) - 1, ny = ty + (k / 3) % 3 - 1, nz = (ND == 3) ? tz + k / 9 - 1 : 0;
        if (k == nn / 2 || nx < 0 || nx >= ntx || ny < 0 || ny >= nty || nz < 0 || nz >= ntz) continue;
        dirty_out[nx + ny * ntx + nz * ntx * nty] = 1;
      }
      if (tid == 0) atomicOr(changed, 1);
    }
    __syncthreads();
  }
}

// ---- single-pass form: one bit-row tile pass, a halo check, a global frontier walk -----------
//
// A tile's walk is complete for every item of its interior (all of an item's rule
// reaches lies within 2 cells), so after one pass over all tiles the only missing
// marks are those a tile made in its halo that the halo's owner did not make itself.
// The pass records, per tile, the halo cells its closure holds lower than the .grad
// held them; the check kernel lowers every such cell that its owner still holds
// higher and queues the lowered items, whose walks may continue beyond that tile's
// box; the walk kernel finishes those walks in global memory.  Concurrent lowering of
// a byte uses a compare-and-swap on its aligned 32-bit word (the low five bits never
// change, so the ldir field only ever decreases); bytes whose word is not wholly
// inside the .grad array go through a bounded spin lock instead.

struct GradView {
  uint8_t* g;
  uintptr_t lo, hi;  // [first, last) byte address of the array
  int* lock;
  int* err;
};

// ldir(c) = min(ldir(c), val); true if this call lowered it
__device__ __forceinline__ bool lower_ldir(const GradView& G, int64_t c, unsigned val) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(G.g + c);
  const uintptr_t wa = a & ~uintptr_t(3);
  if (wa >= G.lo && wa + 4 <= G.hi) {
    uint32_t* w = reinterpret_cast<uint32_t*>(wa);
    const int sh = (int)(a & 3u) * 8;
    uint32_t cur = *reinterpret_cast<volatile uint32_t*>(w);
    for (int guard = 0; guard < 64; guard++) {
      const uint32_t b = (cur >> sh) & 0xFFu;
      if ((b >> 5) <= val) return false;
      const uint32_t nb = (b & 0x1Fu) | (val << 5);
      const uint32_t nw = (cur & ~(0xFFu << sh)) | (nb << sh);
      const uint32_t prev = atomicCAS(w, cur, nw);
      if (prev == cur) return true;
      cur = prev;
    }
    atomicOr(G.err, kErrPassLimit);
    return false;
  }
  // a word that reaches outside the array: serialise on the lock
  bool got = false;
  for (int guard = 0; guard < (1 << 20) && !got; guard++) got = atomicCAS(G.lock, 0, 1) == 0;
  if (!got) {
    atomicOr(G.err, kErrPassLimit);
    return false;
  }
  __threadfence();
  volatile uint8_t* p = G.g + c;
  const uint8_t b = *p;
  const bool lowered = (unsigned)(b >> 5) > val;
  if (lowered) *p = (uint8_t)((b & 0x1Fu) | (val << 5));
  __threadfence();
  atomicExch(G.lock, 0);
  return lowered;
}

// lower_ldir in steps, so that a thread can have the swaps of two cells in flight.  The
// word comes through L1 and may be out of date.  What the walk reads from it stays true:
// the pairs do not change while the ldir stage runs and the ldir field only decreases, so
// a cell that an old word holds low enough is; and a swap against an old word fails and
// returns the present one, from which finish() goes on.  A word that reaches out of the
// array is left to lower_ldir.
struct LdirCell {
  uint32_t* w;
  int sh;
  uint32_t cur, got;
  bool inside, tried;
  __device__ __forceinline__ LdirCell(const GradView& G, int64_t c) : got(0), tried(false) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(G.g + c), wa = a & ~uintptr_t(3);
    inside = wa >= G.lo && wa + 4 <= G.hi;
    w = reinterpret_cast<uint32_t*>(wa);
    sh = (int)(a & 3u) * 8;
    cur = inside ? __ldca(w) : (uint32_t)*reinterpret_cast<volatile uint8_t*>(G.g + c) << sh;
  }
  __device__ __forceinline__ unsigned byte() const { return (cur >> sh) & 0xFFu; }
  __device__ __forceinline__ uint32_t lowered(uint32_t word, unsigned val) const {
    return (word & ~(0xE0u << sh)) | (val << (sh + 5));
  }
  __device__ __forceinline__ void swap(unsigned val) {
    tried = inside && (byte() >> 5) > val;
    if (tried) got = atomicCAS(w, cur, lowered(cur, val));
  }
  // whether this cell was lowered here
  __device__ __forceinline__ bool finish(const GradView& G, int64_t c, unsigned val) {
    if (!inside) return lower_ldir(G, c, val);
    if (!tried) return false;  // held as low already
    for (int guard = 0; guard < 64; guard++) {
      if (got == cur) return true;
      cur = got;
      if ((byte() >> 5) <= val) return false;
      got = atomicCAS(w, cur, lowered(cur, val));
    }
    atomicOr(G.err, kErrPassLimit);
    return false;
  }
  // swap() and finish() of this cell and of t, whose word is the same
  __device__ __forceinline__ bool pair(const GradView& G, const LdirCell& t, unsigned val) {
    for (int guard = 0; guard < 64; guard++) {
      const bool low = (byte() >> 5) > val, low_t = ((cur >> t.sh) & 0xFFu) >> 5 > val;
      if (!low && !low_t) return false;
      uint32_t to = low ? lowered(cur, val) : cur;
      if (low_t) to = t.lowered(to, val);
      got = atomicCAS(w, cur, to);
      if (got == cur) return low;
      cur = got;
    }
    atomicOr(G.err, kErrPassLimit);
    return false;
  }
};

__device__ __forceinline__ int batch_volume(const LdirBatch& B, int64_t flat_tile) {
  int lo = 0, hi = B.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (B.v[mid].tile0 <= flat_tile) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The tile pass works on bit rows.  A box is 32 cells along x (28 owned plus the
// 2-cell halo on each side) by LY x LZ rows, and every per-cell property the walks
// need is one 32-bit word per row (bit = x offset in the box).  Both closures advance
// one BFS level at a time over every row at once:
//   T = NC & cof(F)     cofacets of the frontier along its even axes: bit shifts within
//                       a row for x, the neighbour rows for y and z
//   P = partner(T)      for each pair direction, T & PC[direction] moved one cell
//   value 2 marks the quads of T, the hexes of P and the new edges of P
//   value 1 marks the hexes of T and the new quads of P
// The frontier F is the new edges (value-2 items) and quads (value-1 items): the two
// walks' items, cofacets and partners never share a dimension, so one frontier and
// one partner step serve both.  Visiting order does not change a monotone closure, so
// the marks equal those of the item-by-item walk.  The closures of rough fields are
// shallow (14 levels for value 2, 12 for value 1 over a whole 128^3 k^-3 volume).
//
// A lane holds the row at its own y, a register a word of it, so that a warp's
// registers hold a slab of 32 x 32 cells and a row's y neighbours are one shuffle away.
// 3D: a box of 32 x 32 x 32, eight warps of four slabs each, one above the other: only
// the words that cross from warp to warp go through shared memory.  2D: a warp works on
// a box of 32 x 128 alone.
// A lane reads its row with three 16-byte loads and turns the 32 bytes into bit planes by
// 8 x 8 bit transposes (~130 operations a row).  A warp per row with a ballot per
// property and the word planes in shared memory took 371 K warp instructions a tile, most
// of them staging: 15.4 ms at 512^3 (ALU pipe 75%).
constexpr int kBitLX = 32;
template <int ND, int LY, int LZ>
struct BitTile {
  static constexpr int TX = kBitLX - 4, TY = LY - 4, TZ = ND == 3 ? LZ - 4 : 1;
  static constexpr int R = LY * LZ;  // rows of the box
  // halo rows (every cell in the halo) and inner rows (halo cells at x = 0, 1, 30, 31)
  static constexpr int NHR = ND == 3 ? 4 * LY + 4 * (LZ - 4) : 4;
  static constexpr int NIR = ND == 3 ? (LY - 4) * (LZ - 4) : LY - 4;
  // a tile's record: the {value 2, value 1} masks of each halo row's lowered cells,
  // then one byte per inner row (bits 0-3: value 2 at x = 0, 1, 30, 31; 4-7: value 1)
  static constexpr int64_t REC = ((int64_t)NHR * 8 + NIR + 15) / 16 * 16;
  static_assert(ND == 3 || LZ == 1, "2D boxes have one z row");
  static_assert(LY % 2 == 0 && LZ % 2 == (ND == 3 ? 0 : 1), "tile origins must be even");
};

// record slot of halo row (ly, lz); -1 for an inner row
template <int ND, int LY, int LZ>
__device__ __forceinline__ int halo_row_slot(int ly, int lz) {
  if (ND == 3) {
    if (lz < 2) return lz * LY + ly;
    if (lz >= LZ - 2) return (lz - (LZ - 4)) * LY + ly;
  }
  const int base = ND == 3 ? 4 * LY + (lz - 2) * 4 : 0;
  if (ly < 2) return base + ly;
  if (ly >= LY - 2) return base + ly - (LY - 4);
  return -1;
}

template <int ND, int LY, int LZ>
__device__ __forceinline__ void halo_row_of(int h, int& ly, int& lz) {
  if (ND == 3 && h < 4 * LY) {
    const int s = h / LY;
    lz = s < 2 ? s : LZ - 4 + s;
    ly = h % LY;
    return;
  }
  const int k = ND == 3 ? h - 4 * LY : h;
  const int q = k & 3;
  lz = ND == 3 ? 2 + (k >> 2) : 0;
  ly = q < 2 ? q : LY - 4 + q;
}

constexpr int kSlabs = 4;        // slabs of 32 x 32 cells per warp
constexpr int kTileWarps = 8;    // 3D: warps per tile
constexpr uint32_t kEvenX = 0x55555555u, kOddX = 0xAAAAAAAAu;

// 16 bytes at p (16-byte aligned); bytes outside [lo, hi) read as 0
__device__ __forceinline__ uint4 load_granule(const uint8_t* p, const uint8_t* lo, const uint8_t* hi) {
  if (p >= lo && p + 16 <= hi) return *reinterpret_cast<const uint4*>(p);
  uint32_t w[4] = {0u, 0u, 0u, 0u};
  for (int k = 0; k < 16; k++)  // the array's first and last bytes
    if (p + k >= lo && p + k < hi) w[k >> 2] |= (uint32_t)p[k] << (8 * (k & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// 8 x 8 bit transpose of eight bytes (lo: bytes 0-3): byte b of the result holds bit b of
// every byte.  The method of halves: 1 x 1, 2 x 2, then 4 x 4 blocks change places across the
// diagonal (Warren, Hacker's Delight, "Transposing a Bit Matrix").
__device__ __forceinline__ void transpose8(uint32_t& lo, uint32_t& hi) {
  uint32_t t = (lo ^ (lo >> 7)) & 0x00AA00AAu;
  lo ^= t ^ (t << 7);
  t = (hi ^ (hi >> 7)) & 0x00AA00AAu;
  hi ^= t ^ (t << 7);
  t = (lo ^ (lo >> 14)) & 0x0000CCCCu;
  lo ^= t ^ (t << 14);
  t = (hi ^ (hi >> 14)) & 0x0000CCCCu;
  hi ^= t ^ (t << 14);
  t = (lo & 0x0F0F0F0Fu) | ((hi << 4) & 0xF0F0F0F0u);
  hi = (hi & 0xF0F0F0F0u) | ((lo >> 4) & 0x0F0F0F0Fu);
  lo = t;
}
// byte k of w[0..3] gathered into p[k]
__device__ __forceinline__ void gather_bytes(const uint32_t w[4], uint32_t p[4]) {
  const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);
  const uint32_t c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);
  p[0] = __byte_perm(a, b, 0x5410);
  p[1] = __byte_perm(a, b, 0x7632);
  p[2] = __byte_perm(c, d, 0x5410);
  p[3] = __byte_perm(c, d, 0x7632);
}

// The bit planes of the 32 cells at p (which may reach past both ends of the array)
__device__ __forceinline__ void load_planes(const uint8_t* p, const uint8_t* lo, const uint8_t* hi, uint32_t pl[8]) {
  const int s = (int)(reinterpret_cast<uintptr_t>(p) & 15u);
  const uint8_t* q = p - s;
  const uint4 a = load_granule(q, lo, hi), b = load_granule(q + 16, lo, hi);
  uint4 c = make_uint4(0u, 0u, 0u, 0u);
  if (s > 0) c = load_granule(q + 32, lo, hi);
  uint32_t w[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
#pragma unroll
  for (int i = 0; i < 10; i++) w[i] = (s & 8) ? w[i + 2] : w[i];
#pragma unroll
  for (int i = 0; i < 9; i++) w[i] = (s & 4) ? w[i + 1] : w[i];
  const int sh = 8 * (s & 3);
  uint32_t l[4], h[4];
#pragma unroll
  for (int g = 0; g < 4; g++) {
    l[g] = __funnelshift_r(w[2 * g], w[2 * g + 1], sh);
    h[g] = __funnelshift_r(w[2 * g + 1], w[2 * g + 2], sh);
    transpose8(l[g], h[g]);
  }
  gather_bytes(l, pl);
  gather_bytes(h, pl + 4);
}

// A row's words.
struct LdirRow {
  uint32_t nc;        // assigned, not critical
  uint32_t pc[6];     // paired to +x, -x, +y, -y, +z, -z
  uint32_t m2, m1;    // marked by the value-2 / value-1 walk
  uint32_t f;         // frontier
  uint32_t gt2, gt1;  // assigned, and ldir above 2 / above 1 in the .grad
};
// edges, quads, hexes: the row's cells of that dimension
__device__ __forceinline__ void load_row(LdirRow& R, const uint8_t* p, const uint8_t* lo, const uint8_t* hi,
                                         uint32_t valid, uint32_t dec_map, uint32_t edges, uint32_t quads) {
  uint32_t b[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  if (valid) load_planes(p, lo, hi, b);
  const uint32_t asg = b[0] & valid;
  const uint32_t c0 = b[2], c1 = b[3], c2 = b[4];
  R.nc = asg & ~(c0 & c1 & c2);
  const uint32_t e0 = R.nc & ~c0, e1 = R.nc & c0;
  R.pc[0] = e0 & ~c1 & ~c2;
  R.pc[1] = e1 & ~c1 & ~c2;
  R.pc[2] = e0 & c1 & ~c2;
  R.pc[3] = e1 & c1 & ~c2;
  R.pc[4] = e0 & ~c1 & c2;
  R.pc[5] = e1 & ~c1 & c2;
  if (dec_map != 0x2C688u) {  // a single-vertex axis: the stored code names another axis
    uint32_t t[6];
#pragma unroll
    for (int c = 0; c < 6; c++) t[c] = R.pc[c];
#pragma unroll
    for (int c = 0; c < 6; c++) {
      R.pc[c] = 0;
#pragma unroll
      for (int k = 0; k < 6; k++)
        if (map3(dec_map, k) == c) R.pc[c] |= t[k];
    }
  }
  R.gt2 = asg & (b[7] | (b[6] & b[5]));
  R.gt1 = asg & (b[7] | b[6]);
  R.m2 = asg & edges & b[6] & ~b[5] & ~b[7];
  R.m1 = asg & quads & b[5] & ~b[6] & ~b[7];
  R.f = R.m2 | R.m1;
}
// one level's marks of a row: t the cofacets, p the partners
__device__ __forceinline__ void mark_row(LdirRow& R, uint32_t t, uint32_t p, uint32_t edges, uint32_t quads,
                                         uint32_t hexes) {
  const uint32_t e2 = p & edges & ~R.m2, e1 = p & quads & ~R.m1;
  R.m2 |= (t & quads) | (p & hexes) | e2;
  R.m1 |= (t & hexes) | e1;
  R.f = e2 | e1;
}
// The owned cells of 28 rows (lanes 2-29 hold them) that the walks lowered: a lane per
// cell, four rows in flight.  gp: the slab's first cell of lane 0's row; rows cs1 apart.
__device__ __forceinline__ void write_rows(uint8_t* gp, int64_t cs1, int lane, uint32_t chg, uint32_t low1, int first,
                                           int last) {
#pragma unroll 1
  for (int r0 = first; r0 < last; r0 += 4) {
    uint8_t old[4];
    bool want[4];
    uint32_t one[4];
    uint8_t* q = gp + (int64_t)r0 * cs1 + lane;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t c = __shfl_sync(~0u, chg, r0 + k);
      one[k] = __shfl_sync(~0u, low1, r0 + k);
      want[k] = (c >> lane) & 1u;
      old[k] = 0;
      if (want[k]) old[k] = q[k * cs1];
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (want[k]) q[k * cs1] = (uint8_t)((old[k] & 0x1Fu) | (((one[k] >> lane) & 1u) ? 0x20u : 0x40u));
  }
}
// the four halo cells of an inner row, as the record keeps them
__device__ __forceinline__ uint8_t inner_record(uint32_t low2, uint32_t low1) {
  const uint32_t q2 = (low2 & 3u) | ((low2 >> 28) & 0xCu), q1 = (low1 & 3u) | ((low1 >> 28) & 0xCu);
  return (uint8_t)(q2 | (q1 << 4));
}
// the cells of a row of 32 from x0 that lie inside the complex
__device__ __forceinline__ uint32_t valid_cells(int64_t x0, int64_t dX) {
  const uint32_t below = x0 < 0 ? ~0u << (int)(-x0) : ~0u;
  const int64_t n = dX - x0;
  return below & (n >= 32 ? ~0u : (n <= 0 ? 0u : (1u << (int)n) - 1u));
}

// 3D: a block of eight warps per tile.  BLOCKS per SM: with 3 the warps wait for their rows'
// bytes and the levels' barriers half of the time (47% of the issue slots); with 4, at 64
// instead of 80 registers, they wait less but a block alone takes longer.
template <int BLOCKS>
__global__ void __launch_bounds__(32 * kTileWarps, BLOCKS) ldir_tile3_kernel(const LdirBatch B,
                                                                             uint8_t* __restrict__ rec,
                                                                             int* __restrict__ err) {
  using T = BitTile<3, 32, 32>;
  __shared__ uint32_t s_f[kTileWarps + 1][32];   // the frontier of each warp's first slab
  __shared__ uint32_t s_up[kTileWarps + 1][32];  // partners above a warp's last slab (of warp w at w + 1)
  __shared__ uint32_t s_dn[kTileWarps + 1][32];  // partners below a warp's first slab
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (w == 0) {  // beyond the box: nothing
    s_f[kTileWarps][lane] = 0;
    s_up[0][lane] = 0;
    s_dn[kTileWarps][lane] = 0;
  }
  const uint32_t yo = (lane & 1) ? ~0u : 0u, n0 = lane > 0 ? ~0u : 0u, n31 = lane < 31 ? ~0u : 0u;
  const bool yhalo = lane < 2 || lane >= 30;

  for (int64_t flat = blockIdx.x; flat < B.total_tiles; flat += gridDim.x) {
    const LdirVol& vol = B.v[batch_volume(B, flat)];
    uint8_t* __restrict__ g = vol.g;
    const GradDims& D = vol.D;
    const int64_t dX = D.d[0], dY = D.d[1], dZ = D.d[2];
    const int64_t ntx = (dX + T::TX - 1) / T::TX, nty = (dY + T::TY - 1) / T::TY;
    const int64_t tile = flat - vol.tile0;
    const int64_t tx = tile % ntx, ty = (tile / ntx) % nty, tz = tile / (ntx * nty);
    const int64_t x0 = tx * T::TX - 2, y0 = ty * T::TY - 2, z0 = tz * T::TZ - 2 + kSlabs * w;
    const bool yin = y0 + lane >= 0 && y0 + lane < dY;
    const uint32_t vx = valid_cells(x0, dX);
    const int64_t row0 = x0 + (y0 + lane) * D.cs[1] + z0 * D.cs[2];

    LdirRow R[kSlabs];
#pragma unroll
    for (int j = 0; j < kSlabs; j++) {
      const bool in = yin && z0 + j >= 0 && z0 + j < dZ;
      const uint32_t edges = (j & 1) ? kEvenX & ~yo : kOddX ^ yo, quads = (j & 1) ? kOddX ^ yo : kOddX & yo;
      load_row(R[j], g + (row0 + j * D.cs[2]), g, g + D.ncells, in ? vx : 0u, D.dec_map, edges, quads);
    }
    s_f[w][lane] = R[0].f;
    __syncthreads();

    // BFS levels until no row gains an item; every level adds an item, so the bound
    // is never reached by a valid gradient
    for (int level = 0;; level++) {
      uint32_t t[kSlabs] = {0u, 0u, 0u, 0u};
      const uint32_t above = s_f[w + 1][lane];
      const bool act = __any_sync(~0u, (R[0].f | R[1].f | R[2].f | R[3].f | above) != 0u);
      if (act) {
#pragma unroll
        for (int j = 0; j < kSlabs; j++) {
          const uint32_t f = R[j].f, fe = f & kEvenX;
          const uint32_t fu = __shfl_up_sync(~0u, f, 1), fd = __shfl_down_sync(~0u, f, 1) & n31;
          uint32_t c = (fe << 1) | (fe >> 1) | ((fu | fd) & yo);
          if (j & 1) c |= R[j - 1].f | (j + 1 < kSlabs ? R[j + 1 < kSlabs ? j + 1 : j].f : above);
          t[j] = c & R[j].nc;
        }
      }
      s_up[w + 1][lane] = t[kSlabs - 1] & R[kSlabs - 1].pc[4];
      s_dn[w][lane] = t[0] & R[0].pc[5];
      __syncthreads();
      const uint32_t from_up = s_dn[w + 1][lane], from_dn = s_up[w][lane];
      uint32_t grew = 0;
      if (act || __any_sync(~0u, (from_up | from_dn) != 0u)) {
#pragma unroll
        for (int j = 0; j < kSlabs; j++) {
          const uint32_t tj = t[j];
          uint32_t p = ((tj & R[j].pc[0]) << 1) | ((tj & R[j].pc[1]) >> 1);
          p |= __shfl_up_sync(~0u, tj & R[j].pc[2], 1) & n0;
          p |= __shfl_down_sync(~0u, tj & R[j].pc[3], 1) & n31;
          p |= j > 0 ? t[j > 0 ? j - 1 : 0] & R[j > 0 ? j - 1 : 0].pc[4] : from_dn;
          p |= j + 1 < kSlabs ? t[j + 1 < kSlabs ? j + 1 : j] & R[j + 1 < kSlabs ? j + 1 : j].pc[5] : from_up;
          const uint32_t edges = (j & 1) ? kEvenX & ~yo : kOddX ^ yo, quads = (j & 1) ? kOddX ^ yo : kOddX & yo;
          mark_row(R[j], tj, p, edges, quads, (j & 1) ? kOddX & yo : 0u);
          grew |= R[j].f;
        }
      }
      s_f[w][lane] = R[0].f;
      if (!__syncthreads_or(grew != 0u)) break;
      if (level > 64 * T::R) {
        if (threadIdx.x == 0) atomicOr(err, kErrPassLimit);
        break;
      }
    }

    // write back the owned cells this tile lowered and record the halo cells it holds
    // lower than the .grad did when it was staged (their owners may hold them lower by
    // now: the check compares again)
    uint8_t* trec = rec + flat * T::REC;
#pragma unroll
    for (int j = 0; j < kSlabs; j++) {
      const int lz = kSlabs * w + j;
      const uint32_t low2 = R[j].m2 & R[j].gt2, low1 = R[j].m1 & R[j].gt1;
      const bool zhalo = lz < 2 || lz >= 30;
      if (zhalo || yhalo)
        reinterpret_cast<uint2*>(trec)[halo_row_slot<3, 32, 32>(lane, lz)] = make_uint2(low2, low1);
      else
        trec[T::NHR * 8 + (lz - 2) * T::TY + (lane - 2)] = inner_record(low2, low1);
      if (!zhalo)
        write_rows(g + (x0 + y0 * D.cs[1] + (z0 + j) * D.cs[2]), D.cs[1], lane, (low2 | low1) & 0x3FFFFFFCu, low1, 2,
                   30);
    }
    __syncthreads();
  }
}

// 2D: a warp per tile of 32 x 128 cells, its slabs one below the other along y.
__global__ void __launch_bounds__(256) ldir_tile2_kernel(const LdirBatch B, uint8_t* __restrict__ rec,
                                                         int* __restrict__ err) {
  using T = BitTile<2, 32 * kSlabs, 1>;
  const int lane = threadIdx.x & 31;
  const uint32_t yo = (lane & 1) ? ~0u : 0u;
  const uint32_t edges = kOddX ^ yo, quads = kOddX & yo;
  const int64_t nwarp = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t flat = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); flat < B.total_tiles;
       flat += nwarp) {
    const LdirVol& vol = B.v[batch_volume(B, flat)];
    uint8_t* __restrict__ g = vol.g;
    const GradDims& D = vol.D;
    const int64_t dX = D.d[0], dY = D.d[1];
    const int64_t ntx = (dX + T::TX - 1) / T::TX;
    const int64_t tile = flat - vol.tile0;
    const int64_t tx = tile % ntx, ty = tile / ntx;
    const int64_t x0 = tx * T::TX - 2, y0 = ty * T::TY - 2;
    const uint32_t vx = valid_cells(x0, dX);
    LdirRow R[kSlabs];
#pragma unroll
    for (int j = 0; j < kSlabs; j++) {
      const int64_t y = y0 + 32 * j + lane;
      load_row(R[j], g + (x0 + y * D.cs[1]), g, g + D.ncells, (y >= 0 && y < dY) ? vx : 0u, D.dec_map, edges, quads);
    }
    for (int level = 0;; level++) {
      uint32_t t[kSlabs], up[kSlabs], dn[kSlabs];
      // the rows above and below: a rotation within the slab, the ends from its neighbours
#pragma unroll
      for (int j = 0; j < kSlabs; j++) {
        up[j] = __shfl_sync(~0u, R[j].f, (lane + 31) & 31);
        dn[j] = __shfl_sync(~0u, R[j].f, (lane + 1) & 31);
      }
#pragma unroll
      for (int j = 0; j < kSlabs; j++) {
        const uint32_t fe = R[j].f & kEvenX;
        const uint32_t fu = lane > 0 ? up[j] : (j > 0 ? up[j > 0 ? j - 1 : 0] : 0u);
        const uint32_t fd = lane < 31 ? dn[j] : (j + 1 < kSlabs ? dn[j + 1 < kSlabs ? j + 1 : j] : 0u);
        t[j] = ((fe << 1) | (fe >> 1) | ((fu | fd) & yo)) & R[j].nc;
      }
#pragma unroll
      for (int j = 0; j < kSlabs; j++) {
        up[j] = __shfl_sync(~0u, t[j] & R[j].pc[2], (lane + 31) & 31);
        dn[j] = __shfl_sync(~0u, t[j] & R[j].pc[3], (lane + 1) & 31);
      }
      uint32_t grew = 0;
#pragma unroll
      for (int j = 0; j < kSlabs; j++) {
        uint32_t p = ((t[j] & R[j].pc[0]) << 1) | ((t[j] & R[j].pc[1]) >> 1);
        p |= lane > 0 ? up[j] : (j > 0 ? up[j > 0 ? j - 1 : 0] : 0u);
        p |= lane < 31 ? dn[j] : (j + 1 < kSlabs ? dn[j + 1 < kSlabs ? j + 1 : j] : 0u);
        mark_row(R[j], t[j], p, edges, quads, 0u);
        grew |= R[j].f;
      }
      if (!__any_sync(~0u, grew != 0u)) break;
      if (level > 64 * T::R) {
        if (lane == 0) atomicOr(err, kErrPassLimit);
        break;
      }
    }
    uint8_t* trec = rec + flat * T::REC;
#pragma unroll
    for (int j = 0; j < kSlabs; j++) {
      const int ly = 32 * j + lane;
      const uint32_t low2 = R[j].m2 & R[j].gt2, low1 = R[j].m1 & R[j].gt1;
      const bool halo = ly < 2 || ly >= T::TY + 2;
      if (halo)
        reinterpret_cast<uint2*>(trec)[halo_row_slot<2, 32 * kSlabs, 1>(ly, 0)] = make_uint2(low2, low1);
      else
        trec[T::NHR * 8 + ly - 2] = inner_record(low2, low1);
      write_rows(g + (x0 + (y0 + 32 * j) * D.cs[1]), D.cs[1], lane, halo ? 0u : (low2 | low1) & 0x3FFFFFFCu, low1, 0,
                 32);
    }
  }
}

__device__ __forceinline__ void push_item(int64_t* q, int* n, int cap, int* err, int64_t c) {
  const int slot = atomicAdd(n, 1);
  if (slot < cap) q[slot] = c; else atomicOr(err, kErrLocalQueue);
}

// frontier entries carry their volume above the cell id (bits 57-62, so entries stay
// non-negative for every volume index below kMaxBatch = 64)
constexpr int kVolShift = 57;
constexpr int64_t kCellMask = ((int64_t)1 << kVolShift) - 1;
static_assert(kMaxBatch <= 64, "six volume bits");
__device__ __forceinline__ int entry_volume(int64_t e) { return (int)((uint64_t)e >> kVolShift); }

__device__ __forceinline__ GradView volume_view(const LdirVol& v, int* lock, int* err) {
  return GradView{v.g, reinterpret_cast<uintptr_t>(v.g), reinterpret_cast<uintptr_t>(v.g + v.D.ncells), lock, err};
}

// A tile's box origin and volume, found once per record unit by the whole warp.
struct TileAt {
  int vi;
  int64_t o[3];
};
template <int ND, int LY, int LZ>
__device__ __forceinline__ TileAt tile_at(const LdirBatch& B, int64_t flat) {
  using T = BitTile<ND, LY, LZ>;
  TileAt t;
  t.vi = batch_volume(B, flat);
  const LdirVol& vol = B.v[t.vi];
  const int64_t ntx = (vol.D.d[0] + T::TX - 1) / T::TX, nty = (vol.D.d[1] + T::TY - 1) / T::TY;
  const int64_t tile = flat - vol.tile0;
  int64_t tx, ty, tz;
  if (tile < ((int64_t)1 << 32)) {  // 32-bit division (tile counts of real volumes)
    const uint32_t u = (uint32_t)tile, nx = (uint32_t)ntx, ny = (uint32_t)nty;
    const uint32_t r = u / nx;
    tx = u - r * nx;
    ty = ND == 3 ? r % ny : r;
    tz = ND == 3 ? r / ny : 0;
  } else {
    const int64_t r = tile / ntx;
    tx = tile - r * ntx;
    ty = ND == 3 ? r % nty : r;
    tz = ND == 3 ? r / nty : 0;
  }
  t.o[0] = tx * T::TX - 2;
  t.o[1] = ty * T::TY - 2;
  t.o[2] = ND == 3 ? tz * T::TZ - 2 : 0;
  return t;
}

// A lane per row of a tile's record, 32 rows a warp: a halo row's owner bytes come as bit
// planes (load_planes), so the few cells that the owner holds higher fall out of two word
// operations; an inner row's four halo cells are read byte by byte.  (A warp per halo row
// with a lane per cell spent ~30 warp instructions on a row and waited for one row's
// bytes at a time; with a lane's cells lowered one after another the warp waited for the
// row with the most: 2.0 ms at 512^3 either way, 1.2-1.4 ms with the list below.)
template <int ND, int LY, int LZ>
__global__ void __launch_bounds__(256) ldir_check_kernel(const LdirBatch B, const uint8_t* __restrict__ rec,
                                                         int64_t* __restrict__ queue, int* __restrict__ n_queue,
                                                         int cap, int* lock, int* err) {
  using T = BitTile<ND, LY, LZ>;
  constexpr int UNITS = (T::NHR + T::NIR + 31) / 32;  // warps' rounds per tile
  __shared__ uint16_t s_cell[8][1024];  // per warp: source lane, x, value 1
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t nwarp = (int64_t)gridDim.x * (blockDim.x >> 5), total = B.total_tiles * UNITS;
  for (int64_t u = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); u < total; u += nwarp) {
    const int64_t flat = u / UNITS;
    const int row = (int)(u - flat * UNITS) * 32 + lane;
    const uint8_t* trec = rec + flat * T::REC;
    uint32_t w2 = 0, w1 = 0;  // cells held at 2 / at 1 by the tile
    int ly = 0, lz = 0;
    if (row < T::NHR) {
      const uint2 w = reinterpret_cast<const uint2*>(trec)[row];
      w2 = w.x;
      w1 = w.y;
      halo_row_of<ND, LY, LZ>(row, ly, lz);
    } else if (row < T::NHR + T::NIR) {
      const uint32_t m = trec[T::NHR * 8 + (row - T::NHR)];
      w2 = (m & 3u) | ((m & 0xCu) << 28);
      w1 = ((m >> 4) & 3u) | ((m & 0xC0u) << 24);
      const int i = row - T::NHR;
      ly = 2 + i % (LY - 4);
      lz = ND == 3 ? 2 + i / (LY - 4) : 0;
    }
    if (!__any_sync(~0u, (w2 | w1) != 0u)) continue;
    const TileAt t = tile_at<ND, LY, LZ>(B, flat);
    const LdirVol& vol = B.v[t.vi];
    const int64_t c0 = t.o[0] + (t.o[1] + ly) * vol.D.cs[1] + (t.o[2] + lz) * vol.D.cs[2];
    uint32_t todo = 0;
    if ((w2 | w1) && row < T::NHR) {
      uint32_t b[8];
      load_planes(vol.g + c0, vol.g, vol.g + vol.D.ncells, b);
      todo = (w1 & (b[7] | b[6])) | (w2 & (b[7] | (b[6] & b[5])));
    } else if (w2 | w1) {
      uint8_t own[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int lx = q < 2 ? q : kBitLX - 4 + q;
        own[q] = 0;
        if (((w2 | w1) >> lx) & 1u) own[q] = vol.g[c0 + lx];
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int lx = q < 2 ? q : kBitLX - 4 + q;
        if ((unsigned)(own[q] >> 5) > (((w1 >> lx) & 1u) ? 1u : 2u)) todo |= 1u << lx;
      }
    }
    // the cells of all 32 rows in one list, so that every lane lowers one: most rows have
    // none and a few have several
    const int cnt = __popc(todo);
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(~0u, incl, o);
      if (lane >= o) incl += v;
    }
    const int n = __shfl_sync(~0u, incl, 31);
    if (n == 0) continue;
    for (int slot = incl - cnt; todo; slot++) {
      const int lx = __ffs(todo) - 1;
      todo &= todo - 1;
      s_cell[warp][slot] = (uint16_t)(lane << 5 | lx | ((w1 >> lx) & 1u) << 15);
    }
    __syncwarp();
    const int dim0 = (int)(((t.o[1] + ly) & 1) + ((t.o[2] + lz) & 1));  // (t.o[0] is even)
    for (int k0 = 0; k0 < n; k0 += 32) {
      const bool has = k0 + lane < n;
      const uint32_t e = has ? s_cell[warp][k0 + lane] : 0u;
      const int src = (int)(e >> 5) & 31, lx = (int)(e & 31u);
      const int64_t c = __shfl_sync(~0u, c0, src) + lx;
      const int dim = __shfl_sync(~0u, dim0, src) + (lx & 1);
      const unsigned v = (e >> 15) ? 1u : 2u;
      const bool item = has && lower_ldir(volume_view(vol, lock, err), c, v) && dim == 3 - (int)v;
      // one append per warp: one per item would serialise on the counter in L2
      const unsigned m = __ballot_sync(~0u, item);
      if (!m) continue;
      int base = 0;
      if (lane == __ffs(m) - 1) base = atomicAdd(n_queue, __popc(m));
      base = __shfl_sync(~0u, base, __ffs(m) - 1);
      if (item) {
        const int slot = base + __popc(m & ((1u << lane) - 1u));
        if (slot < cap) queue[slot] = ((int64_t)t.vi << kVolShift) | c; else atomicOr(err, kErrLocalQueue);
      }
    }
    __syncwarp();
  }
}

// Finish the walks of queued items in global memory.  The walks of a smooth field are
// long, and what bounds them is the latency of one step (the cofacet's byte, its
// compare-and-swap, the partner's: ~1.5 us through L2) times the steps that follow one
// another.  So a block shares one stack: it takes up to kWalkItems items at a time, a
// thread per (item, cofacet), and takes new ones from the queue while its own stack is
// short.  (A thread per item with a stack of its own followed every branch of a walk
// alone: 6.0 of the 6.3 ms of a 64^3 Gaussian-sum .grad.)  A block that has worked
// kWalkTail turns past the queue's end and still has work for several turns hands its
// stack to the next round, which deals it out to all blocks again.  A step's reads come
// through L1 (LdirCell), the first one while the item's coordinates are divided out, and
// the swaps of two cells in one word go out as one: 252 -> 220 us for the walk of a 64^3
// Gaussian sum, 258 -> 228 us at 223 x 187 x 241.  The queue's length is read on the device (0 after an
// overflow: the host finishes with tile passes) and it is dealt out through *cursor.
constexpr int kWalkThreads = 384;
constexpr int kWalkItems = 128;   // items a turn at most: the 64 of a long chain's turn are one pass in 3D
constexpr int kWalkStack = 1024;  // items on the block's stack
constexpr int kWalkTail = 16;     // (4 / 16 / 64: 387 / 381 / 381 us a 64^3 Gaussian sum's .grad, 2.15 ms the
                                  // conforming one of 223 x 187 x 241 with each)

template <int ND>
__global__ void __launch_bounds__(kWalkThreads) ldir_walk_kernel(const LdirBatch B, const int64_t* __restrict__ qin,
                                                                 const int* __restrict__ n_in,
                                                                 uint32_t* __restrict__ cursor,
                                                                 int64_t* __restrict__ qout, int* __restrict__ n_out,
                                                                 int cap, int* lock, int* err) {
  __shared__ int64_t s_stack[kWalkStack];
  __shared__ int64_t s_item[kWalkItems];
  __shared__ int s_top, s_base, s_got, s_out;
  const int tid = threadIdx.x;
  const int n = *n_in;
  if (n <= 0 || n > cap) return;
  const int per = (n + (int)gridDim.x - 1) / (int)gridDim.x;
  const int fetch = per < 8 ? 8 : (per < kWalkItems ? per : kWalkItems);
  bool more = true;
  int tail = 0;
  if (tid == 0) s_top = 0;
  __syncthreads();
  while (true) {
    const int top = s_top;
    if (tid == 0) {
      s_got = 0;
      if (more && top < kWalkItems) {
        const uint32_t b = atomicAdd(cursor, (uint32_t)fetch);
        s_base = (int)b;
        s_got = b >= (uint32_t)n ? -1 : (n - (int)b < fetch ? n - (int)b : fetch);
      }
    }
    __syncthreads();
    const int got = s_got > 0 ? s_got : 0;
    if (s_got < 0) more = false;
    if (!more) tail++;
    if (top + got == 0) break;  // (with more of the queue left, some of it was taken)
    if (tail > kWalkTail && top > kWalkItems) {  // the rest goes to the next round
      if (tid == 0) s_out = atomicAdd(n_out, top);
      __syncthreads();
      for (int i = tid; i < top; i += kWalkThreads) {
        const int slot = s_out + i;
        if (slot < cap) qout[slot] = s_stack[i]; else atomicOr(err, kErrLocalQueue);
      }
      break;
    }
    const int take = top < kWalkItems - got ? top : kWalkItems - got;
    const int m = take + got;
    if (tid < m) s_item[tid] = tid < take ? s_stack[top - 1 - tid] : qin[s_base + tid - take];
    if (tid == 0) s_top = top - take;
    __syncthreads();
    for (int p = tid; p < 2 * ND * m; p += kWalkThreads) {
      const int k = p / (2 * ND), j = p - 2 * ND * k, a = j >> 1;
      const int64_t entry = s_item[k];
      const int vi = entry_volume(entry);
      if (vi >= B.n) {  // not an entry this launch wrote
        atomicOr(err, kErrPassLimit);
        continue;
      }
      const LdirVol& vol = B.v[vi];
      const GradDims& D = vol.D;
      const int64_t i = entry & kCellMask;
      const int sgn = (j & 1) ? -1 : 1;
      const int64_t t = i + sgn * D.cs[a];
      if (t < 0 || t >= D.ncells) continue;
      const GradView G = volume_view(vol, lock, err);
      LdirCell ct(G, t);  // on its way while the coordinates are divided out
      int64_t l[3];
      if (D.ncells <= (int64_t)0xFFFFFFFF) {
        const uint32_t u = (uint32_t)i, d0 = (uint32_t)D.d[0], d1 = (uint32_t)D.d[1];
        const uint32_t r = u / d0;
        l[0] = u - r * d0;
        l[1] = ND == 3 ? r % d1 : r;
        l[2] = ND == 3 ? r / d1 : 0;
      } else {
        l[0] = i % D.d[0];
        l[1] = (i / D.d[0]) % D.d[1];
        l[2] = ND == 3 ? i / (D.d[0] * D.d[1]) : 0;
      }
      const int dim = (int)((l[0] & 1) + (l[1] & 1) + (l[2] & 1));
      const unsigned value = dim == 1 ? 2u : 1u;  // edges walk the value-2 closure, quads value 1
      const int64_t ca = a == 0 ? l[0] : (a == 1 ? l[1] : l[2]);
      if (ca & 1) continue;  // cofacets only along even axes
      if (ca + sgn < 0 || ca + sgn >= D.d[a]) continue;
      const unsigned bt = ct.byte(), code = (bt >> 2) & 7u;
      if (!(bt & 1u) || code == 7u) continue;
      const int pc = map3(D.dec_map, (int)code);
      const int pa = pc >> 1, ps = (pc & 1) ? -1 : 1;
      const int64_t tp = t + ps * D.cs[pa];
      // the partner's coordinate along the pair's axis, and its dimension
      const int64_t cp = (pa == 0 ? l[0] : (pa == 1 ? l[1] : l[2])) + (pa == a ? sgn : 0) + ps;
      if (tp == i || cp < 0 || cp >= D.d[pa]) {  // (a pair code pointing out of the complex)
        lower_ldir(G, t, value);
        continue;
      }
      const int pdim = pa == a ? dim : (((cp & 1) != 0) ? dim + 2 : dim);
      const bool item = value != 2u || pdim == 1;  // a hex ends the value-2 path
      // the cofacet's and the partner's swaps go out together, as one where they share a word
      LdirCell cq(G, tp);
      bool won;
      if (cq.inside && cq.w == ct.w) {
        cq.cur = ct.cur;
        won = cq.pair(G, ct, value);
      } else {
        ct.swap(value);
        cq.swap(value);
        ct.finish(G, t, value);
        won = cq.finish(G, tp, value);
      }
      if (!won || !item) continue;
      const int slot = atomicAdd(&s_top, 1);
      if (slot < kWalkStack) s_stack[slot] = ((int64_t)vi << kVolShift) | tp;
      else push_item(qout, n_out, cap, err, ((int64_t)vi << kVolShift) | tp);
    }
    __syncthreads();
    if (tid == 0 && s_top > kWalkStack) s_top = kWalkStack;
    __syncthreads();
  }
}

namespace {
// multi-pass tiles
constexpr int kTX3 = 32, kTY3 = 32, kTZ3 = 16, kBS3 = 512;
constexpr int kTX2 = 128, kTY2 = 64, kBS2 = 256;
using Tile3 = LdirTile<3, kTX3, kTY3, kTZ3>;
using Tile2 = LdirTile<2, kTX2, kTY2, 1>;
// single-pass bit-row tiles: 28 x 28 x 28 owned cells in 3D, 28 x 124 in 2D
constexpr int kBitLY3 = 32, kBitLZ3 = 32;
constexpr int kBitLY2 = 32 * kSlabs;
using Bit3 = BitTile<3, kBitLY3, kBitLZ3>;
using Bit2 = BitTile<2, kBitLY2, 1>;
static_assert(kBitLZ3 == kSlabs * kTileWarps, "the block's slabs make the box");
}  // namespace

int64_t ldir_num_tiles(int nd, const GradDims& D) {
  if (nd == 3) return ((D.d[0] + kTX3 - 1) / kTX3) * ((D.d[1] + kTY3 - 1) / kTY3) * ((D.d[2] + kTZ3 - 1) / kTZ3);
  return ((D.d[0] + kTX2 - 1) / kTX2) * ((D.d[1] + kTY2 - 1) / kTY2);
}

int64_t ldir_bit_tiles(int nd, const GradDims& D) {
  if (nd == 3)
    return ((D.d[0] + Bit3::TX - 1) / Bit3::TX) * ((D.d[1] + Bit3::TY - 1) / Bit3::TY) *
           ((D.d[2] + Bit3::TZ - 1) / Bit3::TZ);
  return ((D.d[0] + Bit2::TX - 1) / Bit2::TX) * ((D.d[1] + Bit2::TY - 1) / Bit2::TY);
}

int64_t ldir_halo_bytes(int nd) { return nd == 3 ? Bit3::REC : Bit2::REC; }

cudaError_t make_ldir_batch(int nd, int n, uint8_t* const* g, const GradDims* D, LdirBatch* B) {
  if (n < 1 || n > kMaxBatch || (nd == 2 && n != 1)) return cudaErrorInvalidValue;
  B->n = n;
  int64_t off = 0;
  for (int i = 0; i < n; i++) {
    B->v[i].g = g[i];
    B->v[i].D = D[i];
    B->v[i].tile0 = off;
    off += ldir_bit_tiles(nd, D[i]);
  }
  B->total_tiles = off;
  return cudaSuccess;
}

cudaError_t launch_ldir_tile(int nd, const LdirBatch& B, uint8_t* rec, int* err, int num_sms, cudaStream_t stream,
                             int ctas_per_sm) {
  const int64_t blocks = nd == 3 ? B.total_tiles : (B.total_tiles + 7) / 8;  // 2D: a warp per tile
  const int64_t cap = ctas_per_sm > 0 ? (int64_t)num_sms * ctas_per_sm : 0x7FFFFFFF;  // 0: a block per tile
  const int grid = (int)(blocks < cap ? blocks : cap);
  if (grid <= 0) return cudaSuccess;
  ::msc::count_launch();
  // 4 blocks per SM where there are blocks for them (4.10 -> 3.51 ms at 512^3), 3 where
  // every tile has its place at once anyhow (30.5 instead of 35 us at 64^3)
  if (nd == 3 && B.total_tiles > 3 * (int64_t)num_sms)
    ldir_tile3_kernel<4><<<grid, 32 * kTileWarps, 0, stream>>>(B, rec, err);
  else if (nd == 3)
    ldir_tile3_kernel<3><<<grid, 32 * kTileWarps, 0, stream>>>(B, rec, err);
  else
    ldir_tile2_kernel<<<grid, 256, 0, stream>>>(B, rec, err);
  return cudaGetLastError();
}

// eight warps a block, a warp per 32 rows of a tile's record
static int check_grid(int nd, const LdirBatch& B, int num_sms) {
  const int64_t cap = (int64_t)num_sms * 8;
  const int64_t rows = nd == 3 ? Bit3::NHR + Bit3::NIR : Bit2::NHR + Bit2::NIR;
  const int64_t blocks = (B.total_tiles * ((rows + 31) / 32) + 7) / 8;
  return (int)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

cudaError_t launch_ldir_check(int nd, const LdirBatch& B, const uint8_t* rec, int64_t* queue, int* n_queue, int cap,
                              int* lock, int* err, int num_sms, cudaStream_t stream) {
  ::msc::count_launch();
  if (nd == 3)
    ldir_check_kernel<3, kBitLY3, kBitLZ3><<<check_grid(nd, B, num_sms), 256, 0, stream>>>(B, rec, queue, n_queue, cap,
                                                                                       lock, err);
  else
    ldir_check_kernel<2, kBitLY2, 1><<<check_grid(nd, B, num_sms), 256, 0, stream>>>(B, rec, queue, n_queue, cap, lock,
                                                                                 err);
  return cudaGetLastError();
}

cudaError_t launch_ldir_walk(int nd, const LdirBatch& B, const int64_t* qin, const int* n_in, int* cursor,
                             int64_t* qout, int* n_out, int cap, int* lock, int* err, int num_sms,
                             cudaStream_t stream) {
  if (cudaError_t e = cudaMemsetAsync(n_out, 0, sizeof(int), stream)) return e;
  if (cudaError_t e = cudaMemsetAsync(cursor, 0, sizeof(int), stream)) return e;
  uint32_t* cur = reinterpret_cast<uint32_t*>(cursor);
  ::msc::count_launch();
  if (nd == 3)
    ldir_walk_kernel<3><<<num_sms * 5, kWalkThreads, 0, stream>>>(B, qin, n_in, cur, qout, n_out, cap, lock, err);
  else
    ldir_walk_kernel<2><<<num_sms * 5, kWalkThreads, 0, stream>>>(B, qin, n_in, cur, qout, n_out, cap, lock, err);
  return cudaGetLastError();
}

cudaError_t launch_ldir_pass(int nd, uint8_t* g, const GradDims& D, const uint8_t* dirty_in, uint8_t* dirty_out,
                             int* changed, int* err, int num_sms, cudaStream_t stream) {
  const int64_t nt = ldir_num_tiles(nd, D);
  const int64_t cap = (int64_t)num_sms * 4;
  const int grid = (int)(nt < cap ? nt : cap);
  if (grid <= 0) return cudaSuccess;
  if (nd == 3) {
    auto k = ldir_pass_kernel<3, kTX3, kTY3, kTZ3, kBS3>;
    const size_t sm = Tile3::smem_bytes();
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    ::msc::count_launch();
    k<<<grid, kBS3, sm, stream>>>(g, D, dirty_in, dirty_out, changed, err);
  } else {
    auto k = ldir_pass_kernel<2, kTX2, kTY2, 1, kBS2>;
    const size_t sm = Tile2::smem_bytes();
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    ::msc::count_launch();
    k<<<grid, kBS2, sm, stream>>>(g, D, dirty_in, dirty_out, changed, err);
  }
  return cudaGetLastError();
}

}  // namespace msc
