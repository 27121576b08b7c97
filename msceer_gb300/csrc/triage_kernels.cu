// Learned triage: a 3x3x3 convolutional network (Cin -> 16 -> 16 -> 2 channels) that
// flags the vertices whose integrated destination differs from their combinatorial
// steepest-path destination.  Forward and input-gradient convolutions are BF16
// implicit GEMMs on the tcgen05 tensor cores with FP32 accumulation in TMEM, and so is the
// weight gradient; loss and optimiser run on the CUDA cores in FP32.
//
// Activation layout ("row-planar"): [Z][Y][2][X][8] BF16.  Each (y, z) row of the
// volume holds two planes, channels 0-7 and channels 8-15, each X x 16 bytes.  That
// is the K-major, no-swizzle operand layout of the MMA (8-row x 16-byte core
// matrices, rows 16 bytes apart), so an operand is a plain address into a staged
// row: output vertices x0..x0+127 under tap (dx, dy, dz) read the staged row of
// (y+dy, z+dz) starting at x0+dx.
//
// A convolution's tile is 128 (x) x 8 (y) output vertices at one z, and its accumulator 128
// x 128: a TMEM lane is an output row and one of 16 output channels, a column a vertex.  An
// input row belongs to up to three of the eight output rows, at dy = -1, 0, +1, so one MMA
// (M = eight rows x 16 channels, N = 128 vertices, K = 16 input channels) takes it to all of
// them: the weights of dy = +1, 0, -1 lie one after the other, so that the operand of input
// row yy, at the block of dy = yy, holds for output row j the weights of dy = yy - j; the
// lanes of the other rows are switched off.  97 MMAs for a tile's 8 x 27 taps (3 x 10 x 3, and
// seven output rows start with one of their own), each output row's in the order dz, dy, dx,
// all of one shape on one accumulator and so in order.
// One CTA per SM keeps the weights in shared memory and works through a run of tiles along
// z, each with one new plane of input rows (10 x 130, staged by bulk copies, one per
// 8-channel plane of a row, zeros outside the volume) in a ring of four, and two
// accumulators, so that the load of a plane, the MMAs of a tile and the epilogue of the one
// before run side by side.  The epilogue turns lanes of channels into rows of vertices in
// shared memory.
// (One MMA per tap and output row, M = 128 vertices and N = 16 channels, took the same 95
// cycles, 108 of them for 4 x 128 vertices: 152-159 us a layer at 128^3, and with a CTA per
// tile 181-217 us; so 79-89 us.  A layer's activations in and out take 20 us of HBM time.)
#include <cuda_bf16.h>

#include "tc_sm100.cuh"
#include "triage.cuh"

namespace msc {

namespace {
constexpr int kBX = 128;                            // vertices of a tile along x
constexpr int kInX = kBX + 2;
constexpr int kPlaneB = kInX * 16;                  // one staged 8-channel plane of a row
constexpr int kRowB = 2 * kPlaneB;                  // one staged row
// convolution
constexpr int kCY = 8, kCInY = kCY + 2;             // output rows, input rows per z
constexpr int kSlotB = kCInY * kRowB;               // a ring slot: the input rows of one z
constexpr int kSlots = 4;
constexpr int kTapB = 256;                          // 16 rows (output channels) x 8 BF16 of a tap
constexpr int kHalfB = 27 * kTapB;                  // of one 8-channel half of K
constexpr int kWeightB = 2 * kHalfB;
constexpr int kWPadB = (kCY - 1) * kTapB;           // the operands reach so far to either side of the weights
constexpr int kOutPlaneB = kBX * 16 + 32;           // epilogue: a row's 8-channel plane, clear of the others' banks
constexpr int kOutB = 4 * kOutPlaneB;               // of one warp: two rows
constexpr int kSmemConv = 1024 + kSlots * kSlotB + 2 * kWPadB + kWeightB + 4 * kOutB + 128;
constexpr uint32_t kSetCols = kBX;                  // columns of an accumulator
constexpr uint32_t kTmemCols = 2 * kSetCols;
constexpr int kConvThreads = 192;                   // four epilogue warps, the MMAs', the loads'
static_assert(kSlotB % 16 == 0 && kWPadB % 16 == 0 && kWeightB % 16 == 0 && kOutB % 16 == 0, "16-byte copies");
static_assert(kSmemConv <= 227 * 1024, "shared memory of a block");
static_assert(2 * kBX * 2 * 4 <= kOutB, "two rows' logits fit a warp's staging");
}  // namespace

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   tc::smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(tc::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(bar)), "r"(bytes)
               : "memory");
}

// Epilogue kinds
//   kEpiReluBf16  out = bf16(relu(acc + bias))                         (hidden layers)
//   kEpiLogits    logits[c][v] = acc[c] + bias[c], c < 2, FP32 planar  (output layer)
//   kEpiMaskBf16  out = bf16(acc * (mask_act > 0))                     (input gradient)
// Stages NX x NY x NZ vertices of a row-planar activation from (xs, ys, zs) on, both planes
// of a row one after the other, zeros outside the volume; `bar` gets one arrival with the
// bytes to come (and `more` bytes besides).  One whole warp calls it, after the stage's
// last reader is done.
template <int NX, int NY, int NZ>
__device__ __forceinline__ void stage_rows(unsigned char* dst, const __nv_bfloat16* __restrict__ act, const ConvDims& D,
                                           int xs, int ys, int zs, uint32_t more, uint64_t* bar) {
  constexpr int ROWS = NY * NZ * 2, PLANE = NX * 16;
  const int lane = threadIdx.x & 31;
  const int xa = max(xs, 0), xb = (int)min((int64_t)(xs + NX), D.X);
  auto row_of = [&](int p, int& y, int& z) {
    y = ys + (p >> 1) % NY;
    z = zs + (p >> 1) / NY;
    return y >= 0 && y < D.Y && z >= 0 && z < D.Z;
  };
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  int y, z;
  if (xa > xs || xb < xs + NX)
    for (int p = lane; p < ROWS; p += 32) {
      uint4* r = reinterpret_cast<uint4*>(dst + p * PLANE);
      for (int x = 0; x < xa - xs; x++) r[x] = zero;
      for (int x = xb - xs; x < NX; x++) r[x] = zero;
    }
  if (ys < 0 || ys + NY > D.Y || zs < 0 || zs + NZ > D.Z)
    for (int p = 0; p < ROWS; p++) {
      if (row_of(p, y, z)) continue;
      for (int x = lane; x < NX; x += 32) reinterpret_cast<uint4*>(dst + p * PLANE)[x] = zero;
    }
  tc::fence_proxy_async_smem();
  __syncwarp();
  const int ny = (int)min((int64_t)(ys + NY), D.Y) - max(ys, 0), nz = (int)min((int64_t)(zs + NZ), D.Z) - max(zs, 0);
  const uint32_t bytes = (uint32_t)(xb - xa) * 16u;
  if (lane == 0) mbar_expect_tx(bar, (uint32_t)(ny * nz * 2) * bytes + more);
  __syncwarp();
  for (int p = lane; p < ROWS; p += 32)
    if (row_of(p, y, z))
      bulk_load(dst + p * PLANE + (xa - xs) * 16,
                act + ((((int64_t)z * D.Y + y) * 2 + (p & 1)) * D.X + xa) * 8, bytes, bar);
}

// Tiles of a convolution, z fastest.
struct ConvColumns {
  int nx, ny;
  int64_t Z, n;
  __device__ __forceinline__ void at(int64_t t, int& x0, int& y0, int& z) const {
    const int64_t c = t / Z, r = c / nx;
    z = (int)(t - c * Z);
    x0 = (int)(c - r * nx) * kBX;
    y0 = (int)r * kCY;
  }
  // tiles of block b of g
  __device__ __forceinline__ int64_t first(int b, int g) const { return n / g * b + (n % g * b) / g; }
};

// The mask's values for one warp's share of a tile, as conv_epilogue writes it.  They are
// asked for before the wait for the tile's MMAs: loaded where they are used, the mask held
// up the epilogue (164 us a layer at 128^3 instead of 87; 89 with the marks below).
__device__ __forceinline__ void load_mask(uint4 (&m)[16], const __nv_bfloat16* __restrict__ mask_act, int x0, int y,
                                          int z, const ConvDims& D) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const int q = i >> 2, x = x0 + lane + 32 * (i & 3);  // q: row, plane
    m[i] = make_uint4(0u, 0u, 0u, 0u);
    if (y + (q >> 1) < D.Y && x < D.X)
      m[i] = *reinterpret_cast<const uint4*>(mask_act +
                                             ((((int64_t)z * D.Y + y + (q >> 1)) * 2 + (q & 1)) * D.X + x) * 8);
  }
}

// The mask multiplies the FP32 gradient, but meets it only after it has been rounded: one
// that is finite and rounds to infinity waits in the staging under this mark (a NaN that no
// conversion makes), so that masked it is zero, while an infinite or NaN gradient stays NaN.
constexpr uint32_t kOverflowMark = 0x7F81u;
constexpr float kRoundsToInf = 0x1.FFp127f;

// One warp's share of a tile: the accumulator lanes of output rows 2 w and 2 w + 1.
// `done` gets an arrival when they have been read.
template <int EPI>
__device__ __forceinline__ void conv_epilogue(uint32_t tl, unsigned char* s_out, int x0, int y, int z, float bias,
                                              const ConvDims& D, __nv_bfloat16* __restrict__ out_act,
                                              float* __restrict__ out_logits,
                                              const uint4 (&mask)[16], uint64_t* done) {
  const int lane = threadIdx.x & 31, row = lane >> 4, ch = lane & 15;
  const bool odd = lane & 1;
  unsigned char* mine = s_out + (2 * row + (ch >> 3)) * kOutPlaneB + (odd ? 16 : 0) + (ch & 6) * 2;
  bool marked = false;
  __syncwarp();  // the tile before has left the staging
  while (true) {
    float most[4] = {0.f, 0.f, 0.f, 0.f};  // largest magnitudes, four chains of them
#pragma unroll 1
    for (int c = 0; c < kBX; c += 16) {
      float v[16];
      tc::tmem_ld16(tl + c, v);
      if (EPI == kEpiLogits) {
        if (ch < 2) {
          float4* o = reinterpret_cast<float4*>(s_out + (2 * row + ch) * kBX * 4 + c * 4);
#pragma unroll
          for (int k = 0; k < 4; k++)
            o[k] = make_float4(v[4 * k] + bias, v[4 * k + 1] + bias, v[4 * k + 2] + bias, v[4 * k + 3] + bias);
        }
      } else {
        uint32_t h[16];
#pragma unroll
        for (int k = 0; k < 16; k++) {
          const float a = EPI == kEpiReluBf16 ? fmaxf(v[k] + bias, 0.f) : v[k];
          h[k] = __bfloat16_as_ushort(__float2bfloat16_rn(a));
        }
        if (EPI == kEpiMaskBf16) {
#pragma unroll
          for (int k = 0; k < 16; k++) most[k & 3] = fmaxf(most[k & 3], fabsf(v[k]));
          if (marked)
#pragma unroll
            for (int k = 0; k < 16; k++)
              if (isfinite(v[k]) && fabsf(v[k]) >= kRoundsToInf) h[k] = (h[k] & 0x8000u) | kOverflowMark;
        }
        // two channels to a word: the even lane of a pair takes the even vertices
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? h[k] : h[k + 1], 1);
          *reinterpret_cast<uint32_t*>(mine + (c + k) * 16) = odd ? (got | (h[k + 1] << 16)) : (h[k] | (got << 16));
        }
      }
    }
    if (EPI != kEpiMaskBf16 || marked) break;
    marked = __any_sync(0xffffffffu, fmaxf(fmaxf(most[0], most[1]), fmaxf(most[2], most[3])) >= kRoundsToInf);
    if (!marked) break;
    __syncwarp();  // once more, with the marks
  }
  tc::fence_before_sync();
  __syncwarp();
  if (lane == 0) tc::mbar_arrive(done);
  if constexpr (EPI == kEpiLogits) {
#pragma unroll
    for (int q = 0; q < 4; q++) {  // row, channel
      if (y + (q >> 1) >= D.Y) continue;
      const float* sv = reinterpret_cast<const float*>(s_out) + q * kBX;
      float* o = out_logits + (q & 1) * D.N + ((int64_t)z * D.Y + y + (q >> 1)) * D.X + x0;
      for (int x = lane; x < kBX && x0 + x < D.X; x += 32) o[x] = sv[x];
    }
  } else {
    if (marked)  // apart from the loop below, whose loads go out together
#pragma unroll
      for (int i = 0; i < 16; i++) {
        unsigned short* r = reinterpret_cast<unsigned short*>(s_out + (i >> 2) * kOutPlaneB + (lane + 32 * (i & 3)) * 16);
        const __nv_bfloat16* mh = reinterpret_cast<const __nv_bfloat16*>(&mask[i]);
#pragma unroll
        for (int c = 0; c < 8; c++)
          if ((r[c] & 0x7FFFu) == kOverflowMark)
            r[c] = (unsigned short)((r[c] & 0x8000u) | (__bfloat162float(mh[c]) > 0.f ? 0x7F80u : 0u));
      }
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const int q = i >> 2, x = lane + 32 * (i & 3);  // q: row, plane
      if (y + (q >> 1) >= D.Y || x0 + x >= D.X) continue;
      uint4 r = *reinterpret_cast<const uint4*>(s_out + q * kOutPlaneB + x * 16);
      if (EPI == kEpiMaskBf16) {
        const __nv_bfloat16* mh = reinterpret_cast<const __nv_bfloat16*>(&mask[i]);
        __nv_bfloat16* rh = reinterpret_cast<__nv_bfloat16*>(&r);
#pragma unroll
        for (int c = 0; c < 8; c++)
          rh[c] = __float2bfloat16_rn(__bfloat162float(rh[c]) * (__bfloat162float(mh[c]) > 0.f ? 1.f : 0.f));
      }
      *reinterpret_cast<uint4*>(out_act + ((((int64_t)z * D.Y + y + (q >> 1)) * 2 + (q & 1)) * D.X + x0 + x) * 8) = r;
    }
  }
}

// Every wait is bounded; a role whose wait runs out reports it in err and ends, and the
// others' waits run out after it.
template <int EPI>
__global__ void __launch_bounds__(kConvThreads, 1) conv3_tc_kernel(const __nv_bfloat16* __restrict__ in_act,
                                                                const uint8_t* __restrict__ wblob,
                                                                const float* __restrict__ bias, const ConvDims D,
                                                                const ConvColumns T,
                                                                __nv_bfloat16* __restrict__ out_act,
                                                                float* __restrict__ out_logits,
                                                                const __nv_bfloat16* __restrict__ mask_act,
                                                                int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* s_in = sm;
  unsigned char* s_w = sm + kSlots * kSlotB + kWPadB;
  unsigned char* s_out = s_w + kWeightB + kWPadB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_out + 4 * kOutB);
  uint64_t* full = bars;                // a slot's input rows (and, with the first, the weights) have come
  uint64_t* empty = bars + kSlots;      // the MMAs that read it are done
  uint64_t* tfull = bars + 2 * kSlots;  // an accumulator is ready
  uint64_t* tempty = tfull + 2;         // and read
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(tempty + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int q = 0; q < kSlots; q++) {
      tc::mbar_init(&full[q], 1);
      tc::mbar_init(&empty[q], 1);
    }
    for (int q = 0; q < 2; q++) {
      tc::mbar_init(&tfull[q], 1);
      tc::mbar_init(&tempty[q], 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4) tc::tmem_alloc<kTmemCols>(s_tmem);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *s_tmem;
  const int64_t t0 = T.first(blockIdx.x, gridDim.x), t1 = T.first(blockIdx.x + 1, gridDim.x);

  if (warp == 5) {  // loads: a tile's three planes, or its third where the tile before had the others
    int64_t i = 0;
    bool ok = true;
    for (int64_t t = t0; t < t1 && ok; t++) {
      int x0, y0, z;
      T.at(t, x0, y0, z);
      for (int dz = (t == t0 || z == 0) ? -1 : 1; dz <= 1 && ok; dz++, i++) {
        const int q = (int)(i % kSlots);
        ok = i < kSlots || tc::mbar_wait(&empty[q], (uint32_t)(i / kSlots - 1) & 1u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) atomicOr(err, 1);
          break;
        }
        if (i == 0 && lane == 0) bulk_load(s_w, wblob, (uint32_t)kWeightB, &full[q]);
        stage_rows<kInX, kCInY, 1>(s_in + q * kSlotB, in_act, D, x0 - 1, y0 - 1, z + dz,
                                   i == 0 ? (uint32_t)kWeightB : 0u, &full[q]);
      }
    }
    // every load has landed before the block ends, also where the MMAs gave up on it
    for (int64_t k = i > kSlots ? i - kSlots : 0; k < i; k++)
      if (!tc::mbar_wait(&full[k % kSlots], (uint32_t)(k / kSlots) & 1u) && lane == 0) atomicOr(err, 1);
  } else if (warp == 4) {  // MMAs
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(128, kBX);
      const uint32_t w0 = tc::smem_u32(s_w), i0 = tc::smem_u32(s_in);
      int64_t s = 0, have = 0;  // the tile's first plane, planes that have come
      for (int64_t t = t0; t < t1; t++) {
        int x0, y0, z;
        T.at(t, x0, y0, z);
        const int q = (int)((t - t0) & 1);
        const uint32_t use = (uint32_t)((t - t0) >> 1);
        bool ok = use == 0 || tc::mbar_wait(&tempty[q], (use - 1) & 1u);
        for (; have < s + 3 && ok; have++) ok = tc::mbar_wait(&full[have % kSlots], (uint32_t)(have / kSlots) & 1u);
        if (!ok) {
          atomicOr(err, 1);
          break;
        }
        tc::fence_after_sync();
        const uint32_t d = tbase + q * kSetCols;
#pragma unroll 1
        for (int dz = 0; dz < 3; dz++) {
          const uint32_t rows = i0 + (uint32_t)((s + dz) % kSlots) * kSlotB;
#pragma unroll
          for (int yy = 0; yy < kCInY; yy++) {
            // output rows lo .. hi take this input row, at dy = yy - j
            const int lo = yy > 2 ? yy - 2 : 0, hi = yy < kCY ? yy : kCY - 1;
            uint32_t off[4], old[4], fresh[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
              off[k] = old[k] = fresh[k] = 0;
              for (int j = 2 * k; j < 2 * k + 2; j++) {
                const uint32_t m = 0xFFFFu << (16 * (j & 1));
                if (j < lo || j > hi) off[k] |= m;
                if (j < lo || j >= yy) old[k] |= m;
                if (j != yy) fresh[k] |= m;
              }
            }
#pragma unroll
            for (int dx = 0; dx < 3; dx++) {
              const uint64_t a =
                  tc::smem_desc(w0 + (uint32_t)(((dz * 3 + dx) * 3 + 2 - yy) * kTapB), kHalfB, 128);
              const uint64_t b = tc::smem_desc(rows + (uint32_t)(yy * kRowB + dx * 16), kPlaneB, 128);
              if (dx == 0 && yy < kCY && dz == 0) {  // output row yy starts here
                if (yy > 0) tc::mma_bf16_lanes(d, a, b, idesc, old, true);
                tc::mma_bf16_lanes(d, a, b, idesc, fresh, false);
              } else {
                tc::mma_bf16_lanes(d, a, b, idesc, off, true);
              }
            }
          }
        }
        // planes that no further tile reads: one, or all at the end of a column
        const int last = (z == D.Z - 1 || t == t1 - 1) ? 3 : 1;
        for (int k = 0; k < last; k++) tc::mma_commit(&empty[(s + k) % kSlots]);
        tc::mma_commit(&tfull[q]);
        s += last;
      }
    }
  } else {  // epilogue
    const int ch = lane & 15;
    const float b = EPI == kEpiMaskBf16 ? 0.f : (EPI == kEpiLogits && ch >= 2 ? 0.f : bias[ch]);
    for (int64_t t = t0; t < t1; t++) {
      const int q = (int)((t - t0) & 1);
      int x0, y0, z;
      T.at(t, x0, y0, z);
      uint4 mask[16];
      if (EPI == kEpiMaskBf16) load_mask(mask, mask_act, x0, y0 + 2 * warp, z, D);
      const bool ok = tc::mbar_wait(&tfull[q], (uint32_t)((t - t0) >> 1) & 1u);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicOr(err, 2);
        break;
      }
      tc::fence_after_sync();
      conv_epilogue<EPI>(tbase + q * kSetCols + ((uint32_t)(32 * warp) << 16), s_out + warp * kOutB, x0, y0 + 2 * warp,
                         z, b, D, out_act, out_logits, mask, &tempty[q]);
    }
  }
  __syncwarp();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 4) tc::tmem_dealloc<kTmemCols>(tbase);
}

// ---- weight gradient ----------------------------------------------------------------------
//
// dW[tap][cin][cout] = sum over the vertices v of X[v + tap][cin] * dY[v][cout], db[cout] =
// sum dY[v][cout]: the vertices are the MMA's K, so both operands are MN-major as the
// row-planar rows lie (a core matrix is 8 channels x 8 vertices).  A tile is 128 (x) x 2 (y)
// x 2 (z) vertices; its staged X is the 4 x 4 rows around, all 8-channel planes kPlaneB
// apart, so M = 128 spans eight rows, and its dY the four rows, N = 64.  With dx as a shift
// of 16 bytes, six MMAs per 16 vertices (three dx, two halves of the rows) give the products
// of every input row with every output row; those with -1 <= dy, dz <= 1 are read.  An MMA
// takes some 95 cycles whatever its N up to 128, so few and wide ones bound it least: with
// one output row (N = 16) it took four times as many.
// The tensor core's FP32 accumulation loses up to an ulp per MMA, so an accumulator runs
// over one tile only, eight MMAs, and is added to FP32 registers: 16 warps, each with the
// lanes of its quarter, one half of the rows and one z of dY.  Against 64 bits the layer-3
// gradient at 128^3 is off by 2.5e-7 (4.4e-7 with FP32 FMAs, 4.3e-6 with the accumulators kept
// in TMEM over all tiles).
// The CUDA-core form (27 x 2 accumulators per thread, X and dY staged as FP32) took 1.0 ms
// a layer at 128^3, one output row to an MMA 197-211 us; so 95 us.
constexpr int kGY = 2, kGZ = 2;                     // output rows of a tile
constexpr int kGRows = (kGY + 2) * (kGZ + 2);       // its input rows
constexpr int kXB = kGRows * kRowB, kDyB = kGY * kGZ * 2 * kBX * 16;
constexpr int kGStageB = kXB + kDyB;
constexpr int kSmemWgrad = 1024 + 2 * kGStageB + 64;
constexpr int kWgradThreads = 512;
constexpr uint32_t kAccCols = 16 * kGY * kGZ;       // columns of one of the six accumulators
constexpr uint32_t kWgradCols = 512;
static_assert(kGRows == 16 && 6 * kAccCols <= kWgradCols, "two operands of eight rows");
static_assert(27 * 256 * 4 + 16 * 8 * 4 <= kGStageB, "the final sums fit a stage");
// A tile's vertices along x (what lies past the volume is not multiplied), and whether its
// second output row along y or z lies past the volume: their products are not read, since a
// zero times an infinite input is none.
constexpr int kEdgeY = 1 << 8, kEdgeZ = 1 << 9;
static_assert(kGY == 2 && kGZ == 2 && kBX <= 0xFF, "the edge word");
struct WgradTiles {
  int nx, ny;
  int64_t n;
  __device__ __forceinline__ void at(int64_t t, int& x0, int& y0, int& z0) const {
    const int64_t r = t / nx;
    x0 = (int)(t - r * nx) * kBX;
    y0 = (int)(r % ny) * kGY;
    z0 = (int)(r / ny) * kGZ;
  }
};

__global__ void __launch_bounds__(kWgradThreads, 1) conv_wgrad_tc_kernel(const __nv_bfloat16* __restrict__ X,
                                                                         const __nv_bfloat16* __restrict__ dY,
                                                                         const ConvDims D, const WgradTiles T,
                                                                         float* __restrict__ dW,
                                                                         float* __restrict__ db,
                                                                         int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + 2 * kGStageB);  // [0], [1] a stage's loads, [2] the MMAs
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + 3);
  int* s_edge = reinterpret_cast<int*>(s_tmem + 1);  // of a stage's tile
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    tc::mbar_init(&bars[0], 2);
    tc::mbar_init(&bars[1], 2);
    tc::mbar_init(&bars[2], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc::tmem_alloc<kWgradCols>(s_tmem);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *s_tmem;
  // this warp's part of the accumulators: TMEM lane = 16 r + channel of the r-th of eight
  // input rows; columns by output row jz, jy
  const int half = (warp >> 2) & 1, jz = warp >> 3;
  const int zz = 2 * half + ((warp & 3) >> 1), yy = 2 * (warp & 1) + (lane >> 4);  // input row
  const int dz = zz - jz;                                                          // warp-uniform
  const uint32_t tl = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + 3 * kAccCols * half + 16 * kGY * jz;
  constexpr uint32_t idesc = tc::idesc_bf16_f32(128, kAccCols, true);

  float acc[3][kGY][16];  // [dx][jy][cout] of the thread's input row and channel
  float bsum[2] = {0.f, 0.f};
#pragma unroll
  for (int q = 0; q < 3 * kGY; q++)
#pragma unroll
    for (int c = 0; c < 16; c++) acc[q / kGY][q % kGY][c] = 0.f;

  auto stage = [&](int64_t t, int64_t i) {  // warps 1 and 2
    int x0, y0, z0;
    T.at(t, x0, y0, z0);
    unsigned char* s = sm + (i & 1) * kGStageB;
    if (warp == 1 && lane == 0)  // (what this thread's arrival below makes visible)
      s_edge[i & 1] = (int)min((int64_t)kBX, D.X - x0) | (y0 + 1 < D.Y ? 0 : kEdgeY) | (z0 + 1 < D.Z ? 0 : kEdgeZ);
    if (warp == 1) stage_rows<kInX, kGY + 2, kGZ + 2>(s, X, D, x0 - 1, y0 - 1, z0 - 1, 0u, &bars[i & 1]);
    if (warp == 2) stage_rows<kBX, kGY, kGZ>(s + kXB, dY, D, x0, y0, z0, 0u, &bars[i & 1]);
  };
  int64_t t = blockIdx.x, i = 0;
  bool ok = true;
  if (t < T.n) stage(t, 0);
  for (; t < T.n && ok; t += gridDim.x, i++) {
    const unsigned char* s_dy = sm + (i & 1) * kGStageB + kXB;
    // (the other stage's MMAs ended with the tile before)
    const bool more = t + gridDim.x < T.n;
    if (more) stage(t + gridDim.x, i + 1);
    ok = tc::mbar_wait(&bars[i & 1], (uint32_t)(i >> 1) & 1u);
    if (!ok && lane == 0) atomicOr(err, 1);
    const int edge = s_edge[i & 1];
    if (warp == 0) {
      ok = __all_sync(0xffffffffu, ok);
      if (ok && lane == 0) {
        tc::fence_after_sync();
        const uint32_t a0 = tc::smem_u32(sm + (i & 1) * kGStageB), b0 = a0 + kXB;
#pragma unroll 1
        for (int k = 0; k < (edge & 0xFF); k += 16) {
          // N groups of 8 channels: (row, plane), kBX x 16 bytes apart
          const uint64_t bd = tc::smem_desc(b0 + (uint32_t)(k * 16), 128, kBX * 16);
#pragma unroll
          for (int q = 0; q < 6; q++) {
            const uint32_t a = a0 + (uint32_t)((8 * (q / 3)) * kRowB + (k + q % 3) * 16);
            tc::mma_bf16(tbase + kAccCols * q, tc::smem_desc(a, 128, kPlaneB), bd, idesc, k > 0);
          }
        }
        tc::mma_commit(&bars[2]);
      }
      __syncwarp();
    }
    // the bias gradient while the MMAs run: a warp has 64 vertices of an output row's plane,
    // a thread two channels of every eighth
    if (ok) {
      const unsigned char* p = s_dy + (((warp >> 1) & 3) * 2 + (warp & 1)) * (kBX * 16) + (warp >> 3) * 64 * 16 + lane * 4;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(p + k * 128);
        bsum[0] += __low2float(h);
        bsum[1] += __high2float(h);
      }
    }
    const bool done = tc::mbar_wait(&bars[2], (uint32_t)i & 1u);
    if (!done && lane == 0) atomicOr(err, 2);
    ok = __all_sync(0xffffffffu, ok && done);
    if (ok && dz >= 0 && dz <= 2 && !(jz == 1 && (edge & kEdgeZ))) {
      tc::fence_after_sync();
#pragma unroll
      for (int jy = 0; jy < kGY; jy++) {
        if (jy == 1 && (edge & kEdgeY)) break;
#pragma unroll
        for (int dx = 0; dx < 3; dx++) {
          float v[16];
          tc::tmem_ld16(tl + kAccCols * dx + 16 * jy, v);
#pragma unroll
          for (int c = 0; c < 16; c++) acc[dx][jy][c] += v[c];
        }
      }
    }
    tc::fence_before_sync();
    ok = __syncthreads_and(ok);  // the accumulators and this stage are free
    tc::fence_after_sync();
    if (!ok && more && tid == 0) tc::mbar_wait(&bars[(i + 1) & 1], (uint32_t)((i + 1) >> 1) & 1u);  // nothing in flight
  }
  if (ok) {
    // the block's sums in shared memory, an output row at a time: within one, every weight
    // has one writer
    float* s_w = reinterpret_cast<float*>(sm);  // [tap][cout][cin]
    float* s_b = s_w + 27 * 256;                // [warp][channel of the plane]
    for (int k = tid; k < 27 * 256; k += kWgradThreads) s_w[k] = 0.f;
#pragma unroll
    for (int c = 0; c < 2; c++) {
      float v = bsum[c];
#pragma unroll
      for (int o = 16; o >= 4; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < 4) s_b[warp * 8 + 2 * lane + c] = v;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kGY * kGZ; j++) {
      const int dy = yy - j % kGY;
      if (jz == j / kGY && dz >= 0 && dz <= 2 && dy >= 0 && dy <= 2)
#pragma unroll
        for (int dx = 0; dx < 3; dx++)
#pragma unroll
          for (int c = 0; c < 16; c++) s_w[((dx + 3 * dy + 9 * dz) * 16 + c) * 16 + (lane & 15)] += acc[dx][j % kGY][c];
      __syncthreads();
    }
    for (int k = tid; k < 27 * 256; k += kWgradThreads)
      atomicAdd(&dW[(k & ~255) + (k & 15) * 16 + ((k >> 4) & 15)], s_w[k]);
    if (tid < 16) {
      float v = 0.f;
      for (int w = tid >> 3; w < 16; w += 2) v += s_b[w * 8 + (tid & 7)];
      atomicAdd(&db[tid], v);
    }
  }
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc<kWgradCols>(tbase);
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <int EPI>
static cudaError_t launch_conv(const __nv_bfloat16* in_act, const uint8_t* wblob, const float* bias, const ConvDims& D,
                               __nv_bfloat16* out_act, float* out_logits, const __nv_bfloat16* mask_act, int* err,
                               int num_sms, cudaStream_t st) {
  ConvColumns T;
  T.nx = (int)((D.X + kBX - 1) / kBX);
  T.ny = (int)((D.Y + kCY - 1) / kCY);
  T.Z = D.Z;
  T.n = (int64_t)T.nx * T.ny * D.Z;
  cudaError_t e = cudaFuncSetAttribute(conv3_tc_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemConv);
  if (e != cudaSuccess) return e;
  ::msc::count_launch();
  conv3_tc_kernel<EPI><<<(unsigned)(T.n < num_sms ? T.n : num_sms), kConvThreads, kSmemConv, st>>>(
      in_act, wblob, bias, D, T, out_act, out_logits, mask_act, err);
  return cudaGetLastError();
}

cudaError_t launch_conv3_tc(int epi, const __nv_bfloat16* in_act, const uint8_t* wblob, const float* bias,
                            const ConvDims& D, __nv_bfloat16* out_act, float* out_logits,
                            const __nv_bfloat16* mask_act, int* err, int num_sms, cudaStream_t st) {
  // bulk copies in, 16-byte loads of the mask, 16-byte stores out
  if (!aligned16(in_act) || !aligned16(wblob) || !aligned16(out_act) || !aligned16(mask_act))
    return cudaErrorInvalidValue;
  // (262,140 rows: what a grid of four rows a block along y takes)
  if ((D.Y + 3) / 4 > 65535) return cudaErrorInvalidConfiguration;
  if (epi == kEpiReluBf16)
    return launch_conv<kEpiReluBf16>(in_act, wblob, bias, D, out_act, out_logits, mask_act, err, num_sms, st);
  if (epi == kEpiLogits)
    return launch_conv<kEpiLogits>(in_act, wblob, bias, D, out_act, out_logits, mask_act, err, num_sms, st);
  return launch_conv<kEpiMaskBf16>(in_act, wblob, bias, D, out_act, out_logits, mask_act, err, num_sms, st);
}

cudaError_t launch_conv_wgrad(const __nv_bfloat16* X, const __nv_bfloat16* dY, const ConvDims& D, float* dW, float* db,
                              int* err, int num_sms, cudaStream_t st) {
  if (!aligned16(X) || !aligned16(dY)) return cudaErrorInvalidValue;  // bulk copies
  WgradTiles T;
  T.nx = (int)((D.X + kBX - 1) / kBX);
  T.ny = (int)((D.Y + kGY - 1) / kGY);
  T.n = (int64_t)T.nx * T.ny * ((D.Z + kGZ - 1) / kGZ);
  cudaError_t e = cudaFuncSetAttribute(conv_wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemWgrad);
  if (e != cudaSuccess) return e;
  ::msc::count_launch();
  conv_wgrad_tc_kernel<<<(unsigned)(T.n < num_sms ? T.n : num_sms), kWgradThreads, kSmemWgrad, st>>>(X, dY, D, T, dW, db,
                                                                                                     err);
  return cudaGetLastError();
}

}  // namespace msc
