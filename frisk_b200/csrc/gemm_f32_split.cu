// fp32 GEMM on the tensor cores: C <- (clear_accum ? 0 : C) + op(A).op(B) with fp32 accuracy, any size, pitch and
// alignment, in ONE launch.  Contract: `frisk.gemm` with f32 operands (lib/Dialect/Frisk/IR/FriskOps.cpp:406-426).
//
// Every element x of a tile is multiplied by 2^24 and split into three bf16 terms while it travels from global to shared
// memory (x 2^24 = x0 + x1 + x2: 3 x 8 significant bits plus the signs, exact for every x below 2^104; the
// factor keeps the terms of small elements out of the subnormals), and six of the nine term products run as
// tcgen05.mma 128 x 128 x 16: A0B0, A0B1, A1B0, A1B1, A0B2, A2B0.  The three left out are at most 2^-26 |a||b| together,
// a quarter of what ONE fp32 rounding of the product may lose.  Products of bf16 terms are exact in fp32.
//
// Accuracy is decided by the accumulation: tensor memory truncates every addition, a bias of half a unit per MMA along
// a sum (1.0e-6 relative error at K = 1024 when the whole K stayed there).  So one 64-k block is
// summed in tensor memory, small terms first, so that only the four A0B0 steps see a large accumulator, and then
// added to fp32 registers with round-to-nearest: 1.0e-7 at K = 1024, 2.6e-7 on the CUDA cores.  Sums whose terms share a
// sign feel the truncations more: below K = 640 a block is summed in two halves, each in an accumulator of its own
// (TWO; 2.7 % of the time at 1024^3), and below K = 320 the CUDA cores are the more accurate (split_accurate).
//
// An element that is not finite, or so large that x 2^24 or a sum overflows, makes the result non-finite.  The 32 x 16
// piece of C it lies in is noted, and when a CTA's tiles are done (no wait of the pipeline is open any more, however long
// K is) all its warps compute such results as plain fp32 sums over k, so infinities and NaN come out as IEEE arithmetic
// gives them.
//
// One CTA per SM, 16 warps with fixed roles (128 registers each, all of the SM's):
//   warps 0-7   promotion: tensor memory -> fp32 registers (64 columns of one row per thread), stores.  Warp 0 also issues
//               the MMAs of block i, a quarter at a time between the quarters of block i - 1 that it adds up
//   warps 8-15  loaders: global -> registers (one block ahead) -> split -> shared memory, in the 128-byte-swizzle image
//               tcgen05 reads (K-major or MN-major, whichever way the operand lies in global memory), or tensor memory
// What bounds a block is the loaders' chain: a warp makes the terms of A, asks for the next A, does the same for B, waits and fences,
// one after the other, 3100 clk a block wherever the terms go and in whatever order they are made.  It is latency: a scheduler's
// two warps fill 1100 of its 3100 issue slots with ~550 instructions each; the MMAs take 1560 (2000 as issued), shared memory
// 2300, or 1150 with A in tensor memory.  1024^3 takes 21.1 us (22.0 with the MMAs of a block issued in one piece instead of
// quarters; 23.1 with operands from HBM), 2000 x 2000 x 400 35.4 (38.1), 2048^3 126, 4096^3 840 to 930 (448 blocks a CTA, at the
// power limit).  Tried: four stages of 32 k instead of two of 64 (2048^3 154), 16 warps that load, split and add up (1024^3 27.0), a
// warp of its own for the MMAs (96 registers a thread then: spills).
//
// Where the tiles are fewer than half the SMs a cluster of 2 to 8 CTAs shares a tile's K; every CTA leaves its fp32 part
// in its own shared memory and each finishes a share of the tile's 32-row pieces, adding the parts over distributed
// shared memory in rank order (reproducible, no scratch).  Otherwise a CTA walks whole tiles.
#include <cuda_bf16.h>
#include <limits.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "gemm_common.cuh"
#include "ptx.cuh"

namespace fb {
namespace {
using gemm_detail::TileCoord;
using gemm_detail::tile_coord;

constexpr int BT = 128;                       // tile edge
constexpr int BK = 64;                        // k per block
constexpr int kPlane = BT * BK * 2;           // one bf16 plane of an operand: 16 KB
constexpr int kStageBytes = 6 * kPlane;       // three planes of A, three of B
constexpr int kStages = 2;
constexpr int kPromoWarps = 8, kLoadWarps = 8;
constexpr int kThreads = 32 * (kPromoWarps + kLoadWarps);
constexpr int kOutOffset = kStages * kStageBytes;
constexpr int kOutPitch = 20;                 // floats: [32 rows][16 columns] per promotion warp, rows 16-byte aligned
constexpr int kOutWarpBytes = 32 * kOutPitch * 4;
constexpr int kRedoOffset = kOutOffset + kPromoWarps * kOutWarpBytes;
constexpr int kMaxTilesPerCta = 2048;         // a word of noted pieces each; larger products take several launches
constexpr int kBarOffset = kRedoOffset + kMaxTilesPerCta * 4;
constexpr int kSmemTotal = kBarOffset + 256 + 1024;
static_assert(kSmemTotal <= 232448, "stages and output buffers must fit");
static_assert(kStages == 2, "stages and accumulators alternate together");
constexpr float kScale = 16777216.f;          // 2^24, for both operands
constexpr float kUnscale = 1.f / (kScale * kScale);
constexpr float kFloatMax = 3.402823466e38f;

struct Operand {
  const float* p;
  int64_t ld;
  int rows, cols;  // as stored
};

struct SplitArgs {
  Operand a, b;
  float* C;
  int64_t ldc;
  int M, N, K, accumulate, vec_c;
  int tiles_m, tiles_n, kb;  // tiles, 64-k blocks per tile
  int tile0, tile1;          // the tiles of this launch
  int splits;                // CTAs of a cluster, which share a tile's K
  unsigned* status;
};

// (x, y) 2^24 as three pairs of bf16 terms (packed arithmetic: 10 instructions instead of 14)
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&w)[3]) {
  float2 v = mul2_rn(make_float2(x, y), make_float2(kScale, kScale));
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
    w[t] = *reinterpret_cast<const uint32_t*>(&h);
    // exact
    if (t < 2) v = fma2_rn(make_float2(__uint_as_float(w[t] << 16), __uint_as_float(w[t] & 0xffff0000u)), make_float2(-1.f, -1.f), v);
  }
}

// An A whose terms go to tensor memory: 128 rows of a tile are its lanes, two k of a plane a column.  It is contiguous along
// its rows, so a loader warp reads 32 rows of one k at a time and nothing is turned round on the way: warp w has rows
// 32 (w % 4).., the first or the second 32 k of the block.  Any alignment.
struct LaneLoader {
  float r[32];
  const float* base;  // this thread's first element of the block the next fetch() takes
  int k, row;         // its place

  __device__ __forceinline__ void place(const Operand& o, int row0, int k0, int tid) {
    row = row0 + (tid & 127);
    k = k0 + (tid >> 7) * 32;
    base = o.p + (int64_t)k * o.ld + row;
  }
  __device__ __forceinline__ void fetch(const Operand& o, bool inside) {
    if (inside) {
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = __ldg(base + j * o.ld);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = row < o.cols && k + j < o.rows ? __ldg(base + j * o.ld) : 0.f;
    }
    base += BK * o.ld;
    k += BK;
  }
  // the three planes of the block, 32 columns each from `tmem` on (this warp's lanes)
  __device__ __forceinline__ void store(uint32_t tmem, int tid) const {
    const uint32_t at = tmem + (tid >> 7) * 16;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t w[3][8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint32_t x[3];
        split_pair(r[h * 16 + 2 * j], r[h * 16 + 2 * j + 1], x);
#pragma unroll
        for (int t = 0; t < 3; ++t) w[t][j] = x[t];
      }
#pragma unroll
      for (int t = 0; t < 3; ++t) tmem_st_32x32b_x8(at + t * 32 + h * 8, w[t]);
    }
  }
};

// A block of an operand is 128 box rows of 64 elements: rows = MN and columns = k for an operand contiguous along K;
// for one contiguous along MN, 64 rows = k of columns mn0..+63, then 64 rows of columns mn0+64..+127.  A loader thread
// takes 32 elements of it, eight groups of four columns (a warp has two rows of 256 bytes at a time): as 16-byte loads where
// the rows are aligned (VEC), otherwise as four loads of 32 bits (spread over whole rows, one element a lane, the loads
// touch fewer lines each but the halves have to be exchanged and stored in pieces: 1151 x 2047 x 1023 69 us so, 43 this way,
// 37 for the aligned neighbour).
template <bool MN, bool VEC>
struct Loader {
  static constexpr int kSteps = 8;
  static constexpr int kRowStep = 128 / kSteps;  // box rows from one step to the next
  float r[32];
  const float* base;  // this thread's first element of the block the next fetch() takes
  int row, col;       // its place in the operand

  __device__ __forceinline__ static int first_row(int tid) { return tid >> 4; }
  __device__ __forceinline__ static int first_col(int tid) { return (tid & 15) * 4; }
  __device__ __forceinline__ void place(const Operand& o, int mn0, int k0, int tid) {
    row = (MN ? k0 : mn0) + first_row(tid);
    col = (MN ? mn0 : k0) + first_col(tid);
    base = o.p + (int64_t)row * o.ld + col;
  }
  // `inside`: the whole block lies in the operand
  __device__ __forceinline__ void fetch(const Operand& o, bool inside) {
    const int64_t step = kRowStep * o.ld;
#pragma unroll
    for (int v = 0; v < kSteps; ++v) {
      const int rv = MN ? v % (kSteps / 2) : v, cv = MN ? v / (kSteps / 2) * 64 : 0;
      const float* p = base + rv * step + cv;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      const int left = row + rv * kRowStep < o.rows ? o.cols - (col + cv) : 0;  // columns of the row from here on
      if (VEC && (inside || left > 3)) {
        x = __ldg(reinterpret_cast<const float4*>(p));
      } else {
        if (inside || left > 0) x.x = __ldg(p);
        if (inside || left > 1) x.y = __ldg(p + 1);
        if (inside || left > 2) x.z = __ldg(p + 2);
        if (inside || left > 3) x.w = __ldg(p + 3);
      }
      r[4 * v] = x.x; r[4 * v + 1] = x.y; r[4 * v + 2] = x.z; r[4 * v + 3] = x.w;
    }
    base += MN ? BK * o.ld : (int64_t)BK;
    if (MN) row += BK; else col += BK;
  }
  // the three planes of the block in the 128-byte-swizzle image: box row br at br * 128 bytes, 16-byte piece c at c ^ (br % 8)
  __device__ __forceinline__ void store(unsigned char* s, int tid) const {
    const int br = first_row(tid), c4 = tid & 15;  // (steps of 16 rows leave br % 8 as it is)
    unsigned char* d = s + br * 128 + ((((c4 >> 1) ^ (br & 7)) << 4) | ((c4 & 1) << 3));
#pragma unroll
    for (int v = 0; v < kSteps; ++v) {
      uint32_t lo[3], hi[3];
      split_pair(r[4 * v], r[4 * v + 1], lo);
      split_pair(r[4 * v + 2], r[4 * v + 3], hi);
#pragma unroll
      for (int t = 0; t < 3; ++t) *reinterpret_cast<uint2*>(d + v * (kRowStep * 128) + t * kPlane) = make_uint2(lo[t], hi[t]);
    }
  }
};

// The 32 x 16 piece of C at (r0, c0), lane = row: unscaled, added to C or written.  Four lanes write 64 consecutive
// bytes of a row, through `out` ([32 rows][16 columns] of shared memory).  Returns false where a result is not finite: the
// piece then stands in C as it is, or has not been added to C.
__device__ __forceinline__ bool store_piece(const SplitArgs& p, float (&v)[16], float* out, int r0, int c0, int lane) {
  if (r0 >= p.M || c0 >= p.N) return true;
  bool finite = true;
#pragma unroll
  for (int i = 0; i < 16; ++i) finite = finite && fabsf(v[i]) <= kFloatMax;
  const bool whole = !__any_sync(0xffffffffu, !finite && r0 + lane < p.M);
  if (!whole && p.accumulate) return false;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(out + lane * kOutPitch + 4 * i) =
        make_float4(v[4 * i] * kUnscale, v[4 * i + 1] * kUnscale, v[4 * i + 2] * kUnscale, v[4 * i + 3] * kUnscale);
  __syncwarp();
  if (p.vec_c) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rl = j * 8 + (lane >> 2), row = r0 + rl, col = c0 + (lane & 3) * 4;
      if (row >= p.M || col >= p.N) continue;
      float4 x = *reinterpret_cast<const float4*>(out + rl * kOutPitch + (lane & 3) * 4);
      float* dst = p.C + (int64_t)row * p.ldc + col;
      if (col + 3 < p.N) {
        if (p.accumulate) {
          const float4 old = *reinterpret_cast<const float4*>(dst);
          x.x += old.x; x.y += old.y; x.z += old.z; x.w += old.w;
        }
        *reinterpret_cast<float4*>(dst) = x;
      } else {
        const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int e = 0; e < 3; ++e)
          if (col + e < p.N) dst[e] = p.accumulate ? dst[e] + xs[e] : xs[e];
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int rl = j * 2 + (lane >> 4), row = r0 + rl, col = c0 + (lane & 15);
      if (row >= p.M || col >= p.N) continue;
      const float x = out[rl * kOutPitch + (lane & 15)];
      float* dst = p.C + (int64_t)row * p.ldc + col;
      *dst = p.accumulate ? *dst + x : x;
    }
  }
  __syncwarp();
  return whole;
}

// The non-finite results (where C is added to: all) of the noted pieces of this CTA's tiles, bit 16 h + w of a tile's word:
// columns 64h + 16 (w / 4), rows 32 (w % 4).  Plain fp32 sums by all 16 warps, half a tile at a time, a lane with 4 x 4
// results of a piece; where few pieces are noted, two or four warps share a block's k and their sums are added in order.
// 4096^3 takes 0.83 ms, with one infinite element 1.5 and with every result above 2^80 8.4 (53 and 451 when the thread that
// met such a result summed it up on the spot); 1024^3 21 us, 167 and 232.
template <bool A_MN, bool B_MN>
__device__ __noinline__ void redo_pieces(const SplitArgs& p, unsigned char* smem, const uint32_t* noted, int first, int step,
                                         int count) {
  constexpr int kPitchA = BT + 4, kPitchB = BT / 2 + 4;  // 4 banks from one k to the next
  float* sa = reinterpret_cast<float*>(smem);            // [64 k][128 rows]
  float* sb = sa + BK * kPitchA;                         // [64 k][64 columns]
  float* sums = sb + BK * kPitchB;                       // [16 warps][16 results][32 lanes]
  static_assert((BK * (kPitchA + kPitchB) + 16 * 512) * 4 <= kOutOffset, "a block and the sums must fit in the stages");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = 0; t < 2 * count; ++t) {
    const uint32_t mask = (noted[t >> 1] >> (16 * (t & 1))) & 0xffffu;
    if (mask == 0) continue;  // (the same for every thread)
    const TileCoord tc = tile_coord(first + (t >> 1) * step, p.tiles_m, p.tiles_n);
    const int m0 = tc.m * BT, n0 = tc.n * BT + (t & 1) * (BT / 2);
    // A thread's elements of a block: where k is contiguous, 8 k of 4 rows a warp (32-byte sectors, all banks); otherwise rows
    auto row_of = [&](bool mn, int rows, int j) { return mn ? (int)threadIdx.x % rows : (lane >> 3) + 4 * warp + 64 * (j >> 3); };
    auto k_of = [&](bool mn, int rows, int j) {
      return mn ? (int)threadIdx.x / rows + j * (kThreads / rows) : (lane & 7) + 8 * (j & 7);
    };
    auto element = [&](const Operand& o, bool mn, int r, int k, int rows) {
      return r < rows && k < p.K ? __ldg(o.p + (mn ? (int64_t)k * o.ld + r : (int64_t)r * o.ld + k)) : 0.f;
    };
    float pa[16], pb[8];
    auto fetch = [&](int k0) {
#pragma unroll
      for (int j = 0; j < 16; ++j) pa[j] = element(p.a, A_MN, m0 + row_of(A_MN, BT, j), k0 + k_of(A_MN, BT, j), p.M);
#pragma unroll
      for (int j = 0; j < 8; ++j) pb[j] = element(p.b, B_MN, n0 + row_of(B_MN, BT / 2, j), k0 + k_of(B_MN, BT / 2, j), p.N);
    };
    const int pieces = __popc(mask), sharers = pieces <= 4 ? 4 : pieces <= 8 ? 2 : 1;  // warps of a piece
    const int slot = warp / sharers, part = warp % sharers;
    const int piece = slot < pieces ? (int)__fns(mask, 0, slot + 1) : -1;  // the slot-th noted piece
    const int row = (piece & 3) * 32 + (lane & 7) * 4, col = (piece >> 2) * 16 + (lane >> 3) * 4;
    const int k_first = part * (BK / sharers), k_last = k_first + BK / sharers;
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    fetch(0);
    for (int kb = 0; kb < p.kb; ++kb) {
      __syncthreads();  // the block before this one has been read
#pragma unroll
      for (int j = 0; j < 16; ++j) sa[k_of(A_MN, BT, j) * kPitchA + row_of(A_MN, BT, j)] = pa[j];
#pragma unroll
      for (int j = 0; j < 8; ++j) sb[k_of(B_MN, BT / 2, j) * kPitchB + row_of(B_MN, BT / 2, j)] = pb[j];
      __syncthreads();
      if (kb + 1 < p.kb) fetch((kb + 1) * BK);
      if (piece >= 0) {
#pragma unroll 4
        for (int k = k_first; k < k_last; ++k) {
          const float4 a4 = *reinterpret_cast<const float4*>(sa + k * kPitchA + row);
          const float4 b4 = *reinterpret_cast<const float4*>(sb + k * kPitchB + col);
          const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[i] = fmaf(a[i >> 2], b[i & 3], acc[i]);
        }
      }
    }
    if (sharers > 1) {
#pragma unroll
      for (int i = 0; i < 16; ++i) sums[(warp * 16 + i) * 32 + lane] = acc[i];
      __syncthreads();
      for (int q = 1; q < sharers; ++q)
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (part == 0) acc[i] += sums[((warp + q) * 16 + i) * 32 + lane];
    }
    if (piece >= 0 && part == 0)
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int r = m0 + row + (i >> 2), c = n0 + col + (i & 3);
        if (r >= p.M || c >= p.N) continue;
        float* dst = p.C + (int64_t)r * p.ldc + c;
        if (p.accumulate)
          *dst += acc[i];
        else if (!(fabsf(*dst) <= kFloatMax))
          *dst = acc[i];
      }
    __syncthreads();
  }
}

// TWO: a block's 32-k halves are summed in accumulators of their own
template <bool A_MN, bool B_MN, bool VEC, bool TWO>
__global__ void __launch_bounds__(kThreads, 1) gemm_f32_split_kernel(const __grid_constant__ SplitArgs p) {
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kBarOffset);
  uint64_t* done_bar = full_bar + kStages;   // [2] a block's MMAs are complete: its stage is free, its accumulator full
  uint64_t* acc_empty = done_bar + kStages;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* any_noted = tmem_slot + 2;
  uint32_t* noted = reinterpret_cast<uint32_t*>(smem + kRedoOffset);  // pieces of each of this CTA's tiles to compute again
  constexpr int kHalves = TWO ? 2 : 1, kAccCols = kHalves * BT;  // of an accumulator
  // The terms of an A that is stored transposed go to tensor memory, behind the two accumulators, where there is room (two
  // stages of three planes): their MMAs then read only B from shared memory: 3 % at 1024^3 with both operands transposed,
  // 515 x 771 x 1003 21.6 -> 20.0 us, 128 x 1500 x 700 15.4 -> 14.9.  (Any operand contiguous along its rows would do, with the
  // product turned round for B; for an A contiguous along K that was 1 % slower at 1024^3.)
  constexpr bool LANES = A_MN && !TWO;
  constexpr uint32_t kPlanesAt = 2 * BT, kPlanesCols = 3 * BK / 2, kTmemCols = LANES ? 512 : 2 * kAccCols;
  static_assert(kPlanesAt + 2 * kPlanesCols <= 512, "accumulators and planes must fit");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = p.splits, rank = splits > 1 ? (int)cluster_ctarank() : 0;
  // this CTA's tiles (one, if K is shared) and its blocks of each
  const int tile_first = p.tile0 + (int)blockIdx.x / splits, tile_step = splits > 1 ? INT_MAX / 2 : (int)gridDim.x;
  const int tiles = p.tile1;
  const int n_mine = tile_first < tiles ? (tiles - 1 - tile_first) / tile_step + 1 : 0;
  const int kb0 = (int)((int64_t)p.kb * rank / splits), kb1 = (int)((int64_t)p.kb * (rank + 1) / splits);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full_bar[i], kLoadWarps);
      mbar_init(&done_bar[i], 1);
      mbar_init(&acc_empty[i], kPromoWarps);
    }
    *abort_flag = 0;
    *any_noted = 0;
    mbar_fence_init();
  }
  for (int i = threadIdx.x; i < n_mine; i += kThreads) noted[i] = 0;
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // Launched with programmatic stream serialization: the set-up above may overlap the kernel before this one.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp < kPromoWarps) {
    // ------------------------------------------------------------------ promotion and epilogue
    const int quad = warp & 3, half = warp >> 2;  // tensor-memory lanes 32*quad.., columns 64*half..
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    float* out = reinterpret_cast<float*>(smem + kOutOffset + warp * kOutWarpBytes);
    int blocks = 0, issued = 0;  // blocks added up, blocks handed to the tensor core (by warp 0), over all tiles
    const int64_t total = (int64_t)n_mine * (kb1 - kb0);
    bool ok = true;
    auto note = [&](int tile, int piece) {
      if (lane == 0) {
        atomicOr(&noted[(tile - tile_first) / tile_step], 1u << piece);
        *any_noted = 1;
      }
    };
    // The MMAs of the next block, by warp 0: stage and accumulator alternate with the block's number.  The tensor core queues
    // only a few of them, so the warp is busy for as long as they run, and what else it did in one piece left the tensor core
    // idle.  So it issues a quarter of a block, adds up a quarter of the one before, which the queue covers, and so on.
    constexpr uint32_t idesc = umma_idesc_f16(BT, BT, true, A_MN && !LANES, B_MN);
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    constexpr int kParts = 4, kPartMmas = 6 * (BK / 16) / kParts;
    auto may_issue = [&]() -> bool {
      const int i = issued & 1;
      const uint32_t phase = (issued >> 1) & 1;
      const bool there = __all_sync(0xffffffffu, mbar_wait_both(&full_bar[i], phase, &acc_empty[i], phase ^ 1, abort_flag, p.status,
                                                                ST_TIMEOUT_FULL, ST_TIMEOUT_ACC_EMPTY));
      tc_fence_after_sync();
      return there;
    };
    auto issue_part = [&](int part) {
      // term products, smallest first; (term of A, term of B)
      constexpr int ta[6] = {2, 0, 1, 1, 0, 0}, tb[6] = {0, 2, 1, 0, 1, 0};
      const int i = issued & 1;
      const uint32_t sa = smem_u32(smem + i * kStageBytes), sb = sa + 3 * kPlane;
      // descriptors differ only in the start address
      const uint64_t da = A_MN ? umma_desc_mnmajor_sw128(sa, BK * 128, 1024) : umma_desc_kmajor_sw128(sa);
      const uint64_t db = B_MN ? umma_desc_mnmajor_sw128(sb, BK * 128, 1024) : umma_desc_kmajor_sw128(sb);
      if (elect_one()) {
#pragma unroll
        for (int m = part * kPartMmas; m < (part + 1) * kPartMmas; ++m) {
          const int t = m / (BK / 16), k = m % (BK / 16);
          const uint32_t acc = tmem + i * kAccCols + (TWO && k >= 2 ? BT : 0), add = (t | (TWO ? k & 1 : k)) != 0 ? 1u : 0u;
          const uint64_t b = db + ((tb[t] * kPlane + k * (B_MN ? 16 * 128 : 32)) >> 4);
          if (LANES)
            umma_f16_ts(acc, tmem + kPlanesAt + i * kPlanesCols + ta[t] * (BK / 2) + k * 8, b, idesc, add);
          else
            umma_f16_ss(acc, da + ((ta[t] * kPlane + k * (A_MN ? 16 * 128 : 32)) >> 4), b, idesc, add);
        }
        if (part == kParts - 1) umma_commit(&done_bar[i]);
      }
      __syncwarp();
    };
    if (warp == 0 && total > 0 && may_issue()) {
#pragma unroll
      for (int part = 0; part < kParts; ++part) issue_part(part);
      ++issued;
    }
    for (int tile = tile_first; tile < tiles && ok; tile += tile_step) {
      float v[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) v[i] = 0.f;
      for (int kb = kb0; kb < kb1; ++kb) {
        const bool issues = warp == 0 && issued < total && may_issue();
        const int acc = blocks & 1;
#pragma unroll
        for (int part = 0; part < kParts; ++part) {
          if (issues) issue_part(part);
          if (part == 0) {
            ok = mbar_wait_warp(&done_bar[acc], (blocks >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_ACC_FULL);
            if (!ok) break;
            tc_fence_after_sync();
          }
          uint32_t t[kHalves][16];
#pragma unroll
          for (int h = 0; h < kHalves; ++h)
            tmem_ld_32x32b_x16(tmem_base + acc * kAccCols + h * BT + half * 64 + part * 16 + lane_addr, t[h]);
          tmem_ld_wait();
          if (part == kParts - 1) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
          }
#pragma unroll
          for (int h = 0; h < kHalves; ++h)
#pragma unroll
            for (int i = 0; i < 16; ++i) v[part * 16 + i] += __uint_as_float(t[h][i]);
        }
        if (issues) ++issued;
        if (!ok) break;
        ++blocks;
      }
      if (!ok) break;
      if (splits > 1) {
        // the part goes into this CTA's shared memory, [32 groups of 4 columns][128 rows] float4.  The ring is free: the last
        // accumulator is complete, so every MMA has read its stage, and no block follows.
        float4* part = reinterpret_cast<float4*>(smem) + quad * 32 + lane;
#pragma unroll
        for (int i = 0; i < 16; ++i)
          part[(half * 16 + i) * BT] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      } else {
        const TileCoord tc = tile_coord(tile, p.tiles_m, p.tiles_n);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float x[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = v[u * 16 + i];
          if (!store_piece(p, x, out, tc.m * BT + quad * 32, tc.n * BT + half * 64 + u * 16, lane))
            note(tile, half * 16 + u * 4 + quad);
        }
      }
    }
    if (splits > 1) {
      // every role of every CTA of the cluster ends (its waits are bounded), so this meeting is reached
      __syncwarp();
      cluster_sync_all();
      const TileCoord tc = tile_coord(tile_first, p.tiles_m, p.tiles_n);
      // the tile's 32 pieces (32 rows x 16 columns) over the cluster's promotion warps
      for (int x = rank * kPromoWarps + warp; x < 32; x += kPromoWarps * splits) {
        const int g = x & 3, u = x >> 2;
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.f;
        const uint32_t at = smem_u32(smem) + ((u * 4) * BT + g * 32 + lane) * 16;
        for (int c = 0; c < splits; ++c) {
          const uint32_t peer = mapa_addr(at, c);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 t = ld_cluster_f4(peer + i * (BT * 16));
            v[4 * i] += t.x; v[4 * i + 1] += t.y; v[4 * i + 2] += t.z; v[4 * i + 3] += t.w;
          }
        }
        if (!store_piece(p, v, out, tc.m * BT + g * 32, tc.n * BT + u * 16, lane)) note(tile_first, x);
      }
      __syncwarp();
      cluster_sync_all();  // the peers have read this CTA's part
    }
  } else {
    // ------------------------------------------------------------------ loaders
    const int tid = threadIdx.x - kPromoWarps * 32;
    std::conditional_t<LANES, LaneLoader, Loader<A_MN, VEC>> la;
    const uint32_t planes = tmem_base + kPlanesAt + (static_cast<uint32_t>((warp & 3) * 32) << 16);  // (LANES)
    Loader<B_MN, VEC> lb;
    int tile = tile_first, kb = kb0, stage = 0;
    uint32_t phase = 0;
    bool a_in = false, b_in = false;  // the tile's rows of A, columns of B lie inside the operands
    auto place = [&]() {
      const TileCoord tc = tile_coord(tile, p.tiles_m, p.tiles_n);
      la.place(p.a, tc.m * BT, kb0 * BK, tid);
      lb.place(p.b, tc.n * BT, kb0 * BK, tid);
      a_in = (tc.m + 1) * BT <= p.M;
      b_in = (tc.n + 1) * BT <= p.N;
    };
    bool more = tile < tiles;
    if (more) {
      place();
      const bool k_in = (unsigned)(kb + 1) * BK <= (unsigned)p.K;
      la.fetch(p.a, a_in && k_in);
      lb.fetch(p.b, b_in && k_in);
    }
    while (more) {
      if (++kb == kb1) {  // the block after the one in registers
        kb = kb0;
        tile += tile_step;
        more = tile < tiles;
        if (more) place();
      }
      if (!mbar_wait_warp(&done_bar[stage], phase ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
      __syncwarp();
      unsigned char* sa = smem + stage * kStageBytes;
      const bool k_in = (unsigned)(kb + 1) * BK <= (unsigned)p.K;
      if constexpr (LANES) {
        tc_fence_after_sync();
        la.store(planes + stage * kPlanesCols, tid);
      } else {
        la.store(sa, tid);
      }
      if (more) la.fetch(p.a, a_in && k_in);
      lb.store(sa + 3 * kPlane, tid);
      if (more) lb.fetch(p.b, b_in && k_in);
      fence_proxy_async_smem();  // the planes are read by the tensor core
      if (LANES) {
        __syncwarp();  // (at an edge of B every lane loads as far as it goes)
        tmem_st_wait();
        tc_fence_before_sync();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[stage]);
      if (++stage == kStages) {
        stage = 0;
        phase ^= 1;
      }
    }
    if (splits > 1) {
      __syncwarp();
      cluster_sync_all();
      cluster_sync_all();
    }
  }

  // ------------------------------------------------------------------ results the split cannot carry
  __syncthreads();  // every role is done, and the peers of a cluster with this CTA's shared memory
  if (*any_noted && !*abort_flag) redo_pieces<A_MN, B_MN>(p, smem, noted, tile_first, tile_step, n_mine);

  // ------------------------------------------------------------------ teardown
  if (*abort_flag) {
    unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// How many CTAs of a cluster share a tile's K: as many as leave every CTA an SM and two blocks of its own (adding the
// parts up takes about as long as one: 512 x 512 x 512 in 11.6 us with 2 blocks each on 4 CTAs a tile), and of those the
// fewest that give the same number of blocks.  `fits(n)`: the device runs a cluster of n for every tile at a time.
template <typename F>
int split_of(int64_t tiles, int64_t kb, int sms, F&& fits) {
  int best = 1;
  for (int n = 2; n <= kMaxCluster && tiles * n <= sms && kb >= 2 * n; ++n)
    if ((kb + n - 1) / n < (kb + best - 1) / best && fits(n)) best = n;
  return best;
}

constexpr int kTwoBelowK = 640;
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <bool A_MN, bool B_MN, bool VEC, bool TWO>
int launch_one(frisk_b200_ctx* ctx, SplitArgs a, cudaStream_t s) {
  auto kern = gemm_f32_split_kernel<A_MN, B_MN, VEC, TWO>;
  static PerDeviceOnce opt_in;
  if (opt_in(ctx->device, [&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemTotal) == cudaSuccess ? 0 : 1;
      }))
    return FRISK_B200_E_CUDA;
  static ClusterCapacity capacity;
  const int sms = std::min(ctx->num_sms, kNumSMsDefault), tiles = a.tiles_m * a.tiles_n;
  a.splits = split_of(tiles, a.kb, sms, [&](int n) { return capacity(ctx->device, kern, kThreads, kSmemTotal, n) >= tiles; });
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemTotal;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // the kernel waits (griddepcontrol.wait) itself
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)a.splits;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.splits > 1 ? 2 : 1;
  for (a.tile0 = 0; a.tile0 < tiles; a.tile0 = a.tile1) {
    a.tile1 = (int)std::min<int64_t>(tiles, (int64_t)a.tile0 + (int64_t)sms * kMaxTilesPerCta);
    const int n = a.tile1 - a.tile0;
    cfg.gridDim = dim3((unsigned)(a.splits > 1 ? n * a.splits : std::min(n, sms)));
    FB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, a));
  }
  return 0;
}

template <bool A_MN, bool B_MN>
int launch_vec(frisk_b200_ctx* ctx, const SplitArgs& a, bool vec, cudaStream_t s) {
  if (a.K < kTwoBelowK)
    return vec ? launch_one<A_MN, B_MN, true, true>(ctx, a, s) : launch_one<A_MN, B_MN, false, true>(ctx, a, s);
  return vec ? launch_one<A_MN, B_MN, true, false>(ctx, a, s) : launch_one<A_MN, B_MN, false, false>(ctx, a, s);
}

}  // namespace

// what `algo = FRISK_B200_ALGO_F32_SPLIT` accepts
bool f32_split_supported(const frisk_b200_gemm_desc& d) {
  if (d.dtype_ab != FRISK_B200_F32 || d.dtype_c != FRISK_B200_F32) return false;
  if (d.M % 8 || d.N % 8 || d.K % 8) return false;
  return 3 * d.M <= INT32_MAX && 3 * d.N <= INT32_MAX && d.K <= INT32_MAX;
}

bool f32_split_preferred(const frisk_b200_gemm_desc& d) {
  return f32_split_supported(d) && d.M >= 256 && d.N >= 256 && d.K >= 256;
}

// Where the error is no larger than that of the CUDA cores' fp32 sums, whatever the signs.  Relative to theirs it is, for
// terms of either sign / of one sign / of sizes e^3 apart: 0.9 / 1.7 / 1.4 at K = 64, 0.8 / 1.5 / 1.2 at 128 with one
// accumulator a block; 0.54 / 1.06 / 0.7 at 256, 0.52 / 0.96 / 0.65 at 320, 0.45 / 0.87 / 0.57 at 512 with two; 0.45 / 0.98 /
// 0.7 at 640, 0.38 / 0.86 / 0.6 at 1024 with one (1024 x 1024 x K, 2-norm; CUDA cores 8e-8 at 64, 2.6e-7 at 1024).
bool split_accurate(const frisk_b200_gemm_desc& d) { return d.K >= 320 || f32_split_preferred(d); }

// Both kernels estimated in microseconds from measurements.  CUDA cores: 4.3 for 64 x 64 x 64 and about 2.0 more for
// every further 64 x 64 x 64 unit an SM takes, 2 to add up the parts of a shared tile (512^3 13.5, 1024^3 57, 2048^3 401).
// Tensor cores: 5.5 and 2.1 for every 128 x 128 x 64 block a CTA takes, 2 more to add up the parts of a shared tile; 2.4 per block
// where rows are not 16-byte aligned.  That was fitted when a block's MMAs were issued in one piece and is 5 to 15 % too much today (512^3
// 11.1, 1024^3 21.1, 2048^3 126, 1151 x 2047 x 1023 43), more for a transposed A off 16 bytes from K = 640 on, whose lane-wise loads do
// not care: where the two are close the CUDA cores are taken a little too often.
bool f32_split_beats_simt(const frisk_b200_gemm_desc& d) {
  if (d.dtype_ab != FRISK_B200_F32 || d.dtype_c != FRISK_B200_F32 || !split_accurate(d)) return false;
  if (d.M > INT32_MAX / 4 || d.N > INT32_MAX / 4 || d.K > INT32_MAX / 4) return false;
  const GemmDims g = resolve_dims(d);
  const double sms = kNumSMsDefault;
  const int64_t kb = (g.K + BK - 1) / BK, tiles = ((g.M + BT - 1) / BT) * ((g.N + BT - 1) / BT);
  if (tiles > (int64_t)1 << 30) return false;
  const double units = std::ceil((double)(((g.M + 63) / 64) * ((g.N + 63) / 64)) * (double)kb / sms);
  const double simt = 4.3 + 2.0 * (units - 1) + (units < (double)kb ? 2.0 : 0.0);
  const int splits = split_of(tiles, kb, kNumSMsDefault, [](int) { return true; });
  const double blocks = std::ceil((double)tiles / sms) * std::ceil((double)kb / splits);
  const double block = g.lda % 4 || g.ldb % 4 ? 2.4 : 2.1;
  return 5.5 + block * blocks + (splits > 1 ? 2.0 : 0.0) < simt;
}

int launch_gemm_f32_split(frisk_b200_ctx* ctx, const frisk_b200_gemm_desc& d, const float* A, const float* B,
                          float* C, cudaStream_t s) {
  const GemmDims g = resolve_dims(d);
  SplitArgs a;
  a.a = Operand{A, g.lda, (int)(d.trans_a ? g.K : g.M), (int)(d.trans_a ? g.M : g.K)};
  a.b = Operand{B, g.ldb, (int)(d.trans_b ? g.N : g.K), (int)(d.trans_b ? g.K : g.N)};
  const bool vec = aligned16(A) && g.lda % 4 == 0 && aligned16(B) && g.ldb % 4 == 0;
  a.C = C;
  a.ldc = g.ldc;
  a.M = (int)g.M; a.N = (int)g.N; a.K = (int)g.K;
  a.accumulate = d.clear_accum ? 0 : 1;
  a.vec_c = aligned16(C) && g.ldc % 4 == 0;
  const int64_t tiles_m = (g.M + BT - 1) / BT, tiles_n = (g.N + BT - 1) / BT;
  if (tiles_m * tiles_n > (int64_t)1 << 30) return FRISK_B200_E_UNSUPPORTED;
  a.tiles_m = (int)tiles_m;
  a.tiles_n = (int)tiles_n;
  a.kb = (int)((g.K + BK - 1) / BK);
  a.status = ctx->d_status;
  const bool a_mn = d.trans_a != 0, b_mn = d.trans_b == 0;
  if (a_mn) return b_mn ? launch_vec<true, true>(ctx, a, vec, s) : launch_vec<true, false>(ctx, a, vec, s);
  return b_mn ? launch_vec<false, true>(ctx, a, vec, s) : launch_vec<false, false>(ctx, a, vec, s);
}

}  // namespace fb
