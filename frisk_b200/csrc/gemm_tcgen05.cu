// fp16 / bf16 GEMM on the 5th-generation tensor cores (tcgen05), fp32 accumulation in
// tensor memory.  Contract: `frisk.gemm` with f16/bf16 operands and a C of the same type or
// f32 (lib/Dialect/Frisk/IR/FriskOps.cpp:406-426,
// lib/Dialect/Frisk/IR/LegacyImportSemantics.cpp:26-44).
//
// One persistent CTA per SM, 6 warps with fixed roles:
//   warp 0    TMA producer: A and B tiles -> shared-memory ring of 192 KB (full/empty mbarriers)
//   warp 1    MMA issuer:   one thread issues tcgen05.mma (128 x BN x 16) per k16 slice,
//                           tcgen05.commit releases the stage / publishes the accumulator
//   warps 2-5 epilogue:     tcgen05.ld of the finished accumulator, conversion, stores
// Two accumulators (2 x BN TMEM columns) let the epilogue of tile i overlap the main loop of
// tile i+1.  Output tiles are 128 x 256 (12 KB of operands per 128 clk of MMA) or, where those are too few, 128 x 128
// (8 KB per 64 clk, all that shared memory delivers) or 128 x 64.
//
// Whole rounds of tiles are dealt out tile by tile.  The tiles of a partial last round (all of them, where there are
// fewer tiles than SMs) are shared by clusters of 2, 4 or 8 CTAs, each multiplying its part of K: every CTA leaves its fp32
// accumulator in its own shared memory (the operand ring has done its work by then), and the parts are added up over
// distributed shared memory, in rank order, for the CTAs that finish the tile's boxes of C (reproducible, no scratch, no
// CTA waits for one outside its cluster).
//
// Every form of C leaves through a shared-memory box of 32 rows x 128 bytes per epilogue warp: an aligned C by TMA
// stores (and its old values, where they are added, come in by TMA loads), any other C by whole-row accesses of the warp.
// `frisk.fill` before and a row reduction after the gemm are folded in: the fill value is added in registers, every
// (row, box of columns) leaves one fp32 partial of the reduction, and the CTA that finishes a row block's last column
// tile combines them in column order.
//
// Shared-memory operand images are the canonical 128-byte-swizzle layouts (rows of 64
// 16-bit elements, 1024-byte aligned stages): K-major for an operand that is contiguous
// along K in global memory, MN-major otherwise.  These are the images Frisk's layout
// inference proposes for 16-bit MMA operands
// (lib/Dialect/Frisk/Target/SM90/SM90GemmConstraints.cpp:121-138); TMA writes them directly.
// No TMA load uses cluster multicast.
#include <limits.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"

#include "gemm_common.cuh"
#include "ptx.cuh"
#include "work_split.cuh"

namespace fb {
namespace {
using namespace gemm_detail;

constexpr int BM = 128;
constexpr int BK = 64;       // one 128-byte swizzle span of 16-bit elements
constexpr int UMMA_K = 16;
constexpr int kThreads = 192;
constexpr int kBoxBytes = 32 * 128;

template <int BN>
struct SmemLayout {
  static constexpr int kABytes = BM * BK * 2;
  static constexpr int kBBytes = BN * BK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = 196608 / kStageBytes;  // 4 at BN = 256, 6 at BN = 128, 8 at BN = 64
  static constexpr int kBoxRowsB = BN < 128 ? BN : 128;  // rows of B that one TMA instruction brings
  static constexpr int kBarOffset = kStages * kStageBytes;
  // two [32 rows][128 bytes] boxes of C per epilogue warp, 1024-byte aligned
  static constexpr int kOutOffset = kBarOffset + 1024;
  static constexpr int kTotal = kOutOffset + 4 * 2 * kBoxBytes + 1024;
  static_assert(kTotal <= 232448, "the boxes of C must fit next to the operand ring");
  // a shared tile: this CTA's part [BN/4][128 rows] float4, then the sums of the columns it finishes (at most half, but at
  // BN = 64 and 16 bits, a single box wide, all)
  static constexpr int kSumOffset = BM * BN * 4;
  static_assert(kSumOffset + BM * (BN == 64 ? BN : BN / 2) * 4 <= kBarOffset, "the parts and sums of a shared tile must fit in the ring");
};

struct GemmArgs {
  void* C;
  int64_t ldc;
  int M, N, K;
  int accumulate;  // the old C is added
  int tma_c;       // C goes through the TMA unit
  int n_whole;     // tiles [0, n_whole) are walked whole, one by one
  int splits;      // CTAs of a cluster, which share the K of one of the other tiles
  RowEpilogue epi;
  unsigned* status;
};

// A 32-row box (128 bytes a row, a 32-bit word a lane) of a C that the TMA unit cannot address: its rows begin on a multiple
// of the element's size and no more.  16-bit elements go in pairs wherever they lie on 4 bytes: of a row that begins
// there lane l has elements 2l and 2l + 1, of an odd row 2l + 1 and 2l + 2, and its first and last element go by themselves.
// Which rows are odd is one of four patterns, the same for the whole box: an epilogue warp has its scheduler to itself, so its
// time is the number of instructions, and rows that decide for themselves took 1200 of them a box (1.9 us).  With 2-byte accesses
// 4000 x 4092 x 512 took 51.7 us, 33.3 so, 22.9 with 4096 columns by TMA; 4095 columns 51.7 and 39.8.  The old values used to be
// loaded one after the other, each behind the shared-memory store of the one before: two panels of 6543 x 4546 x 2296
// 872 us, 359 so; fp32 3000 x 2055 x 1032 186 and 73.
struct BoxRows {
  bool first_odd, second_odd;
  template <typename TO>
  __device__ __forceinline__ BoxRows(const TO* row, int64_t pitch)
      : first_odd(sizeof(TO) == 2 && (reinterpret_cast<uintptr_t>(row) & 2u)),
        second_odd(sizeof(TO) == 2 && (reinterpret_cast<uintptr_t>(row + pitch) & 2u)) {}
  // f(first row odd, second row odd), the answers as types
  template <typename F>
  __device__ __forceinline__ void pattern(F&& f) const {
    if (first_odd) {
      if (second_odd) f(std::true_type(), std::true_type()); else f(std::true_type(), std::false_type());
    } else {
      if (second_odd) f(std::false_type(), std::true_type()); else f(std::false_type(), std::false_type());
    }
  }
};
// the old values of a box, cols x rows of which lie in C (all loads on their way before the first is used), into its image:
// put(r, word of row r)
template <typename TO, typename Put>
__device__ __forceinline__ void load_box_rows(const TO* row, int64_t pitch, int rows, int cols, int lane, Put&& put) {
  uint32_t w[32];
  if (sizeof(TO) == 4) {
#pragma unroll
    for (int r = 0; r < 32; ++r) w[r] = r < rows && lane < cols ? *reinterpret_cast<const uint32_t*>(row + r * pitch + lane) : 0u;
#pragma unroll
    for (int r = 0; r < 32; ++r) put(r, w[r]);
    return;
  }
  const unsigned short* p = reinterpret_cast<const unsigned short*>(row);
  // lane r: the first element of row r
  const uint32_t firsts = lane < rows ? p[lane * pitch] : 0u;
  BoxRows(row, pitch).pattern([&](auto odd0, auto odd1) {
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      const bool odd = r % 2 ? decltype(odd1)::value : decltype(odd0)::value;
      const int j = 2 * lane + (odd ? 1 : 0);
      w[r] = 0u;
      if (r < rows && j + 1 < cols) w[r] = *reinterpret_cast<const uint32_t*>(p + r * pitch + j);
      if (r < rows && j + 1 == cols) w[r] = p[r * pitch + j];
    }
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      const bool odd = r % 2 ? decltype(odd1)::value : decltype(odd0)::value;
      if (odd) {
        const uint32_t before = __shfl_up_sync(0xffffffffu, w[r], 1), first = __shfl_sync(0xffffffffu, firsts, r);
        w[r] = (lane == 0 ? first : before >> 16) | (w[r] << 16);
      }
      put(r, w[r]);
    }
  });
}
// a box back to C: get(r) gives this lane's word of row r
template <typename TO, typename Get>
__device__ __forceinline__ void store_box_rows(TO* row, int64_t pitch, int rows, int cols, int lane, Get&& get) {
  constexpr int kStep = 8;
  if (sizeof(TO) == 4) {
#pragma unroll 1
    for (int r = 0; r < rows; r += kStep, row += kStep * pitch) {
      uint32_t w[kStep];
#pragma unroll
      for (int i = 0; i < kStep; ++i) w[i] = get(r + i);
#pragma unroll
      for (int i = 0; i < kStep; ++i)
        if (r + i < rows && lane < cols) *reinterpret_cast<uint32_t*>(row + i * pitch + lane) = w[i];
    }
    return;
  }
  unsigned short* p = reinterpret_cast<unsigned short*>(row);
  // an odd row's pairs, and what is left over: lane 0 has the first element, the lane of the last column the last where cols is even
  const bool pair_even = 2 * lane + 1 < cols, pair_odd = 2 * lane + 2 < cols, one_even = 2 * lane + 1 == cols;
  const bool one_odd = lane == 0 || 2 * lane + 2 == cols;
  const int one_at = lane == 0 ? 0 : 2 * lane + 1;
  BoxRows(row, pitch).pattern([&](auto odd0, auto odd1) {
#pragma unroll 1
    for (int r = 0; r < rows; r += kStep, p += kStep * pitch) {
      uint32_t w[kStep];
#pragma unroll
      for (int i = 0; i < kStep; ++i) w[i] = get(r + i);
#pragma unroll
      for (int i = 0; i < kStep; ++i) {
        const bool odd = i % 2 ? decltype(odd1)::value : decltype(odd0)::value;
        unsigned short* q = p + i * pitch;
        const bool in = r + i < rows;
        if (odd) {
          const uint32_t after = __shfl_down_sync(0xffffffffu, w[i], 1);
          if (in && pair_odd) *reinterpret_cast<uint32_t*>(q + 2 * lane + 1) = __funnelshift_r(w[i], after, 16);
          if (in && one_odd) q[one_at] = (unsigned short)(lane == 0 ? w[i] : w[i] >> 16);
        } else {
          if (in && pair_even) *reinterpret_cast<uint32_t*>(q + 2 * lane) = w[i];
          if (in && one_even) q[2 * lane] = (unsigned short)w[i];
        }
      }
    }
    // (cols = 2: lane 0 has both ends of an odd row)
    if (cols == 2 && (decltype(odd0)::value || decltype(odd1)::value)) {
      unsigned short* q = reinterpret_cast<unsigned short*>(row);
      for (int r = 0; r < rows; ++r) {
        const uint32_t w = get(r);
        if (lane == 0 && (r % 2 ? decltype(odd1)::value : decltype(odd0)::value)) q[r * pitch + 1] = (unsigned short)(w >> 16);
      }
    }
  });
}

// A_MN / B_MN: the operand is contiguous along M / N in global memory (MN-major image).
// PLAIN: an overwriting store of an aligned C, the usual call, without the code of every other epilogue.
template <typename TO, int BN, bool BF16, bool A_MN, bool B_MN, bool PLAIN>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                        const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ GemmArgs p) {
  using L = SmemLayout<BN>;
  const bool tma_c = PLAIN || p.tma_c, accumulate = !PLAIN && p.accumulate, has_fill = !PLAIN && p.epi.has_fill;
  const int reduce_kind = PLAIN ? FRISK_B200_REDUCE_NONE : p.epi.reduce_kind;
  constexpr int kStages = L::kStages;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* acc_full = empty_bar + kStages;   // [2]
  uint64_t* acc_empty = acc_full + 2;         // [2]
  uint64_t* box_bar = acc_empty + 2;          // [4 warps][2] old values of C have landed in a box
  uint64_t* epi_bar = box_bar + 8;            // the epilogue threads among themselves
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(epi_bar + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* epi_word = tmem_slot + 2;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (p.M + BM - 1) / BM, tiles_n = (p.N + BN - 1) / BN, tiles = tiles_m * tiles_n;
  const int splits = p.splits, rank = splits > 1 ? (int)cluster_ctarank() : 0;
  const int num_kb = (p.K + BK - 1) / BK;
  // this CTA's work, item by item
  const TileWalk walk{tiles, num_kb, p.n_whole, splits, (int)gridDim.x};
  auto get_item = [&](int i, TileItem& it) { return walk.get((int)blockIdx.x, rank, i, it); };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 4);
    }
    for (int i = 0; i < 8; ++i) mbar_init(&box_bar[i], 1);
    mbar_init(epi_bar, 128);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    if (tma_c) tma_prefetch_desc(&tmap_c);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // Launched with programmatic stream serialization: the set-up above may run while the kernel in front of
  // this one drains; nothing touches global memory before that kernel is complete.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      TileItem it;
      for (int i = 0; ok && get_item(i, it); ++i) {
        const TileCoord tc = tile_coord(it.tile, tiles_m, tiles_n);
        const int m0 = tc.m * BM, n0 = tc.n * BN;
        for (int kb = it.kb0; kb < it.kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) {
            ok = false;
            break;
          }
          unsigned char* sa = smem + stage * L::kStageBytes;
          unsigned char* sb = sa + L::kABytes;
          mbar_expect_tx(&full_bar[stage], L::kStageBytes);
          const int k0 = kb * BK;
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              tma_load_2d(sa + j * (BK * 128), &tmap_a, &full_bar[stage], m0 + j * 64, k0);
          } else {
            tma_load_2d(sa, &tmap_a, &full_bar[stage], k0, m0);
          }
          if (B_MN) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_2d(sb + j * (BK * 128), &tmap_b, &full_bar[stage], n0 + j * 64, k0);
          } else {
            // boxes of at most 128 rows: stacked 8-row groups, the same image as one taller box
#pragma unroll
            for (int j = 0; j < BN / L::kBoxRowsB; ++j)
              tma_load_2d(sb + j * (L::kBoxRowsB * BK * 2), &tmap_b, &full_bar[stage], k0, n0 + j * L::kBoxRowsB);
          }
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // Run by the whole warp, so that descriptors and counters are uniform; one elected lane issues.  A k-block of 128 columns takes
    // 427 clk so, 501 as one lane's code (wait, four MMAs of 65, commit; with 256 columns the MMAs hide the rest): 512 x 512 x 4096
    // 11.6 -> 11.1 us, 128 x 2048 x 2048 9.1 -> 8.8.  One wait and one commit for two k-blocks were slower (256 x 4096 x 4096 18.3 -> 19.2).
    constexpr uint32_t idesc = umma_idesc_f16(BM, BN, BF16, A_MN, B_MN);
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    TileItem it;
    for (int i = 0; ok && get_item(i, it); ++i) {
      ok = mbar_wait_warp(&acc_empty[acc], acc_phase ^ 1, abort_flag, p.status, ST_TIMEOUT_ACC_EMPTY);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t d_tmem = tmem + acc * BN;
      for (int kb = it.kb0; kb < it.kb1; ++kb) {
        ok = mbar_wait_warp(&full_bar[stage], phase, abort_flag, p.status, ST_TIMEOUT_FULL);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t sa = smem_u32(smem + stage * L::kStageBytes);
        const uint32_t sb = sa + L::kABytes;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            uint64_t da = A_MN ? umma_desc_mnmajor_sw128(sa + k * (UMMA_K * 128), BK * 128, 1024)
                               : umma_desc_kmajor_sw128(sa + k * (UMMA_K * 2));
            uint64_t db = B_MN ? umma_desc_mnmajor_sw128(sb + k * (UMMA_K * 128), BK * 128, 1024)
                               : umma_desc_kmajor_sw128(sb + k * (UMMA_K * 2));
            umma_f16_ss(d_tmem, da, db, idesc, (kb > it.kb0 || k != 0) ? 1u : 0u);
          }
          umma_commit(&empty_bar[stage]);                     // stage reusable once these MMAs have read it
          if (kb + 1 == it.kb1) umma_commit(&acc_full[acc]);  // accumulator complete (an item has a k-block or more)
        }
        __syncwarp();
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quad = warp & 3;  // TMEM lanes [32*quad, 32*quad+32) are this warp's
    constexpr int U = 128 / (int)sizeof(TO);     // columns of a box
    constexpr int kPer = 4 / (int)sizeof(TO);    // of a lane's 32-bit word of a box row
    unsigned char* boxes = smem + L::kOutOffset + quad * 2 * kBoxBytes;
    uint64_t* bars = box_bar + quad * 2;
    TO* const C = static_cast<TO*>(p.C);
    int box_sel = 0;              // the box the next unit uses
    uint32_t box_phases = 0;      // bit b: the phase box b's barrier is in
    int acc = 0;
    uint32_t acc_phase = 0, epi_phase = 0;
    bool ok = true;
    // bounded meeting point of this CTA's 128 epilogue threads
    auto epi_sync = [&]() {
      mbar_arrive(epi_bar);
      if (ok) ok = mbar_wait_warp(epi_bar, epi_phase, abort_flag, p.status, ST_TIMEOUT_MISC);
      epi_phase ^= 1;
    };
    // byte offset of column j of a box's row r: 128-byte rows in the 128-byte-swizzle image
    auto box_at = [](int r, int j) {
      const int byte = j * (int)sizeof(TO);
      return r * 128 + (((byte >> 4) ^ (r & 7)) << 4) + (byte & 15);
    };
    // the old values of the box at (r0, c0) on their way into box `sel`, whose last store has been read (one lane)
    auto fetch_old = [&](int sel, int r0, int c0) {
      tma_store_wait_read<0>();
      mbar_expect_tx(&bars[sel], kBoxBytes);
      tma_load_2d(boxes + sel * kBoxBytes, &tmap_c, &bars[sel], c0, r0);
    };
    // Finishes the box of C at (r0, c0): lane = row; values(h, v) gives the row's fp32 results of columns c0 + 32h..+31.
    // Where the old C comes by TMA its load has been issued.
    auto finish_box = [&](int r0, int c0, auto&& values) {
      unsigned char* box = boxes + box_sel * kBoxBytes;
      uint4* const my_row = reinterpret_cast<uint4*>(box + lane * 128);
      float row_acc = reduce_identity(reduce_kind);
      if (tma_c) {
        if (!accumulate && lane == 0) tma_store_wait_read<1>();  // the store before the last one used this box
      } else if (accumulate) {
        // old values of C, a row at a time, into the same image; all loads are on their way before the first is stored
        load_box_rows(C + (int64_t)r0 * p.ldc + c0, p.ldc, min(32, p.M - r0), min(U, p.N - c0), lane, [&](int r, uint32_t w) {
          *reinterpret_cast<uint32_t*>(box + box_at(r, lane * kPer)) = w;
        });
      }
      __syncwarp();
      uint32_t w[32];
#pragma unroll
      for (int h = 0; h < U / 32; ++h) {
        float v[32];
        values(h, v);
        if (accumulate) {
          if (h == 0 && tma_c) {
            if (ok) ok = mbar_wait_warp(&bars[box_sel], (box_phases >> box_sel) & 1, abort_flag, p.status, ST_TIMEOUT_MISC);
            box_phases ^= 1u << box_sel;
            __syncwarp();
          }
          if (sizeof(TO) == 4) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint4 o = my_row[j ^ (lane & 7)];
              v[4 * j] += __uint_as_float(o.x); v[4 * j + 1] += __uint_as_float(o.y);
              v[4 * j + 2] += __uint_as_float(o.z); v[4 * j + 3] += __uint_as_float(o.w);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 o = my_row[(h * 4 + j) ^ (lane & 7)];
              const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 f = unpack_out<TO>(ow[e]);
                v[8 * j + 2 * e] += f.x;
                v[8 * j + 2 * e + 1] += f.y;
              }
            }
          }
        } else if (has_fill) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] += p.epi.fill;
        }
        if (sizeof(TO) == 4) {
#pragma unroll
          for (int i = 0; i < 32; ++i) w[i] = __float_as_uint(v[i]);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) w[(h & 1) * 16 + i] = pack_out<TO>(v[2 * i], v[2 * i + 1]);
        }
        if (reduce_kind) {  // over the values as they are stored
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c0 + h * 32 + i < p.N) row_acc = reduce_combine(reduce_kind, row_acc, rounded_as<TO>(v[i]));
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) my_row[j ^ (lane & 7)] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
      if (tma_c) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tmap_c, box, c0, r0);  // clipped at the edges of C (its rows end on 16 bytes, tma_writes_c)
          tma_store_commit();
        }
      } else {
        __syncwarp();
        store_box_rows(C + (int64_t)r0 * p.ldc + c0, p.ldc, min(32, p.M - r0), min(U, p.N - c0), lane, [&](int r) {
          return *reinterpret_cast<const uint32_t*>(box + box_at(r, lane * kPer));
        });
        __syncwarp();
      }
      box_sel ^= 1;
      if (reduce_kind && r0 + lane < p.M) __stcg(p.epi.row_partials + (int64_t)(c0 / U) * p.M + r0 + lane, row_acc);
    };
    // (one thread) a draw of row block m's ticket; true for the last of its column tiles
    auto draw_row = [&](int m) {
      const bool last = atomicAdd(p.epi.row_tickets + m, 1u) == (unsigned)tiles_n - 1;
      if (last) p.epi.row_tickets[m] = 0;  // clean for the next launch
      return last;
    };
    int drawn = 0;  // items whose tickets this CTA has drawn
    // A column tile of row block tc.m has left its partials: whoever draws the last ticket combines the row block's
    auto combine_rows = [&](const TileCoord& tc) {
      epi_sync();
      if (warp == 2 && lane == 0) {
        __threadfence();
        const bool last = draw_row(tc.m);
        if (last) __threadfence();
        *epi_word = last ? 1u : 0u;
      }
      ++drawn;
      epi_sync();
      const bool combine = ok && *epi_word != 0;
      epi_sync();  // everybody has read it
      const int row = tc.m * BM + quad * 32 + lane;
      if (combine && row < p.M) {
        TO* const dst = static_cast<TO*>(p.epi.reduce_dst);
        float r = p.epi.reduce_clear ? reduce_identity(reduce_kind) : static_cast<float>(dst[row]);
        const int n = (p.N + U - 1) / U;
#pragma unroll 4
        for (int t = 0; t < n; ++t) r = reduce_combine(reduce_kind, r, __ldcg(p.epi.row_partials + (int64_t)t * p.M + row));
        dst[row] = static_cast<TO>(r);
      }
    };

    TileItem it;
    TileCoord shared_tile{-1, -1};
    for (int i = 0; ok && get_item(i, it); ++i) {
      const TileCoord tc = tile_coord(it.tile, tiles_m, tiles_n);
      const int m0 = tc.m * BM, n0 = tc.n * BN;
      if (!mbar_wait_warp(&acc_full[acc], acc_phase, abort_flag, p.status, ST_TIMEOUT_ACC_FULL)) break;
      tc_fence_after_sync();
      __syncwarp();
      const uint32_t taddr = tmem_base + acc * BN + (static_cast<uint32_t>(quad * 32) << 16);
      if (it.shared) {
        // this CTA's last item: its part goes into the ring, every stage of which has been read
        float4* part = reinterpret_cast<float4*>(smem) + quad * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(taddr + c * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            part[(c * 8 + i) * BM] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                                 __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
        }
        shared_tile = tc;
        break;
      }
      const int r0 = m0 + quad * 32;
      const int units = r0 < p.M ? (min(BN, p.N - n0) + U - 1) / U : 0;
      const bool old_by_tma = accumulate && tma_c;
      if (old_by_tma && units > 0 && lane == 0) fetch_old(box_sel, r0, n0);
#pragma unroll 1
      for (int u = 0; u < units; ++u) {
        if (old_by_tma && u + 1 < units && lane == 0) fetch_old(box_sel ^ 1, r0, n0 + (u + 1) * U);
        finish_box(r0, n0 + u * U, [&](int h, float (&v)[32]) {
          uint32_t t[32];
          tmem_ld_32x32b_x32(taddr + u * U + h * 32, t);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(t[i]);
        });
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
      if (reduce_kind) combine_rows(tc);
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (splits > 1) {
      // every role of every CTA of the cluster ends (its waits are bounded), so these meetings are reached
      __syncwarp();
      cluster_sync_all();  // the parts are complete
      const TileCoord tc = shared_tile;
      const bool shared = tc.m >= 0;  // (the same for the whole cluster, unless a wait ran out)
      const int r0 = tc.m * BM + quad * 32;
      // Column groups (4 columns) rank, rank + splits, ...: the parts of this warp's rows, S x kDeep loads in flight, summed
      // in rank order and handed to the CTA that finishes their box (boxes are dealt out column by column)
      auto add_up = [&](auto splits_c) {
        constexpr int S = decltype(splits_c)::value, kDeep = 16 / S;
        const uint32_t own = smem_u32(smem) + (quad * 32 + lane) * 16;
        for (int cg0 = rank; cg0 < BN / 4; cg0 += S * kDeep) {
          float4 t[kDeep][S];
#pragma unroll
          for (int j = 0; j < kDeep; ++j)
#pragma unroll
            for (int c = 0; c < S; ++c) t[j][c] = ld_cluster_f4(mapa_addr(own + (cg0 + j * S) * (BM * 16), c));
#pragma unroll
          for (int j = 0; j < kDeep; ++j) {
            float4 sum = t[j][0];
#pragma unroll
            for (int c = 1; c < S; ++c) {
              sum.x += t[j][c].x; sum.y += t[j][c].y; sum.z += t[j][c].z; sum.w += t[j][c].w;
            }
            const int cg = cg0 + j * S, u = cg / (U / 4);  // box column u: finished by CTA u % S, as its u / S-th
            st_cluster_f4(mapa_addr(own + L::kSumOffset + ((u / S) * (U / 4) + cg % (U / 4)) * (BM * 16), u % S), sum);
          }
        }
      };
      // Where every CTA finishes a box column, it reads the parts of its boxes itself; otherwise (more CTAs than box
      // columns) all of them add up first.
      const bool direct = BN / U >= splits;
      if (shared && r0 < p.M && !direct) {
        if (splits == 2) add_up(std::integral_constant<int, 2>());
        else if (splits == 4) add_up(std::integral_constant<int, 4>());
        else add_up(std::integral_constant<int, 8>());
      }
      if (!direct) {
        __syncwarp();
        cluster_sync_all();  // the sums are complete
      }
      if (shared) {
#pragma unroll 1
        for (int u = rank; u < BN / U; u += splits) {
          const int c0 = tc.n * BN + u * U;
          if (r0 >= p.M || c0 >= p.N) continue;
          if (accumulate && tma_c && lane == 0) fetch_old(box_sel, r0, c0);
          finish_box(r0, c0, [&](int h, float (&v)[32]) {
            if (direct) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = 0.f;
              const uint32_t at = smem_u32(smem) + ((u * U + h * 32) / 4 * BM + quad * 32 + lane) * 16;
              for (int c = 0; c < splits; c += 2) {  // two parts' loads in flight, added in rank order
                float4 t[2][8];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                  const uint32_t peer = mapa_addr(at, c + j);
#pragma unroll
                  for (int i = 0; i < 8; ++i) t[j][i] = ld_cluster_f4(peer + i * (BM * 16));
                }
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                  for (int i = 0; i < 8; ++i) {
                    v[4 * i] += t[j][i].x; v[4 * i + 1] += t[j][i].y; v[4 * i + 2] += t[j][i].z; v[4 * i + 3] += t[j][i].w;
                  }
              }
              return;
            }
            const float4* sums = reinterpret_cast<const float4*>(smem + L::kSumOffset) +
                                 ((u / splits) * (U / 4) + h * 8) * BM + quad * 32 + lane;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 t = sums[i * BM];
              v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
            }
          });
        }
      }
      if (reduce_kind) __threadfence();  // the row partials, before rank 0 takes the ticket for the cluster
      __syncwarp();
      cluster_sync_all();  // nobody reads a peer any more
      if (reduce_kind && shared && rank == 0) combine_rows(tc);
    }
    // what a wait that ran out has left over: the tickets are zero again however the launch ends
    if (reduce_kind && warp == 2 && lane == 0)
      walk.draw_owed((int)blockIdx.x, rank, drawn, [&](int tile) { draw_row(tile_coord(tile, tiles_m, tiles_n).m); });
    if (tma_c && lane == 0) tma_store_wait<0>();  // the boxes are read and written out before the CTA leaves
  }
  if (warp < 2 && splits > 1) {
    __syncwarp();
    cluster_sync_all();
    if (BN * (int)sizeof(TO) / 128 < splits) cluster_sync_all();
    cluster_sync_all();
  }

  // ------------------------------------------------------------------ teardown
  if (*abort_flag) {
    // a wait ran out somewhere: give copies that are still in flight time to land
    unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Which tile, and how many CTAs share the K of a tile of the last round: the least of these estimates, in clocks of about
// 1.9 GHz beyond the launch.
struct Plan {
  int bn, splits, n_whole, grid;
  double clocks;
};
// The plan for tiles of bn columns and clusters of `splits` CTAs, of which the device runs `clusters`.  A 64-k block takes
// its MMAs (512 clk at 256 columns) or the issuing warp's work (below) and, the more SMs are at it, what L2 adds: 770 at 2048^3
// and 4096^3 with the chip full, 1100 where rows begin off 128-byte lines (3000^3: two requests of the TMA unit a row).  Sharing costs
// barriers, parts and sums: 3.5 us at 128 rows (128 x 512 x 512 over clusters of four took 8.7 us, whole 6.7), less
// with fewer rows (17 x 1024 x 1024 6.8, 128 x 1024 x 1024 9.1 over clusters of eight).  Tiles of 64 columns take as long for a
// block (410 clk, 427 with 128 columns: the issuing warp's wait, four MMAs and commit set the pace, not the MMAs) but put twice the SMs
// to work and have half the parts to add up: they are for products with few columns and rows (128 x 2048 x 2048
// in clusters of four 9.9 us, 11.2 with 128 columns; 64 x 2048 x 4096 11.4, 12.3;
// 256 x 1024 x 4096 12.1, 13.4; whole 300 x 1000 x 1000 9.2, 9.9).
Plan plan_of(const GemmDims& g, int64_t tiles, int sms, int bn, int splits, int clusters) {
  const int64_t kb = (g.K + BK - 1) / BK;
  const bool aligned = g.lda % 64 == 0 && g.ldb % 64 == 0;
  Plan p{bn, splits, 0, 0, 1e300};
  double blocks, extra;
  if (splits == 1) {
    p.n_whole = (int)tiles;
    p.grid = (int)std::min<int64_t>(tiles, sms);
    blocks = std::ceil((double)tiles / sms) * (double)kb;
    extra = bn == 256 ? 3500 : bn == 128 ? 1800 : 1500;
  } else {
    const int grid = splits * std::min(clusters, sms / splits);
    if (grid == 0 || kb < 2 * splits) return p;
    const int64_t rounds = tiles / grid, rest = tiles % grid;
    if (rest == 0 || rest > grid / splits) return p;
    p.n_whole = (int)(rounds * grid);
    p.grid = rounds > 0 ? grid : (int)rest * splits;
    blocks = (double)rounds * (double)kb + std::ceil((double)kb / splits);
    extra = (bn == 256 ? 4500 : bn == 128 ? 3500 : 2500) + (bn == 64 ? 1500.0 : 3000.0) * (double)std::min<int64_t>(g.M, BM) / BM;
  }
  const double busy = (double)p.grid / sms;
  // (Fitted to whole calls together with `l2` and `extra`, when one lane issued the MMAs: 270 and 250 are shares of an estimate, and lie
  // below the 427 and 410 clk that a block takes an issuing warp.)
  const double mma = bn == 256 ? 520 : bn == 128 ? 270 : 250;
  const double l2 = bn == 256 ? (aligned ? 250 : 580) : bn == 128 ? (aligned ? 200 : 450) : aligned ? 150 : 340;
  p.clocks = blocks * (mma + l2 * busy) + extra;
  return p;
}
template <typename F>
Plan make_plan(const GemmDims& g, int sms, F&& clusters) {
  Plan best{256, 1, 0, 0, 1e300};
  const int64_t kb = (g.K + BK - 1) / BK;
  for (int bn : {256, 128, 64}) {
    const int64_t tiles = ((g.M + BM - 1) / BM) * ((g.N + bn - 1) / bn);
    if (tiles > INT32_MAX / 2) continue;
    if (bn == 64 && tiles > 2 * sms) continue;  // (wider ones fill the SMs; the call that asks has a launch to make)
    for (int splits : {1, 2, 4, 8}) {
      if (splits > 1 && kb < 2 * splits) break;
      const Plan p = plan_of(g, tiles, sms, bn, splits, splits > 1 ? clusters(bn, splits) : 0);
      if (p.clocks < best.clocks) best = p;
    }
  }
  return best;
}

template <typename TO, int BN, bool BF16, bool A_MN, bool B_MN>
int launch_cfg(frisk_b200_ctx* ctx, const frisk_b200_gemm_desc& d, const void* A, const void* B, void* C,
               const Plan& plan, const RowEpilogue* epi, cudaStream_t s) {
  GemmDims g = resolve_dims(d);
  CUtensorMap ta, tb;
  int rc;
  // A: K-major -> dims {K, M}, box {64, 128};  MN-major (stored [K,M]) -> dims {M, K}, box {64, 64}
  if (A_MN)
    rc = encode_tmap_2d(ctx, &ta, d.dtype_ab, A, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.lda * 2, 64, BK, true);
  else
    rc = encode_tmap_2d(ctx, &ta, d.dtype_ab, A, (uint64_t)g.K, (uint64_t)g.M, (uint64_t)g.lda * 2, BK, BM, true);
  if (rc) { ctx->last_cuda = rc; return FRISK_B200_E_CUDA; }
  if (B_MN)
    rc = encode_tmap_2d(ctx, &tb, d.dtype_ab, B, (uint64_t)g.N, (uint64_t)g.K, (uint64_t)g.ldb * 2, 64, BK, true);
  else
    rc = encode_tmap_2d(ctx, &tb, d.dtype_ab, B, (uint64_t)g.K, (uint64_t)g.N, (uint64_t)g.ldb * 2, BK,
                        SmemLayout<BN>::kBoxRowsB, true);
  if (rc) { ctx->last_cuda = rc; return FRISK_B200_E_CUDA; }

  GemmArgs a{};
  a.tma_c = tma_writes_c(d, C);
  CUtensorMap tc = ta;  // unused otherwise
  if (a.tma_c) {
    const int out_dtype = sizeof(TO) == 4 ? FRISK_B200_F32 : (std::is_same<TO, __half>::value ? FRISK_B200_F16 : FRISK_B200_BF16);
    rc = encode_tmap_2d(ctx, &tc, out_dtype, C, (uint64_t)g.N, (uint64_t)g.M, (uint64_t)g.ldc * sizeof(TO),
                        128 / sizeof(TO), 32, true);
    if (rc) { ctx->last_cuda = rc; return FRISK_B200_E_CUDA; }
  }
  a.C = C;
  a.ldc = g.ldc;
  a.M = (int)g.M; a.N = (int)g.N; a.K = (int)g.K;
  a.accumulate = d.clear_accum || (epi && epi->has_fill) ? 0 : 1;
  if (epi) a.epi = *epi;
  a.status = ctx->d_status;
  a.splits = plan.splits;
  a.n_whole = plan.n_whole;
  using L = SmemLayout<BN>;
  auto launch = [&](auto kern, PerDeviceOnce& opt_in) -> int {
    if (opt_in(ctx->device, [&] {
          return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal) == cudaSuccess ? 0 : 1;
        }))
      return FRISK_B200_E_CUDA;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)plan.grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = L::kTotal;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // the kernel waits (griddepcontrol.wait) itself
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)plan.splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = plan.splits > 1 ? 2 : 1;
    FB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, ta, tb, tc, a));
    return 0;
  };
  static PerDeviceOnce opt_in_plain, opt_in_general;  // one pair per instantiation
  if (a.tma_c && !a.accumulate && !a.epi.has_fill && !a.epi.reduce_kind)
    return launch(gemm_tcgen05_kernel<TO, BN, BF16, A_MN, B_MN, true>, opt_in_plain);
  return launch(gemm_tcgen05_kernel<TO, BN, BF16, A_MN, B_MN, false>, opt_in_general);
}

template <typename TO, bool BF16, int BN>
int launch_major(frisk_b200_ctx* ctx, const frisk_b200_gemm_desc& d, const void* A, const void* B, void* C,
                 const Plan& plan, const RowEpilogue* epi, cudaStream_t s) {
  bool a_mn = d.trans_a != 0;   // A stored [K,M]
  bool b_mn = d.trans_b == 0;   // B stored [K,N]
  if (a_mn) {
    if (b_mn) return launch_cfg<TO, BN, BF16, true, true>(ctx, d, A, B, C, plan, epi, s);
    return launch_cfg<TO, BN, BF16, true, false>(ctx, d, A, B, C, plan, epi, s);
  }
  if (b_mn) return launch_cfg<TO, BN, BF16, false, true>(ctx, d, A, B, C, plan, epi, s);
  return launch_cfg<TO, BN, BF16, false, false>(ctx, d, A, B, C, plan, epi, s);
}

// Clusters the device runs at a time.  Every instantiation has one CTA per SM (shared memory decides), so one of them
// answers for all of the same tile.
int clusters_of(int device, int bn, int splits) {
  static ClusterCapacity wide, narrow, thin;
  static PerDeviceOnce opt_wide, opt_narrow, opt_thin;
  auto ask = [&](auto kern, int smem, ClusterCapacity& capacity, PerDeviceOnce& opt_in) {
    if (opt_in(device, [&] {
          return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess ? 0 : 1;
        }))
      return 0;
    return capacity(device, kern, kThreads, smem, splits);
  };
  if (bn == 256) return ask(gemm_tcgen05_kernel<__half, 256, false, false, false, true>, SmemLayout<256>::kTotal, wide, opt_wide);
  if (bn == 128) return ask(gemm_tcgen05_kernel<__half, 128, false, false, false, true>, SmemLayout<128>::kTotal, narrow, opt_narrow);
  return ask(gemm_tcgen05_kernel<__half, 64, false, false, false, true>, SmemLayout<64>::kTotal, thin, opt_thin);
}
Plan plan_for(frisk_b200_ctx* ctx, const frisk_b200_gemm_desc& d) {
  return make_plan(resolve_dims(d), std::min(ctx->num_sms, kNumSMsDefault),
                   [&](int bn, int splits) { return clusters_of(ctx->device, bn, splits); });
}

template <typename TO, bool BF16>
int launch_tile(frisk_b200_ctx* ctx, const frisk_b200_gemm_desc& d, const void* A, const void* B, void* C,
                const RowEpilogue* epi, cudaStream_t s) {
  const Plan plan = plan_for(ctx, d);
  if (plan.grid == 0) return FRISK_B200_E_UNSUPPORTED;
  if (plan.bn == 256) return launch_major<TO, BF16, 256>(ctx, d, A, B, C, plan, epi, s);
  if (plan.bn == 128) return launch_major<TO, BF16, 128>(ctx, d, A, B, C, plan, epi, s);
  return launch_major<TO, BF16, 64>(ctx, d, A, B, C, plan, epi, s);
}

}  // namespace

bool tcgen05_supported(const frisk_b200_gemm_desc& d) {
  if (d.dtype_ab != FRISK_B200_F16 && d.dtype_ab != FRISK_B200_BF16) return false;
  GemmDims g = resolve_dims(d);
  // TMA: 16-byte pitches; 32-bit coordinates
  if (g.lda % 8 || g.ldb % 8) return false;
  if (g.M > INT32_MAX || g.N > INT32_MAX || g.K > INT32_MAX) return false;
  return true;
}

// clocks the plan is estimated at (frisk_b200_gemm weighs it against the pair kernel)
double tcgen05_clocks(frisk_b200_ctx* ctx, const frisk_b200_gemm_desc& d) { return plan_for(ctx, d).clocks; }

void tcgen05_describe(frisk_b200_ctx* ctx, const frisk_b200_gemm_desc& d, frisk_b200_gemm_plan_info* out) {
  const Plan p = plan_for(ctx, d);
  const GemmDims g = resolve_dims(d);
  out->tile_n = p.bn;
  out->splits = p.splits;
  out->ctas = p.grid;
  out->tiles = ((g.M + BM - 1) / BM) * ((g.N + p.bn - 1) / p.bn);
  out->whole_tiles = p.n_whole;
  out->clocks = p.clocks;
}

// the row reduction keeps one fp32 per (box of columns, row) and one ticket per row block
bool tcgen05_row_epilogue_fits(const frisk_b200_gemm_desc& d) {
  const GemmDims g = resolve_dims(d);
  const int64_t box = 128 / (int64_t)dtype_size(d.dtype_c);
  return (g.N + box - 1) / box * g.M * 4 <= (int64_t)kRowPartialBytes && (g.M + BM - 1) / BM <= kRowTickets;
}

int launch_gemm_tcgen05(frisk_b200_ctx* ctx, const frisk_b200_gemm_desc& d, const void* A, const void* B,
                        void* C, cudaStream_t s, const RowEpilogue* epi) {
  if (!tcgen05_supported(d)) return FRISK_B200_E_UNSUPPORTED;
  if (!aligned16(A) || !aligned16(B)) return FRISK_B200_E_ALIGN;
  const bool bf = d.dtype_ab == FRISK_B200_BF16;
  if (d.dtype_c == FRISK_B200_F32)
    return bf ? launch_tile<float, true>(ctx, d, A, B, C, epi, s) : launch_tile<float, false>(ctx, d, A, B, C, epi, s);
  if (bf) return launch_tile<__nv_bfloat16, true>(ctx, d, A, B, C, epi, s);
  return launch_tile<__half, false>(ctx, d, A, B, C, epi, s);
}

}  // namespace fb
