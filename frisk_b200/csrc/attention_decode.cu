// Attention forward for a few queries per (batch, head) (S_q <= 16: decoding against a key/value cache), single-pass
// mode.  Same contract and numerics as attention_fwd.cu: fp32 scores and statistics, a running reference maximum that
// moves only when the maximum grew by more than 2^8, probabilities rounded to the input type before they meet V, fp32
// accumulation (benchmark/layout/execution/tiled_attention.py:392,505-515,628-629; compact BHSD, :52-61).
//
// Bound by HBM: every key and value is read once and meets 16 queries at most.  The two-tile kernel gives a head to
// one CTA and walks its keys through a serial chain (S -> softmax -> P.V, ~2 us for 128 keys, 112 of 128 rows
// padding) with 128 KB in flight: 3.8 TB/s at best, and a machine that is empty when there are few heads.  Here
//
//   * the (head, 64-key tile) units are numbered head-major and CTA c takes a contiguous range of them, so every SM
//     streams the same number of bytes whatever the head count and the cache length; a head shared by several CTAs is
//     finished by the contributor that draws the last ticket, which adds the partial results in contributor order
//     (reproducible).  No CTA waits for another, and one whose own wait ran out still draws the tickets it owes, so
//     that they are zero again when the launch ends however it ends;
//   * K and V tiles arrive by TMA in a ring of 192 KB (6 stages of 64 keys at D = 128, 12 at D = 64);
//   * four warps work on every tile, warp w on its keys 16w..16w+15 with its own reference maximum, row sums and fp32
//     O, so nothing but the ring ties them together before the end of a head's range.  The products use
//     mma.sync 16x8x16: 16 queries are exactly its M, the work per byte is far below what tensor memory would pay
//     for (a warp needs ~500 clk for a tile that takes ~1300 to arrive), and scores and probabilities never leave
//     the registers.
// Every mbarrier wait is bounded (ptx.cuh); no TMA load uses cluster multicast.
#include <algorithm>

#include "common.cuh"
#include "ptx.cuh"
#include "work_split.cuh"

#include "attention_common.cuh"

namespace fb {
namespace {
using namespace attn;

constexpr int kQ = 16;            // queries per head, padded
constexpr int kKeys = 64;         // keys per tile
constexpr int kWarps = 4;         // consumer warps
constexpr int kDecThreads = 32 * (kWarps + 1);
constexpr int kRingBytes = 192 * 1024;
constexpr int kMaxHeads = 1 << 16;  // tickets in the context's scratch
constexpr size_t kTicketBytes = (size_t)kMaxHeads * sizeof(unsigned);
constexpr int kPartialFloats = kQ * 128 + 2 * kQ;  // O [16][D], reference maxima [16], row sums [16]

template <int D>
struct DecSmem {
  static constexpr int kTile = kKeys * D * 2;
  static constexpr int kStages = kRingBytes / (2 * kTile);
  static constexpr int kO = kRingBytes;                        // [4 warps][16][D] fp32; contributor weights while merging
  static constexpr int kStat = kO + kWarps * kQ * D * 4;       // [4][16] maxima, [4][16] sums
  static constexpr int kBar = kStat + 2 * kWarps * kQ * 4;
  static constexpr int kTotal = kBar + 512 + 1024;
  static_assert(kTotal <= 232448, "ring and reduction area must fit");
  static_assert(kNumSMsDefault * kQ * 4 <= kWarps * kQ * D * 4, "the weights of all contributors must fit");
};

struct DecParams {
  const void* Q;
  void* O;
  int S_q, S_kv, n_tiles, causal;
  WorkSplit work;  // (head, key tile) units over the CTAs
  float scale_log2;
  unsigned* tickets;  // one per head, zero between launches
  float* partials;    // two per CTA
  unsigned* status;
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
template <bool BF16>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (BF16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// four consecutive results of one row, rounded to the output type
template <bool BF16, bool OUT_F32>
__device__ __forceinline__ void store4(void* O, size_t at, float4 v) {
  if (OUT_F32)
    *reinterpret_cast<float4*>(static_cast<float*>(O) + at) = v;
  else
    *reinterpret_cast<uint2*>(static_cast<uint16_t*>(O) + at) = make_uint2(pack16<BF16>(v.x, v.y), pack16<BF16>(v.z, v.w));
}

template <bool BF16, int D, bool OUT_F32>
__global__ void __launch_bounds__(kDecThreads, 1)
    attention_decode_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                            const DecParams p) {
  using L = DecSmem<D>;
  constexpr int kBoxes = D / 64, kBoxBytes = kKeys * 128;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* empty_bar = full_bar + L::kStages;
  uint64_t* meet_bar = empty_bar + L::kStages;  // the 128 consumer threads among themselves
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(meet_bar + 1);
  volatile uint32_t* ticket_word = abort_flag + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned n_tiles = (unsigned)p.n_tiles;
  const unsigned u_begin = p.work.start(blockIdx.x), u_end = p.work.start(blockIdx.x + 1);

  if (threadIdx.x == 0) {
    for (int i = 0; i < L::kStages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], kWarps);
    }
    mbar_init(meet_bar, kWarps * 32);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
  }
  __syncthreads();
  // Launched with programmatic stream serialization: the set-up above may overlap the kernel before this one.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp == kWarps) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      unsigned head = u_begin / n_tiles, tile = u_begin % n_tiles;
      for (unsigned u = u_begin; u < u_end; ++u) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, ST_ATTN_KV)) break;
        unsigned char* sk = smem + stage * 2 * L::kTile;
        mbar_expect_tx(&full_bar[stage], 2 * L::kTile);  // rows beyond S_kv are filled with zeros and counted
#pragma unroll
        for (int b = 0; b < kBoxes; ++b)
          tma_load_3d(sk + b * kBoxBytes, &tmap_k, &full_bar[stage], b * 64, (int)tile * kKeys, (int)head);
#pragma unroll
        for (int b = 0; b < kBoxes; ++b)
          tma_load_3d(sk + L::kTile + b * kBoxBytes, &tmap_v, &full_bar[stage], b * 64, (int)tile * kKeys, (int)head);
        if (++stage == L::kStages) {
          stage = 0;
          phase ^= 1;
        }
        if (++tile == n_tiles) {
          tile = 0;
          ++head;
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ consumers
    const int g = lane >> 2, tq = lane & 3;  // fragment coordinates: rows g and g + 8, column pair tq
    const int off = p.S_kv - p.S_q;
    float* s_o = reinterpret_cast<float*>(smem + L::kO);
    float* s_m = reinterpret_cast<float*>(smem + L::kStat);
    float* s_l = s_m + kWarps * kQ;
    uint32_t meet_phase = 0;
    bool ok = true;
    auto meet = [&]() {  // bounded meeting point of the consumer threads
      mbar_arrive(meet_bar);
      if (ok) ok = mbar_wait_warp(meet_bar, meet_phase, abort_flag, p.status, ST_TIMEOUT_MISC);
      meet_phase ^= 1;
    };
    // ldmatrix rows of this lane: K as [16 keys][16 d] (key blocks outer), V as [16 keys][16 d] (d blocks outer)
    const int mat = lane >> 3, mrow = lane & 7;
    const int k_row = warp * 16 + (mat >> 1) * 8 + mrow, v_row = warp * 16 + (mat & 1) * 8 + mrow;
    const uint32_t k_off = k_row * 128, v_off = v_row * 128;
    int stage = 0;
    uint32_t phase = 0;
    // (one thread) this CTA's draw of a shared head's ticket; true for the last of the head's contributors
    auto draw = [&](unsigned head, unsigned partners) {
      const bool last = atomicAdd(&p.tickets[head], 1u) == partners;
      if (last) p.tickets[head] = 0;  // clean for the next launch
      return last;
    };

    unsigned u = u_begin;  // the tickets of the units before u are drawn
    while (u < u_end && ok) {
      const unsigned head = u / n_tiles, tile0 = u % n_tiles;
      const unsigned tile1 = min(n_tiles, tile0 + (u_end - u));  // this CTA's tiles of the head: [tile0, tile1)

      uint32_t qf[D / 16][4];
      {
        const uint32_t* Q = static_cast<const uint32_t*>(p.Q) + (size_t)head * p.S_q * (D / 2);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = g + (i & 1) * 8, word = kk * 8 + (i >> 1) * 4 + tq;
            qf[kk][i] = row < p.S_q ? __ldg(Q + (size_t)row * (D / 2) + word) : 0u;
          }
      }
      float o[D / 8][4];
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[n][i] = 0.f;
      float m_ref[2] = {-INFINITY, -INFINITY}, l_sum[2] = {0.f, 0.f};  // rows g and g + 8 (l: this lane's columns)

      for (unsigned tile = tile0; tile < tile1; ++tile) {
        if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag, p.status, ST_ATTN_KV)) {
          ok = false;
          break;
        }
        const uint32_t sk = smem_u32(smem + stage * 2 * L::kTile), sv = sk + L::kTile;
        float s[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) s[n][i] = 0.f;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          uint32_t kf[4];
          ldsm4(kf, sk + (kk >> 2) * kBoxBytes + k_off + ((((kk & 3) * 2 + (mat & 1)) ^ mrow) << 4));
          mma16816<BF16>(s[0], qf[kk], kf[0], kf[1]);
          mma16816<BF16>(s[1], qf[kk], kf[2], kf[3]);
        }
        const int key0 = (int)tile * kKeys + warp * 16 + 2 * tq;
        if ((int)(tile + 1) * kKeys > (p.causal ? min(p.S_kv, off + 1) : p.S_kv)) {
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int limit = p.causal ? min(p.S_kv - 1, g + (i >> 1) * 8 + off) : p.S_kv - 1;
              if (key0 + n * 8 + (i & 1) > limit) s[n][i] = -INFINITY;
            }
        }
        float m_new[2];
        bool grow = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float mx = fmaxf(fmaxf(s[0][2 * h], s[0][2 * h + 1]), fmaxf(s[1][2 * h], s[1][2 * h + 1]));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
          m_new[h] = fmaxf(m_ref[h], mx * p.scale_log2);
          grow |= m_new[h] - m_ref[h] > kRescaleThreshold;  // (false while no key has been seen: -inf - -inf)
        }
        if (__any_sync(0xffffffffu, grow)) {
          float f[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            f[h] = m_ref[h] == -INFINITY ? 0.f : ex2f(m_ref[h] - m_new[h]);
            m_ref[h] = m_new[h];
            l_sum[h] *= f[h];
          }
#pragma unroll
          for (int n = 0; n < D / 8; ++n) {
            o[n][0] *= f[0]; o[n][1] *= f[0];
            o[n][2] *= f[1]; o[n][3] *= f[1];
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float neg_m = m_ref[h] == -INFINITY ? 0.f : -m_ref[h];  // a row that sees no key yet: keep it finite
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 2 * h; i < 2 * h + 2; ++i) {
              s[n][i] = ex2f(fmaf(s[n][i], p.scale_log2, neg_m));
              l_sum[h] += s[n][i];
            }
        }
        const uint32_t pf[4] = {pack16<BF16>(s[0][0], s[0][1]), pack16<BF16>(s[0][2], s[0][3]),
                                pack16<BF16>(s[1][0], s[1][1]), pack16<BF16>(s[1][2], s[1][3])};
#pragma unroll
        for (int j = 0; j < D / 16; ++j) {
          uint32_t vf[4];
          ldsm4_trans(vf, sv + (j >> 2) * kBoxBytes + v_off + ((((j & 3) * 2 + (mat >> 1)) ^ mrow) << 4));
          mma16816<BF16>(o[2 * j], pf, vf[0], vf[1]);
          mma16816<BF16>(o[2 * j + 1], pf, vf[2], vf[3]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[stage]);
        if (++stage == L::kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;

      // ---- the four warps' results meet in shared memory
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        l_sum[h] += __shfl_xor_sync(0xffffffffu, l_sum[h], 1);
        l_sum[h] += __shfl_xor_sync(0xffffffffu, l_sum[h], 2);
        if (tq == 0) {
          s_m[warp * kQ + g + 8 * h] = m_ref[h];
          s_l[warp * kQ + g + 8 * h] = l_sum[h];
        }
        // columns in blocks of 8, block index xor row % 4: the half-warp's four rows fall into different banks
        float* row = s_o + (warp * kQ + g + 8 * h) * D + 2 * tq;
#pragma unroll
        for (int n = 0; n < D / 8; ++n)
          *reinterpret_cast<float2*>(row + ((n ^ (g & 3)) << 3)) = make_float2(o[n][2 * h], o[n][2 * h + 1]);
      }
      meet();
      if (!ok) break;
      const bool whole = tile0 == 0 && tile1 == n_tiles;
      // a CTA leaves at most two partials: slot 0 for the head its range begins in, slot 1 for the one it ends in
      float* part = p.partials + ((size_t)blockIdx.x * 2 + (u == u_begin ? 0 : 1)) * kPartialFloats;
      const int words = p.S_q * (D / 4);  // float4 of the head's result
      for (int e = threadIdx.x; e < words; e += kWarps * 32) {
        const int row = e / (D / 4), c4 = e % (D / 4);
        float m = -INFINITY, l = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) m = fmaxf(m, s_m[w * kQ + row]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          const float mw = s_m[w * kQ + row];
          const float f = mw == -INFINITY ? 0.f : ex2f(mw - m);  // (a warp that saw no key of this row holds zeros)
          const float4 v = *reinterpret_cast<const float4*>(s_o + (w * kQ + row) * D + (((c4 >> 1) ^ (row & 3)) << 3) + (c4 & 1) * 4);
          l = fmaf(s_l[w * kQ + row], f, l);
          acc.x = fmaf(v.x, f, acc.x); acc.y = fmaf(v.y, f, acc.y);
          acc.z = fmaf(v.z, f, acc.z); acc.w = fmaf(v.w, f, acc.w);
        }
        if (whole) {
          const float inv = 1.0f / l;
          store4<BF16, OUT_F32>(p.O, ((size_t)head * p.S_q + row) * D + c4 * 4,
                                make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
        } else {
          __stcg(reinterpret_cast<float4*>(part) + e, acc);
          if (c4 == 0) {
            __stcg(part + kQ * D + row, m);
            __stcg(part + kQ * D + kQ + row, l);
          }
        }
      }
      if (!whole) {
        const unsigned h0 = head * n_tiles, partners = p.work.partners(h0, n_tiles), c_first = p.work.worker_of(h0);
        meet();  // the partial is written ...
        if (threadIdx.x == 0) {
          __threadfence();  // ... and visible device-wide before the ticket is taken
          *ticket_word = draw(head, partners) ? 1u : 0u;
        }
        meet();
        if (ok && *ticket_word) {
          __threadfence();
          const int n_contrib = (int)partners + 1;
          // (a contributor whose range begins before the head has it as the head its range ends in)
          auto slot_of = [&](unsigned c) {
            return p.partials + ((size_t)c * 2 + (p.work.start(c) >= h0 ? 0 : 1)) * kPartialFloats;
          };
          // weights of the contributors, eight threads to a row
          const int row = threadIdx.x >> 3, sub = threadIdx.x & 7;
          float* weight = s_o;  // [contributor][16]
          float m = -INFINITY, l = 0.f;
          if (row < p.S_q)
            for (int i = sub; i < n_contrib; i += 8) m = fmaxf(m, __ldcg(slot_of(c_first + i) + kQ * D + row));
#pragma unroll
          for (int x = 4; x > 0; x >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
          if (row < p.S_q)
            for (int i = sub; i < n_contrib; i += 8) {
              const float* s = slot_of(c_first + i) + kQ * D + row;
              const float mc = __ldcg(s);
              const float f = mc == -INFINITY ? 0.f : ex2f(mc - m);
              weight[i * kQ + row] = f;
              l = fmaf(__ldcg(s + kQ), f, l);
            }
#pragma unroll
          for (int x = 4; x > 0; x >>= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
          if (sub == 0) s_l[row] = 1.0f / l;
          meet();
          for (int e = threadIdx.x; e < words && ok; e += kWarps * 32) {
            const int r = e / (D / 4), c4 = e % (D / 4);
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int i = 0; i < n_contrib; ++i) {
              const float4 v = __ldcg(reinterpret_cast<const float4*>(slot_of(c_first + i)) + e);
              const float f = weight[i * kQ + r];
              acc.x = fmaf(v.x, f, acc.x); acc.y = fmaf(v.y, f, acc.y);
              acc.z = fmaf(v.z, f, acc.z); acc.w = fmaf(v.w, f, acc.w);
            }
            const float inv = s_l[r];
            store4<BF16, OUT_F32>(p.O, ((size_t)head * p.S_q + r) * D + c4 * 4,
                                  make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
          }
        }
      }
      meet();  // the reduction area may be written again
      u += tile1 - tile0;
    }
    // what a wait that ran out has left over
    if (threadIdx.x == 0) p.work.draw_owed(u, u_end, n_tiles, draw);
  }

  // ------------------------------------------------------------------ teardown
  if (*abort_flag) {
    unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncthreads();
}

template <bool BF16, int D, bool OUT_F32>
int launch_cfg(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K, const void* V,
               void* O, cudaStream_t s) {
  CUtensorMap tk, tv;
  const int bh = d.B * d.H;
  const uint64_t row_bytes = (uint64_t)D * 2;
  int rc = encode_tmap_3d(ctx, &tk, d.dtype_in, K, D, d.S_kv, bh, row_bytes, row_bytes * d.S_kv, 64, kKeys, 1, true);
  if (!rc) rc = encode_tmap_3d(ctx, &tv, d.dtype_in, V, D, d.S_kv, bh, row_bytes, row_bytes * d.S_kv, 64, kKeys, 1, true);
  if (rc) {
    ctx->last_cuda = rc;
    return FRISK_B200_E_CUDA;
  }
  auto kern = attention_decode_kernel<BF16, D, OUT_F32>;
  using L = DecSmem<D>;
  static PerDeviceOnce opt_in;
  if (opt_in(ctx->device, [&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal) == cudaSuccess ? 0 : 1;
      }))
    return FRISK_B200_E_CUDA;
  DecParams p;
  p.Q = Q;
  p.O = O;
  p.S_q = d.S_q;
  p.S_kv = d.S_kv;
  p.causal = d.causal ? 1 : 0;
  p.n_tiles = (d.S_kv + kKeys - 1) / kKeys;
  p.scale_log2 = d.scale * 1.4426950408889634f;
  const unsigned units = (unsigned)bh * (unsigned)p.n_tiles;  // < 2^31 (attention_decode_preferred)
  const unsigned grid = std::min<unsigned>(units, (unsigned)std::min(ctx->num_sms, kNumSMsDefault));
  p.work.q = units / grid;
  p.work.r = units % grid;
  p.tickets = static_cast<unsigned*>(ctx->attn_scratch);
  p.partials = reinterpret_cast<float*>(static_cast<unsigned char*>(ctx->attn_scratch) + kTicketBytes);
  p.status = ctx->d_status;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // the kernel waits (griddepcontrol.wait) itself
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, tk, tv, p));
  return 0;
}

template <bool BF16, int D>
int launch_out(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K, const void* V,
               void* O, cudaStream_t s) {
  return d.dtype_out == FRISK_B200_F32 ? launch_cfg<BF16, D, true>(ctx, d, Q, K, V, O, s)
                                       : launch_cfg<BF16, D, false>(ctx, d, Q, K, V, O, s);
}

}  // namespace

size_t attention_decode_scratch_bytes() {
  return kTicketBytes + (size_t)kNumSMsDefault * 2 * kPartialFloats * sizeof(float);
}
size_t attention_decode_ticket_bytes() { return kTicketBytes; }

// Up to 16 queries the padded query tile of the two-tile kernel does at least eight times the work; the normalised
// mode needs the complete row sum before it rounds and stays there.
bool attention_decode_preferred(const frisk_b200_attn_desc& d) {
  const int64_t bh = (int64_t)d.B * d.H;
  return d.S_q <= kQ && !d.normalize_p && bh <= kMaxHeads && bh * ((d.S_kv + kKeys - 1) / kKeys) <= INT32_MAX;
}

int launch_attention_decode(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K,
                            const void* V, void* O, cudaStream_t s) {
  const bool bf = d.dtype_in == FRISK_B200_BF16;
  if (d.D == 128) return bf ? launch_out<true, 128>(ctx, d, Q, K, V, O, s) : launch_out<false, 128>(ctx, d, Q, K, V, O, s);
  if (d.D == 64) return bf ? launch_out<true, 64>(ctx, d, Q, K, V, O, s) : launch_out<false, 64>(ctx, d, Q, K, V, O, s);
  return FRISK_B200_E_ATTN_SHAPE;
}

}  // namespace fb
