// Fused attention forward for sm_100a: O = softmax(scale * Q.K^T [+ causal mask]) . V over
// compact BHSD tensors, fp16/bf16 inputs, fp32 scores and statistics, probabilities rounded to
// the 16-bit input type before P.V.  Numerics contract:
// benchmark/layout/execution/tiled_attention.py:392,505-515,628-629 (scale applied to the fp32
// dot, exp through ex2, P rounded RNE before P.V, fp32 accumulation of P.V); launch contract:
// tiled_attention.py:52-61 (compact BHSD, q/k/v/out pointers).
//
// Unlike the reference's three-pass schedule (tiled_attention.py:697-698) this is a single
// pass with an online softmax, so K and V are read once per query tile:
//
//   * the kernel is persistent: one CTA per SM takes work items from an atomic counter, heavy items first, until none is
//     left.  An item is TWO 128-row query tiles, of one (batch, head) or of two, each with a softmax group and an MMA thread of
//     its own, or ONE (items_estimate, below), whose key tiles the two groups share out (kSplit) or group 0 takes alone.
//     Barriers, tensor memory and the K/V ring live across items, so the next item's Q, K and V are already on their
//     way, and its first scores are computed, while the softmax warps still store the last item's O;
//   * key tiles are 64 keys, and every query tile has two buffers of scores: S of tile b + 2 follows P(b).V on the tensor core
//     while the softmax group works on tile b + 1, whose scores are there.  With one buffer of 128 keys every tile waited for the
//     chain P -> P.V -> next S -> softmax.  An MMA of S takes 49 clk for 64 keys and 65 for 128 (it
//     reads Q's rows from shared memory either way): 1240 clk for both query tiles' step of 64 keys, as measured with the softmax
//     left out, against 1050, the price;
//   * K and V stream through a TMA ring of 4 stages, each what one step of the MMA threads takes;
//   * warp 8 is the TMA producer; warps 9 and 10 issue the tcgen05.mma of softmax group 0 and 1: S_q =
//     Q_q.K^T (SS form, both operands K-major, 128-byte swizzle) into tensor memory and O_q += P_q.V
//     (P read from tensor memory, V as an MN-major shared-memory operand);
//   * warps 0-3 and 4-7 are the two softmax groups: thread r owns row r of its query tile
//     (TMEM lane r), so row max / row sum need no shuffles.  They work freely, one filling the gaps of the other;
//   * the running maximum is applied lazily: O is rescaled in tensor memory only when the
//     maximum grew by more than 2^8, which keeps P within bf16/fp16 range and makes most
//     iterations rescale-free;
//   * causal: key tiles wholly above the diagonal are never loaded; only tiles that touch the
//     diagonal (or the ragged end of the keys) are masked.
// TMEM columns: S0 [0,64) and [64,128), S1 [128,192) and [192,256), O0 [256,256+D) O1 [384,384+D); P_q of a key tile
// aliases the first 32 columns of its scores (two 16-bit values per column).
//
// What bounds it: 8 x 32 heads x 4096 causal at D = 128 (1050 us, 1120 with 128-key tiles, one buffer and softmax groups in
// turn) the power limit, at which it runs at 1.5 instead of 1.7 GHz; short runs the softmax groups, 1700 clk for a step of both
// where the exponentials take 1024 and the MMAs 1240.
// Every mbarrier wait is bounded (ptx.cuh); no TMA load uses cluster multicast.
#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "ptx.cuh"

#include "attention_common.cuh"

namespace fb {
namespace {
using namespace attn;

constexpr int BN = 64;  // keys per K/V tile

// number of key tiles query tile `m0` needs
__device__ __forceinline__ int kv_tiles_for(int m0, int S_q, int S_kv, int causal) {
  if (m0 >= S_q) return 0;
  int all = (S_kv + BN - 1) / BN;
  if (!causal) return all;
  int last_key = min(S_kv - 1, m0 + BM - 1 + (S_kv - S_q));  // visible to the tile's last row
  return min(all, last_key / BN + 1);
}

constexpr int kHeadChunk = 16;  // heads whose K and V are worked on together (they stay in L2: 16 x 2 MB at S = 4096)
template <int D>
struct AttnSmem {
  static constexpr int kTileBytes = BM * D * 2;        // one Q tile
  static constexpr int kKvBytes = BN * D * 2;          // one K or V tile
  static constexpr int kStagesKV = 4;                  // of the K/V ring; two may belong to either MMA thread
  static constexpr int kQ = 0;                         // Q0, Q1
  static constexpr int kStageBytes = 2 * kKvBytes;     // a K tile, then a V tile
  static constexpr int kKV = 2 * kTileBytes;           // the ring
  static constexpr int kBar = kKV + kStagesKV * kStageBytes;
  // 16-bit outputs: one [32 rows][128 bytes] box per softmax warp for the TMA stores of O, 1024-byte aligned
  static constexpr int kOut = kBar + 1024;
  static constexpr int kTotal = kOut + 8 * (32 * 128) + 1024;
  static_assert(kTotal <= 232448, "the output boxes must fit next to the Q, K and V tiles");
};


// What the two softmax groups (and MMA threads) make of a work item
enum Mode {
  kPair,   // two query tiles of one head, which share the K and V tiles
  kSplit,  // ONE query tile, whose key tiles they take in turn, even and odd ones, each with its own S, P, O and statistics; at the
           // end the halves are put together
  kTwin    // two heads of one query tile each, with K and V of their own
};

template <bool BF16, int D, bool OUT_F32, bool NORM, Mode MODE>
__global__ void __launch_bounds__(kThreads, 1)
    attention_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                         const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o,
                         const AttnParams p) {
  constexpr bool SPLIT = MODE == kSplit, TWIN = MODE == kTwin;
  constexpr bool OWN_KV = MODE != kPair;  // each MMA thread has key tiles, and stages of the ring, of its own
  using L = AttnSmem<D>;
  constexpr int kBoxes = D / 64;            // 64-element (128-byte) column blocks per tile
  constexpr int kBoxBytes = BM * 128;       // one [128 rows][128 B] block of Q
  constexpr int kKvBoxBytes = BN * 128;     // one [64 keys][128 B] block of K or V
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* q_full = bars;              // [1]
  uint64_t* q_empty = bars + 1;         // [1] both MMA threads are done with the Q tiles
  uint64_t* kv_full = bars + 2;         // [4]
  uint64_t* kv_empty = bars + 6;        // [4]
  uint64_t* s_full = bars + 10;         // [2 groups][2 buffers] the scores of a key tile are complete
  uint64_t* p_ready = bars + 14;        // [2 groups][2 buffers] its probabilities are written (statistics pass: the scores read)
  uint64_t* o_done = bars + 18;         // [2 groups][2] of an item all P.V but the last, all P.V are complete
  uint64_t* item_full = bars + 22;      // [2] the producer has published the id of a work item
  uint64_t* item_empty = bars + 24;     // [2] every consumer has read it
  uint64_t* turn = bars + 26;           // [2] the MMA threads issue in turn
  uint64_t* xchg = bars + 28;           // [1] the two softmax groups meet (SPLIT only)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 29);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile int* item_slot = reinterpret_cast<volatile int*>(tmem_slot + 2);  // [2]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Work items in the order they are handed out: heads in chunks of kHeadChunk (their K and V stay in L2
  // together); inside a chunk the heavy (late) query tiles of every head first, so that the machine
  // drains on light items.
  struct Item {
    int bh, m0;
    int nq[2];  // key tiles of softmax group 0 and 1
    int n_max;  // key tiles that are loaded
  };
  const int bh_total = (int)(p.total_items / p.n_groups);
  auto decode = [&](int t) {
    const int per_chunk = kHeadChunk * p.n_groups;
    const int chunk = t / per_chunk;
    const int within = t - chunk * per_chunk;
    const int heads_here = min(kHeadChunk, bh_total - chunk * kHeadChunk);
    const int group = p.n_groups - 1 - within / heads_here;
    Item it;
    if (TWIN) {
      it.bh = 2 * t;
      it.m0 = 0;
      it.nq[0] = it.n_max = kv_tiles_for(0, p.S_q, p.S_kv, p.causal);
      it.nq[1] = it.bh + 1 < p.heads ? it.nq[0] : 0;
      return it;
    }
    it.bh = chunk * kHeadChunk + within % heads_here;
    it.m0 = group * p.group_rows;
    const int n0 = kv_tiles_for(it.m0, p.S_q, p.S_kv, p.causal);
    if (SPLIT) {
      it.nq[0] = (n0 + 1) / 2;
      it.nq[1] = n0 / 2;
      it.n_max = n0;
    } else {
      it.nq[0] = n0;
      it.nq[1] = p.group_rows > BM ? kv_tiles_for(it.m0 + BM, p.S_q, p.S_kv, p.causal) : 0;
      it.n_max = max(it.nq[0], it.nq[1]);
    }
    return it;
  };
  // Consumers (the two MMA threads, the softmax warps) learn the n-th item of this CTA from the producer:
  // returns its id, or -1 when the work has run out or a wait was abandoned.  The slot is written again once the warp's one arrival
  // is in, so no lane may read it after that: lane 0 reads it for the warp, or all lanes before the arrival.  The latter is compiled into
  // faster loops for the normalised mode (16 heads x 1025 22.1 against 22.4 us), the former for the others (split keys, 4 heads x 4096 at
  // D = 64 33.1 against 35.1, causal at D = 128 32.6 against 33.4).
  auto next_item = [&](int n) -> int {
    int t = -1;
    if (NORM) {
      if (!mbar_wait_warp(&item_full[n & 1], (n >> 1) & 1, abort_flag, p.status, ST_ATTN_Q)) return -1;
      t = item_slot[n & 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(&item_empty[n & 1]);
      return t;
    }
    if (lane == 0 && mbar_wait(&item_full[n & 1], (n >> 1) & 1, abort_flag, p.status, ST_ATTN_Q)) {
      t = item_slot[n & 1];
      mbar_arrive(&item_empty[n & 1]);
    }
    return __shfl_sync(0xffffffffu, t, 0);
  };
  // The ring of K and V.  What an MMA thread takes in one step, the V of key tile b and the K of tile b + 2, makes a stage: one
  // barrier to wait for and one to release (each costs the thread about a hundred clocks).  The n-th goes to stage n % kStages, and
  // both MMA threads follow all of them.  OWN_KV: two stages belong to either MMA thread and n counts that thread's,
  // because a thread that does not follow all uses of a stage can mistake an earlier phase of its barrier for its own.
  constexpr int kStages = L::kStagesKV, kOwnStages = OWN_KV ? kStages / 2 : kStages;
  auto ring_stage = [](int n, int group) -> int { return (OWN_KV ? group * kOwnStages : 0) + n % kOwnStages; };
  auto ring_phase = [](int n) -> uint32_t { return (n / kOwnStages) & 1; };
  // Normalised mode runs the key loop twice: pass 0 only gathers row maxima and row sums, pass 1
  // is the pass every mode has.  Barrier phases keep counting across passes and items.
  constexpr int first_pass = NORM ? 0 : 1;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], OWN_KV ? 1 : 2);  // one arrival per MMA-issuing thread that reads the stage
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 128);
      mbar_init(&o_done[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&turn[i], 1);
      mbar_init(&item_full[i], 1);
      mbar_init(&item_empty[i], 10);  // two MMA threads, one lane of each of the eight softmax warps
    }
    mbar_init(q_empty, 2);
    mbar_init(xchg, 256);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
  }
  if (warp == kWarpMma) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // Launched with programmatic stream serialization: the set-up above may run while the kernel in front of this one
  // drains; nothing touches global memory (the operands, the work counter) before that kernel is complete.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // the TMA/MMA warpgroup hands registers to the two softmax warpgroups (a full row of S per thread)
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
  if (warp == kWarpTma) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int loaded[2] = {0, 0};  // stages filled so far, over all items; OWN_KV: for either MMA thread
      bool ok = true;
      for (int n = 0; ok; ++n) {
        // take the next item and tell the other roles (slot n & 1 was last used by item n - 2)
        if (n >= 2 && !mbar_wait(&item_empty[n & 1], ((n >> 1) & 1) ^ 1, abort_flag, p.status, ST_ATTN_Q)) break;
        int t = (int)atomicAdd(p.work, 1u);
        if (t >= (int)p.total_items) t = -1;
        item_slot[n & 1] = t;
        mbar_arrive(&item_full[n & 1]);
        if (t < 0) break;
        const Item it = decode(t);
        // the Q tiles of the item before are free when both MMA threads have issued their last S of it
        if (n > 0 && !mbar_wait(q_empty, (n - 1) & 1, abort_flag, p.status, ST_ATTN_Q)) break;
        const int q_tiles = it.nq[1] > 0 && !SPLIT ? 2 : 1;  // (no query reads the second tile's place where there is none)
        mbar_expect_tx(q_full, q_tiles * L::kTileBytes);
        for (int q = 0; q < q_tiles; ++q)
#pragma unroll
          for (int b = 0; b < kBoxes; ++b)
            tma_load_3d(smem + L::kQ + q * L::kTileBytes + b * kBoxBytes, &tmap_q, q_full, b * 64, TWIN ? 0 : it.m0 + q * BM,
                        it.bh + (TWIN ? q : 0));
        for (int pass = first_pass; pass < 2 && ok; ++pass) {
          const int n_keys = OWN_KV ? it.nq[0] : it.n_max;  // (group 0 has no fewer key tiles than group 1)
          for (int b = -2; b < n_keys && ok; ++b) {
#pragma unroll
            for (int g = 0; g < (OWN_KV ? 2 : 1); ++g) {
              const int n_mine = OWN_KV ? it.nq[g] : it.n_max, bh = it.bh + (TWIN ? g : 0);
              const bool has_k = b + 2 < n_mine, has_v = pass == 1 && b >= 0 && b < n_mine;  // (statistics need no values)
              if (!ok || !(has_k || has_v)) continue;
              const int st = ring_stage(loaded[g], g);
              ok = mbar_wait(&kv_empty[st], ring_phase(loaded[g]) ^ 1, abort_flag, p.status, ST_ATTN_KV);
              if (!ok) continue;
              ++loaded[g];
              mbar_expect_tx(&kv_full[st], (has_k && has_v ? 2 : 1) * L::kKvBytes);
              unsigned char* at = smem + L::kKV + st * L::kStageBytes;
#pragma unroll
              for (int x = 0; x < kBoxes; ++x) {
                if (has_k)
                  tma_load_3d(at + x * kKvBoxBytes, &tmap_k, &kv_full[st], x * 64, (SPLIT ? 2 * (b + 2) + g : b + 2) * BN, bh);
                if (has_v)
                  tma_load_3d(at + L::kKvBytes + x * kKvBoxBytes, &tmap_v, &kv_full[st], x * 64, (SPLIT ? 2 * b + g : b) * BN, bh);
              }
            }
          }
        }
      }
    }
  } else if (warp == kWarpMma || warp == kWarpMma + 1) {
    // ------------------------------------------------------------------ MMA issuers, one warp per query tile
    // tcgen05 operations of ONE thread execute in issue order, which is all the ordering a query tile needs: S_q(b + 2) overwrites
    // P_q(b) after P_q(b).V(b) has read it.  The tensor core queues only a few MMAs, so an issuing thread is busy for as long as
    // its MMAs run and everything else it does (a wait or a commit costs 100 clk or more, ~500 a step) leaves the pipe idle,
    // unless the other thread issues meanwhile.  Two threads that issue freely fall into step, MMA by MMA, and do everything
    // else at the same time too: 1840 clk a step.  So they issue in turn (1240 clk where the softmax is left out), and there
    // is little else to do: one wait for P and the stage of the ring, two commits.  The loop is run by whole warps, so that
    // descriptors and counters are uniform; one elected lane issues.
    const int mq = __shfl_sync(0xffffffffu, warp - kWarpMma, 0);
    constexpr uint32_t idesc_s = umma_idesc_f16(BM, BN, BF16, false, false);
    constexpr uint32_t idesc_o = umma_idesc_f16(BM, D, BF16, false, true);
    // descriptors differ only in the start address
    const uint64_t dq = umma_desc_kmajor_sw128(smem_u32(smem + L::kQ) + (SPLIT ? 0 : mq * L::kTileBytes));
    const uint64_t dk = umma_desc_kmajor_sw128(smem_u32(smem + L::kKV));
    const uint64_t dv = umma_desc_mnmajor_sw128(smem_u32(smem + L::kKV + L::kKvBytes), kKvBoxBytes, 1024);
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t t_sq = tmem + mq * 128;        // the two buffers of S_q, 64 columns each
    const uint32_t t_oq = tmem + 256 + mq * 128;  // O_q
    int turns = 0;     // steps in turn so far, over all items
    int taken = 0;     // stages of the ring followed so far, over all items
    int begun = 0;     // S_q begun so far, over all items: its buffer
    int finished = 0;  // P_q taken so far, over all items: its buffer and the phase of p_ready
    bool ok = true;
    for (int n = 0; ok; ++n) {
      const int t = next_item(n);
      if (t < 0) break;
      const Item it = decode(t);
      const int n_mine = it.nq[mq], n_max = OWN_KV ? n_mine : it.n_max;  // key tiles: used, followed
      const int n_steps = OWN_KV ? it.nq[0] : it.n_max;  // the same for both MMA threads
      const bool in_turn = it.nq[1] > 0;                // a lone thread issues as it comes
      ok = mbar_wait_warp(q_full, n & 1, abort_flag, p.status, ST_ATTN_Q);
      for (int pass = first_pass; pass < 2 && ok; ++pass) {
        const bool stats_pass = pass == 0;  // the pass that only gathers statistics issues no P.V
        // S runs two key tiles ahead of P.V: the scores of tile b + 1 are complete (or on their way) while the softmax
        // group works on tile b, and those of tile b + 2 take their place as soon as P(b).V has read P(b) there.
        for (int b = -2; b < n_steps && ok; ++b) {
          const bool staged = b + 2 < n_max || (!stats_pass && b >= 0 && b < n_max);  // a stage of the ring comes with this step
          const bool use_p = b >= 0 && b < n_mine, use_s = b + 2 < n_mine;
          const int st = ring_stage(taken, mq), buf = finished & 1;
          uint64_t* const p_bar = &p_ready[2 * mq + buf];
          if (use_p && staged)
            ok = mbar_wait_both(p_bar, (finished >> 1) & 1, &kv_full[st], ring_phase(taken), abort_flag, p.status, ST_ATTN_P,
                                ST_ATTN_KV);
          else if (use_p)
            ok = mbar_wait(p_bar, (finished >> 1) & 1, abort_flag, p.status, ST_ATTN_P);
          else if (staged)
            ok = mbar_wait(&kv_full[st], ring_phase(taken), abort_flag, p.status, ST_ATTN_KV);
          if (ok && in_turn) ok = mbar_wait(&turn[mq], (turns & 1) ^ (mq ^ 1), abort_flag, p.status, ST_ATTN_S);
          turns += in_turn;
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t at = static_cast<uint64_t>((st * L::kStageBytes) >> 4);
          if (use_p) {
            ++finished;
            if (!stats_pass && elect_one()) {
#pragma unroll
              for (int kk = 0; kk < BN / 16; ++kk)
                umma_f16_ts(t_oq, t_sq + buf * BN + kk * 8, dv + at + static_cast<uint64_t>((kk * 2048) >> 4), idesc_o,
                            (b > 0 || kk > 0) ? 1u : 0u);
            }
          }
          if (use_s) {
            const int s_buf = begun & 1;
            ++begun;
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < D / 16; ++kk)
                umma_f16_ss(t_sq + s_buf * BN, dq + static_cast<uint64_t>(((kk / 4) * kBoxBytes + (kk % 4) * 32) >> 4),
                            dk + at + static_cast<uint64_t>(((kk / 4) * kKvBoxBytes + (kk % 4) * 32) >> 4), idesc_s, kk != 0);
              if (in_turn) mbar_arrive(&turn[mq ^ 1]);
              umma_commit(&s_full[2 * mq + s_buf]);
              if (pass == 1 && b + 2 == n_mine - 1) umma_commit(q_empty);  // this thread's last use of the Q tiles
            }
          } else if (in_turn && elect_one()) {
            mbar_arrive(&turn[mq ^ 1]);
          }
          if (use_p && !stats_pass && b >= n_mine - 2 && elect_one()) umma_commit(&o_done[2 * mq + (b == n_mine - 1)]);
          if (staged) {
            // this thread's use of the stage ends when these MMAs have read it
            if (elect_one()) {
              if (use_p || use_s) umma_commit(&kv_empty[st]); else mbar_arrive(&kv_empty[st]);
            }
            ++taken;
          }
        }
      }
      if (ok && n_mine == 0 && lane == 0) mbar_arrive(q_empty);  // (a query tile beyond the end of the sequence)
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    // ------------------------------------------------------------------ softmax groups
    const int q = warp >> 2;         // this group: its query tile, or its share of the key tiles
    const int quad = warp & 3;       // TMEM lane quadrant this warp may touch
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = tmem_base + q * 128 + lane_addr;
    const uint32_t t_o = tmem_base + 256 + q * 128 + lane_addr;
    const int off = p.S_kv - p.S_q;
    int steps = 0;    // (pass, key tile) steps of this group so far, over all items: buffer and phase of s_full
    int ends[2] = {0, 0};  // items with two key tiles or more, with one or more so far: the phases of o_done
    int meets = 0;    // meetings of the two groups so far: the phase of xchg
    bool ok = true;
    // Waits of this lane that have not run out.  A vote of its own on every wait for scores costs the single pass 0.7 % (8 x 32 x 4096
    // causal) to 3 % (150 x 2586).  So a lane whose wait has run out goes on with what it finds until the warp votes on whether to
    // rescale, for every key tile.  Split keys at D = 64 have such a vote for the waits at the end of an item too, before O is read
    // (16 heads x 1025 14.2 -> 14.0 us, 12 x 2048 causal 18.9 -> 18.7); at D = 128 each of those waits is voted on, which is as fast.
    bool there = true;
    constexpr bool END_VOTE = SPLIT && D == 64;
    // Split keys: the two groups meet, and each thread learns what the other group's thread of its row brings.  The
    // statistics lie in the second query tile's place, which nothing else uses then, in two sets that alternate: a set is
    // written again only when everybody has arrived at the meeting in between, after reading it.
    auto meet = [&](float2 mine_v) -> float2 {
      float2* set = reinterpret_cast<float2*>(smem + L::kQ + L::kTileBytes) + (meets & 1) * 2 * BM;
      set[q * BM + row] = mine_v;
      tc_fence_before_sync();
      mbar_arrive(xchg);
      if (END_VOTE)
        there &= mbar_wait(xchg, meets & 1, abort_flag, p.status, ST_ATTN_O);
      else if (!mbar_wait_warp(xchg, meets & 1, abort_flag, p.status, ST_ATTN_O))
        ok = false;
      ++meets;
      tc_fence_after_sync();
      return set[(q ^ 1) * BM + row];
    };

    for (int n = 0; ok; ++n) {
      const int item_id = next_item(n);
      if (item_id < 0) break;
      const Item it = decode(item_id);
      const int bh = it.bh + (TWIN ? q : 0);
      const int n_tiles = it.nq[q];
      const int m_tile = it.m0 + (MODE == kPair ? q * BM : 0);
      // (only END_VOTE carries it on to the next item; said so, the loops are faster here, 12 x 2048 at D = 64 33.9 -> 33.5 us, and slower
      // elsewhere: 24 x 1000 at D = 128 21.9 -> 22.1)
      if (SPLIT ? D == 128 : D == 64) there = true;
      // (both groups have read both O of the item before)
      if (SPLIT && n > 0) meet(make_float2(0.f, 0.f));
      const int g_row = m_tile + row;  // query index within the head
      float m_ref = -INFINITY;  // reference maximum (scaled, log2 units) the stored P and O are relative to
      float l_sum = 0.f;

      uint32_t sr[2][32];  // the scores of a key tile
      auto load_scores = [&]() {  // of step `steps`
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < 2; ++c) tmem_ld_32x32b_x32(t_s + (steps & 1) * BN + c * 32, sr[c]);
      };
      auto scores_there = [&](bool more) -> bool {  // (the vote is taken in any case: behind a branch on `more` the loop is 13 % slower)
        return __all_sync(0xffffffffu, more && mbar_test(&s_full[2 * q + (steps & 1)], (steps >> 1) & 1));
      };
      auto wait_scores = [&]() {
        if (NORM) {
          if (ok) ok = mbar_wait_warp(&s_full[2 * q + (steps & 1)], (steps >> 1) & 1, abort_flag, p.status, ST_ATTN_S);
          if (!ok) return;
        } else {
          there = mbar_wait(&s_full[2 * q + (steps & 1)], (steps >> 1) & 1, abort_flag, p.status, ST_ATTN_S);
        }
        load_scores();
      };
      auto mask_scores = [&](int n0) {  // of keys n0..
        if ((n0 + BN > p.S_kv) || (p.causal && (n0 + BN - 1 > m_tile + off))) {
          int limit = p.S_kv - 1;
          if (p.causal) limit = min(limit, g_row + off);
          limit -= n0;  // columns > limit are hidden
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i > limit) sr[c][i] = 0xff800000u;  // -inf
        }
      };
      auto row_max = [&](float (&m)[4]) {  // in four chains
#pragma unroll
        for (int e = 0; e < 16; ++e)
#pragma unroll
          for (int c = 0; c < 2; ++c)
            m[2 * c + (e & 1)] = max3f(m[2 * c + (e & 1)], __uint_as_float(sr[c][2 * e]), __uint_as_float(sr[c][2 * e + 1]));
      };

      if (NORM) {
        // The reference's semantics (benchmark/layout/execution/tiled_attention.py:697-698,
        // tail_attention_reference.py:74-78): score = fp32(dot) * scale; subtract the maximum of the
        // WHOLE row; e = ex2((score - max) * log2e); p = e / (sum of e over the whole row), IEEE
        // division; p rounded to 16 bits; then P.V.  Pass 0 finds max and sum, pass 1 forms P.
        // The row of a key tile is worked on in packed pairs without branches: an IEEE division per element
        // (__fdiv_rn branches) made this mode latency-bound, 16 heads x 1025 rows x D 64 took 154 us, 31 so.
        const float kLog2e = 1.44269504088896340736f;
        const float2 scale2 = make_float2(p.scale, p.scale), log2e2 = make_float2(kLog2e, kLog2e);
        auto exp2_of = [](float x) { return BF16 ? ex2f_ieee_range(x) : ex2f(x); };
        float m_run = -INFINITY, l_run = 0.f;
        for (int pass = 0; pass < 2 && ok; ++pass) {
          if (SPLIT && pass == 1) {
            // the other group's half of the keys
            const float2 o = meet(make_float2(m_run, l_run));
            const float m_all = fmaxf(m_run, o.x);
            auto share = [&](float m, float l) {
              return m == -INFINITY ? 0.f : l * ex2f_ieee_range(__fmul_rn(__fsub_rn(m, m_all), kLog2e));
            };
            const float a = share(m_run, l_run), b = share(o.x, o.y);
            l_run = a + b;
            m_run = m_all;
            if (END_VOTE && !__all_sync(0xffffffffu, there)) ok = false;
            if (!ok) break;
          }
          const float inv_l = __frcp_rn(l_run);  // (of use in pass 1 only)
          const float2 inv2 = make_float2(inv_l, inv_l), negl2 = make_float2(-l_run, -l_run);
          for (int i = 0; i < n_tiles; ++i) {
            const int buf = steps & 1;
            wait_scores();
            if (!ok) break;
            ++steps;
            tmem_ld_wait();
            if (pass == 0) {
              // the scores are in registers: the MMA warp may overwrite them
              tc_fence_before_sync();
              mbar_arrive(&p_ready[2 * q + buf]);
            }
            mask_scores((SPLIT ? 2 * i + q : i) * BN);
            // (score - m) * log2e of a pair, rounded step by step; the scale is positive, so it keeps the order and
            // the maximum of the scaled scores is the scaled maximum
            auto arg2 = [&](int c, int i, float2 negm2) {
              const float2 s2 = make_float2(__uint_as_float(sr[c][2 * i]), __uint_as_float(sr[c][2 * i + 1]));
              return mul2_rn(add2_rn(mul2_rn(s2, scale2), negm2), log2e2);
            };
            if (pass == 0) {
              float mxc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
              row_max(mxc);
              const float mx = __fmul_rn(max3f(mxc[0], mxc[1], fmaxf(mxc[2], mxc[3])), p.scale);
              const float m_new = fmaxf(m_run, mx);
              if (m_new != -INFINITY) {
                const float2 negm2 = make_float2(-m_new, -m_new);
                float2 sum[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) sum[c] = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 16; ++i)
#pragma unroll
                  for (int c = 0; c < 2; ++c) {
                    const float2 x = arg2(c, i, negm2);
                    sum[2 * c + (i & 1)] = add2_rn(sum[2 * c + (i & 1)], make_float2(exp2_of(x.x), exp2_of(x.y)));
                  }
                const float2 all = add2_rn(add2_rn(sum[0], sum[1]), add2_rn(sum[2], sum[3]));
                const float carry = (m_run == -INFINITY) ? 0.f : l_run * ex2f_ieee_range(__fmul_rn(__fsub_rn(m_run, m_new), kLog2e));
                l_run = carry + (all.x + all.y);
                m_run = m_new;
              }
            } else {
              const float2 negm2 = make_float2(-m_run, -m_run);
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  const float2 x = arg2(c, i, negm2);
                  const float2 pv = div2_by(make_float2(exp2_of(x.x), exp2_of(x.y)), negl2, inv2);
                  pk[i] = pack16<BF16>(pv.x, pv.y);
                }
                tmem_st_32x32b_x16(t_s + buf * BN + c * 16, pk);
              }
              tmem_st_wait();
              tc_fence_before_sync();
              mbar_arrive(&p_ready[2 * q + buf]);
            }
          }
        }
        l_sum = 1.0f;  // P is already normalised
        m_ref = 0.f;
      } else {
      // The scores of a key tile are read as soon as those of the tile before are used up, if they are there by then (usually
      // they are), and else after that tile's P has been handed over.
      if (n_tiles > 0) {
        // The first reference is the maximum of two key tiles: more rows then have their largest probability at 1, which loses
        // nothing when it is rounded (2.10e-3 from 64 bits at 8 x 32 x 4096; with one key tile's 2.11e-3).
        float mx = -INFINITY;
        for (int t = 0; t < min(n_tiles, 2); ++t) {
          const int n0 = (SPLIT ? 2 * t + q : t) * BN, step = steps + t;
          there &= mbar_wait(&s_full[2 * q + (step & 1)], (step >> 1) & 1, abort_flag, p.status, ST_ATTN_S);
          tc_fence_after_sync();
#pragma unroll
          for (int c = 0; c < 2; ++c) tmem_ld_32x32b_x32(t_s + (step & 1) * BN + c * 32, sr[c]);
          tmem_ld_wait();
          mask_scores(n0);
#pragma unroll
          for (int e = 0; e < 32; ++e) mx = max3f(mx, __uint_as_float(sr[0][e]), __uint_as_float(sr[1][e]));
        }
        // A row that has seen no key, or only scores of -inf: the lowest finite reference, so that its exponentials are 0 and the
        // first finite score moves it (0 would let lower scores vanish; a group's first key tiles may be any row's -inf).
        m_ref = fmaxf(mx * p.scale_log2, -FLT_MAX);
        // The groups begin a CTA's first item at the same time, and two that work in step leave the special-function unit idle
        // together between their key tiles.  So at D = 64 and with split keys group 1 begins later, by about a third of its work on a
        // tile.  (Later items begin as far apart as the ones before ended; where tiles are short and equally many it pays for every item.)
        // Without and with: 12 x 2048 34.1 and 33.1 us, 16 x 1025 14.6 and 13.8, 48 x 300 against 1024 keys 13.9 and 13.1, 150 x 2586 404
        // and 398, 132 x 1075 causal 59.2 and 59.3; split at D = 128, 4 x 4096 37.6 and 36.6, causal 32.9 and 32.6, 2 x 8192 causal 58.1
        // and 57.8.  Pairs at D = 128 it costs more than it gives (8 x 8192 261 and 268, causal 137.5 and 140, 62 x 6308 causal 599 and
        // 605), and two heads an item (512 x 128 against 256 15.75 and 16.05).
        if ((SPLIT || (D == 64 && !TWIN)) && q == 1 && n_tiles > 3 && (n == 0 || (D == 64 && !p.causal))) {
          const long long from = clock64();
          while (clock64() - from < 300) {
          }
        }
        __syncwarp();
        load_scores();
      }
      for (int i = 0; i < n_tiles && ok; ++i) {
        const int buf = steps & 1;
        ++steps;
        tmem_ld_wait();
        mask_scores((SPLIT ? 2 * i + q : i) * BN);
        const bool more = i + 1 < n_tiles;
        const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
        float mxc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // four chains of the row maximum
        // Takes the row maximum into the reference.  O is rescaled only when the maximum grew by more than the threshold: rare.
        auto settle = [&]() {
          const float mx = max3f(mxc[0], mxc[1], fmaxf(mxc[2], mxc[3]));
          const float m_new = fmaxf(m_ref, mx * p.scale_log2);
          // (warp-uniform decision because the TMEM accesses are warp-collective)
          if (!__any_sync(0xffffffffu, !there || m_new - m_ref > kRescaleThreshold)) return;
          ok = __all_sync(0xffffffffu, there);
          if (!ok) return;
          const float factor = ex2f(m_ref - m_new);
          m_ref = m_new;
          l_sum *= factor;
          // O_q must be complete up to the key tile before this one before it is scaled
          // (the scores of the next key tile come after that product)
          ok = i + 1 < n_tiles ? mbar_wait_warp(&s_full[2 * q + (buf ^ 1)], (steps >> 1) & 1, abort_flag, p.status, ST_ATTN_S)
                               : mbar_wait_warp(&o_done[2 * q], ends[0] & 1, abort_flag, p.status, ST_ATTN_O);
          if (!ok) return;
          tc_fence_after_sync();
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(t_o + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * factor);
            tmem_st_32x32b_x32(t_o + c * 32, o);
          }
        };
        row_max(mxc);
        settle();
        if (!ok) break;
        // P = 2^(s*scale_log2 - m_ref) with packed fp32 FMAs, row sum in fp32, P rounded to 16 bits.  The two 32-key halves are
        // interleaved pair by pair so that the special-function unit always has independent work.
        uint32_t pk0[16], pk1[16];
        const float2 negm2 = make_float2(-m_ref, -m_ref);
        float2 sa = make_float2(0.f, 0.f), sb = make_float2(0.f, 0.f);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float2 xa = fma2(make_float2(__uint_as_float(sr[0][2 * e]), __uint_as_float(sr[0][2 * e + 1])), scale2, negm2);
          const float2 xb = fma2(make_float2(__uint_as_float(sr[1][2 * e]), __uint_as_float(sr[1][2 * e + 1])), scale2, negm2);
          const float2 ea = make_float2(ex2f(xa.x), ex2f(xa.y));
          const float2 eb = make_float2(ex2f(xb.x), ex2f(xb.y));
          sa = add2(sa, ea);
          sb = add2(sb, eb);
          pk0[e] = pack16<BF16>(ea.x, ea.y);
          pk1[e] = pack16<BF16>(eb.x, eb.y);
        }
        const float2 tot = add2(sa, sb);
        const bool ahead = scores_there(more);
        if (ahead) load_scores();
        // P is written over the first half of the scores it comes from
        tmem_st_32x32b_x16(t_s + buf * BN, pk0);
        tmem_st_32x32b_x16(t_s + buf * BN + 16, pk1);
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(&p_ready[2 * q + buf]);
        l_sum += tot.x + tot.y;
        if (more && !ahead) wait_scores();
      }
      }

      // ---- epilogue: O / l
      if (ok && n_tiles > 0) {
        if (END_VOTE) there &= mbar_wait(&o_done[2 * q + 1], ends[1] & 1, abort_flag, p.status, ST_ATTN_O);
        else ok = mbar_wait_warp(&o_done[2 * q + 1], ends[1] & 1, abort_flag, p.status, ST_ATTN_O);
      }
      float f_first = 0.f, f_second = 0.f;
      int c_begin = 0, c_end = D / 32;  // 32-column chunks of O this group stores
      if (SPLIT) {
        const float2 other = meet(make_float2(m_ref, l_sum));
        if (NORM) {
          f_first = f_second = 1.0f;
        } else {
          // O = (O0 2^(m0 - m) + O1 2^(m1 - m)) / (l0 2^(m0 - m) + l1 2^(m1 - m)); a half that saw no key counts for nothing
          const float l0 = q == 0 ? l_sum : other.y, l1 = q == 0 ? other.y : l_sum;
          const float m0 = l0 == 0.f ? -INFINITY : (q == 0 ? m_ref : other.x);
          const float m1 = l1 == 0.f ? -INFINITY : (q == 0 ? other.x : m_ref);
          const float m = fmaxf(m0, m1);
          const float w0 = m0 == -INFINITY ? 0.f : ex2f(m0 - m), w1 = m1 == -INFINITY ? 0.f : ex2f(m1 - m);
          const float l = l0 * w0 + l1 * w1;
          f_first = w0 / l;
          f_second = w1 / l;
        }
        // each group stores half of the columns, but a 16-bit row of D = 64 is one box, which group 0 stores
        if (D == 64 && !OUT_F32) {
          c_end = q == 0 ? D / 32 : 0;
        } else {
          c_begin = q * (D / 64);
          c_end = c_begin + D / 64;
        }
      }
      if (END_VOTE && !__all_sync(0xffffffffu, there)) ok = false;
      if (ok && (SPLIT || n_tiles > 0)) {
        tc_fence_after_sync();
        const float inv = SPLIT ? 1.0f : 1.0f / l_sum;  // (the halves are scaled as they are put together)
        const bool valid = g_row < p.S_q;
        const size_t row_off = ((size_t)bh * p.S_q + (size_t)min(g_row, p.S_q - 1)) * D;
        uint32_t packed[32];
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          __syncwarp();
          if (SPLIT && (c < c_begin || c >= c_end)) continue;
          uint32_t o[32];
          tmem_ld_32x32b_x32((SPLIT ? t_o - q * 128 : t_o) + c * 32, o);
          tmem_ld_wait();
          if (SPLIT) {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f_first);
            if (it.nq[1] > 0) {  // (group 0 always has a key tile)
              uint32_t o1[32];
              tmem_ld_32x32b_x32(t_o - q * 128 + 128 + c * 32, o1);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i)
                o[i] = __float_as_uint(__fmaf_rn(__uint_as_float(o1[i]), f_second, __uint_as_float(o[i])));
            }
          }
          if (valid) {
            if (OUT_F32) {
              float4* dst = reinterpret_cast<float4*>(static_cast<float*>(p.O) + row_off + c * 32);
#pragma unroll
              for (int i = 0; i < 8; ++i)
                dst[i] = make_float4(__uint_as_float(o[4 * i]) * inv, __uint_as_float(o[4 * i + 1]) * inv,
                                     __uint_as_float(o[4 * i + 2]) * inv, __uint_as_float(o[4 * i + 3]) * inv);
            }
          }
          if (!OUT_F32) {
            // the 32 scaled values of this lane's row, rounded: half of a 128-byte box row
#pragma unroll
            for (int i = 0; i < 16; ++i)
              packed[(c & 1) * 16 + i] = pack16<BF16>(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
            if (c & 1) {
              // A lane holds 128 bytes of ONE row: the warp writes its 32 rows as a 128-byte-swizzle box and one
              // lane hands it to the TMA unit, which writes whole lines and leaves out rows beyond S_q.
              unsigned char* box = smem + L::kOut + warp * (32 * 128);
              if (lane == 0) tma_store_wait_read<0>();  // the previous store from this box has read it
              __syncwarp();
#pragma unroll
              for (int j = 0; j < 8; ++j)
                *reinterpret_cast<uint4*>(box + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                    make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
              fence_proxy_async_smem();
              __syncwarp();
              const int row0 = g_row - lane;
              if (lane == 0 && row0 < p.S_q) {
                tma_store_3d(&tmap_o, box, (c >> 1) * 64, row0, bh);
                tma_store_commit();
              }
            }
          }
        }
      }
      ends[0] += n_tiles > 1;
      ends[1] += n_tiles > 0;
    }
  }

  // ------------------------------------------------------------------ teardown
  if (!OUT_F32 && warp < 8 && lane == 0) tma_store_wait<0>();  // the output boxes are read and written out
  if (*abort_flag) {
    unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kWarpMma) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
  // the last CTA to leave puts the work counter back to zero for the next launch
  if (threadIdx.x == 0) {
    if (atomicAdd(p.work + 1, 1u) == gridDim.x - 1) {
      p.work[0] = 0;
      p.work[1] = 0;
      __threadfence();
    }
  }
}

// Items of ONE query tile or of two.  A lone tile has half of its SM's softmax and MMA threads idle where its keys are not split
// (split_keys_pay: one key tile, two in the single pass), but more items balance better.  So lone tiles are taken where that leaves at most one item per SM, and
// beyond that where this estimate is clearly better: in steps (128 keys of two query tiles side by side, 1.8 us at D = 128), a pair of
// tiles takes its key tiles, a split lone tile 0.56 a step, either 1.9 more to begin and end; equal items go round by round,
// causal ones heavy first.  Estimated / measured ratios: 12 heads x 2048 causal 0.67 / 0.61 (34.5 against 21.2 us; D = 64 32.5
// against 20.9), 15 x 2013 causal 0.79 / 0.65, 10 x 4096 causal 0.87 / 0.72, 64 x 700 normalised 0.93 / 0.88, 64 x 1025 0.80 / 0.85;
// 64 x 2048 causal 1.14 / 1.16.  Of 63 shapes the choice costs more than 2 % in 6, at most 8 %.  The estimate is too low for
// causal ones of few key tiles (50 x 612 0.93 / 1.16) and too high in the normalised mode (36 x 978 1.21 / 1.05): hence 0.9 and 0.95.
double items_estimate(const frisk_b200_attn_desc& d, int sms, int tiles_per_item) {
  constexpr double kSplitStep = 0.56, kItem = 1.9;
  const int64_t heads = (int64_t)d.B * d.H, tiles = (d.S_q + BM - 1) / BM;
  const int64_t groups = (tiles + tiles_per_item - 1) / tiles_per_item, items = groups * heads;
  const double step = (tiles_per_item == 1 ? kSplitStep : 1.0) * (d.normalize_p ? 2 : 1);
  const int64_t all = (d.S_kv + 127) / 128, off = (int64_t)d.S_kv - d.S_q;
  const double heaviest = step * (double)all + kItem;
  if (!d.causal) return (double)((items + sms - 1) / sms) * heaviest;
  if (items <= sms) return heaviest;
  double total = 0;
  for (int64_t g = 0; g < groups; ++g) {
    const int64_t last_row = std::min<int64_t>((g + 1) * tiles_per_item * BM, d.S_q) - 1;
    total += step * (double)std::min<int64_t>(all, std::max<int64_t>(0, last_row + off) / 128 + 1) + kItem;
  }
  return std::max(heaviest, (double)heads * total / sms + 0.5 * total / (double)groups);
}
// A lone tile's keys are worth sharing beyond 128 in the normalised mode (33 heads x 251 11.8 -> 10.4 us) and beyond 256 in the
// single pass, where with fewer the meeting of the groups costs what it saves (16 heads x 256 and 48 x 159 as fast either way).
bool split_keys_pay(const frisk_b200_attn_desc& d) { return d.S_kv > (d.normalize_p ? 128 : 256); }

bool one_tile_items(const frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d) {
  const int64_t tiles = (d.S_q + BM - 1) / BM * d.B * d.H;
  if (tiles <= ctx->num_sms) return true;
  // (four rounds of pairs balance by themselves)
  if (!split_keys_pay(d) || tiles > 8 * (int64_t)ctx->num_sms) return false;
  return items_estimate(d, ctx->num_sms, 1) < (d.normalize_p ? 0.95 : 0.9) * items_estimate(d, ctx->num_sms, 2);
}

template <bool BF16, int D, bool OUT_F32, bool NORM, Mode MODE>
int launch_cfg(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K, const void* V,
               void* O, cudaStream_t s) {
  CUtensorMap tq, tk, tv;
  const int bh = d.B * d.H;
  const uint64_t row_bytes = (uint64_t)D * 2;
  int rc = encode_tmap_3d(ctx, &tq, d.dtype_in, Q, D, d.S_q, bh, row_bytes, row_bytes * d.S_q, 64, BM, 1, true);
  if (!rc) rc = encode_tmap_3d(ctx, &tk, d.dtype_in, K, D, d.S_kv, bh, row_bytes, row_bytes * d.S_kv, 64, BN, 1, true);
  if (!rc) rc = encode_tmap_3d(ctx, &tv, d.dtype_in, V, D, d.S_kv, bh, row_bytes, row_bytes * d.S_kv, 64, BN, 1, true);
  CUtensorMap to = tq;  // unused for fp32 outputs
  if (!rc && !OUT_F32)
    rc = encode_tmap_3d(ctx, &to, d.dtype_out, O, D, d.S_q, bh, row_bytes, row_bytes * d.S_q, 64, 32, 1, true);
  if (rc) {
    ctx->last_cuda = rc;
    return FRISK_B200_E_CUDA;
  }
  AttnParams p;
  p.S_q = d.S_q;
  p.S_kv = d.S_kv;
  p.group_rows = MODE == kTwin || one_tile_items(ctx, d) ? BM : 2 * BM;
  p.n_groups = (d.S_q + p.group_rows - 1) / p.group_rows;
  p.causal = d.causal ? 1 : 0;
  p.heads = bh;
  p.total_items = MODE == kTwin ? ((int64_t)bh + 1) / 2 : (int64_t)p.n_groups * bh;
  p.scale_log2 = d.scale * 1.4426950408889634f;
  p.scale = d.scale;
  p.normalized = d.normalize_p ? 1 : 0;
  p.O = O;
  p.status = ctx->d_status;
  p.work = ctx->d_status + 16;  // work counter and exit counter of the persistent grid (zero between launches)
  if (p.total_items > INT32_MAX) return FRISK_B200_E_ATTN_SHAPE;
  auto kern = attention_fwd_kernel<BF16, D, OUT_F32, NORM, MODE>;
  using L = AttnSmem<D>;
  // setmaxnreg.inc waits (without a bound) until the CTA's own register pool holds what it
  // asks for: the registers the TMA/MMA warpgroup (128 threads) gives up must cover what the
  // two softmax warpgroups (256 threads) take, or the kernel would never start.  Checked
  // against the compiled register count before every launch.
  static PerDeviceOnce set_up;  // one per instantiation; a failed check is repeated (and fails) every call
  const int bad = set_up(ctx->device, [&] {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return (int)FRISK_B200_E_CUDA;
    if (fa.numRegs < kRegsOther || fa.numRegs > kRegsSoftmax ||
        (fa.numRegs - kRegsOther) * 128 < (kRegsSoftmax - fa.numRegs) * 256)
      return (int)FRISK_B200_E_UNSUPPORTED;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal) != cudaSuccess)
      return (int)FRISK_B200_E_CUDA;
    return 0;
  });
  if (bad) return bad;
  const unsigned grid = (unsigned)std::min<int64_t>(p.total_items, ctx->num_sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // the kernel waits (griddepcontrol.wait) itself
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, tq, tk, tv, to, p));
  return 0;
}

Mode mode_of(const frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d) {
  // A lone query tile's key tiles go to the two softmax groups in turn: one group alone leaves the schedulers idle while it
  // waits for tensor memory and barriers (with one buffer of scores: 16 heads x 1025 normalised 29.2 -> 23.4 us, 4 heads x 4096
  // causal at D = 128 62.1 -> 40.4; with two 22.1 and 32.9).
  if (split_keys_pay(d) && one_tile_items(ctx, d)) return kSplit;
  // Heads of one query tile, more of them than SMs, whose keys are not split: two at a time, since a pair's second group would be
  // idle (512 heads x 128, D = 64 13.9 -> 11.9 us, D = 128 19.2 -> 16.5).  That is up to 256 keys, or more than 8 heads an SM:
  // between, the estimate above knows no item of two heads and always prefers split keys.  In the normalised mode a lone tile is
  // as fast.
  if (!d.normalize_p && d.S_q <= BM && (int64_t)d.B * d.H > ctx->num_sms) return kTwin;
  return kPair;
}

template <bool BF16, int D, bool OUT_F32, bool NORM>
int launch_mode(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K, const void* V,
                 void* O, cudaStream_t s) {
  switch (mode_of(ctx, d)) {
    case kSplit: return launch_cfg<BF16, D, OUT_F32, NORM, kSplit>(ctx, d, Q, K, V, O, s);
    case kTwin: return launch_cfg<BF16, D, OUT_F32, NORM, NORM ? kPair : kTwin>(ctx, d, Q, K, V, O, s);
    default: return launch_cfg<BF16, D, OUT_F32, NORM, kPair>(ctx, d, Q, K, V, O, s);
  }
}

template <bool BF16, int D>
int launch_out(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K, const void* V,
               void* O, cudaStream_t s) {
  if (d.normalize_p) {
    if (d.dtype_out == FRISK_B200_F32) return launch_mode<BF16, D, true, true>(ctx, d, Q, K, V, O, s);
    return launch_mode<BF16, D, false, true>(ctx, d, Q, K, V, O, s);
  }
  if (d.dtype_out == FRISK_B200_F32) return launch_mode<BF16, D, true, false>(ctx, d, Q, K, V, O, s);
  return launch_mode<BF16, D, false, false>(ctx, d, Q, K, V, O, s);
}

}  // namespace

int attention_form(const frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d) {
  if (attention_decode_preferred(d)) return FRISK_B200_ATTN_FEW_QUERIES;
  const Mode mode = mode_of(ctx, d);
  return mode == kSplit ? FRISK_B200_ATTN_SPLIT_KEYS : mode == kTwin ? FRISK_B200_ATTN_TWO_HEADS : FRISK_B200_ATTN_PAIRS;
}

int launch_attention_fwd(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K,
                         const void* V, void* O, cudaStream_t s) {
  if (attention_decode_preferred(d)) return launch_attention_decode(ctx, d, Q, K, V, O, s);
  const bool bf = d.dtype_in == FRISK_B200_BF16;
  if (d.D == 128) return bf ? launch_out<true, 128>(ctx, d, Q, K, V, O, s) : launch_out<false, 128>(ctx, d, Q, K, V, O, s);
  if (d.D == 64) return bf ? launch_out<true, 64>(ctx, d, Q, K, V, O, s) : launch_out<false, 64>(ctx, d, Q, K, V, O, s);
  return FRISK_B200_E_ATTN_SHAPE;
}

}  // namespace fb
