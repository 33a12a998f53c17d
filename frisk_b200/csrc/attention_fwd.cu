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
//     left.  An item is TWO 128-row query tiles of one (batch, head), each with a softmax group and an MMA thread of its own, or
//     ONE (items_estimate, below), whose key tiles the two groups share out (SPLIT) or group 0 takes alone.  Barriers, tensor
//     memory and the K/V ring live across items, so the next item's Q, K and V are already on their
//     way, and its first scores are computed, while the softmax warps still store the last item's O;
//   * 128-key K/V tiles stream through a 2-stage TMA ring (K and V have separate full/empty mbarriers).  Both MMA threads read
//     every tile; SPLIT: the even key tiles are in stage 0, for the first thread alone, the odd ones in stage 1, for the second;
//   * warp 8 is the TMA producer; warps 9 and 10 issue the tcgen05.mma of softmax group 0 and 1: S_q =
//     Q_q.K^T (SS form, both operands K-major, 128-byte swizzle) into tensor memory and O_q += P_q.V
//     (P read from tensor memory, V as an MN-major shared-memory operand);
//   * warps 0-3 and 4-7 are the two softmax groups: thread r owns row r of its query tile
//     (TMEM lane r), so row max / row sum need no shuffles.  In the single pass the two groups take turns, so
//     the tensor core works on one group's MMAs while the other exponentiates.  The row maximum is taken within the turn, through
//     the first exponentials, or before it (kMaxFirst);
//   * the running maximum is applied lazily: O is rescaled in tensor memory only when the
//     maximum grew by more than 2^8, which keeps P within bf16/fp16 range and makes most
//     iterations rescale-free;
//   * causal: key tiles wholly above the diagonal are never loaded; only tiles that touch the
//     diagonal (or the ragged end of the keys) are masked.
// TMEM columns: S0 [0,128) S1 [128,256) O0 [256,256+D) O1 [384,384+D); P_q aliases the first
// 64 columns of S_q (two 16-bit values per column).
// Every mbarrier wait is bounded (ptx.cuh); no TMA load uses cluster multicast.
#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

#include "attention_common.cuh"

namespace fb {
namespace {
using namespace attn;

constexpr int kStagesKV = 2;
constexpr int kHeadChunk = 16;  // heads whose K and V are worked on together (they stay in L2: 16 x 2 MB at S = 4096)
template <int D>
struct AttnSmem {
  static constexpr int kTileBytes = BM * D * 2;       // one Q, K or V tile
  static constexpr int kQ = 0;                         // Q0, Q1
  static constexpr int kK = 2 * kTileBytes;            // K stages
  static constexpr int kV = kK + kStagesKV * kTileBytes;
  static constexpr int kBar = kV + kStagesKV * kTileBytes;
  // 16-bit outputs: one [32 rows][128 bytes] box per softmax warp for the TMA stores of O, 1024-byte aligned
  static constexpr int kOut = kBar + 1024;
  static constexpr int kTotal = kOut + 8 * (32 * 128) + 1024;
  static_assert(kTotal <= 232448, "the output boxes must fit next to the Q, K and V tiles");
};


// SPLIT: an item is ONE query tile, whose key tiles the two softmax groups (and MMA threads) take in turn, even and odd
// ones, each with its own S, P, O and statistics; at the end the halves are put together.
template <bool BF16, int D, bool OUT_F32, bool NORM, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
    attention_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                         const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o,
                         const AttnParams p) {
  using L = AttnSmem<D>;
  constexpr int kBoxes = D / 64;            // 64-element (128-byte) column blocks per tile
  constexpr int kBoxBytes = BM * 128;       // one [128 rows][128 B] block
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  uint64_t* q_full = bars;              // [1]
  uint64_t* k_full = bars + 1;          // [2]
  uint64_t* k_empty = bars + 3;         // [2]
  uint64_t* v_full = bars + 5;          // [2]
  uint64_t* v_empty = bars + 7;         // [2]
  uint64_t* s_full = bars + 9;          // [2] per query tile
  uint64_t* p_ready = bars + 11;        // [2] first half of P_q (keys 0-63) written
  uint64_t* p_ready_hi = bars + 16;     // [2] second half written
  uint64_t* o_done = bars + 13;         // [2]
  uint64_t* turn = bars + 18;           // [2] hand-over of the exponential section between the two softmax groups
  uint64_t* item_full = bars + 20;      // [2] the producer has published the id of a work item
  uint64_t* item_empty = bars + 22;     // [2] every consumer has read it
  uint64_t* q_empty = bars + 24;        // [1] both MMA threads are done with the Q tiles
  uint64_t* xchg = bars + 26;           // [1] the two softmax groups meet (SPLIT only)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 27);
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
  // returns its id, or -1 when the work has run out or a wait was abandoned.
  auto next_item = [&](int n, bool arrive) -> int {
    if (!mbar_wait(&item_full[n & 1], (n >> 1) & 1, abort_flag, p.status, ST_ATTN_Q)) return -1;
    const int t = item_slot[n & 1];
    if (arrive) mbar_arrive(&item_empty[n & 1]);
    return t;
  };
  // The ring of K and V: tile n goes to stage n % 2, and both MMA threads follow every tile.  SPLIT: each stage belongs to one MMA
  // thread and n counts that stage's tiles, because a thread that does not follow all uses of a stage can mistake an earlier
  // phase of its barrier for its own (with an odd number of key tiles the threads would change stages from pass to pass).
  auto ring_phase = [](int n) -> uint32_t { return (SPLIT ? n : n / kStagesKV) & 1; };
  // Normalised mode runs the key loop twice: pass 0 only gathers row maxima and row sums, pass 1
  // is the pass every mode has.  Barrier phases keep counting across passes and items.
  constexpr int first_pass = NORM ? 0 : 1;
  // Where the row maximum is taken: before the group's turn, on the ALU while the other group keeps the special-function
  // unit busy, or within it, run through the first exponentials.  Before is faster where the turns set the pace: D = 64, whose
  // MMAs are half as long (8 x 32 heads x 2048 causal 274 -> 251 us, 3 x 16 x 1500 57.8 -> 51.7), and a lone query tile.  At
  // D = 128 P.V and the next S set it, and long runs the power limit (930 W): before is slower there (8 x 32 x 4096 causal 1120
  // -> 1145 us, 8 heads x 8192 272 -> 284).
  constexpr bool kMaxFirst = D == 64 || SPLIT;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], SPLIT ? 1 : 2);  // one arrival per MMA-issuing thread that reads the stage
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], SPLIT ? 1 : 2);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_ready[i], 128);
      mbar_init(&p_ready_hi[i], 128);
      mbar_init(&o_done[i], 1);
      mbar_init(&turn[i], 128);
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
      // K / V tiles loaded so far, over all items (K is streamed once per pass); SPLIT: into either stage
      int kt = 0, vt = 0, kt_odd = 0, vt_odd = 0;
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
            tma_load_3d(smem + L::kQ + q * L::kTileBytes + b * kBoxBytes, &tmap_q, q_full, b * 64, it.m0 + q * BM, it.bh);
        for (int pass = first_pass; pass < 2 && ok; ++pass) {
          for (int j = 0; j < it.n_max; ++j) {
            const bool odd = SPLIT && (j & 1);  // the second group's key tile
            const int kp = odd ? kt_odd++ : kt++, vp = odd ? vt_odd : vt;
            const int ks = SPLIT ? (int)odd : kp % kStagesKV;
            if (!mbar_wait(&k_empty[ks], ring_phase(kp) ^ 1, abort_flag, p.status, ST_ATTN_KV)) {
              ok = false;
              break;
            }
            mbar_expect_tx(&k_full[ks], L::kTileBytes);
#pragma unroll
            for (int b = 0; b < kBoxes; ++b)
              tma_load_3d(smem + L::kK + ks * L::kTileBytes + b * kBoxBytes, &tmap_k, &k_full[ks], b * 64, j * BN, it.bh);
            if (pass == 0) continue;  // the statistics pass needs no values
            (odd ? vt_odd : vt)++;
            const int vs = SPLIT ? (int)odd : vp % kStagesKV;
            if (!mbar_wait(&v_empty[vs], ring_phase(vp) ^ 1, abort_flag, p.status, ST_ATTN_KV)) {
              ok = false;
              break;
            }
            mbar_expect_tx(&v_full[vs], L::kTileBytes);
#pragma unroll
            for (int b = 0; b < kBoxes; ++b)
              tma_load_3d(smem + L::kV + vs * L::kTileBytes + b * kBoxBytes, &tmap_v, &v_full[vs], b * 64, j * BN, it.bh);
          }
        }
      }
    }
  } else if (warp == kWarpMma || warp == kWarpMma + 1) {
    // ------------------------------------------------------------------ MMA issuers, one thread per query tile
    // Each query tile has its own issuing thread (warps 9 and 10).  One thread for both tiles was the
    // kernel's bottleneck: besides the 32 MMAs of a key tile it has a dozen barrier waits, fences and commits
    // to execute, each a round trip of ~100 clocks for a single thread, and the two tiles' chains
    // (S -> softmax -> P.V -> next S) queued behind each other in it.  tcgen05 operations of ONE thread execute
    // in issue order, which is all the ordering a query tile needs (S_q(j+1) overwrites P_q(j) only after
    // P_q(j).V(j) has read it); the two tiles share only the read-only K and V stages, which each thread
    // releases with its own arrival (the empty barriers count two).
    const int mq = warp - kWarpMma;
    if (lane == 0) {
      constexpr uint32_t idesc_s = umma_idesc_f16(BM, BN, BF16, false, false);
      constexpr uint32_t idesc_o = umma_idesc_f16(BM, D, BF16, false, true);
      const uint32_t sq = smem_u32(smem + L::kQ), sk = smem_u32(smem + L::kK), sv = smem_u32(smem + L::kV);
      // descriptors are built once; the k16 slices only add a constant to the start-address field
      const uint64_t dq = umma_desc_kmajor_sw128(sq + (SPLIT ? 0 : mq * L::kTileBytes));
      const uint64_t dk[2] = {umma_desc_kmajor_sw128(sk), umma_desc_kmajor_sw128(sk + L::kTileBytes)};
      const uint64_t dv[2] = {umma_desc_mnmajor_sw128(sv, kBoxBytes, 1024),
                              umma_desc_mnmajor_sw128(sv + L::kTileBytes, kBoxBytes, 1024)};
      const uint32_t t_sq = tmem_base + mq * 128;        // S_q; P_q aliases its first 64 columns (8 per k16 slice)
      const uint32_t t_oq = tmem_base + 256 + mq * 128;  // O_q
      int kt = 0, vt = 0;    // K / V tiles seen so far, over all items (ring positions; K is streamed once per pass)
      int steps = 0;         // (pass, key tile) steps of THIS softmax group so far: the phase of s_full / p_ready
      auto ring_stage = [&](int n) -> int { return SPLIT ? mq : n % kStagesKV; };
      bool ok = true;
      for (int n = 0; ok; ++n) {
        const int t = next_item(n, true);
        if (t < 0) break;
        const Item it = decode(t);
        const int n_mine = it.nq[mq], n_max = SPLIT ? n_mine : it.n_max;  // key tiles: used, followed
        ok = mbar_wait(q_full, n & 1, abort_flag, p.status, ST_ATTN_Q);
        for (int pass = first_pass; pass < 2 && ok; ++pass) {
          const bool stats_pass = pass == 0;  // the pass that only gathers statistics issues no P.V
          // Per key tile and query tile the dependent chain is: softmax publishes P(j) -> P(j).V(j) -> S(j+1) ->
          // softmax.  Everything this thread can do off that chain is done off it: the wait for K(j+1) happens
          // before the wait for P(j), and the commits that release V(j), K(j+1) and publish O come after the
          // MMAs of S(j+1) have been issued (a commit covers everything issued before it, so they only fire a
          // little later than strictly possible).
          bool have_k = false;  // K(j) of the current pass is known to have landed
          for (int j = 0; j < n_max && ok; ++j, ++kt) {
            const int ks = ring_stage(kt);
            if (!have_k) ok = mbar_wait(&k_full[ks], ring_phase(kt), abort_flag, p.status, ST_ATTN_KV);
            have_k = false;
            if (!ok) break;
            if (j < n_mine) {
              tc_fence_after_sync();
#pragma unroll
              for (int kk = 0; kk < D / 16; ++kk) {
                const uint64_t off = static_cast<uint64_t>(((kk / 4) * kBoxBytes + (kk % 4) * 32) >> 4);
                umma_f16_ss(t_sq, dq + off, dk[ks] + off, idesc_s, kk != 0);
              }
              umma_commit(&s_full[mq]);
              umma_commit(&k_empty[ks]);  // this tile's use of the K stage ends when these MMAs have read it
              if (j > 0 && !stats_pass && !SPLIT) {  // (deferred from the previous tile)
                umma_commit(&o_done[mq]);
                umma_commit(&v_empty[(vt - 1) % kStagesKV]);
              }
              if (pass == 1 && j == n_mine - 1) umma_commit(q_empty);  // this thread's last use of the Q tiles
            } else {
              mbar_arrive(&k_empty[ks]);  // a key tile only the other query tile needs
            }
            const int vs = ring_stage(vt);
            if (j < n_mine) {
              // the next K tile, while the softmax group works on this one (SPLIT: it comes behind a V tile whose stage the
              // other thread has yet to release, and must not hold up this thread's P.V)
              if (!SPLIT && j + 1 < n_max) {
                ok = mbar_wait(&k_full[ring_stage(kt + 1)], ring_phase(kt + 1), abort_flag, p.status, ST_ATTN_KV);
                have_k = ok;
              }
              if (!stats_pass && ok) ok = mbar_wait(&v_full[vs], ring_phase(vt), abort_flag, p.status, ST_ATTN_KV);
              // O_q += P_q(j) . V(j).  The softmax group publishes P in two halves (64 keys each), so the first
              // four k16 slices start while the second half is still being exponentiated.  In the statistics
              // pass the two waits only tell that the softmax group is done with S_q.
              const uint32_t parity = steps & 1;
              ++steps;
#pragma unroll
              for (int half = 0; half < 2; ++half) {
                if (ok) ok = mbar_wait(half ? &p_ready_hi[mq] : &p_ready[mq], parity, abort_flag, p.status, ST_ATTN_P);
                if (stats_pass) continue;
                if (!ok) break;
                tc_fence_after_sync();
#pragma unroll
                for (int kk = half * 4; kk < half * 4 + 4; ++kk)
                  umma_f16_ts(t_oq, t_sq + kk * 8, dv[vs] + static_cast<uint64_t>((kk * 2048) >> 4), idesc_o,
                              (j | kk) != 0);
              }
              if (!ok) break;
              // no further S of this item follows, or the next V tile of this group waits for the stage: publish now
              if (!stats_pass && (SPLIT || j + 1 >= n_mine)) {
                umma_commit(&o_done[mq]);
                umma_commit(&v_empty[vs]);
              }
            } else if (!stats_pass) {
              ok = mbar_wait(&v_full[vs], ring_phase(vt), abort_flag, p.status, ST_ATTN_KV);
              if (ok) mbar_arrive(&v_empty[vs]);
            }
            if (!stats_pass) ++vt;
          }
        }
        if (ok && n_mine == 0) mbar_arrive(q_empty);  // (a query tile beyond the end of the sequence)
      }
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
    int steps = 0;    // (pass, key tile) steps of this query tile so far, over all items: the phase of s_full
    int turns = 0;    // key-tile iterations so far: the phase of the turn barriers
    int pv_base = 0;  // key tiles whose P.V was issued for earlier items: the phase of o_done
    int meets = 0;    // meetings of the two groups so far: the phase of xchg
    bool ok = true;
    // Split keys: the two groups meet, and each thread learns what the other group's thread of its row brings.  The
    // statistics lie in the second query tile's place, which nothing else uses then, in two sets that alternate: a set is
    // written again only when everybody has arrived at the meeting in between, after reading it.
    auto meet = [&](float2 mine_v) -> float2 {
      float2* set = reinterpret_cast<float2*>(smem + L::kQ + L::kTileBytes) + (meets & 1) * 2 * BM;
      set[q * BM + row] = mine_v;
      tc_fence_before_sync();
      mbar_arrive(xchg);
      if (!mbar_wait(xchg, meets & 1, abort_flag, p.status, ST_ATTN_O)) ok = false;
      ++meets;
      tc_fence_after_sync();
      return set[(q ^ 1) * BM + row];
    };

    for (int n = 0; ok; ++n) {
      const int item_id = next_item(n, lane == 0);
      if (item_id < 0) break;
      const Item it = decode(item_id);
      const int bh = it.bh, n_max = max(it.nq[0], it.nq[1]);
      const int n_tiles = it.nq[q];
      const int m_tile = it.m0 + (SPLIT ? 0 : q * BM);
      // (both groups have read both O of the item before)
      if (SPLIT && n > 0) meet(make_float2(0.f, 0.f));
      const int g_row = m_tile + row;  // query index within the head
      float m_ref = -INFINITY;  // reference maximum (scaled, log2 units) the stored P and O are relative to
      float l_sum = 0.f;

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
            if (!ok) break;
          }
          const float inv_l = __frcp_rn(l_run);  // (of use in pass 1 only)
          const float2 inv2 = make_float2(inv_l, inv_l), negl2 = make_float2(-l_run, -l_run);
          for (int i = 0; i < n_tiles; ++i) {
            const int j = SPLIT ? 2 * i + q : i;
            if (!mbar_wait(&s_full[q], steps & 1, abort_flag, p.status, ST_ATTN_S)) {
              ok = false;
              break;
            }
            ++steps;
            tc_fence_after_sync();
            uint32_t sr[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(t_s + c * 32, sr[c]);
            tmem_ld_wait();
            if (pass == 0) {
              // S_q is in registers: the MMA warp may overwrite it
              tc_fence_before_sync();
              mbar_arrive(&p_ready[q]);
              mbar_arrive(&p_ready_hi[q]);
            }
            const int n0 = j * BN;
            if ((n0 + BN > p.S_kv) || (p.causal && (n0 + BN - 1 > m_tile + off))) {
              int limit = p.S_kv - 1;
              if (p.causal) limit = min(limit, g_row + off);
              limit -= n0;  // columns > limit are hidden
#pragma unroll
              for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (c * 32 + i > limit) sr[c][i] = 0xff800000u;  // -inf
            }
            // (score - m) * log2e of a pair, rounded step by step; the scale is positive, so it keeps the order and
            // the maximum of the scaled scores is the scaled maximum
            auto arg2 = [&](int c, int i, float2 negm2) {
              const float2 s2 = make_float2(__uint_as_float(sr[c][2 * i]), __uint_as_float(sr[c][2 * i + 1]));
              return mul2_rn(add2_rn(mul2_rn(s2, scale2), negm2), log2e2);
            };
            if (pass == 0) {
              float mxc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
              for (int i = 0; i < 16; ++i)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                  mxc[c] = max3f(mxc[c], __uint_as_float(sr[c][2 * i]), __uint_as_float(sr[c][2 * i + 1]));
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
                  for (int c = 0; c < 4; ++c) {
                    const float2 x = arg2(c, i, negm2);
                    sum[c] = add2_rn(sum[c], make_float2(exp2_of(x.x), exp2_of(x.y)));
                  }
                const float2 all = add2_rn(add2_rn(sum[0], sum[1]), add2_rn(sum[2], sum[3]));
                const float carry = (m_run == -INFINITY) ? 0.f : l_run * ex2f_ieee_range(__fmul_rn(__fsub_rn(m_run, m_new), kLog2e));
                l_run = carry + (all.x + all.y);
                m_run = m_new;
              }
            } else {
              const float2 negm2 = make_float2(-m_run, -m_run);
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  const float2 x = arg2(c, i, negm2);
                  const float2 pv = div2_by(make_float2(exp2_of(x.x), exp2_of(x.y)), negl2, inv2);
                  pk[i] = pack16<BF16>(pv.x, pv.y);
                }
                tmem_st_32x32b_x16(t_s + c * 16, pk);
                if (c & 1) {
                  tmem_st_wait();
                  tc_fence_before_sync();
                  mbar_arrive(c == 1 ? &p_ready[q] : &p_ready_hi[q]);
                }
              }
            }
          }
        }
        l_sum = 1.0f;  // P is already normalised
        m_ref = 0.f;
      } else
      // The two softmax groups take turns: group 1 starts the arithmetic of its key tile j when group 0 has
      // finished that of its tile j (all 128 keys: handing over after the first 64 measured 3 % slower), and group 0
      // starts tile j+1 when group 1 has finished tile j.  Left alone the
      // two groups fall into step (they share the K/V ring and the tensor pipe), exponentiate at the same time
      // on the same four schedulers and then both sit idle while their MMAs run; taking turns, one group works
      // alone (a third faster) while the other group's P.V and next S are in flight.  A group with fewer key
      // tiles than the other keeps passing the turn on until the other is done.
      for (int i = 0; i < n_max; ++i) {
        const bool mine = i < n_tiles;
        uint32_t sr[4][32];
        if (mine) {
          if (!mbar_wait(&s_full[q], steps & 1, abort_flag, p.status, ST_ATTN_S)) {
            ok = false;
            break;
          }
          ++steps;
          tc_fence_after_sync();
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(t_s + c * 32, sr[c]);
          tmem_ld_wait();

          const int n0 = (SPLIT ? 2 * i + q : i) * BN;
          const bool needs_mask = (n0 + BN > p.S_kv) || (p.causal && (n0 + BN - 1 > m_tile + off));
          if (needs_mask) {
            int limit = p.S_kv - 1;
            if (p.causal) limit = min(limit, g_row + off);
            limit -= n0;  // columns > limit are hidden
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c * 32 + i > limit) sr[c][i] = 0xff800000u;  // -inf
          }
        }
        const float2 scale2 = make_float2(p.scale_log2, p.scale_log2);
        float mxc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // four chains of the row maximum
        auto max_step = [&](int i) {  // two keys of every 32
#pragma unroll
          for (int c = 0; c < 4; ++c)
            mxc[c] = max3f(mxc[c], __uint_as_float(sr[c][2 * i]), __uint_as_float(sr[c][2 * i + 1]));
        };
        // Takes the row maximum into the reference; true where that has moved (exponentials relative to the one before are
        // void).  O is rescaled only when the maximum grew by more than the threshold: rare after the first tiles.
        auto settle = [&]() -> bool {
          const float mx = max3f(mxc[0], mxc[1], fmaxf(mxc[2], mxc[3]));
          float m_new = fmaxf(m_ref, mx * p.scale_log2);
          // A row that has seen no key, or only scores of -inf: the lowest finite reference, so that its exponentials are 0 and the
          // first finite score moves it (0 would let lower scores vanish; a group's first key tile may be any row's -inf).
          if (m_new == -INFINITY) m_new = -FLT_MAX;
          if (i == 0) {
            m_ref = m_new;
            return true;
          }
          // (warp-uniform decision because the TMEM accesses are warp-collective)
          if (!__any_sync(0xffffffffu, m_new - m_ref > kRescaleThreshold)) return false;
          const float factor = ex2f(m_ref - m_new);
          m_ref = m_new;
          l_sum *= factor;
          // O_q must be complete up to the key tile before this one before it is scaled
          ok = mbar_wait(&o_done[q], (pv_base + i - 1) & 1, abort_flag, p.status, ST_ATTN_O);
          if (!ok) return true;
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
          return true;
        };
        if (kMaxFirst && mine) {
#pragma unroll
          for (int e = 0; e < 16; ++e) max_step(e);
          settle();
          if (!ok) break;
        }
        if (!mbar_wait(&turn[q], q == 0 ? ((turns & 1) ^ 1) : (turns & 1), abort_flag, p.status, ST_ATTN_S)) {
          ok = false;
          break;
        }
        ++turns;
        if (!mine) {
          mbar_arrive(&turn[q ^ 1]);
          continue;
        }

        // P = 2^(s*scale_log2 - m_ref) with packed fp32 FMAs, row sum in fp32, P rounded to 16 bits.
        // Two 32-key chunks at a time, interleaved pair by pair so that the special-function unit always has
        // independent work.  WITH_MAX also runs the row maximum of all 128 keys through the same loop: the maximum is a
        // chain on the ALU, the exponentials are bound by the special-function unit, and neither waits for the other.
        auto exp_chunks = [&](int c0, uint32_t (&pa)[16], uint32_t (&pb)[16], float2& sum, auto with_max) {
          const float2 negm2 = make_float2(-m_ref, -m_ref);
          float2 sa = make_float2(0.f, 0.f), sb = make_float2(0.f, 0.f);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 xa = fma2(make_float2(__uint_as_float(sr[c0][2 * e]), __uint_as_float(sr[c0][2 * e + 1])), scale2, negm2);
            const float2 xb = fma2(make_float2(__uint_as_float(sr[c0 + 1][2 * e]), __uint_as_float(sr[c0 + 1][2 * e + 1])), scale2, negm2);
            if (decltype(with_max)::value) max_step(e);
            const float2 ea = make_float2(ex2f(xa.x), ex2f(xa.y));
            const float2 eb = make_float2(ex2f(xb.x), ex2f(xb.y));
            sa = add2(sa, ea);
            sb = add2(sb, eb);
            pa[e] = pack16<BF16>(ea.x, ea.y);
            pb[e] = pack16<BF16>(eb.x, eb.y);
          }
          sum = add2(sa, sb);
        };
        uint32_t pk0[16], pk1[16];
        float2 sum01;
        if (kMaxFirst) {
          exp_chunks(0, pk0, pk1, sum01, std::false_type());
        } else {
          // Optimistic first half: the exponentials of keys 0-63 are taken relative to the reference maximum the row
          // already has, so they do not wait for the row maximum, and are computed again where that moves it (always on
          // the first tile, whose reference is -infinity).  The stale reference cannot overflow what is kept: a value
          // that would exceed 2^threshold is by construction one that moves it.
          exp_chunks(0, pk0, pk1, sum01, std::true_type());
          const bool redo = settle();
          if (!ok) break;
          if (redo) exp_chunks(0, pk0, pk1, sum01, std::false_type());
        }
        // P is written back over S chunk by chunk; a half of P (64 keys) that is complete lets the MMA warp start on it
        tmem_st_32x32b_x16(t_s, pk0);
        tmem_st_32x32b_x16(t_s + 16, pk1);
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(&p_ready[q]);
        float2 sum23;
        exp_chunks(2, pk0, pk1, sum23, std::false_type());
        tmem_st_32x32b_x16(t_s + 32, pk0);
        tmem_st_32x32b_x16(t_s + 48, pk1);
        tmem_st_wait();
        tc_fence_before_sync();
        mbar_arrive(&p_ready_hi[q]);
        mbar_arrive(&turn[q ^ 1]);  // the other group's turn: its scores arrived while this one worked alone
        const float2 tot = add2(sum01, sum23);
        l_sum += tot.x + tot.y;
      }

      // ---- epilogue: O / l
      if (ok && n_tiles > 0) ok = mbar_wait(&o_done[q], (pv_base + n_tiles - 1) & 1, abort_flag, p.status, ST_ATTN_O);
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
      if (ok && (SPLIT || n_tiles > 0)) {
        tc_fence_after_sync();
        const float inv = SPLIT ? 1.0f : 1.0f / l_sum;  // (the halves are scaled as they are put together)
        const bool valid = g_row < p.S_q;
        const size_t row_off = ((size_t)bh * p.S_q + (size_t)min(g_row, p.S_q - 1)) * D;
        uint32_t packed[32];
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
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
      pv_base += n_tiles;
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
// beyond that where this estimate is clearly better: in steps (one key tile of two query tiles side by side, 2.1 us at D = 128), a pair of
// tiles takes its key tiles, a split lone tile 0.56 a key tile (304 us for 8 x 8192 where pairs take 273), either 1.9 more to
// begin and end; equal items go round by round, causal ones heavy first.  Estimated / measured ratios: 12 heads x 2048 causal 0.66 / 0.66
// (44.2 -> 29.0 us; D = 64 34.9 -> 21.5), 15 x 2013 causal 0.79 / 0.72, 10 x 4096 causal 0.87 / 0.78, 64 x 700 normalised 0.93 / 0.84,
// 64 x 1025 0.80 / 0.85; 24 x 1000 1.29 / 1.18, 8 x 8192 1.14 / 1.12, 64 x 2048 causal 1.14 / 1.23.  Of 68 shapes the estimate
// is too low only for causal ones of few key tiles (50 x 612 0.93 / 1.18), and too high in the normalised mode (36 x 978 1.21 / 1.06):
// hence 0.9 and 0.95.
double items_estimate(const frisk_b200_attn_desc& d, int sms, int tiles_per_item) {
  constexpr double kSplitStep = 0.56, kItem = 1.9;
  const int64_t heads = (int64_t)d.B * d.H, tiles = (d.S_q + BM - 1) / BM;
  const int64_t groups = (tiles + tiles_per_item - 1) / tiles_per_item, items = groups * heads;
  const double step = (tiles_per_item == 1 ? kSplitStep : 1.0) * (d.normalize_p ? 2 : 1);
  const int64_t all = (d.S_kv + BN - 1) / BN, off = (int64_t)d.S_kv - d.S_q;
  const double heaviest = step * (double)all + kItem;
  if (!d.causal) return (double)((items + sms - 1) / sms) * heaviest;
  if (items <= sms) return heaviest;
  double total = 0;
  for (int64_t g = 0; g < groups; ++g) {
    const int64_t last_row = std::min<int64_t>((g + 1) * tiles_per_item * BM, d.S_q) - 1;
    total += step * (double)std::min<int64_t>(all, std::max<int64_t>(0, last_row + off) / BN + 1) + kItem;
  }
  return std::max(heaviest, (double)heads * total / sms + 0.5 * total / (double)groups);
}
// A lone tile's key tiles are worth sharing from two on in the normalised mode (33 heads x 251 11.8 -> 10.4 us) and from three
// on in the single pass, where with two the meeting of the groups costs what it saves (48 heads x 159 9.4 us, 9.7 split).
bool split_keys_pay(const frisk_b200_attn_desc& d) { return d.S_kv > (d.normalize_p ? BN : 2 * BN); }

bool one_tile_items(const frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d) {
  const int64_t tiles = (d.S_q + BM - 1) / BM * d.B * d.H;
  if (tiles <= ctx->num_sms) return true;
  // (four rounds of pairs balance by themselves)
  if (!split_keys_pay(d) || tiles > 8 * (int64_t)ctx->num_sms) return false;
  return items_estimate(d, ctx->num_sms, 1) < (d.normalize_p ? 0.95 : 0.9) * items_estimate(d, ctx->num_sms, 2);
}

template <bool BF16, int D, bool OUT_F32, bool NORM, bool SPLIT>
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
  p.group_rows = one_tile_items(ctx, d) ? BM : 2 * BM;
  p.n_groups = (d.S_q + p.group_rows - 1) / p.group_rows;
  p.causal = d.causal ? 1 : 0;
  p.total_items = (int64_t)p.n_groups * bh;
  p.scale_log2 = d.scale * 1.4426950408889634f;
  p.scale = d.scale;
  p.normalized = d.normalize_p ? 1 : 0;
  p.O = O;
  p.status = ctx->d_status;
  p.work = ctx->d_status + 16;  // work counter and exit counter of the persistent grid (zero between launches)
  if (p.total_items > INT32_MAX) return FRISK_B200_E_ATTN_SHAPE;
  auto kern = attention_fwd_kernel<BF16, D, OUT_F32, NORM, SPLIT>;
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

template <bool BF16, int D, bool OUT_F32, bool NORM>
int launch_split(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K, const void* V,
                 void* O, cudaStream_t s) {
  // A lone query tile's key tiles go to the two softmax groups in turn: one group alone is
  // bound by the chain S -> softmax -> P.V -> next S (1.4 us a key tile at D = 64 normalised), and two such chains overlap.
  // 16 heads x 1025 normalised 29.2 -> 23.4 us; single pass, D = 128: 4 heads x 4096 causal 62.1 -> 40.4, 2 x 8192 121.4 -> 75.3,
  // 8 x 1000 19.8 -> 15.2; D = 64: 4 x 3000 42.5 -> 27.5.
  if (split_keys_pay(d) && one_tile_items(ctx, d)) return launch_cfg<BF16, D, OUT_F32, NORM, true>(ctx, d, Q, K, V, O, s);
  return launch_cfg<BF16, D, OUT_F32, NORM, false>(ctx, d, Q, K, V, O, s);
}

template <bool BF16, int D>
int launch_out(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K, const void* V,
               void* O, cudaStream_t s) {
  if (d.normalize_p) {
    if (d.dtype_out == FRISK_B200_F32) return launch_split<BF16, D, true, true>(ctx, d, Q, K, V, O, s);
    return launch_split<BF16, D, false, true>(ctx, d, Q, K, V, O, s);
  }
  if (d.dtype_out == FRISK_B200_F32) return launch_split<BF16, D, true, false>(ctx, d, Q, K, V, O, s);
  return launch_split<BF16, D, false, false>(ctx, d, Q, K, V, O, s);
}

}  // namespace

int launch_attention_fwd(frisk_b200_ctx* ctx, const frisk_b200_attn_desc& d, const void* Q, const void* K,
                         const void* V, void* O, cudaStream_t s) {
  if (attention_decode_preferred(d)) return launch_attention_decode(ctx, d, Q, K, V, O, s);
  const bool bf = d.dtype_in == FRISK_B200_BF16;
  if (d.D == 128) return bf ? launch_out<true, 128>(ctx, d, Q, K, V, O, s) : launch_out<false, 128>(ctx, d, Q, K, V, O, s);
  if (d.D == 64) return bf ? launch_out<true, 64>(ctx, d, Q, K, V, O, s) : launch_out<false, 64>(ctx, d, Q, K, V, O, s);
  return FRISK_B200_E_ATTN_SHAPE;
}

}  // namespace fb
