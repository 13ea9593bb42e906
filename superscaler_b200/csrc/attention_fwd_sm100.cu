// Flash-attention forward for sm_100a: two query tiles per CTA in ping-pong, probabilities kept in tensor memory.
//
// Replaces four reference ops and three CUDA extensions at once: ParallelAttentionScoreOp (baddbmm),
// ParallelSoftmaxFusionOp (scaled [causal|masked] softmax), ParallelSoftmaxDropoutOp and ParallelContextOp (bmm) --
// runtime/megatron/model/flex_ops.py:711-1015 -- without ever writing the [b, np, sq, sk] score matrix to memory.
//
// A work item is 256 queries of one (batch, head), two tiles of 128; where that leaves SMs idle or unequally loaded, one tile
// whose even and odd key blocks go to the two slots, each with a maximum, a sum and an accumulator of its own that are brought
// together at the end (one sequence of 16 causal heads of 2048 x 128: 41.4 -> 27.5 us, 4 of 1024 22.7 -> 15.1).  Every slot has
// eight softmax warps; two threads share a query row (64 keys of a block each) and exchange one maximum per block through
// shared memory.
// Per key block of 128 and tile:
//   S   = Q . K_j^T       fp32 accumulator in TMEM columns [128 t, 128 t + 128)
//   softmax warps: S -> registers, running maximum, P = exp2(..) as bf16 -> TMEM, each half over its own columns of S
//   O  += P . V_j         P is the A operand straight from TMEM; accumulator in columns [256 + 128 t, .. + HD)
// While the tensor core runs O += P V and the next S of one tile, the softmax warps of the other tile work: both units
// stay busy and P never passes through shared memory.  (Published ideas: two query tiles in ping-pong, FlashAttention-3; P as an
// operand in tensor memory, FlashAttention-4.)
// The accumulator O stays in TMEM in the frame of the running maximum; where that grew for a row of a warp, the warp rescales
// its columns of O itself, after its exponentials, when the registers of the scores are free again.  The row's largest
// probability is then exactly one when it is rounded to bf16.  A reference that may lag by 2^8 saves most of these passes, but
// rounds that probability: 2048 keys with scores of spread 3, relative error of O 2.24e-3 instead of 1.78e-3.  It gains 3 %
// unmasked (510 instead of 525 us, 16 x 16 heads of 2048 x 128) and nothing under the causal mask (348 instead of 340); one
// sequence takes 41.0 either way, 43.6 with the pass in front of the exponentials.  P is a bf16 operand; the sums of the
// unrounded probabilities and the products are fp32.
//
// The kernel is persistent (one CTA per SM): the loads and the first product of the next item run under the epilogue
// of the previous one.  Under the causal mask items are numbered heavy (late) query blocks first over all heads and
// dealt out in snake order: the busiest SM gets 1.01 to 1.09 of the mean for 64 to 256 heads of 2048 tokens, without a
// counter in memory (grouping heads for the L2 instead left 1.15 to 1.33; K and V at 3 TB/s do not bound the kernel).
// Without the mask all items cost the same and neighbours share a head.
//
// Measured against the one-tile kernel it replaces (128 queries a CTA, P through shared memory, four threads a row): causal,
// 16 x 16 heads of 2048 x 128: 589 -> 340 us (808 TFLOP/s), with dropout 803 -> 395 us, unmasked 931 -> 525 us (1045 TFLOP/s);
// one sequence of 16 heads 58.9 -> 41.0 us.  With one thread per row and four warps per tile the dropout form took 434 to
// 449 us and T5's (bias, dropout, head size 64) 160 instead of 137: two warps per SM sub-partition could not cover the chain
// S -> maximum -> exponentials -> P.  Tried on top, no gain: starting P.V on three quarters of the keys; slower: a separate
// warpgroup for the masks (664 us, its hashes take longer than a step).
//
// Warps: 0 = TMA producer, 1 = TMEM allocator + MMA issuer, 2 and 3 idle, then per tile 8 softmax warps (4 per half row).
#include "attention_device.cuh"

namespace ssb {

int make_tma_batched_bf16(CUtensorMap* map, const void* base, uint64_t batches, uint64_t rows, uint64_t ld,
                          uint32_t box_rows, uint32_t box_cols);

namespace {

using namespace attn;
// The thread that issues the products looks at its barriers without a suspend-time hint: its wake-up is on the path of every step
// (16 x 16 heads of 2048 x 128 causal 346 -> 342 us; looking without suspending at all takes issue slots from the softmax warps,
// 384 -> 400 with dropout).
constexpr MbarLook kIssueLook = MbarLook::kBrief;

constexpr int kFwdThreads = 640;   // five warpgroups: {TMA, MMA, 2 idle}, then two (column halves) per tile
// Register split: 640 threads are launched with 96 registers each (61440 in all); the first warpgroup keeps 64 and the four
// softmax warpgroups take 104: 128 * 64 + 512 * 104 = 61440.
constexpr int kFwdRegsOther = 64, kFwdRegsSoftmax = 104;

template <int HD>
struct FwdCfg {
  static constexpr int kCh = HD / 64;
  static constexpr int kTile = 128 * HD * 2;               // Q / K / V tile of 128 rows
  static constexpr int kStages = HD == 128 ? 4 : 6;        // K and V tiles in flight, in the order K0 V0 K1 V1 ...
  static constexpr int kOutBytes = 16 * 32 * 64;           // per softmax warp: 32 rows x 32 output columns
  static constexpr int kXchBytes = 2 * 2 * 128 * 4;        // row maxima: [tile][half][row]
  static constexpr int kBarBytes = 256;
  // Score bias, per softmax warp: the distances of its 32 queries x 64 keys (32 x 16 heads of 512 x 64 with bias and dropout 121 ->
  // 101 us).  No room at head size 128 (read from global memory).
  static constexpr int kBiasBytes = HD == 64 ? 16 * 96 * 4 : 0;
  static constexpr int kSmem = 2 * kTile + kStages * kTile + kOutBytes + kXchBytes + kBarBytes + kBiasBytes;
  static constexpr int kTmemCols = 512;                    // S/P 0, S/P 1, O 0, O 1: 128 columns each
};

struct FwdItems {
  int total, n_qb, heads;  // work items, query blocks per head, B * NH
  int split;               // 0: a block is two tiles of 128 queries; 1: one tile, its key blocks dealt to the two slots in turn
};

struct FwdItem {
  int head, b, q0, kv_len, n[2];
};

__device__ __forceinline__ FwdItem fwd_item(int idx, const FwdItems& it, const AttnParams& p) {
  FwdItem w;
  const int outer = idx / (p.causal ? it.heads : it.n_qb), inner = idx - outer * (p.causal ? it.heads : it.n_qb);
  const int qb = p.causal ? it.n_qb - 1 - outer : inner;
  const int hh = p.causal ? inner : outer;
  w.b = hh / p.NH;
  w.head = hh - w.b * p.NH;
  w.q0 = qb * (it.split ? 128 : 256);
  w.kv_len = p.kv_lens ? max(0, min(p.kv_lens[w.b], p.SK)) : p.SK;
  const int n_kv = (w.kv_len + 127) >> 7;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int qt = w.q0 + (it.split ? 0 : t * 128);
    const int n = qt >= p.SQ ? 0 : (p.causal ? min(n_kv, (qt >> 7) + 1) : n_kv);
    w.n[t] = it.split ? (n + 1 - t) >> 1 : n;
  }
  return w;
}

// Index of this CTA's k-th item, or -1 past the end (odd rounds run backwards through the CTAs).
__device__ __forceinline__ int fwd_item_index(int k, int total) {
  const int base = k * static_cast<int>(gridDim.x);
  if (base >= total) return -1;
  return base + ((k & 1) ? static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x));
}

// Bytes of four keys for this lane's query: lane `sub` of a query quad holds the hash of key `sub` (byte i decides query
// i); a 4 x 4 byte transpose inside the quad leaves byte e = the byte of key e for this lane's query.
__device__ __forceinline__ uint32_t quad_transpose(uint32_t h, uint32_t sel1, uint32_t sel2) {
  const uint32_t r1 = __shfl_xor_sync(0xffffffffu, h, 1);
  const uint32_t x = __byte_perm(h, r1, sel1);
  const uint32_t r2 = __shfl_xor_sync(0xffffffffu, x, 2);
  return __byte_perm(x, r2, sel2);
}

template <int HD, bool DROPOUT, bool BIAS, bool SPLIT>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const AttnParams p, const FwdItems items) {
  using Cfg = FwdCfg<HD>;
  constexpr int CH = Cfg::kCh, NS = Cfg::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;                          // 2 tiles
  uint8_t* sKV = sQ + 2 * Cfg::kTile;          // NS stages
  uint8_t* sOut = sKV + NS * Cfg::kTile;
  float* sXch = reinterpret_cast<float*>(sOut + Cfg::kOutBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + Cfg::kOutBytes + Cfg::kXchBytes);
  uint64_t* q_full = bars;             // 2
  uint64_t* q_empty = bars + 2;        // 2: the last S of the tile retired
  uint64_t* s_full = bars + 4;         // 2: S of a block complete (and with it P.V of the block before)
  uint64_t* p_full = bars + 6;         // 2 (one arrival per softmax warp): P written, O rescaled if need be
  uint64_t* o_full = bars + 8;         // 2: last P.V of the item complete
  uint64_t* kv_full = bars + 10;       // NS
  uint64_t* kv_empty = bars + 10 + NS; // NS
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10 + 2 * NS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1);
      mbar_init(&q_empty[t], 1);
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t], 8);
      mbar_init(&o_full[t], 1);
    }
    for (int s = 0; s < NS; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 4) {
    reg_dealloc<kFwdRegsOther>();  // one instruction for the whole warpgroup
    // ------------------------------------------ TMA producer ------------------------------------------
    if (warp == 0 && elect_one()) {
      Pipe pp;
      uint32_t qn[2] = {0, 0};  // items loaded per tile
      bool ok = true;
      auto load_kv = [&](const CUtensorMap* tm, int col0, int row, int b) {
        if (!mbar_wait(&kv_empty[pp.stage], pp.phase ^ 1, abort_flag)) return false;
        mbar_arrive_expect_tx(&kv_full[pp.stage], Cfg::kTile);
#pragma unroll
        for (int c = 0; c < CH; ++c)
          tma_load_3d(sKV + pp.stage * Cfg::kTile + c * 16384, tm, &kv_full[pp.stage], col0 + c * 64, row, b);
        pp.advance(NS);
        return true;
      };
      for (int k = 0, idx; ok && (idx = fwd_item_index(k, items.total)) >= 0; ++k) {
        if (idx >= items.total) continue;
        const FwdItem w = fwd_item(idx, items, p);
        const int kcol = p.k_col0 + w.head * HD, vcol = p.v_col0 + w.head * HD;
        if constexpr (SPLIT) {  // Q K0 K1 V0 K2 V1 K3 ...
          const int n = w.n[0] + w.n[1];
          if (n == 0) continue;
          if (!mbar_wait(&q_empty[0], (qn[0] & 1) ^ 1, abort_flag)) { ok = false; break; }
          mbar_arrive_expect_tx(&q_full[0], Cfg::kTile);
#pragma unroll
          for (int c = 0; c < CH; ++c)
            tma_load_3d(sQ + c * 16384, &tm_q, &q_full[0], p.q_col0 + w.head * HD + c * 64, w.q0, w.b);
          ++qn[0];
          ok = load_kv(&tm_k, kcol, 0, w.b);
          if (ok && n > 1) ok = load_kv(&tm_k, kcol, 128, w.b);
          for (int j = 0; j < n && ok; ++j) {
            ok = load_kv(&tm_v, vcol, j * 128, w.b);
            if (ok && j + 2 < n) ok = load_kv(&tm_k, kcol, (j + 2) * 128, w.b);
          }
          continue;
        }
        const int n = max(w.n[0], w.n[1]);
        for (int t = 0; t < 2 && ok && n > 0; ++t) {
          if (w.n[t] > 0) {
            if (!mbar_wait(&q_empty[t], (qn[t] & 1) ^ 1, abort_flag)) { ok = false; break; }
            mbar_arrive_expect_tx(&q_full[t], Cfg::kTile);
#pragma unroll
            for (int c = 0; c < CH; ++c)
              tma_load_3d(sQ + t * Cfg::kTile + c * 16384, &tm_q, &q_full[t], p.q_col0 + w.head * HD + c * 64,
                          w.q0 + t * 128, w.b);
            ++qn[t];
          }
          if (t == 0) ok = load_kv(&tm_k, kcol, 0, w.b);
        }
        for (int j = 0; j < n && ok; ++j) {
          ok = load_kv(&tm_v, vcol, j * 128, w.b);
          if (ok && j + 1 < n) ok = load_kv(&tm_k, kcol, (j + 1) * 128, w.b);
        }
      }
      if (!ok) {  // let the copies in flight land before the CTA leaves
        for (int t = 0; t < 2; ++t)
          for (uint32_t it = 0; qn[t] > 0 && it < (1u << 20); ++it)
            if (mbar_try_wait(&q_full[t], (qn[t] - 1) & 1)) break;
        for (int s = 0; s < NS; ++s) {
          const uint32_t armed = (s < pp.stage) ? pp.phase : (pp.phase ^ 1);
          for (uint32_t it = 0; it < (1u << 20); ++it)
            if (mbar_try_wait(&kv_full[s], armed)) break;
        }
      }
    }
    // ------------------------------------------ MMA issuer --------------------------------------------
    if (warp == 1 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, false, false);
      constexpr uint32_t idesc_o = umma_idesc_bf16(128, HD, false, true);
      // one descriptor per operand; a step along it is an addition to the address field
      const uint64_t q_k = umma_desc_sw128(smem_u32(sQ), 16, 1024), kv_k = umma_desc_sw128(smem_u32(sKV), 16, 1024);
      const uint64_t kv_mn = umma_desc_sw128(smem_u32(sKV), 16384, 1024);
      constexpr uint64_t kStep = Cfg::kTile >> 4;
      Pipe pp;                               // next K / V stage to consume
      uint32_t qn[2] = {0, 0}, pn[2] = {0, 0};
      bool ok = true;
      auto issue_s = [&](int t, int qtile, int stage) {
        const uint64_t a = q_k + qtile * kStep, bb = kv_k + stage * kStep;
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          umma_f16_ss(tmem_base + t * 128, a + off, bb + off, idesc_s, kk != 0);
        }
        umma_commit(&s_full[t]);
      };
      auto issue_o = [&](int t, int stage, bool accumulate) {
        const uint64_t bb = kv_mn + stage * kStep;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)  // 128 keys = 8 steps of 16 (8 TMEM columns of packed bf16 pairs)
          umma_f16_ts(tmem_base + 256 + t * 128, tmem_base + t * 128 + (kk >> 2) * 64 + (kk & 3) * 8, bb + (kk * 2048 >> 4),
                      idesc_o, accumulate || kk != 0);
      };
      for (int k = 0, idx; ok && (idx = fwd_item_index(k, items.total)) >= 0; ++k) {
        if (idx >= items.total) continue;
        const FwdItem w = fwd_item(idx, items, p);
        if constexpr (SPLIT) {
          const int n = w.n[0] + w.n[1];
          if (n == 0) continue;
          if (!(ok = mbar_wait<kIssueLook>(&q_full[0], qn[0] & 1, abort_flag))) break;
          ++qn[0];
          auto next_s = [&](int j) {  // scores of key block j
            if (!(ok = mbar_wait<kIssueLook>(&kv_full[pp.stage], pp.phase, abort_flag))) return;
            tc_fence_after_sync();
            issue_s(j & 1, 0, pp.stage);
            umma_commit(&kv_empty[pp.stage]);
            if (j + 1 == n) umma_commit(&q_empty[0]);
            pp.advance(NS);
          };
          for (int j = 0; j < min(n, 2) && ok; ++j) next_s(j);
          for (int j = 0; j < n && ok; ++j) {
            const int t = j & 1;
            if (!(ok = mbar_wait<kIssueLook>(&kv_full[pp.stage], pp.phase, abort_flag))) break;
            if (!(ok = mbar_wait<kIssueLook>(&p_full[t], pn[t] & 1, abort_flag))) break;
            ++pn[t];
            tc_fence_after_sync();
            issue_o(t, pp.stage, j >= 2);
            umma_commit(&kv_empty[pp.stage]);
            pp.advance(NS);
            if (j + 2 < n) next_s(j + 2);  // overwrites S / P of the slot: products retire in issue order
            else umma_commit(&o_full[t]);
          }
          continue;
        }
        const int n = max(w.n[0], w.n[1]);
        if (n == 0) continue;
        int sk = pp.stage;
        if (!mbar_wait<kIssueLook>(&kv_full[sk], pp.phase, abort_flag)) break;
        for (int t = 0; t < 2 && ok; ++t) {
          if (w.n[t] == 0) continue;
          if (!mbar_wait<kIssueLook>(&q_full[t], qn[t] & 1, abort_flag)) { ok = false; break; }
          ++qn[t];
          tc_fence_after_sync();
          issue_s(t, t, sk);
          if (w.n[t] == 1) umma_commit(&q_empty[t]);
        }
        if (!ok) break;
        umma_commit(&kv_empty[sk]);
        pp.advance(NS);
        for (int j = 0; j < n && ok; ++j) {
          const int sv = pp.stage;
          const uint32_t phv = pp.phase;
          pp.advance(NS);
          sk = pp.stage;
          bool have_v = false, have_k = false;
          for (int t = 0; t < 2; ++t) {
            if (j >= w.n[t]) continue;
            if (!have_v && !mbar_wait<kIssueLook>(&kv_full[sv], phv, abort_flag)) { ok = false; break; }
            have_v = true;
            if (!mbar_wait<kIssueLook>(&p_full[t], pn[t] & 1, abort_flag)) { ok = false; break; }
            ++pn[t];
            tc_fence_after_sync();
            issue_o(t, sv, j != 0);
            if (j + 1 == w.n[t]) {
              umma_commit(&o_full[t]);
            } else {
              if (!have_k && !mbar_wait<kIssueLook>(&kv_full[sk], pp.phase, abort_flag)) { ok = false; break; }
              have_k = true;
              tc_fence_after_sync();
              issue_s(t, t, sk);  // overwrites S / P of the tile: products retire in issue order
              if (j + 2 == w.n[t]) umma_commit(&q_empty[t]);
            }
          }
          if (!ok) break;
          umma_commit(&kv_empty[sv]);
          if (j + 1 < n) {
            umma_commit(&kv_empty[sk]);
            pp.advance(NS);
          }
        }
      }
    }
  } else {
    // ------------------------------------------ softmax warps -----------------------------------------
    reg_alloc<kFwdRegsSoftmax>();
    const int quarter = warp & 3;
    const int t = (warp - 4) >> 3, half = ((warp - 4) >> 2) & 1;  // tile; keys [64 half, 64 half + 64) of a block
    const int r = quarter * 32 + lane;
    const uint32_t tm_row = tmem_base + t * 128 + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t tm_s = tm_row + half * 64, tm_o = tm_row + 256 + half * (HD / 2);
    uint8_t* stage = sOut + (warp - 4) * 2048;
    float* xch = sXch + t * 256 + r;   // + half * 128
    float* sBias = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + Cfg::kBarBytes) + (warp - 4) * 96;
    // The two warps that share these 32 rows meet once per key block and twice per item.
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + t * 4 + quarter) : "memory"); };
    // The end of an item: with split keys the four warps of both slots that hold partial results of these rows.
    auto end_sync = [&]() {
      if constexpr (SPLIT) asm volatile("bar.sync %0, 128;" ::"r"(9 + quarter) : "memory");
      else pair_sync();
    };
    // A warp whose bounded wait ran out in its k-th item, `left` blocks before the item's end, still comes to all the
    // meetings ahead: its partner may pass the same wait a moment later and must not be left waiting (its own next wait runs
    // out too, P of this warp being missing).  An mbarrier with the bounded wait at every meeting costs 10 % (one sequence of
    // 16 heads 41.0 -> 45.1 us), a barrier that tells both whether one gave up 5 % (43.0).
    auto meet_to_the_end = [&](int k, int left) {
      for (int idx;;) {
        for (; left > 0; --left) pair_sync();
        end_sync();
        end_sync();
        FwdItem w;
        do {
          if ((idx = fwd_item_index(++k, items.total)) < 0) return;
          if (idx < items.total) w = fwd_item(idx, items, p);
        } while (idx >= items.total || (!SPLIT && w.q0 + t * 128 >= p.SQ));
        left = w.n[t];
      }
    };
    const float c = p.scale * kLog2e;
    // With a bias the logits are brought into the log2 domain first (x c + bias log2 e) and everything below works on
    // them with a factor of one; without it the raw accumulator is used and the factor is c.
    const float cc = BIAS ? 1.0f : c;
    const uint32_t keep8 = dropout_keep8(p.dropout_p);
    const float inv_keep = DROPOUT ? 256.0f / static_cast<float>(keep8) : 1.0f;  // applied once, to O
    const uint32_t qquads = (p.SQ + 3) >> 2;
    const int sub = lane & 3;
    const uint32_t sel1 = (lane & 1) ? 0x3715u : 0x6240u, sel2 = (lane & 2) ? 0x3276u : 0x5410u;
    const uint32_t drop_c = (256u - keep8) * 0x01010101u;  // byte + drop_c carries out <=> byte >= keep8
    uint32_t sn = 0, on0 = 0, on1 = 0;  // blocks of this slot so far; items with work for slot 0 and slot 1
    bool ok = true;
    for (int k = 0, idx; ok && (idx = fwd_item_index(k, items.total)) >= 0; ++k) {
      if (idx >= items.total) continue;
      const FwdItem w = fwd_item(idx, items, p);
      const int qt = w.q0 + (SPLIT ? 0 : t * 128), q = qt + r;
      if (qt >= p.SQ) continue;
      const int j0 = SPLIT ? t : 0, dj = SPLIT ? 2 : 1;  // key blocks of this slot: j0, j0 + dj, ...
      const int nt = w.n[t];
      uint32_t hash_base = 0, hash_step = 0;
      if constexpr (DROPOUT) {
        // attn_col_hash mixes (key qquads + quad) * 0x9E3779B1 + seed: linear in the key, so a step of four keys is an add
        const uint32_t bh_seed = static_cast<uint32_t>(hash64(p.dropout_seed, static_cast<uint64_t>(w.b) * p.NH + w.head));
        hash_base = (static_cast<uint32_t>(half * 64 + sub) * qquads + (static_cast<uint32_t>(q) >> 2)) * 0x9E3779B1u + bh_seed;
        hash_step = 4u * qquads * 0x9E3779B1u;
        hash_base += static_cast<uint32_t>(32 * j0) * hash_step;
      }
      const float* bias_row = BIAS ? p.bias_table + static_cast<size_t>(w.head) * (p.SQ + p.SK - 1) + (p.SQ - 1) - min(q, p.SQ - 1)
                                   : nullptr;
      float m = -INFINITY, l = 0.f;
      for (int j = 0; j < nt; ++j) {
        const int kv0 = (j0 + j * dj) * 128 + half * 64;
        if constexpr (BIAS && HD == 64) {  // (the reads of the block before are behind this warp's arrival)
          const float* head_row = p.bias_table + static_cast<size_t>(w.head) * (p.SQ + p.SK - 1);
          const int d = p.SQ - 32 - (qt + quarter * 32) + kv0 + lane;  // distance of (query 31, key 0) of this warp, + lane
#pragma unroll
          for (int i = 0; i < 3; ++i) sBias[i * 32 + lane] = __ldg(head_row + min(max(d + i * 32, 0), p.SQ + p.SK - 2));
          __syncwarp();
        }
        if (!mbar_wait_warp(&s_full[t], sn & 1, abort_flag)) {
          meet_to_the_end(k, nt - j);
          ok = false;
          break;
        }
        ++sn;
        tc_fence_after_sync();
        const bool masked = (p.causal && kv0 + 63 > qt) || kv0 + 64 > w.kv_len;  // diagonal block or ragged end
        const int lim = min(w.kv_len - 1, p.causal ? q : w.kv_len) - kv0;        // last visible key of this row
        auto prepare = [&](uint32_t (&x)[32], int k0) {
          if constexpr (BIAS && HD == 64) {
            const float* br = sBias + 31 - lane + k0;
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = __float_as_uint(fmaf(__uint_as_float(x[i]), c, br[i] * kLog2e));
          } else if constexpr (BIAS) {
            const float* br = bias_row + kv0 + k0;
            if (kv0 + 64 <= p.SK) {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                x[i] = __float_as_uint(fmaf(__uint_as_float(x[i]), c, __ldg(br + i) * kLog2e));
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                x[i] = __float_as_uint(fmaf(__uint_as_float(x[i]), c, __ldg(bias_row + min(kv0 + k0 + i, p.SK - 1)) * kLog2e));
            }
          }
          if (masked) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (k0 + i > lim) x[i] = 0xff800000u;  // -inf
          }
        };
        auto row_max = [&](const uint32_t (&x)[32], const uint32_t (&y)[32], float start) {  // four independent chains
          float mm[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            mm[e] = fmaxf(__uint_as_float(x[e]), __uint_as_float(y[e]));
#pragma unroll
            for (int i = 4; i < 32; i += 4) mm[e] = fmaxf(mm[e], fmaxf(__uint_as_float(x[e + i]), __uint_as_float(y[e + i])));
          }
          return fmaxf(fmaxf(fmaxf(mm[0], mm[1]), fmaxf(mm[2], mm[3])), start);
        };
        uint32_t x0[32], x1[32];
        tmem_ld_32x32(tm_s, x0);
        tmem_ld_32x32(tm_s + 32, x1);
        tmem_ld_wait();
        prepare(x0, 0);
        prepare(x1, 32);
        float mx = row_max(x0, x1, -INFINITY);
        // The other half of the row: its maximum.  The slot is free again for the next block: its scores (s_full) follow
        // this block's P of both halves, hence both reads.
        xch[half * 128] = mx;
        pair_sync();
        mx = fmaxf(mx, xch[(half ^ 1) * 128]);
        const bool grown = j > 0 && __any_sync(0xffffffffu, mx > m);
        const float mn = fmaxf(m, mx);
        const float alpha = grown && mn != -INFINITY ? ex2((m - mn) * cc) : 1.f;  // from m = -inf: 0 (O and l are zero)
        m = mn;
        const float mc = (m == -INFINITY) ? 0.f : m * cc;  // no visible key: keep the exponents finite
        float2 rs[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        const float2 c2 = make_float2(cc, cc), nm2 = make_float2(-mc, -mc);
        auto exponentials = [&](const uint32_t (&x)[32], int ch) {
          uint32_t pw[8];
          uint32_t hash = hash_base + static_cast<uint32_t>(ch * 8) * hash_step;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float2 a = fma_f32x2(make_float2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])), c2, nm2);
            float2 b2 = fma_f32x2(make_float2(__uint_as_float(x[i + 2]), __uint_as_float(x[i + 3])), c2, nm2);
            a.x = ex2(a.x);  // masked entries: ex2(-inf) = 0
            a.y = ex2(a.y);
            b2.x = ex2(b2.x);
            b2.y = ex2(b2.y);
            rs[0] = add_f32x2(rs[0], a);
            rs[1] = add_f32x2(rs[1], b2);
            uint32_t w0 = pack_bf16x2(a.x, a.y), w1 = pack_bf16x2(b2.x, b2.y);
            if constexpr (DROPOUT) {
              const uint32_t xb = quad_transpose(fmix32(hash), sel1, sel2);
              hash += hash_step;
              const uint32_t cs = (xb & 0x7f7f7f7fu) + (drop_c & 0x7f7f7f7fu);
              const uint32_t d = (xb & drop_c) | ((xb | drop_c) & cs);  // bit 7 of byte e: carry out of that byte
              w0 &= ~spread_sign_bytes(d, 0x9988);                        // sign bits of bytes 0, 1 spread over a half each
              w1 &= ~spread_sign_bytes(d, 0xBBAA);
            }
            pw[(i >> 1) & 7] = w0;
            pw[((i >> 1) + 1) & 7] = w1;
            if ((i & 15) == 12) tmem_st_32x8(tm_s + ch * 16 + (i >> 4) * 8, pw);
          }
        };
        exponentials(x0, 0);
        exponentials(x1, 1);
        hash_base += static_cast<uint32_t>(32 * dj) * hash_step;
        if (grown) {  // into the new frame; P.V of the block before completed with s_full (products retire in issue order)
          const float2 a2 = make_float2(alpha, alpha);
#pragma unroll
          for (int ch = 0; ch < HD / 64; ++ch) {  // this half's columns of O
            uint32_t oo[32];
            tmem_ld_32x32(tm_o + ch * 32, oo);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float2 o2 = mul_f32x2(make_float2(__uint_as_float(oo[i]), __uint_as_float(oo[i + 1])), a2);
              oo[i] = __float_as_uint(o2.x);
              oo[i + 1] = __float_as_uint(o2.y);
            }
            tmem_st_32x32(tm_o + ch * 32, oo);
          }
        }
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrive(&p_full[t], lane);
        l = l * alpha + ((rs[0].x + rs[0].y) + (rs[1].x + rs[1].y));
      }
      if (!ok) break;
      // (both slots' sums where they share the tile)
      if constexpr (SPLIT) {
        if (w.n[0] > 0) ok = mbar_wait_warp(&o_full[0], on0++ & 1, abort_flag);
        if (ok && w.n[1] > 0) ok = mbar_wait_warp(&o_full[1], on1++ & 1, abort_flag);
      } else if (nt > 0) {
        ok = mbar_wait_warp(&o_full[t], on0++ & 1, abort_flag);
      }
      if (!ok) {
        meet_to_the_end(k, 0);
        break;
      }
      tc_fence_after_sync();
      // Row sums of the halves, added in one order by all (in the staging tiles, which are free here); with split keys also
      // the other slot's frame: factor f[u] brings slot u's sum and O into the common one.
      float f0 = 1.f, f1 = 0.f;
      {
        float* mine = reinterpret_cast<float*>(stage) + lane;
        auto of = [&](int slot, int hf) { return reinterpret_cast<const float*>(sOut + (slot * 8 + hf * 4 + ((warp - 4) & 3)) * 2048) + lane; };
        mine[0] = l;
        if constexpr (SPLIT) mine[32] = m;
        end_sync();
        const int own = SPLIT ? 0 : t;
        l = of(own, 0)[0] + of(own, 1)[0];
        if constexpr (SPLIT) {
          const float m0 = of(0, 0)[32], m1 = of(1, 0)[32];
          m = fmaxf(m0, m1);
          f0 = m0 == -INFINITY ? 0.f : ex2((m0 - m) * cc);
          f1 = m1 == -INFINITY ? 0.f : ex2((m1 - m) * cc);
          l = l * f0 + (of(1, 0)[0] + of(1, 1)[0]) * f1;
        } else {
          end_sync();
        }
      }
      const float inv_l = l > 0.f ? inv_keep / l : 0.f;
      // 32 (16) columns at a time through shared memory: 64- (32-)byte row segments to memory
      const int rows_left = p.SQ - qt - quarter * 32;
      __nv_bfloat16* obase = reinterpret_cast<__nv_bfloat16*>(p.O) + (static_cast<size_t>(w.b) * p.SQ + qt + quarter * 32) * p.ldo +
                             p.o_col0 + w.head * HD + half * (HD / 2);
      auto put = [&](auto& oo, int col) {  // a row's values -> row segments of O from column `col` of this half
        constexpr int W = sizeof(oo) / 4, PIECES = W / 8, RPI = 32 / PIECES;
        auto cell = [&](int row, int piece) { return stage + row * (W * 2) + ((piece ^ ((row >> (W == 32 ? 1 : 2)) & (PIECES - 1))) << 4); };
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
          uint4 v;
          v.x = pack_bf16x2(__uint_as_float(oo[8 * i + 0]), __uint_as_float(oo[8 * i + 1]));
          v.y = pack_bf16x2(__uint_as_float(oo[8 * i + 2]), __uint_as_float(oo[8 * i + 3]));
          v.z = pack_bf16x2(__uint_as_float(oo[8 * i + 4]), __uint_as_float(oo[8 * i + 5]));
          v.w = pack_bf16x2(__uint_as_float(oo[8 * i + 6]), __uint_as_float(oo[8 * i + 7]));
          *reinterpret_cast<uint4*>(cell(lane, i)) = v;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32 / RPI; ++i) {
          const int row = i * RPI + lane / PIECES, piece = lane % PIECES;
          const uint4 v = *reinterpret_cast<const uint4*>(cell(row, piece));
          if (row < rows_left) *reinterpret_cast<uint4*>(obase + static_cast<size_t>(row) * p.ldo + col + piece * 8) = v;
        }
        __syncwarp();
      };
      if constexpr (SPLIT) {
        // a quarter of the columns per warp: O of both slots, added in the common frame
        constexpr int W = HD / 4;
        const uint32_t src = tmem_base + 256 + (static_cast<uint32_t>(quarter * 32) << 16) + half * (HD / 2) + t * W;
        uint32_t oo[W], ot[W];
#pragma unroll
        for (int i = 0; i < W; ++i) oo[i] = ot[i] = 0u;
        if (w.n[0] > 0) tmem_ld_cols<W>(src, oo);
        if (w.n[1] > 0) tmem_ld_cols<W>(src + 128, ot);
        tmem_ld_wait();
        // everyone's reads of O and of the exchanged sums are done: the staging tiles and, for the next item's first P.V, O
        // are free
        tc_fence_before_sync();
        end_sync();
        tc_fence_after_sync();
        f0 *= inv_l;
        f1 *= inv_l;
#pragma unroll
        for (int i = 0; i < W; ++i)
          oo[i] = __float_as_uint(fmaf(__uint_as_float(ot[i]), f1, __uint_as_float(oo[i]) * f0));
        put(oo, t * W);
      } else {
#pragma unroll
        for (int ch = 0; ch < HD / 64; ++ch) {
          uint32_t oo[32];
          if (nt > 0) {
            tmem_ld_32x32(tm_o + ch * 32, oo);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) oo[i] = 0u;
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) oo[i] = __float_as_uint(__uint_as_float(oo[i]) * inv_l);
          put(oo, ch * 32);
        }
      }
      // rows with no visible key get +inf so that the backward probabilities exp(s - lse) vanish
      if (half == 0 && (!SPLIT || t == 0) && q < p.SQ)
        p.LSE[(static_cast<size_t>(w.b) * p.NH + w.head) * p.SQ + q] =
            l > 0.f ? m * (BIAS ? 1.0f / kLog2e : p.scale) + logf(l) : INFINITY;
      // the reads of O are ordered before the next item's P.V by the p_full arrival of its first block
      tc_fence_before_sync();
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && p.status != nullptr) atomicMax(p.status, static_cast<int>(kStatusMbarTimeout));
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// Pairs of query tiles or single tiles with their key blocks split over the two slots: estimated time of the busiest SM, in tile
// steps.  A split step costs a tenth more (K and V are fetched for 128 queries instead of 256, the slots are brought together at
// the end), an item as much as 2.5 steps.  Without the mask all items are equal and whole rounds count; under it the longest item
// or the mean counts.  Measured, pairs / split in us, head size 128: 16 causal heads of 2048 40.2 / 27.5, 4 of 1024 22.7 / 15.1,
// 32 of 1024 24.2 / 20.2, 64 of 512 16.1 / 16.4, 32 of 2048 45.0 / 49.8; unmasked 16 of 1024 24.1 / 15.8, 16 of 2048 40.5 / 43.8,
// 40 of 2048 111.7 / 103.1, 256 of 1024 142.6 / 163.4.
bool fwd_split(long long heads, int SQ, int SK, int causal, int num_sms) {
  const long long tiles = (SQ + 127) / 128, pairs = (tiles + 1) / 2;
  const double n = (SK + 127) / 128, item = 2.5, step = 1.1;
  if (!causal) {
    const double rounds_pair = static_cast<double>((heads * pairs + num_sms - 1) / num_sms);
    const double rounds_split = static_cast<double>((heads * tiles + num_sms - 1) / num_sms);
    return rounds_split * (step * n + item) < rounds_pair * (2 * n + item);
  }
  const double steps = heads * n * (n + 1) / 2;
  const double longest = tiles % 2 ? (n > 2 * n - 3 ? n : 2 * n - 3) : 2 * n - 1;
  const double mean_pair = (steps + item * heads * pairs) / num_sms, mean_split = (step * steps + item * heads * tiles) / num_sms;
  const double pair = longest + item > mean_pair ? longest + item : mean_pair;
  const double split = step * n + item > mean_split ? step * n + item : mean_split;
  return 1.05 * split < pair;
}

template <int HD, bool DROPOUT, bool BIAS>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnParams& p, int num_sms,
               cudaStream_t stream) {
  FwdItems it;
  it.heads = p.B * p.NH;
  it.split = fwd_split(it.heads, p.SQ, p.SK, p.causal, num_sms);
  it.n_qb = (p.SQ + (it.split ? 127 : 255)) / (it.split ? 128 : 256);
  it.total = it.n_qb * it.heads;
  const int grid = it.total < num_sms ? it.total : num_sms;
  auto kernel = it.split ? attn_fwd_kernel<HD, DROPOUT, BIAS, true> : attn_fwd_kernel<HD, DROPOUT, BIAS, false>;
  const int rc = static_cast<int>(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdCfg<HD>::kSmem));
  if (rc) return rc;
  kernel<<<grid, kFwdThreads, FwdCfg<HD>::kSmem, stream>>>(tq, tk, tv, p, it);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

// Which form the forward takes: true where the key blocks of a query tile are split over the two slots.
bool attn_fwd_split(long long heads, int SQ, int SK, int causal, int num_sms) { return fwd_split(heads, SQ, SK, causal, num_sms); }

// q/k/v: base pointers of the 2-D matrices that hold the heads (see AttnParams); ld in elements.
int attn_fwd_launch(const void* q, int ldq, const void* k, int ldk, const void* v, int ldv, const AttnParams& p,
                    int num_sms, cudaStream_t stream) {
  if (p.HD != 64 && p.HD != 128) return -2;
  if (p.causal && p.SQ != p.SK) return -2;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (p.ldo % 8) || (p.q_col0 % 8) || (p.k_col0 % 8) || (p.v_col0 % 8) ||
      (p.o_col0 % 8))
    return -3;
  // Blocks past the end of a sample read zeros: a probability of zero times whatever the next sample holds there, an
  // infinity or NaN among it, must not enter this one.
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_tma_batched_bf16(&tq, q, p.B, p.SQ, ldq, 128, 64))) return rc;
  if ((rc = make_tma_batched_bf16(&tk, k, p.B, p.SK, ldk, 128, 64))) return rc;
  if ((rc = make_tma_batched_bf16(&tv, v, p.B, p.SK, ldv, 128, 64))) return rc;
  const bool drop = p.dropout_p > 0.f, bias = p.bias_table != nullptr;
#define SSB_FWD(HD, D, BI) launch_fwd<HD, D, BI>(tq, tk, tv, p, num_sms, stream)
  if (p.HD == 128)
    return drop ? (bias ? SSB_FWD(128, true, true) : SSB_FWD(128, true, false))
                : (bias ? SSB_FWD(128, false, true) : SSB_FWD(128, false, false));
  return drop ? (bias ? SSB_FWD(64, true, true) : SSB_FWD(64, true, false))
              : (bias ? SSB_FWD(64, false, true) : SSB_FWD(64, false, false));
#undef SSB_FWD
}

}  // namespace ssb
