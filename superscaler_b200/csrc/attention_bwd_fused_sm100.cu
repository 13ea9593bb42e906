// Flash-attention backward in ONE kernel for sm_100a: five tile GEMMs per (key block, query block) pair on tcgen05
// tensor cores instead of the seven of the dK/dV + dQ kernel pair, and one pass of the exponentials, the dropout mask
// and the dS arithmetic instead of two.
//
// Replaces the autograd of ParallelAttentionScoreOp / SoftmaxFusion / SoftmaxDropout / ContextOp
// (runtime/megatron/model/flex_ops.py:711-1015) together with the softmax backward kernels of the reference
// (runtime/megatron/fused_kernels/scaled_masked_softmax.h:329-423).
//
// A work item is 128 keys of one (batch, head); a CTA walks over the query blocks (128 queries each) that see them:
//   S^T  = K . Q_i^T          [128 keys x 128 queries]    TMEM columns [0, 128)
//   P^T  = exp2(S^T c - lse2) (x dropout mask)            bf16, over the columns of S^T the same warpgroup has read
//   dP^T = V . dO_i^T         [128 keys x 128 queries]    TMEM columns [128, 256)
//   dV  += P^T  . dO_i        [128 keys x HD]             A operand straight from TMEM
//   dS^T = P^T (dP^T mask - delta)                        bf16, shared memory
//   dQ   = dS . K             [128 queries x HD]          same tile read MN-major; over dP^T (HD 128), own columns (HD 64)
//   dK  += dS^T . Q_i         [128 keys x HD]
// The softmax scale is applied once, to dK and dQ, and the dropout scale of P once, to dV, at the end.
//
// dQ is one key block's share: four drain warps bring it from TMEM to shared memory, 64 columns at a time, and bulk
// reductions add it to an fp32 accumulator in global memory, laid out [tile][lane quarter][HD / 4][32 lanes][4] so that a
// warp's share is contiguous in both.  A small kernel scales the accumulator and writes the bf16 dQ matrix afterwards.  (As
// 16-byte reductions from registers the drain kept the load / store queues of all four sub-partitions full: the first product
// issued behind them waited 1000 to 1500 cycles of a step of 5900, and columns were released late.)  The order in which the key
// blocks add their shares is not fixed, so dQ can differ in the last bit from run to run; the two-kernel backward stays
// available for bitwise-reproducible runs.
//
// The kernel is persistent: a CTA takes over the blocks of the grid that have not started yet (cluster launch control), so
// that the loads, scores and probabilities of the next item run while the drain warps write dV and dK of the last one (tiled
// stores of 32 x 64).  With one item per CTA, start and end took 12000 of 22000 cycles at four steps an item.  Where no CTA gets a
// second item (MORE = false: at most as many as SMs) nothing is requested and the math warps, which have nothing else to do then,
// write dV and dK.
//
// Order of the tensor-core work (one issuing thread; products retire in issue order), step i:
//   dV_i (needs P_i) | S_{i+1} | dQ_i, dK_i (need dS_i) | dP_{i+1} (needs dQ_i drained at HD 128)
// The math warps turn S_{i+1} into P_{i+1} while dQ_i, dK_i and dP_{i+1} run, and dP_{i+1} into dS_{i+1} while dV_{i+1}
// and S_{i+2} run.
//
// Threads: warpgroup 0 = {TMA warp, MMA warp, two idle}, 1 .. 4 = math (warpgroup 1 + g: queries [32 g, 32 g + 32) of a block,
// one key row per thread), 5 = drain.  The math of a step is a chain of waits and dependent arithmetic: with two warpgroups
// of twice the columns (two warps per SM sub-partition) it, and not the tensor core, set the pace.
//
// The thread that issues the products waits as in the forward, without a suspend-time hint; looking without suspending at all is
// no faster (530 sizes: 1.000 in the geometric mean), nor in a training step under the power cap (58.7 samples/s either way).
//
// Measured (kernel alone; whole backward in brackets), with one item per CTA and dQ reduced from registers -> now: 16 x 16 heads
// of 2048 x 128 causal with dropout 951 -> 784 us (1111 -> 985), without (1073 -> 963), 4 x 16 unmasked (427 -> 370); 32 x 16
// heads of 512 x 64 with bias and dropout 280 -> 204 (345 -> 252), plain (235 -> 175).  What bounds it now: the reload of a Q stage
// (two fit; a product of the step before is its last reader) and the alternation of the two halves of the math.
#include "attention_device.cuh"

namespace ssb {

int make_tma_batched_bf16(CUtensorMap* map, const void* base, uint64_t batches, uint64_t rows, uint64_t ld,
                          uint32_t box_rows, uint32_t box_cols);

namespace {

using namespace attn;

constexpr MbarLook kIssueLook = MbarLook::kBrief;  // of the thread that issues the products
constexpr int kFusedThreads = 768;
constexpr int kFusedMathWarps = 16;
// Register split of the 768 x 80 registers the block is launched with: 128 (56 + 4 * 80 + 104) = 61440.
constexpr int kFusedRegsIssue = 56, kFusedRegsMath = 80, kFusedRegsDrain = 104;

template <int HD>
struct FusedCfg {
  static constexpr int kCh = HD / 64;
  static constexpr int kTile = 128 * HD * 2;      // K_j, V_j, Q_i (two stages), dO_i
  static constexpr int kDsBytes = 128 * 128 * 2;  // dS^T: two chunks of 64 queries
  static constexpr int kDoStages = HD == 128 ? 1 : 2, kKvStages = HD == 128 ? 1 : 2;
  static constexpr int kDqBytes = 4 * 8192;       // per drain warp: 32 queries x 64 columns of dQ in fp32
  static constexpr int kStatBytes = 2 * 128 * 4;  // -lse2 and -delta of a query block, per Q stage
  static constexpr int kBarBytes = 512;           // answers to item requests, barriers, TMEM address
  // Score bias, per math warp: the 64 distances of its 32 keys x 32 queries.  No room at head size 128 (read from global memory).
  static constexpr int kBiasBytes = HD == 64 ? kFusedMathWarps * 64 * 4 : 0;
  static constexpr int kSmem = (2 * kKvStages + 2 + kDoStages) * kTile + kDsBytes + kDqBytes + 2 * kStatBytes + kBarBytes + kBiasBytes;
  static constexpr int kTmemCols = 512;
  static constexpr int kColS = 0, kColDP = 128, kColDV = 256;
  static constexpr int kColDK = HD == 128 ? 384 : 320, kColDQ = HD == 128 ? kColDP : 384;
};

template <int HD, bool DROPOUT, bool BIAS, bool MORE>
__global__ void __launch_bounds__(kFusedThreads, 1)
attn_bwd_fused_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                      const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                      float* __restrict__ dq_acc, const AttnParams p) {
  using Cfg = FusedCfg<HD>;
  constexpr int CH = Cfg::kCh, NDO = Cfg::kDoStages, NKV = Cfg::kKvStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;                       // NKV stages
  uint8_t* sV = sK + NKV * Cfg::kTile;      // NKV stages
  uint8_t* sQ = sV + NKV * Cfg::kTile;      // 2 stages
  uint8_t* sdO = sQ + 2 * Cfg::kTile;       // NDO stages
  uint8_t* sdS = sdO + NDO * Cfg::kTile;
  uint8_t* sDq = sdS + Cfg::kDsBytes;
  float* sStat = reinterpret_cast<float*>(sDq + Cfg::kDqBytes);  // [2 stages][nlse2: 128, nd: 128]
  uint8_t* ctl = reinterpret_cast<uint8_t*>(sStat) + 2 * Cfg::kStatBytes;
  uint4* next_item = reinterpret_cast<uint4*>(ctl);  // 2: answers to the requests for a further block index
  uint64_t* bars = reinterpret_cast<uint64_t*>(ctl + 32);
  uint64_t* k_full = bars;           // NKV
  uint64_t* k_empty = bars + 2;      // NKV: last dQ of the key block retired
  uint64_t* v_full = bars + 4;       // NKV
  uint64_t* v_empty = bars + 6;      // NKV: last dP^T of the key block retired
  uint64_t* q_full = bars + 8;       // 2 (with the statistics of the block)
  uint64_t* q_empty = bars + 10;     // 2: dK of the block retired, which follows every other reader of the stage
  uint64_t* do_full = bars + 12;     // NDO
  uint64_t* do_empty = bars + 14;    // NDO: dV of the block retired
  uint64_t* s_full = bars + 16;      // 1
  uint64_t* p_full = bars + 17;      // 1 (one arrival per math warp): P^T in TMEM
  uint64_t* dp_full = bars + 18;     // 1 (also: dQ and dK of the block before retired, dS^T free)
  uint64_t* ds_full = bars + 19;     // 1 (one arrival per math warp): dS^T in shared memory, dP^T read
  uint64_t* dq_full = bars + 20;     // 1
  uint64_t* dq_empty = bars + 21;    // 1 (one arrival per drain warp): dQ read from TMEM
  uint64_t* acc_full = bars + 22;    // 1: dV and dK of the key block complete
  uint64_t* acc_empty = bars + 23;   // 1 (one arrival per drain warp): both read from TMEM
  uint64_t* item_full = bars + 24;   // 2
  uint64_t* item_empty = bars + 26;  // 2 (MMA thread, math and drain warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
      mbar_init(&do_full[s], 1);
      mbar_init(&do_empty[s], 1);
      mbar_init(&item_full[s], 1);
      mbar_init(&item_empty[s], 1 + kFusedMathWarps + 4);
    }
    mbar_init(s_full, 1);
    mbar_init(p_full, kFusedMathWarps);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, kFusedMathWarps);
    mbar_init(dq_full, 1);
    mbar_init(dq_empty, 4);
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 4);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_s = tmem_base + Cfg::kColS, tmem_dp = tmem_base + Cfg::kColDP, tmem_dq = tmem_base + Cfg::kColDQ;
  const uint32_t tmem_dv = tmem_base + Cfg::kColDV, tmem_dk = tmem_base + Cfg::kColDK;

  // Work item: one key block of one (batch, head).  The grid has a block per item, the early key blocks of a head first
  // (they see the most queries under the causal mask); a resident CTA goes on with the items of blocks that have not
  // started yet.
  const int n_tiles = (p.SQ + 127) / 128;
  struct Item {
    int jb, head, b, kv_len, i0, n_it;
    size_t tile0;  // first query block of the walk
  };
  auto make_item = [&](uint32_t x, uint32_t y, uint32_t z) {
    Item w;
    w.jb = static_cast<int>(x);
    w.head = static_cast<int>(y);
    w.b = static_cast<int>(z);
    w.kv_len = p.kv_lens ? min(p.kv_lens[w.b], p.SK) : p.SK;
    w.i0 = p.causal ? w.jb : 0;
    w.n_it = (w.jb * 128 < w.kv_len && n_tiles > w.i0) ? n_tiles - w.i0 : 0;
    w.tile0 = (static_cast<size_t>(w.b) * p.NH + w.head) * n_tiles + w.i0;
    return w;
  };
  // Answer to request r: true with the item, false when no block is left (or a wait ran out).
  auto take_item = [&](int r, Item& w) {
    if constexpr (!MORE) return false;
    if (!mbar_wait(&item_full[r & 1], (r >> 1) & 1, abort_flag)) return false;
    uint32_t x, y, z;
    const bool more = launch_cancelled(&next_item[r & 1], x, y, z);
    fence_proxy_async_smem();  // the slot is written through the async proxy again
    if (more) w = make_item(x, y, z);
    return more;
  };

  if (warp < 4) {
    reg_dealloc<kFusedRegsIssue>();
    if (warp == 0 && elect_one()) {
      // ---------------------------------------- TMA producer ----------------------------------------
      Item w = make_item(blockIdx.x, blockIdx.y, blockIdx.z);
      int nq = 0, ndo = 0, nk = 0, nv = 0;  // loads issued so far
      bool ok = true;
      auto load_tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int row) {
#pragma unroll
        for (int c = 0; c < CH; ++c) tma_load_3d(dst + c * 16384, tm, bar, col + c * 64, row, w.b);
      };
      auto load_kv = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* full, uint64_t* empty, int col, int& n) {
        const int st = n % NKV;
        if (!ok || !(ok = mbar_wait(&empty[st], ((n / NKV) & 1) ^ 1, abort_flag))) return;
        mbar_arrive_expect_tx(&full[st], Cfg::kTile);
        load_tile(dst + st * Cfg::kTile, tm, &full[st], col + w.head * HD, w.jb * 128);
        ++n;
      };
      auto load_q = [&](int i) {
        const int st = nq & 1;
        if (!ok || !(ok = mbar_wait(&q_empty[st], ((nq >> 1) & 1) ^ 1, abort_flag))) return;
        mbar_arrive_expect_tx(&q_full[st], Cfg::kTile + Cfg::kStatBytes);
        load_tile(sQ + st * Cfg::kTile, &tm_q, &q_full[st], p.q_col0 + w.head * HD, (w.i0 + i) * 128);
        bulk_load(sStat + st * 256, p.LSE + (w.tile0 + i) * 128, 512, &q_full[st]);
        bulk_load(sStat + st * 256 + 128, p.delta + (w.tile0 + i) * 128, 512, &q_full[st]);
        ++nq;
      };
      auto load_do = [&](int i) {
        const int st = ndo % NDO;
        if (!ok || !(ok = mbar_wait(&do_empty[st], ((ndo / NDO) & 1) ^ 1, abort_flag))) return;
        mbar_arrive_expect_tx(&do_full[st], Cfg::kTile);
        load_tile(sdO + st * Cfg::kTile, &tm_do, &do_full[st], p.o_col0 + w.head * HD, (w.i0 + i) * 128);
        ++ndo;
      };
      for (int r = 0; ok; ++r) {
        if (w.n_it > 0) {  // in the order in which the stages come free at the end of the item before
          load_q(0);
          if (nk == 0 || NKV > 1) load_kv(sK, &tm_k, k_full, k_empty, p.k_col0, nk);  // S can start while V is under way
          load_kv(sV, &tm_v, v_full, v_empty, p.v_col0, nv);
          load_do(0);
          if (nk < nv) load_kv(sK, &tm_k, k_full, k_empty, p.k_col0, nk);
          for (int i = 1; i < w.n_it && ok; ++i) {
            load_q(i);
            load_do(i);
          }
        }
        // The next item, one or two steps ahead of the end of this one.
        if (!MORE) break;
        if (!ok || !(ok = mbar_wait(&item_empty[r & 1], ((r >> 1) & 1) ^ 1, abort_flag))) break;
        mbar_arrive_expect_tx(&item_full[r & 1], 16);
        launch_try_cancel(&next_item[r & 1], &item_full[r & 1]);
        if (!take_item(r, w)) break;
      }
      if (*abort_flag) {  // let the copies in flight land before the CTA leaves
        auto settle = [&](uint64_t* bar, int n, int stages) {
          for (int i = max(n - stages, 0); i < n; ++i)
            for (uint32_t it = 0; it < (1u << 20); ++it)
              if (mbar_try_wait(&bar[i % stages], (i / stages) & 1)) break;
        };
        settle(k_full, nk, NKV);
        settle(v_full, nv, NKV);
        settle(q_full, nq, 2);
        settle(do_full, ndo, NDO);
      }
    }
    if (warp == 1 && elect_one()) {
      // ---------------------------------------- MMA issuer ------------------------------------------
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, false, false);  // [keys x queries], reduce over HD
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, HD, false, true);  // [keys x HD], reduce over queries
      constexpr uint32_t idesc_dq = umma_idesc_bf16(128, HD, true, true);    // [queries x HD], reduce over keys
      // One descriptor per operand and orientation; a step along the operand is an addition to its address field.
      const uint64_t k_k = umma_desc_sw128(smem_u32(sK), 16, 1024), k_mn = umma_desc_sw128(smem_u32(sK), 16384, 1024);
      const uint64_t v_k = umma_desc_sw128(smem_u32(sV), 16, 1024);
      const uint64_t ds_k = umma_desc_sw128(smem_u32(sdS), 16, 1024), ds_mn = umma_desc_sw128(smem_u32(sdS), 16384, 1024);
      const uint64_t q_k = umma_desc_sw128(smem_u32(sQ), 16, 1024), q_mn = umma_desc_sw128(smem_u32(sQ), 16384, 1024);
      const uint64_t do_k = umma_desc_sw128(smem_u32(sdO), 16, 1024), do_mn = umma_desc_sw128(smem_u32(sdO), 16384, 1024);
      constexpr uint64_t kStage = Cfg::kTile >> 4;  // descriptor distance of the Q / dO stages
      auto product = [&](uint32_t d, uint64_t a, uint64_t bb) {  // [128 x 128] = A . B^T over HD, both K-major
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) >> 4;
          umma_f16_ss(d, a + off, bb + off, idesc_s, kk != 0);
        }
      };
      Item w = make_item(blockIdx.x, blockIdx.y, blockIdx.z);
      uint32_t n = 0, m = 0;  // steps and (non-empty) items so far
      bool ok = true;
      for (int r = 0; ok; ++r) {
        if (w.n_it > 0) {
          const int kst = m % NKV;
          const uint32_t kph = (m / NKV) & 1;
          const uint64_t kk_k = k_k + kst * kStage, kk_mn = k_mn + kst * kStage, vv_k = v_k + kst * kStage;
          ok = mbar_wait<kIssueLook>(&k_full[kst], kph, abort_flag) && mbar_wait<kIssueLook>(&q_full[n & 1], (n >> 1) & 1, abort_flag);
          if (!ok) break;
          tc_fence_after_sync();
          product(tmem_s, kk_k, q_k + (n & 1) * kStage);
          umma_commit(s_full);
          ok = mbar_wait<kIssueLook>(&v_full[kst], kph, abort_flag) && mbar_wait<kIssueLook>(&do_full[n % NDO], (n / NDO) & 1, abort_flag) &&
               (HD == 64 || n == 0 || mbar_wait<kIssueLook>(dq_empty, (n - 1) & 1, abort_flag));  // dP^T takes the columns of dQ
          if (!ok) break;
          tc_fence_after_sync();
          product(tmem_dp, vv_k, do_k + (n % NDO) * kStage);
          umma_commit(dp_full);
          for (int i = 0; i < w.n_it; ++i, ++n) {
            const int st = n & 1, nx = st ^ 1, dst = n % NDO, dnx = (n + 1) % NDO;
            const uint32_t ph = n & 1;
            const bool last = i + 1 == w.n_it;
            if (!(ok = mbar_wait<kIssueLook>(p_full, ph, abort_flag))) break;
            if (i == 0 && m > 0 && !(ok = mbar_wait<kIssueLook>(acc_empty, (m - 1) & 1, abort_flag))) break;
            tc_fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)  // 128 queries = 8 steps of 16; the warpgroups' shares of P^T start 32 columns apart
              umma_f16_ts(tmem_dv, tmem_s + (kk >> 1) * 32 + (kk & 1) * 8, do_mn + dst * kStage + (kk * 2048 >> 4), idesc_acc,
                          (i | kk) != 0);
            umma_commit(&do_empty[dst]);
            if (!last) {
              if (!(ok = mbar_wait<kIssueLook>(&q_full[nx], ((n + 1) >> 1) & 1, abort_flag))) break;
              tc_fence_after_sync();
              product(tmem_s, kk_k, q_k + nx * kStage);
              umma_commit(s_full);
            } else {
              umma_commit(&v_empty[kst]);
            }
            if (!(ok = mbar_wait<kIssueLook>(ds_full, ph, abort_flag))) break;
            if (HD == 64 && n >= 1 && !(ok = mbar_wait<kIssueLook>(dq_empty, (n - 1) & 1, abort_flag))) break;
            tc_fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)  // 128 keys = 8 steps of 16
              umma_f16_ss(tmem_dq, ds_mn + (kk * 2048 >> 4), kk_mn + (kk * 2048 >> 4), idesc_dq, kk != 0);
            umma_commit(dq_full);
            if (last) umma_commit(&k_empty[kst]);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_f16_ss(tmem_dk, ds_k + (((kk >> 2) * 16384 + (kk & 3) * 32) >> 4), q_mn + st * kStage + (kk * 2048 >> 4),
                          idesc_acc, (i | kk) != 0);
            umma_commit(&q_empty[st]);
            if (!last) {
              if (!(ok = mbar_wait<kIssueLook>(&do_full[dnx], ((n + 1) / NDO) & 1, abort_flag))) break;
              if (HD == 128 && !(ok = mbar_wait<kIssueLook>(dq_empty, ph, abort_flag))) break;
              tc_fence_after_sync();
              product(tmem_dp, vv_k, do_k + dnx * kStage);
              umma_commit(dp_full);
            } else {
              umma_commit(acc_full);
            }
          }
          ++m;
        }
        if (!ok || !take_item(r, w)) break;
        mbar_arrive(&item_empty[r & 1]);
      }
    }
  } else if (warp >= 20) {
    // -------------- drain warps: dQ of every step -> fp32 accumulator in global memory --------------
    reg_alloc<kFusedRegsDrain>();
    const int quarter = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    uint8_t* stage = sDq + quarter * 8192;
    const uint32_t keep8 = dropout_keep8(p.dropout_p);
    const float inv_keep = DROPOUT ? 256.0f / static_cast<float>(keep8) : 1.0f;
    Item w = make_item(blockIdx.x, blockIdx.y, blockIdx.z);
    uint32_t n = 0, m = 0;
    bool ok = true;
    for (int r = 0;; ++r) {
      // dQ: [HD / 4 column quads][32 lanes][16 bytes], as in the accumulator
      float* dst = dq_acc + w.tile0 * (128 * HD) + quarter * (32 * HD);
      for (int i = 0; i < w.n_it; ++i, ++n) {
        if (!(ok = mbar_wait_warp(dq_full, n & 1, abort_flag))) break;
        tc_fence_after_sync();
#pragma unroll
        for (int half = 0; half < HD / 64; ++half) {
          uint32_t a[2][32];
          tmem_ld_32x32(tmem_dq + lane_addr + half * 64, a[0]);
          tmem_ld_32x32(tmem_dq + lane_addr + half * 64 + 32, a[1]);
          tmem_ld_wait();
          if (half == HD / 64 - 1) {  // the columns are free for dP^T of the next block
            tc_fence_before_sync();
            warp_arrive(dq_empty, lane);
          }
          if (lane == 0) tma_store_wait_read<0>();  // the copy before has read the staging tile
          __syncwarp();
#pragma unroll
          for (int e = 0; e < 16; ++e)
            *reinterpret_cast<uint4*>(stage + e * 512 + lane * 16) =
                make_uint4(a[e >> 3][4 * (e & 7)], a[e >> 3][4 * (e & 7) + 1], a[e >> 3][4 * (e & 7) + 2], a[e >> 3][4 * (e & 7) + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            bulk_add_f32(dst + half * 2048, stage, 8192);
            tma_store_commit();
          }
        }
        dst += 128 * HD;
      }
      if (!ok) break;
      if constexpr (!MORE) break;  // dV and dK: the math warps
      // dV and dK of the key block: 32 rows x 64 columns at a time as tiled stores (which clip at the end of the sample)
      if (w.n_it > 0) {
        if (!(ok = mbar_wait_warp(acc_full, m & 1, abort_flag))) break;
        ++m;
        tc_fence_after_sync();
      }
      if (lane == 0) tma_store_wait_read<0>();
      __syncwarp();
#pragma unroll 1
      for (int part = 0; part < 2 * (HD / 64); ++part) {
        const bool is_dk = part >= HD / 64;
        const int c0 = (part & (HD / 64 - 1)) * 64;
        uint32_t a[2][32];
        if (w.n_it > 0) {
          const uint32_t src = (is_dk ? tmem_dk : tmem_dv) + lane_addr + c0;
          tmem_ld_32x32(src, a[0]);
          tmem_ld_32x32(src + 32, a[1]);
          tmem_ld_wait();
          if (part == 2 * (HD / 64) - 1) {
            tc_fence_before_sync();
            warp_arrive(acc_empty, lane);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) a[0][e] = a[1][e] = 0u;
        }
        const float sc = is_dk ? p.scale : inv_keep;
        uint8_t* half_stage = stage + (part & 1) * 4096;
        if (part >= 2) {
          if (lane == 0) tma_store_wait_read<1>();  // the copy two parts back has read its half
          __syncwarp();
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const uint32_t(&x)[32] = a[e >> 2];
          const int o = (e & 3) * 8;
          uint4 v;
          v.x = pack_bf16x2(__uint_as_float(x[o + 0]) * sc, __uint_as_float(x[o + 1]) * sc);
          v.y = pack_bf16x2(__uint_as_float(x[o + 2]) * sc, __uint_as_float(x[o + 3]) * sc);
          v.z = pack_bf16x2(__uint_as_float(x[o + 4]) * sc, __uint_as_float(x[o + 5]) * sc);
          v.w = pack_bf16x2(__uint_as_float(x[o + 6]) * sc, __uint_as_float(x[o + 7]) * sc);
          *reinterpret_cast<uint4*>(half_stage + lane * 128 + ((e ^ (lane & 7)) << 4)) = v;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_3d(is_dk ? &tm_dk : &tm_dv, half_stage, (is_dk ? p.dk_col0 : p.dv_col0) + w.head * HD + c0,
                       w.jb * 128 + quarter * 32, w.b);
          tma_store_commit();
        }
      }
      const bool more = take_item(r, w);
      if (!__all_sync(0xffffffffu, more)) break;
      warp_arrive(&item_empty[r & 1], lane);
    }
    if (lane == 0) tma_store_wait_read<0>();
  } else {
    // ------------------------------------------ math warps --------------------------------------------
    // (the math warpgroups keep the registers they were launched with)
    const int quarter = warp & 3;
    const int g = (warp - 4) >> 2;      // queries [32 g, 32 g + 32) of a block; without further items columns [g HD/4, ..) of dK and dV
    const int r = quarter * 32 + lane;  // key row inside the tile
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t my_s = tmem_s + lane_addr + g * 32, my_dp = tmem_dp + lane_addr + g * 32;
    const float c = p.scale * kLog2e;
    const uint32_t keep8 = dropout_keep8(p.dropout_p);
    const float inv_keep = DROPOUT ? 256.0f / static_cast<float>(keep8) : 1.0f;
    const uint32_t drop_c = (256u - keep8) * 0x01010101u;  // byte + drop_c carries out <=> byte >= keep8
    const int n_dist = p.SQ + p.SK - 1;
    uint8_t* ds_row = sdS + (g >> 1) * 16384 + r * 128;
    float* sBias = reinterpret_cast<float*>(ctl + Cfg::kBarBytes) + (warp - 4) * 64;
    Item w = make_item(blockIdx.x, blockIdx.y, blockIdx.z);
    uint32_t n = 0;
    bool ok = true;
    for (int t = 0;; ++t) {
      const int kv0 = w.jb * 128, kv = kv0 + r, kv_len = w.kv_len;
      const uint32_t bh_seed = DROPOUT ? static_cast<uint32_t>(hash64(p.dropout_seed, static_cast<uint64_t>(w.b) * p.NH + w.head)) : 0u;
      // attn_col_hash mixes (key quads + quad) * 0x9E3779B1 + seed: linear in the quad
      const uint32_t hash0 = (static_cast<uint32_t>(kv) * ((p.SQ + 3) >> 2) + static_cast<uint32_t>(w.i0 * 32 + g * 8)) * 0x9E3779B1u + bh_seed;
      const bool kv_ok = kv < kv_len;
      // score bias: bias_table[head][kv - q + SQ - 1] log2(e); its gradient is dS summed along the diagonals
      const float* bias_head = BIAS ? p.bias_table + static_cast<size_t>(w.head) * n_dist : nullptr;
      float* dbias_head = BIAS ? p.dbias_table + static_cast<size_t>(w.head) * n_dist : nullptr;

      // Score bias of a block, fetched a block ahead: with the loads in front of their use a step waited 700 cycles for them
      constexpr bool kBiasStaged = BIAS && HD == 64;
      float bias_next[2] = {0.f, 0.f};
      auto fetch_bias = [&](int q0) {
        if constexpr (kBiasStaged) {
          const int d = kv0 + quarter * 32 - q0 + p.SQ - 32 + lane;  // distance of (key 0, query 31) of this warp, + lane
          bias_next[0] = __ldg(bias_head + min(max(d, 0), n_dist - 1));
          bias_next[1] = __ldg(bias_head + min(max(d + 32, 0), n_dist - 1));
        }
      };
      fetch_bias(w.i0 * 128 + g * 32);

      for (int i = 0; i < w.n_it; ++i, ++n) {
        const uint32_t ph = n & 1;
        const int qblk0 = (w.i0 + i) * 128, qbase = qblk0 + g * 32;
        const float* nlse2 = sStat + ph * 256 + g * 32;
        const float* nd = nlse2 + 128;
        const bool need_mask = (p.causal && kv0 + 127 > qblk0) || qblk0 + 128 > p.SQ || kv0 + 128 > kv_len;
        // queries lo .. hi - 1 of this thread's 32 see its key
        const int lo = p.causal ? kv - qbase : 0, hi = kv_ok ? p.SQ - qbase : 0;
        // Nothing to see for the whole warp (above the diagonal or past an end): zeros for P and dS, no arithmetic.  In a
        // last block of 64 queries these are half of the warps: 256 heads of 64 x 64 15.6 -> 13.7 us.
        if (need_mask && (qbase >= p.SQ || kv0 + quarter * 32 >= (p.causal ? min(kv_len, qbase + 32) : kv_len))) {
          uint32_t zero[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) zero[e] = 0u;
          if (!mbar_wait_warp(s_full, ph, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          tmem_st_32x16(my_s, zero);
          tmem_st_wait();
          tc_fence_before_sync();
          warp_arrive(p_full, lane);
          if (!mbar_wait_warp(dp_full, ph, abort_flag)) { ok = false; break; }
#pragma unroll
          for (int e = 0; e < 4; ++e)
            *reinterpret_cast<uint4*>(ds_row + ((((g & 1) * 4 + e) ^ (r & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
          fence_proxy_async_smem();
          warp_arrive(ds_full, lane);
          fetch_bias(qbase + 128);
          continue;
        }
        uint32_t drop = 0u;  // bit 7 - n of byte e: query 4 n + e dropped for this key; hashed before the scores are there
        if constexpr (DROPOUT) {
          uint32_t h = hash0 + static_cast<uint32_t>(i) * (32u * 0x9E3779B1u);
#pragma unroll
          for (int n = 0; n < 8; ++n) {
            const uint32_t x = fmix32(h);
            h += 0x9E3779B1u;
            const uint32_t cs = (x & 0x7f7f7f7fu) + (drop_c & 0x7f7f7f7fu);
            drop |= (((x & drop_c) | ((x | drop_c) & cs)) & 0x80808080u) >> n;
          }
        }
        if constexpr (kBiasStaged) {  // (the reads of the block before are behind this warp's arrivals)
          sBias[lane] = bias_next[0];
          sBias[lane + 32] = bias_next[1];
          __syncwarp();
        }
        if (!mbar_wait_warp(&q_full[ph], (n >> 1) & 1, abort_flag)) { ok = false; break; }  // the statistics
        if (!mbar_wait_warp(s_full, ph, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        float pr[32];
        {
          uint32_t rs[32], w[16];
          tmem_ld_32x32(my_s, rs);
          tmem_ld_wait();
          const float2 c2 = make_float2(c, c);
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            float4 nl = *reinterpret_cast<const float4*>(nlse2 + e);
            if constexpr (kBiasStaged) {
              const float* br = sBias + lane + 31 - e;  // entries run down as the query runs up
              nl.x = fmaf(br[0], kLog2e, nl.x);
              nl.y = fmaf(br[-1], kLog2e, nl.y);
              nl.z = fmaf(br[-2], kLog2e, nl.z);
              nl.w = fmaf(br[-3], kLog2e, nl.w);
            } else if constexpr (BIAS) {
              const int d = kv - (qbase + e) + p.SQ - 1;  // entries run down as the query runs up
              nl.x = fmaf(__ldg(bias_head + min(max(d, 0), n_dist - 1)), kLog2e, nl.x);
              nl.y = fmaf(__ldg(bias_head + min(max(d - 1, 0), n_dist - 1)), kLog2e, nl.y);
              nl.z = fmaf(__ldg(bias_head + min(max(d - 2, 0), n_dist - 1)), kLog2e, nl.z);
              nl.w = fmaf(__ldg(bias_head + min(max(d - 3, 0), n_dist - 1)), kLog2e, nl.w);
            }
            const float2 a = fma_f32x2(make_float2(__uint_as_float(rs[e]), __uint_as_float(rs[e + 1])), c2, make_float2(nl.x, nl.y));
            const float2 b2 = fma_f32x2(make_float2(__uint_as_float(rs[e + 2]), __uint_as_float(rs[e + 3])), c2, make_float2(nl.z, nl.w));
            pr[e] = ex2(a.x);
            pr[e + 1] = ex2(a.y);
            pr[e + 2] = ex2(b2.x);
            pr[e + 3] = ex2(b2.y);
          }
          if (need_mask) {  // uniform branch: only blocks on the diagonal or at the ragged ends pay for the tests
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (e < lo || e >= hi) pr[e] = 0.f;
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            w[e] = pack_bf16x2(pr[2 * e], pr[2 * e + 1]);
            if constexpr (DROPOUT) w[e] &= ~spread_sign_bytes(drop << (e >> 1), (e & 1) ? 0xBBAA : 0x9988);
          }
          tmem_st_32x16(my_s, w);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        warp_arrive(p_full, lane);
        fetch_bias(qbase + 128);
        if (!mbar_wait_warp(dp_full, ph, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        float diag = 0.f, wrap = 0.f;  // BIAS: sums along the diagonals through (lane, 0) and, wrapped, 32 distances below
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          uint32_t rp[16], w[8];
          tmem_ld_32x16(my_dp + ch * 16, rp);
          tmem_ld_wait();
          const float2 k2 = make_float2(inv_keep, inv_keep);
#pragma unroll
          for (int e = 0; e < 16; e += 4) {
            const int q = ch * 16 + e;
            const float4 n4 = *reinterpret_cast<const float4*>(nd + q);
            if constexpr (DROPOUT) {
              const uint32_t d = drop << (q >> 2);
#pragma unroll
              for (int u = 0; u < 4; ++u) rp[e + u] &= ~spread_sign_bytes(d, 0x8888 + 0x1111 * u);
            }
            float2 a = make_float2(__uint_as_float(rp[e]), __uint_as_float(rp[e + 1]));
            float2 b2 = make_float2(__uint_as_float(rp[e + 2]), __uint_as_float(rp[e + 3]));
            if constexpr (DROPOUT) {
              a = fma_f32x2(a, k2, make_float2(n4.x, n4.y));
              b2 = fma_f32x2(b2, k2, make_float2(n4.z, n4.w));
            } else {
              a = add_f32x2(a, make_float2(n4.x, n4.y));
              b2 = add_f32x2(b2, make_float2(n4.z, n4.w));
            }
            a = mul_f32x2(make_float2(pr[q], pr[q + 1]), a);
            b2 = mul_f32x2(make_float2(pr[q + 2], pr[q + 3]), b2);
            if (need_mask) {  // rows and keys outside: not even 0 x NaN (from the padded statistics) may enter
              if (q < lo || q >= hi) a.x = 0.f;
              if (q + 1 < lo || q + 1 >= hi) a.y = 0.f;
              if (q + 2 < lo || q + 2 >= hi) b2.x = 0.f;
              if (q + 3 < lo || q + 3 >= hi) b2.y = 0.f;
            }
            w[e >> 1] = pack_bf16x2(a.x, a.y);
            w[(e >> 1) + 1] = pack_bf16x2(b2.x, b2.y);
            if constexpr (BIAS) {
              // Gradient of the bias table: dS (before the softmax scale) summed along the diagonals key - query.  Lane l
              // takes entry (l + q, q) from lane l + q: all on its own diagonal, or 32 distances below it where the
              // lane index wraps.  Independent shuffles, two coalesced reductions per warp and step.
              const float v4[4] = {a.x, a.y, b2.x, b2.y};
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const float y = __shfl_sync(0xffffffffu, v4[u], (lane + q + u) & 31);
                if (lane + q + u < 32) diag += y;
                else wrap += y;
              }
            }
          }
#pragma unroll
          for (int e = 0; e < 2; ++e)
            *reinterpret_cast<uint4*>(ds_row + ((((g & 1) * 4 + ch * 2 + e) ^ (r & 7)) << 4)) =
                make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
        }
        tc_fence_before_sync();
        fence_proxy_async_smem();
        warp_arrive(ds_full, lane);
        if constexpr (BIAS) {
          const int d = kv - qbase + p.SQ - 1;
          if (d >= 0 && d < n_dist) atomicAdd(dbias_head + d, diag);
          if (lane > 0 && d - 32 >= 0 && d - 32 < n_dist) atomicAdd(dbias_head + d - 32, wrap);
        }
      }
      if (!ok || !MORE) break;
      const bool more = take_item(t, w);
      if (!__all_sync(0xffffffffu, more)) break;
      warp_arrive(&item_empty[t & 1], lane);
    }
    // A single item per CTA: nothing is left for these warps to do, so all sixteen write dV and dK, 32 keys x HD / 4 columns per
    // warp and matrix, through shared memory (every load and product is complete, the Q stages are free).  Written by the four
    // drain warps, as in front of a further item, the backward of 16 heads of 64 x 128 took 18.1 us instead of 16.9.
    if constexpr (!MORE) {
      if (ok && w.n_it > 0) ok = mbar_wait_warp(acc_full, 0, abort_flag);
      if (ok) {
        tc_fence_after_sync();
        constexpr int OC = HD / 4, PIECES = OC / 8, RPI = 32 / PIECES;  // columns, 16-byte pieces, rows per store
        uint8_t* stage = sQ + (warp - 4) * 2048;
        auto cell = [&](int row, int piece) { return stage + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4); };
        const int row0 = w.jb * 128 + quarter * 32, piece = lane % PIECES;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          const float sc = which ? p.scale : inv_keep;
          uint32_t a[OC];
          if (w.n_it > 0) {
            tmem_ld_cols<OC>((which ? tmem_dk : tmem_dv) + lane_addr + g * OC, a);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int e = 0; e < OC; ++e) a[e] = 0u;
          }
#pragma unroll
          for (int e = 0; e < PIECES; ++e) {
            uint4 v;
            v.x = pack_bf16x2(__uint_as_float(a[8 * e + 0]) * sc, __uint_as_float(a[8 * e + 1]) * sc);
            v.y = pack_bf16x2(__uint_as_float(a[8 * e + 2]) * sc, __uint_as_float(a[8 * e + 3]) * sc);
            v.z = pack_bf16x2(__uint_as_float(a[8 * e + 4]) * sc, __uint_as_float(a[8 * e + 5]) * sc);
            v.w = pack_bf16x2(__uint_as_float(a[8 * e + 6]) * sc, __uint_as_float(a[8 * e + 7]) * sc);
            *reinterpret_cast<uint4*>(cell(lane, e)) = v;
          }
          __syncwarp();
          const int ld = which ? p.lddk : p.lddv;
          __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(which ? p.dK : p.dV) + (static_cast<size_t>(w.b) * p.SK + row0) * ld +
                               (which ? p.dk_col0 : p.dv_col0) + w.head * HD + g * OC + piece * 8;
#pragma unroll
          for (int e = 0; e < 32 / RPI; ++e) {
            const int row = e * RPI + lane / PIECES;
            const uint4 v = *reinterpret_cast<const uint4*>(cell(row, piece));
            if (row0 + row < p.SK) *reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * ld) = v;
          }
          __syncwarp();
        }
      }
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

// dQ[b, q, head, :] (bf16) = scale * the fp32 accumulator [b, head, tile][quarter][HD / 4][32][4].  A warp turns 32 queries x
// 32 columns: 512-byte reads, a transpose through shared memory, 64-byte row segments out.  (With 64 columns a warp short
// sequences waited longer for fewer warps: 4 heads of 33 x 64 2.9 us instead of 2.1.)
template <int HD>
__global__ void __launch_bounds__(128)
attn_dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, int lddq, int dq_col0, int NH,
                       int SQ, int n_tiles, float scale) {
  __shared__ __align__(16) uint8_t tile_smem[4][2048];
  const int head = blockIdx.y, b = blockIdx.z;
  const int tile = blockIdx.x / (HD / 32), c0 = (blockIdx.x % (HD / 32)) * 32;
  const int quarter = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q0 = tile * 128 + quarter * 32;
  if (q0 >= SQ) return;
  const float* src = acc + (((static_cast<size_t>(b) * NH + head) * n_tiles + tile) * 4 + quarter) * (32 * HD) + c0 * 32 + lane * 4;
  float4 v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = *reinterpret_cast<const float4*>(src + e * 128);
  uint8_t* stage = tile_smem[quarter];
  auto cell = [&](int row, int piece) { return stage + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4); };
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    uint4 w;
    w.x = pack_bf16x2(v[2 * e].x * scale, v[2 * e].y * scale);
    w.y = pack_bf16x2(v[2 * e].z * scale, v[2 * e].w * scale);
    w.z = pack_bf16x2(v[2 * e + 1].x * scale, v[2 * e + 1].y * scale);
    w.w = pack_bf16x2(v[2 * e + 1].z * scale, v[2 * e + 1].w * scale);
    *reinterpret_cast<uint4*>(cell(lane, e)) = w;
  }
  __syncwarp();
  __nv_bfloat16* out = dq + (static_cast<size_t>(b) * SQ + q0) * lddq + dq_col0 + head * HD + c0 + (lane & 3) * 8;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int row = e * 8 + (lane >> 2);
    const uint4 w = *reinterpret_cast<const uint4*>(cell(row, lane & 3));
    if (q0 + row < SQ) *reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * lddq) = w;
  }
}

// What the fused kernel starts from: the dQ accumulator cleared, and the row statistics in the form it consumes: nd[b, h, q] = -sum_d dO O and nlse2[b, h, q] = -LSE log2(e), rows
// padded to whole query blocks (the padding is read but never used).  A warp takes one head and 32 consecutive queries of one sequence.  LPR = HD / 8 lanes read one (token, head) row
// with 16-byte loads, so one load instruction of the warp covers 32 / LPR tokens; after the butterfly sum inside the
// lane group every lane of the group holds the row's result, and lane L keeps token (L % LPR) * (32 / LPR) + L / LPR.
// Clearing here, under the loads of O and dO, takes the place of a memset in front: backward of 8 x 16 heads of 123 x 64 against 477
// keys 36.0 -> 32.8 us, 4 x 4 of 256 x 128 26.1 -> 23.0, 16 of 2048 x 128 98 -> 91.5, 32 x 16 of 512 x 64 250 -> 247.
template <int HD>
__global__ void __launch_bounds__(128)
attn_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, int ldo, int o_col0, const __nv_bfloat16* __restrict__ dout,
                     int lddo, const float* __restrict__ lse, float* __restrict__ nd, float* __restrict__ nlse2,
                     float* __restrict__ dq_acc, int B, int NH, int SQ, int SQp) {
  constexpr int LPR = HD / 8, TPI = 32 / LPR;
  const int lane = threadIdx.x & 31;
  const int qblocks = (SQ + 31) / 32;
  const long long w = blockIdx.x * 4LL + (threadIdx.x >> 5);
  if (w >= static_cast<long long>(B) * NH * qblocks) return;
  const int qb = static_cast<int>(w % qblocks);
  const int head = static_cast<int>((w / qblocks) % NH);
  const int b = static_cast<int>(w / (static_cast<long long>(qblocks) * NH));
  const int sub = lane % LPR, grp = lane / LPR;
  const size_t col = static_cast<size_t>(o_col0) + head * HD + sub * 8;
  float mine = 0.f;
  uint4 qo[LPR], qd[LPR];
#pragma unroll
  for (int i = 0; i < LPR; ++i) {       // all loads first: 2 * LPR independent 16-byte requests per lane
    const int q = qb * 32 + i * TPI + grp;
    const size_t tok = static_cast<size_t>(b) * SQ + min(q, SQ - 1);
    qo[i] = *reinterpret_cast<const uint4*>(o + tok * ldo + col);
    qd[i] = *reinterpret_cast<const uint4*>(dout + tok * lddo + col);
  }
  float* acc = dq_acc + ((static_cast<size_t>(b) * NH + head) * (SQp / 32) + qb) * (32 * HD) + lane * 4;  // [HD / 4][32][4]
#pragma unroll
  for (int i = 0; i < HD / 4; ++i) *reinterpret_cast<float4*>(acc + i * 128) = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < LPR; ++i) {
    const float2 a0 = unpack_bf16x2(qo[i].x), a1 = unpack_bf16x2(qo[i].y), a2 = unpack_bf16x2(qo[i].z), a3 = unpack_bf16x2(qo[i].w);
    const float2 g0 = unpack_bf16x2(qd[i].x), g1 = unpack_bf16x2(qd[i].y), g2 = unpack_bf16x2(qd[i].z), g3 = unpack_bf16x2(qd[i].w);
    float t = (a0.x * g0.x + a0.y * g0.y) + (a1.x * g1.x + a1.y * g1.y) + (a2.x * g2.x + a2.y * g2.y) +
              (a3.x * g3.x + a3.y * g3.y);
#pragma unroll
    for (int d = LPR / 2; d >= 1; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
    if (sub == i) mine = t;
  }
  const int q = qb * 32 + sub * TPI + grp;
  if (q < SQ) {
    const size_t bh = static_cast<size_t>(b) * NH + head;
    nd[bh * SQp + q] = -mine;
    nlse2[bh * SQp + q] = -lse[bh * SQ + q] * kLog2e;
  }
}

template <typename K>
int set_smem(K kernel, int bytes) {
  return static_cast<int>(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

template <int HD, bool DROPOUT, bool BIAS>
int launch_fused(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                 const CUtensorMap& tdk, const CUtensorMap& tdv, const AttnParams& p, float* dq_acc, int num_sms, cudaStream_t stream) {
  const int n_tiles = (p.SQ + 127) / 128;
  dim3 grid_kv((p.SK + 127) / 128, p.NH, p.B);
  auto kernel = static_cast<long long>(grid_kv.x) * grid_kv.y * grid_kv.z > num_sms ? attn_bwd_fused_kernel<HD, DROPOUT, BIAS, true>
                                                                                    : attn_bwd_fused_kernel<HD, DROPOUT, BIAS, false>;
  const int rc = set_smem(kernel, FusedCfg<HD>::kSmem);
  if (rc) return rc;
  kernel<<<grid_kv, kFusedThreads, FusedCfg<HD>::kSmem, stream>>>(tq, tk, tv, tdo, tdk, tdv, dq_acc, p);
  dim3 grid_cv(n_tiles * (HD / 32), p.NH, p.B);
  attn_dq_convert_kernel<HD><<<grid_cv, 128, 0, stream>>>(dq_acc, reinterpret_cast<__nv_bfloat16*>(p.dQ), p.lddq,
                                                          p.dq_col0, p.NH, p.SQ, n_tiles, p.scale);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace

// Floats of fp32 scratch the fused backward needs: the dQ accumulator, then the two row-statistic arrays (padded rows).
long long attn_bwd_fused_scratch_floats(int B, int NH, int SQ, int HD) {
  return static_cast<long long>(B) * NH * ((SQ + 127) / 128) * 128 * (HD + 2);
}

// dout shares the layout of O (p.ldo / p.o_col0 describe both).  `scratch` holds attn_bwd_fused_scratch_floats()
// floats, 16-byte aligned; what is accumulated into is cleared here, on `stream`.
int attn_bwd_fused_launch(const void* q, int ldq, const void* k, int ldk, const void* v, int ldv, const void* dout,
                          int lddo, const AttnParams& p, float* scratch, int num_sms, cudaStream_t stream) {
  if (p.HD != 64 && p.HD != 128) return -2;
  if (p.causal && p.SQ != p.SK) return -2;
  // 16-byte granularity everywhere: TMA x coordinates (column offsets of Q / K / V / dO), the 16-byte stores of
  // dQ, dK and dV; a misaligned offset would fault on the device instead of failing here
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (lddo % 8) || (p.lddq % 8) || (p.lddk % 8) || (p.lddv % 8) ||
      (p.dq_col0 % 8) || (p.dk_col0 % 8) || (p.dv_col0 % 8) || (p.q_col0 % 8) || (p.k_col0 % 8) || (p.v_col0 % 8))
    return -3;
  int rc;
  const int n_tiles = (p.SQ + 127) / 128;
  const long long acc_rows = static_cast<long long>(p.B) * p.NH * n_tiles * 128;
  const long long acc_floats = acc_rows * p.HD;
  float* dq_acc = scratch;
  float* nd = scratch + acc_floats;
  float* nlse2 = nd + acc_rows;
  {
    if ((p.ldo % 8) || (p.o_col0 % 8)) return -3;
    const long long warps = static_cast<long long>(p.B) * p.NH * ((p.SQ + 31) / 32);
    const auto* ob = reinterpret_cast<const __nv_bfloat16*>(p.O);
    const auto* db = reinterpret_cast<const __nv_bfloat16*>(dout);
    const unsigned blocks = static_cast<unsigned>((warps + 3) / 4);
    if (p.HD == 128)
      attn_bwd_prep_kernel<128><<<blocks, 128, 0, stream>>>(ob, p.ldo, p.o_col0, db, lddo, p.LSE, nd, nlse2, dq_acc, p.B, p.NH, p.SQ, n_tiles * 128);
    else
      attn_bwd_prep_kernel<64><<<blocks, 128, 0, stream>>>(ob, p.ldo, p.o_col0, db, lddo, p.LSE, nd, nlse2, dq_acc, p.B, p.NH, p.SQ, n_tiles * 128);
  }
  AttnParams pp = p;
  pp.delta = nd;
  pp.LSE = nlse2;
  // Blocks past the end of a sample read zeros: P and dS are zero there, and zero times an infinity or NaN of the next
  // sample must not enter this one's gradients.
  CUtensorMap tq, tk, tv, tdo, tdk, tdv;
  if ((rc = make_tma_batched_bf16(&tq, q, p.B, p.SQ, ldq, 128, 64))) return rc;
  if ((rc = make_tma_batched_bf16(&tdo, dout, p.B, p.SQ, lddo, 128, 64))) return rc;
  if ((rc = make_tma_batched_bf16(&tk, k, p.B, p.SK, ldk, 128, 64))) return rc;
  if ((rc = make_tma_batched_bf16(&tv, v, p.B, p.SK, ldv, 128, 64))) return rc;
  if ((rc = make_tma_batched_bf16(&tdk, p.dK, p.B, p.SK, p.lddk, 32, 64))) return rc;
  if ((rc = make_tma_batched_bf16(&tdv, p.dV, p.B, p.SK, p.lddv, 32, 64))) return rc;
  const bool drop = p.dropout_p > 0.f;
  if (p.bias_table != nullptr) {
    if (p.dbias_table == nullptr) return -2;
    if (p.HD == 128)
      return drop ? launch_fused<128, true, true>(tq, tk, tv, tdo, tdk, tdv, pp, dq_acc, num_sms, stream)
                  : launch_fused<128, false, true>(tq, tk, tv, tdo, tdk, tdv, pp, dq_acc, num_sms, stream);
    return drop ? launch_fused<64, true, true>(tq, tk, tv, tdo, tdk, tdv, pp, dq_acc, num_sms, stream)
                : launch_fused<64, false, true>(tq, tk, tv, tdo, tdk, tdv, pp, dq_acc, num_sms, stream);
  }
  if (p.HD == 128)
    return drop ? launch_fused<128, true, false>(tq, tk, tv, tdo, tdk, tdv, pp, dq_acc, num_sms, stream)
                : launch_fused<128, false, false>(tq, tk, tv, tdo, tdk, tdv, pp, dq_acc, num_sms, stream);
  return drop ? launch_fused<64, true, false>(tq, tk, tv, tdo, tdk, tdv, pp, dq_acc, num_sms, stream)
              : launch_fused<64, false, false>(tq, tk, tv, tdo, tdk, tdv, pp, dq_acc, num_sms, stream);
}

}  // namespace ssb
