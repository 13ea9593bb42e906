// Two-SM ("cta_group::2") variant of the bf16 GEMM: a cluster of two CTAs on one SM pair computes a
// 256 x 256 output tile.  Each CTA stages its own 128 rows of A and its own 128 of the tile's 256 B rows
// (columns of the output), the leader CTA issues tcgen05.mma.cta_group::2 instructions that read both
// CTAs' shared memory, and each CTA ends up with its 128 x 256 half of the accumulator in its own TMEM.
//
// Why: with one CTA per 128 x 256 tile the tensor core reads 12 KB of operands from shared memory per
// 128 x 256 x 16 step while TMA writes the same amount, which exceeds what one SM's shared memory delivers
// (measured: tensor pipe 65 % busy, L1/shared pipe 80 %).  Pairing halves the B traffic per SM.
//
//   warp 0     : TMA producer (one elected lane), in both CTAs
//   warp 1     : TMEM allocator in both CTAs; MMA issuer in the leader (cluster rank 0)
//   warps 2..17: epilogue; warp w reads TMEM lanes 32*(w%4)..+31, columns 64*((w-2)/4)..+63 in chunks of 16.
//                Sixteen warps (four per SM sub-partition): with eight, bias + GeLU + pre-activation epilogues took
//                longer than the K = 2048 main loop of the next tile (measured 643 us against 407 us for the same
//                GEMM with a plain epilogue)
//
// Wide tile (NH = 2): 256 x 512, two accumulators of 256 columns that take the whole TMEM.  Long products run into the power cap,
// where what a product costs in energy sets the pace, not idle cycles: a quarter less traffic from the L2 for the same
// arithmetic lets the clock rise (4096 x 2048 over 51200: 1310 -> 1417 MHz at 990 W, tensor pipe 77 % busy either way).
//
// Barriers: `full` lives in the leader and counts the bytes of both CTAs' loads (the peer's TMA signals it
// through the cluster address); `empty` and `tmem_full` exist in both CTAs and are signalled together by a
// multicast tcgen05.commit; `tmem_empty` lives in the leader and collects the epilogue warps of both CTAs.
// Same operation and epilogue as gemm_bf16_kernel (runtime/megatron/mpu/layers.py:363,459,532,593 of the
// reference are the call sites this replaces).
#include <cuda.h>

#include "common.cuh"
#include "gemm_ag_sm100.cuh"
#include "gemm_epilogue.cuh"
#include "gemm_sm100.cuh"
#include "launch_once.cuh"

namespace ssb {

int make_tma_2d_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                     uint32_t box_rows, uint32_t box_cols);
int make_tma_im2col_bf16(CUtensorMap* map, const void* base, int N, int H, int W, int C, int lower_h, int lower_w,
                         int upper_h, int upper_w, int stride, int pixels);

namespace {

constexpr int BM2 = 128;   // rows per CTA (256 per cluster)
constexpr int BNH = 128;   // B rows staged per CTA (256 output columns per cluster)
constexpr int BN2 = 256;
constexpr int BK2 = 64;
constexpr int kStagesPlain = 5;
constexpr int kStagesGather = 4;                 // one stage (32 KB) becomes the pusher's staging area
constexpr int kStagesWide = 4;                   // of 48 KB
// wide tile: K blocks at both ends of a tile that are taken half by half; with one, sustained, 8192 x 2048 over 8192 226.1 -> 227.3 us, fp32
// over 16384 456 -> 460
constexpr int kSwitchGroup = 2;
constexpr int kPushChunk2 = 16384;
constexpr int kEpiWarps = 16;
constexpr int kThreads2 = 64 + kEpiWarps * 32;
constexpr int kThreadsGather = kThreads2 + 32;    // + pusher warp
constexpr int kGroupM2 = 8;
constexpr int kConvNone = 0, kConvA = 1, kConvB = 2;
constexpr int kABytes2 = BM2 * BK2 * 2;
constexpr int kBBytes2 = BNH * BK2 * 2;
constexpr int kStageBytes2 = kABytes2 + kBBytes2;
constexpr int kEpiStage = 32 * 128;                 // per epilogue warp: 32 rows x 64 bf16 columns (wide tile: 32 columns)
constexpr int kSmem2 = kStagesPlain * kStageBytes2 + kEpiWarps * kEpiStage + 1024 + 256;  // all variants
static_assert(kStagesWide * (kABytes2 + 2 * kBBytes2) + kEpiWarps * kEpiStage / 2 + 1024 + 256 <= kSmem2, "wide tile");

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa_smem(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load into this CTA's shared memory whose completion bytes are counted on an mbarrier that may live in
// the other CTA of the pair (no multicast: every CTA fetches its own tile).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
// The same for an im2col map over an NHWC tensor: pixels from (w, h, n) on, 64 channels from c, filter tap (ow, oh).
__device__ __forceinline__ void tma_load_im2col_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                     int c, int w, int h, int n, int ow, int oh) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.im2col.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c), "r"(w), "r"(h), "r"(n),
      "h"(static_cast<uint16_t>(ow)), "h"(static_cast<uint16_t>(oh))
      : "memory");
}
__device__ __forceinline__ void umma_f16_ss_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One arrival on the barrier at this offset in BOTH CTAs once all MMAs issued so far have retired.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}

// TMEM allocation for a CTA pair: warp 1 of BOTH CTAs executes these, with the same shared-memory offset.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// Bounded wait (one thread) until *flag >= epoch.
__device__ __forceinline__ bool wait_flag_one(const uint32_t* flag, uint32_t epoch, volatile int* abort_flag, int* status) {
  uint64_t t0 = 0;
  for (uint32_t it = 0; it < (1u << 30); ++it) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (v >= epoch) return true;
    if ((it & 1023u) == 1023u) {
      if (*abort_flag) return false;
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > 20ull * 1000 * 1000 * 1000) break;
    }
  }
  *abort_flag = 1;
  if (status != nullptr) atomicMax(status, static_cast<int>(kStatusPeerTimeout));
  return false;
}

struct TileCoord2 {
  int m_blk, n_blk;
};
__device__ __forceinline__ TileCoord2 tile_coord2(int tile, int num_m, int num_n) {
  const int per_group = kGroupM2 * num_n;
  const int group = tile / per_group;
  const int first_m = group * kGroupM2;
  const int gsize = min(num_m - first_m, kGroupM2);
  const int in_group = tile - group * per_group;
  TileCoord2 c;
  c.m_blk = first_m + in_group % gsize;
  c.n_blk = in_group / gsize;
  return c;
}

// GATHER = true: the all-gather of A's rows over the tensor-parallel group is part of the kernel (see
// gemm_ag_sm100.cu for the protocol): tma_a addresses this rank's own rows, tma_a2 the local gather buffer, output
// tiles are ordered own rows first, the producer waits for the "arrived" flag of a 128-row block before loading it,
// and warp 18 pushes this rank's rows to every peer.
//
// CONV: one operand is the patch matrix of a k x k convolution that never exists in memory: its tiles are fetched by TMA
// im2col loads straight from the NHWC activation.  Writing the patch matrix (k * k times the activation), reading it
// back and scattering its gradient were a third to a half of a 3 x 3 layer: 640 channels, 16 x 28 x 28, forward and backward
// with BatchNorm 439 -> 317 us; 61 x 7 x 7 of 1280 channels 364 -> 311, stride 2 (64 x 28 x 28 of 640) 462 -> 410.
//   kConvA: A's rows are pixels, the reduction runs over (tap, 64-channel block); forward (B = filter, K-major) and
//           input gradient (A = output gradient, taps flipped, B = filter read MN-major).  A channel block that reaches past C
//           is zero-filled, so what the filter's block holds there (the next tap) does not matter.
//   kConvB: filter gradient; the reduction runs over the pixels, B's columns are (tap, channel), C a multiple of 64.
// NARROW: a tile of `columns`, else of 256 (9472 x 512 over 64 8.1 -> 7.9 us with the width known to the compiler).
// FP32: the staged epilogue of fp32 outputs, else that of bf16 outputs; what does not fit either goes by chunks.  With both in one kernel
// bf16 outputs took longer, the same products 7.9 instead of 7.6 us.
template <bool A_MN, bool B_MN, bool GATHER, int CONV, int NH, bool NARROW, bool FP32>
__global__ void __launch_bounds__(GATHER ? kThreadsGather : kThreads2, 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_a2,
                  const __grid_constant__ CUtensorMap tma_b, const GemmParams p, const GemmAgComm cm, const ConvLoad cv, const int columns) {
  const int bn = NARROW ? columns : BN2;            // of an accumulator
  constexpr int kStages2 = NH == 2 ? kStagesWide : GATHER ? kStagesGather : kStagesPlain;
  const int BNT = NH == 2 ? 2 * BN2 : bn;           // columns of a tile
  constexpr int kStageAll = kABytes2 + NH * kBBytes2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + kStages2 * kABytes2;
  uint8_t* push_buf = smem + kStages2 * kStageAll;              // GATHER only: 2 x 16 KB
  uint8_t* epi_stage = push_buf + (GATHER ? 2 * kPushChunk2 : 0);
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_stage + kEpiWarps * kEpiStage / NH);
  uint64_t* full_bar = bars;                       // leader's are used
  uint64_t* empty_bar = bars + kStages2;           // both CTAs
  uint64_t* tmem_full_bar = bars + 2 * kStages2;   // both CTAs
  uint64_t* tmem_empty_bar = bars + 2 * kStages2 + 2;  // leader's are used
  uint64_t* push_bar = bars + 2 * kStages2 + 4;  // 2 (GATHER only)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages2 + 6);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  const int cluster_id = blockIdx.x >> 1;
  const int num_clusters = gridDim.x >> 1;

  const int num_m = (p.M + 2 * BM2 - 1) / (2 * BM2);
  const int num_n = (p.N + BNT - 1) / BNT;
  const int num_tiles = num_m * num_n;
  const int conv_cblk = CONV == kConvA ? (cv.C + BK2 - 1) / BK2 : 1;  // channel blocks per tap
  const int num_kb = CONV == kConvA ? cv.KH * cv.KW * conv_cblk : (p.K + BK2 - 1) / BK2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages2; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tmem_full_bar[s], 1);
      mbar_init(&tmem_empty_bar[s], 2 * kEpiWarps);
      mbar_init(&push_bar[s], 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anything signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  // GATHER: logical pair-block i (the order tiles are computed in) -> source rank and actual pair-block
  const int pb_per_rank = GATHER ? max(1, num_m / cm.tp) : 1;
  auto src_of = [&](int i) { return GATHER ? (cm.rank + i / pb_per_rank) % cm.tp : 0; };
  auto pblk_of = [&](int i) { return GATHER ? src_of(i) * pb_per_rank + i % pb_per_rank : i; };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = cluster_id; tile < num_tiles && ok; tile += num_clusters) {
        const TileCoord2 tc = tile_coord2(tile, num_m, num_n);
        int m0 = pblk_of(tc.m_blk) * 2 * BM2 + static_cast<int>(cta_rank) * BM2;
        const int n0 = tc.n_blk * BNT + static_cast<int>(cta_rank) * (bn / 2);
        const CUtensorMap* ta = &tma_a;
        if (GATHER) {
          if (src_of(tc.m_blk) == cm.rank) {
            m0 -= cm.rank * pb_per_rank * 2 * BM2;  // own rows: read straight from the local shard
          } else {
            // rows pushed by another rank: wait for this CTA's 128-row block, then order the TMA reads after it
            if (!wait_flag_one(cm.flag_ptrs[cm.rank] + m0 / BM2, cm.epoch, abort_flag, p.status)) { ok = false; break; }
            asm volatile("fence.proxy.async.global;" ::: "memory");
            ta = &tma_a2;
          }
        }
        // base position (w, h, n) of output pixel `pix`
        auto pixel = [&](int pix, int& w, int& h, int& n) {
          const int row = pix / cv.Wo;
          n = row / cv.Ho;
          h = (row - n * cv.Ho) * cv.stride + cv.lower_h;
          w = (pix - row * cv.Wo) * cv.stride + cv.lower_w;
        };
        int pw = 0, ph = 0, pn = 0;       // kConvA: base position of this CTA's first row
        int tap_r = 0, tap_s = 0, cb = 0;  // kConvA: filter tap and channel block of the K block
        int bc[2] = {0, 0}, br[2] = {0, 0}, bs[2] = {0, 0};  // kConvB: channel and tap of the two column chunks
        if (CONV == kConvA) pixel(min(m0, (p.M - 1) & ~(BM2 - 1)), pw, ph, pn);  // a CTA past the last row repeats it
        if (CONV == kConvB) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int col = min(n0 + c * 64, p.N - 64), tap = col / cv.C;  // past the last column: repeated, not stored
            bc[c] = col - tap * cv.C;
            br[c] = tap / cv.KW;
            bs[c] = tap - br[c] * cv.KW;
          }
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * (B_MN ? kStageAll : kABytes2 + NH * (bn / 2) * (BK2 * 2)));
          const uint32_t bar = mapa_smem(smem_u32(&full_bar[stage]), 0);
          uint8_t* sa = smem_a + stage * kABytes2;
          uint8_t* sb = smem_b + stage * (NH * kBBytes2);
          if (CONV == kConvA) {
            const int tap = tap_r * cv.KW + tap_s;
            const int ow = cv.flip ? cv.KW - 1 - tap_s : tap_s, oh = cv.flip ? cv.KH - 1 - tap_r : tap_r;
            tma_load_im2col_pair(sa, ta, bar, cb * BK2, pw, ph, pn, ow, oh);
            if (!B_MN) {
              tma_load_2d_pair(sb, &tma_b, bar, tap * cv.tap_cols + cb * BK2, n0);
            } else {
#pragma unroll
              for (int c = 0; c < BNH / 64; ++c)
                tma_load_2d_pair(sb + c * (64 * BK2 * 2), &tma_b, bar, tap * cv.tap_cols + n0 + c * 64, cb * BK2);
            }
            if (++cb == conv_cblk) {
              cb = 0;
              if (++tap_s == cv.KW) {
                tap_s = 0;
                ++tap_r;
              }
            }
          } else if (!A_MN) {
            tma_load_2d_pair(sa, ta, bar, kb * BK2, m0);
          } else {
#pragma unroll
            for (int c = 0; c < BM2 / 64; ++c) tma_load_2d_pair(sa + c * (64 * BK2 * 2), ta, bar, m0 + c * 64, kb * BK2);
          }
          if (CONV == kConvB) {
            pixel(kb * BK2, pw, ph, pn);
#pragma unroll
            for (int c = 0; c < BNH / 64; ++c)
              tma_load_im2col_pair(sb + c * (64 * BK2 * 2), &tma_b, bar, bc[c], pw, ph, pn, bs[c], br[c]);
          } else if (CONV == kConvNone) {
#pragma unroll
            for (int h = 0; h < NH; ++h) {
              if (!B_MN) {
                tma_load_2d_pair(sb + h * kBBytes2, &tma_b, bar, kb * BK2, n0 + h * BN2);
              } else {
#pragma unroll
                for (int c = 0; c < BNH / 64; ++c)
                  tma_load_2d_pair(sb + h * kBBytes2 + c * (64 * BK2 * 2), &tma_b, bar, n0 + h * BN2 + c * 64, kb * BK2);
              }
            }
          }
          if (++stage == kStages2) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      // The copies issued by this thread have landed once the MMAs that consume them retired, which the
      // epilogue of the last tile waits for; on an aborted run the teardown below waits for them instead.
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    if (leader && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(2 * BM2, bn, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      int iter = 0;
      bool ok = true;
      for (int tile = cluster_id; tile < num_tiles && ok; tile += num_clusters, ++iter) {
        // D (+)= A . B of one stage, 64 of the reduction
        auto products = [&](uint32_t tmem_d, int st, int h, bool first) {
          const uint32_t sa = smem_u32(smem_a + st * kABytes2);
          const uint32_t sb = smem_u32(smem_b + (st * NH + h) * kBBytes2);
#pragma unroll
          for (int k = 0; k < BK2 / 16; ++k) {
            const uint64_t da = A_MN ? umma_desc_sw128(sa + k * 2048, 64 * BK2 * 2, 1024)
                                     : umma_desc_sw128(sa + k * 32, 16, 1024);
            const uint64_t db = B_MN ? umma_desc_sw128(sb + k * 2048, 64 * BK2 * 2, 1024)
                                     : umma_desc_sw128(sb + k * 32, 16, 1024);
            umma_f16_ss_pair(tmem_d, da, db, idesc, !first || k != 0 ? 1u : 0u);
          }
        };
        if constexpr (NH == 2) {
          // Both halves take the whole TMEM, so the next tile waits for the epilogue.  The first and the last K blocks of a tile
          // are taken half by half: the first half is complete, and its columns wanted again, that much earlier.
          for (int kb = 0; kb < num_kb && ok;) {
            const bool last = kb + kSwitchGroup >= num_kb;
            const int g = last ? num_kb - kb : kb == 0 ? kSwitchGroup : 1;
            int st = stage;
            uint32_t ph = phase;
#pragma unroll
            for (int h = 0; h < NH; ++h) {
              if (kb == 0 && !(ok = ok && mbar_wait(&tmem_empty_bar[h], (iter & 1) ^ 1, abort_flag))) break;
              st = stage;
              ph = phase;
              for (int j = 0; j < g; ++j) {
                if (h == 0 && !(ok = mbar_wait(&full_bar[st], ph, abort_flag))) break;
                tc_fence_after_sync();
                products(tmem_base + h * BN2, st, h, kb + j == 0);
                if (h == NH - 1) umma_commit_pair(&empty_bar[st]);
                if (++st == kStages2) {
                  st = 0;
                  ph ^= 1;
                }
              }
              if (!ok) break;
              if (last) umma_commit_pair(&tmem_full_bar[h]);
            }
            stage = st;
            phase = ph;
            kb += g;
          }
          continue;
        }
        const int acc = iter & 1;
        const uint32_t acc_phase = (iter >> 1) & 1;
        if (!mbar_wait(&tmem_empty_bar[acc], acc_phase ^ 1, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          products(tmem_base + acc * BN2, stage, 0, kb == 0);
          umma_commit_pair(&empty_bar[stage]);
          if (++stage == kStages2) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit_pair(&tmem_full_bar[acc]);
      }
    }
  } else if (warp < 2 + kEpiWarps) {
    // -------------------------------- epilogue --------------------------------
    const int quarter = warp & 3;
    const int grp = (warp - 2) >> 2;  // 64-column group of the 256-column tile
    constexpr int kCols = 64 / NH, kPieces = kCols / 8, kRows = 32 / kPieces;  // columns staged at a time, 16-byte pieces of a row, rows per pass
    uint8_t* stg = epi_stage + (warp - 2) * (kEpiStage / NH);
    const uint32_t keep16 = dropout_keep16(p.dropout_p);
    const float drop_scale = p.dropout_p > 0.f ? 65536.0f / static_cast<float>(keep16) : 1.0f;
    int iter = 0;
    bool ok = true;
    for (int tile = cluster_id; tile < num_tiles && ok; tile += num_clusters, ++iter) {
      const TileCoord2 tc = tile_coord2(tile, num_m, num_n);
      const int row0 = pblk_of(tc.m_blk) * 2 * BM2 + static_cast<int>(cta_rank) * BM2 + quarter * 32;  // first row of this warp
      const int row = row0 + lane;
      const bool row_ok = row < p.M;
#pragma unroll 1
      for (int h = 0; h < NH && ok; ++h) {
        const int acc = NH == 2 ? h : iter & 1;
        const uint32_t acc_phase = (NH == 2 ? iter : iter >> 1) & 1;
        const int col0 = tc.n_blk * BNT + h * BN2 + grp * 64;  // first column
        const int col_end = min(p.N, tc.n_blk * BNT + h * BN2 + bn);
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BN2 + grp * 64;
        auto release = [&]() {  // the accumulator columns are free
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_smem(smem_u32(&tmem_empty_bar[acc]), 0));
        };
        // Staged path: bf16 output, no accumulate, the warp's 64 columns inside the matrix, at most one row operand.
        // Row operands enter and results leave through a swizzled staging tile, so every global access of the warp is four
        // full 128-byte row segments (wide tile: eight of 64 bytes) instead of 32 scattered 32-byte pieces.
        const bool has_operand = p.residual != nullptr || p.act == kActDGelu || p.act == kActDRelu;
        const bool staged = !FP32 && !p.out_fp32 && !p.accumulate && col0 + 64 <= col_end &&
                            !(p.residual != nullptr && (p.act == kActDGelu || p.act == kActDRelu)) &&
                            !(p.preact_out != nullptr && has_operand);
        if (staged) {
          const int srow = lane / kPieces, spiece = lane % kPieces;  // coalesced phase
          auto cell = [&](int rr, int piece) {
            return stg + rr * (kCols * 2) + ((piece ^ ((NH == 2 ? rr >> 1 : rr) & (kPieces - 1))) << 4);
          };
          auto fetch = [&](int c0) {
            const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(p.residual != nullptr ? p.residual : p.aux);
            const int ld = p.residual != nullptr ? p.ldres : p.ldaux;
#pragma unroll
            for (int it = 0; it < kPieces; ++it) {
              const int rr = it * kRows + srow;
              if (row0 + rr < p.M)
                *reinterpret_cast<uint4*>(cell(rr, spiece)) =
                    __ldg(reinterpret_cast<const uint4*>(src + static_cast<size_t>(row0 + rr) * ld + c0) + spiece);
            }
            __syncwarp();
          };
          auto flush = [&](void* base, int ld, int c0) {  // staging tile -> global
            __syncwarp();
#pragma unroll
            for (int it = 0; it < kPieces; ++it) {
              const int rr = it * kRows + srow;
              if (row0 + rr < p.M)
                *(reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(base) + static_cast<size_t>(row0 + rr) * ld + c0) +
                  spiece) = *reinterpret_cast<const uint4*>(cell(rr, spiece));
            }
            __syncwarp();
          };
          if (has_operand) fetch(col0);  // while the tensor cores still work on this tile
          if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full_bar[acc], acc_phase, abort_flag))) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
#pragma unroll 1
          for (int part = 0; part < NH; ++part) {
            const int c0 = col0 + part * kCols;
            if (part > 0 && has_operand) fetch(c0);
            if (p.preact_out != nullptr) {  // first pass: the pre-activation tile
#pragma unroll 1
              for (int c = 0; c < kCols / 16; ++c) {
                uint32_t r[16];
                tmem_ld_32x16(taddr + part * kCols + c * 16, r);
                tmem_ld_wait();
                const uint4 none[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
                float pre[16], v[16];
                gemm_epilogue_math16(p, row, c0 + c * 16, r, none, keep16, drop_scale, pre, v);
                *reinterpret_cast<uint4*>(cell(lane, 2 * c)) = pack8(pre);
                *reinterpret_cast<uint4*>(cell(lane, 2 * c + 1)) = pack8(pre + 8);
              }
              flush(p.preact_out, p.ldpre, c0);
            }
#pragma unroll 1
            for (int c = 0; c < kCols / 16; ++c) {
              uint32_t r[16];
              tmem_ld_32x16(taddr + part * kCols + c * 16, r);
              tmem_ld_wait();
              if (part == NH - 1 && c == kCols / 16 - 1) release();  // its last columns are in registers
              uint4 operand[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
              if (has_operand) {
                operand[0] = *reinterpret_cast<const uint4*>(cell(lane, 2 * c));
                operand[1] = *reinterpret_cast<const uint4*>(cell(lane, 2 * c + 1));
              }
              float pre[16], v[16];
              gemm_epilogue_math16(p, row, c0 + c * 16, r, operand, keep16, drop_scale, pre, v);
              *reinterpret_cast<uint4*>(cell(lane, 2 * c)) = pack8(v);
              *reinterpret_cast<uint4*>(cell(lane, 2 * c + 1)) = pack8(v + 8);
            }
            flush(p.D, p.ldd, c0);
          }
          continue;
        }
        // fp32 output: 16 columns at a time through the staging tile, 64-byte row segments to memory; what is there already
        // (gradients are added to) is read in the same pieces, one ahead; the first while the tensor cores still work on this tile.
        // A thread with a row of its own moved 16 of every 32-byte sector at a time and waited for each 16 columns of old values
        // in turn; with a reduction of 4096 that took longer than the main loop of the next tile.  Alone / sustained under the
        // power cap: weight gradients 51200 x 2048 over 4096 rows 649 -> 600 / 805 -> 754 us, 8192 x 2048 over 8192 216 -> 209 /
        // 255 -> 248.
        if (FP32 && p.out_fp32 && col0 + 64 <= col_end && !has_operand && p.preact_out == nullptr) {
          const int srow = lane >> 2, spiece = lane & 3;
          float* out = reinterpret_cast<float*>(p.D) + static_cast<size_t>(row0 + srow) * p.ldd + col0 + spiece * 4;
          auto cell = [&](int rr, int piece) { return stg + rr * 64 + ((piece ^ ((rr >> 1) & 3)) << 4); };
          auto old_values = [&](float4 (&o)[4], int c) {
#pragma unroll
            for (int it = 0; it < 4; ++it)
              if (row0 + it * 8 + srow < p.M) o[it] = *reinterpret_cast<const float4*>(out + static_cast<size_t>(it * 8) * p.ldd + c * 16);
          };
          float4 old[4] = {}, next[4] = {};
          if (p.accumulate) old_values(old, 0);
          if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full_bar[acc], acc_phase, abort_flag))) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            if (p.accumulate && c < 3) old_values(next, c + 1);
            uint32_t r[16];
            tmem_ld_32x16(taddr + c * 16, r);
            tmem_ld_wait();
            if (c == 3) release();
            const uint4 none[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
            float pre[16], v[16];
            gemm_epilogue_math16(p, row, col0 + c * 16, r, none, keep16, drop_scale, pre, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(cell(lane, i)) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            __syncwarp();
#pragma unroll
            for (int it = 0; it < 4; ++it) {
              const int rr = it * 8 + srow;
              float4 q = *reinterpret_cast<const float4*>(cell(rr, spiece));
              if (row0 + rr < p.M) {
                if (p.accumulate) {
                  q.x += old[it].x; q.y += old[it].y; q.z += old[it].z; q.w += old[it].w;
                }
                *reinterpret_cast<float4*>(out + static_cast<size_t>(it * 8) * p.ldd + c * 16) = q;
              }
            }
#pragma unroll
            for (int it = 0; it < 4; ++it) old[it] = next[it];
            __syncwarp();
          }
          continue;
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full_bar[acc], acc_phase, abort_flag))) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          const int n0 = col0 + c * 16;
          if (n0 >= col_end) break;  // uniform across the warp
          uint32_t r[16];
          tmem_ld_32x16(taddr + c * 16, r);
          tmem_ld_wait();
          if (!row_ok) continue;
          gemm_epilogue_chunk<16>(p, row, n0, r, keep16, drop_scale);
        }
        release();
      }
    }
  } else if (GATHER) {
    // --------------------------------- pusher ---------------------------------
    // Copies this rank's rows, 128-row block by block (CTA c takes blocks c, c + grid, ...), through a double-
    // buffered 16 KB staging area into the same rows of every peer's gather buffer, then flags the block there.
    if (lane == 0 && cm.tp > 1) {
      const size_t blk_bytes = static_cast<size_t>(BM2) * p.K * 2;  // shard and gather buffers are dense
      const uint8_t* x = reinterpret_cast<const uint8_t*>(cm.x_local);
      const int blocks_per_rank = pb_per_rank * 2;
      const int pieces_per_blk = static_cast<int>(blk_bytes / kPushChunk2);
      int my_blocks = 0;
      for (int b = blockIdx.x; b < blocks_per_rank; b += gridDim.x) ++my_blocks;
      const int total = my_blocks * pieces_per_blk;
      auto issue_load = [&](int j) {
        const int b = blockIdx.x + (j / pieces_per_blk) * gridDim.x;
        mbar_arrive_expect_tx(&push_bar[j & 1], kPushChunk2);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(push_buf + (j & 1) * kPushChunk2)),
                     "l"(x + static_cast<size_t>(b) * blk_bytes + static_cast<size_t>(j % pieces_per_blk) * kPushChunk2),
                     "r"(kPushChunk2), "r"(smem_u32(&push_bar[j & 1]))
                     : "memory");
      };
      bool okp = true;
      if (total > 0) issue_load(0);
      for (int j = 0; j < total && okp; ++j) {
        if (j + 1 < total) {
          tma_store_wait_read<0>();  // the stores of piece j - 1 have left the other buffer
          issue_load(j + 1);
        }
        if (!mbar_wait(&push_bar[j & 1], (j >> 1) & 1, abort_flag)) { okp = false; break; }
        const int b = blockIdx.x + (j / pieces_per_blk) * gridDim.x;
        const size_t dst_off = (static_cast<size_t>(cm.rank) * blocks_per_rank + b) * blk_bytes +
                               static_cast<size_t>(j % pieces_per_blk) * kPushChunk2;
        for (int pr = 0; pr < cm.tp; ++pr)
          if (pr != cm.rank)
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                             reinterpret_cast<uint8_t*>(cm.gather_ptrs[pr]) + dst_off),
                         "r"(smem_u32(push_buf + (j & 1) * kPushChunk2)), "r"(kPushChunk2)
                         : "memory");
        tma_store_commit();
        if (j % pieces_per_blk == pieces_per_blk - 1) {
          tma_store_wait<0>();  // the whole block has been written on every peer
          for (int pr = 0; pr < cm.tp; ++pr)
            if (pr != cm.rank)
              asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(cm.flag_ptrs[pr] + cm.rank * blocks_per_rank + b),
                           "r"(cm.epoch)
                           : "memory");
        }
      }
      tma_store_wait<0>();
    }
  }

  // ------------------------------- teardown ----------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // Aborted: give the copies in flight into this CTA's shared memory a bounded time to land.
    if (threadIdx.x == 0) {
      if (p.status != nullptr) atomicMax(p.status, static_cast<int>(kStatusMbarTimeout));
      const uint64_t t0 = global_timer_ns();
      for (uint32_t it = 0; it < (1u << 22); ++it)
        if (global_timer_ns() - t0 > 2000000ull) break;
    }
    __syncthreads();
  }
  cluster_sync_all();  // neither CTA leaves (or frees TMEM) while the other may still address it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <bool A_MN, bool B_MN, bool GATHER, int CONV, int NH, bool NARROW, bool FP32>
int launch_maps(const CUtensorMap& ta, const CUtensorMap& ta2, const CUtensorMap& tb, const GemmParams& p,
                const GemmAgComm& cm, const ConvLoad& cv, int bn, int num_sms, cudaStream_t stream) {
  auto kernel = gemm2_bf16_kernel<A_MN, B_MN, GATHER, CONV, NH, NARROW, FP32>;
  constexpr int threads = GATHER ? kThreadsGather : kThreads2;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  static OncePerDevice<> resident;
  int dev = 0, max_clusters = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return static_cast<int>(e);
  const int rc = resident.get(dev, &max_clusters, [&](int* clusters) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem2);
    if (e != cudaSuccess) return static_cast<int>(e);
    cudaLaunchConfig_t q = {};
    q.gridDim = dim3(num_sms & ~1);
    q.blockDim = dim3(threads);
    q.dynamicSmemBytes = kSmem2;
    q.attrs = attr;
    q.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(clusters, kernel, &q);
    if (e != cudaSuccess || *clusters < 1) {
      (void)cudaGetLastError();
      return -5;
    }
    return 0;
  });
  if (rc) return rc;
  const int num_tiles = ((p.M + 2 * BM2 - 1) / (2 * BM2)) * ((p.N + NH * bn - 1) / (NH * bn));
  int clusters = num_sms / 2;
  if (clusters > max_clusters) clusters = max_clusters;
  if (clusters > num_tiles) clusters = num_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = kSmem2;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, ta, ta2, tb, p, cm, cv, bn));
}

// The tile of 256 x 512 takes a product with a long reduction, where its end (the next tile waits for the epilogue) weighs little,
// and where counting in whole rounds of 256 columns costs nothing.  us of a single call / sustained under the power cap, 256 -> 512
// columns, 8192 x 2048 in bf16: over 4096 109 -> 117 / 116 -> 119; 6144 155 -> 160 / 175 -> 172; 8192 207 -> 210 / 235 -> 226; 10240 252 -> 253;
// 12288 303 -> 292 / 349 -> 330.  Over 8192, the first length taken, a single call is slower (4096 x 2048 113 -> 116, 2048 x 8192 203 -> 209)
// and a loop faster (119 -> 114, 231 -> 228); training is loops.  4096 x 2048 over 51200 594 -> 568 / 708 -> 652.  fp32, added to: over 8192
// 210 -> 224 / 251 -> 246; 16384 406 -> 401 / 485 -> 457, 4096 x 2048 208 -> 210 / 243 -> 226; 32768 818 -> 755 / 956 -> 883.
constexpr int kWideK = 8192, kWideKFp32 = 16384;
bool wide_tile(int M, int N, int K, bool out_fp32, int num_sms) {
  const long long m = (M + 255LL) / 256, narrow = m * ((N + 255LL) / 256), wide = m * ((N + 511LL) / 512);
  const int pairs = num_sms / 2;
  return N >= 512 && K >= (out_fp32 ? kWideKFp32 : kWideK) && 2 * ((wide + pairs - 1) / pairs) <= (narrow + pairs - 1) / pairs;
}

// Columns of a tile, in steps of the 32 that a pair's instruction takes: fewer than 256 where the rounds of narrower tiles are enough
// shorter.  A round costs its columns and a part that does not shrink with them (A's rows, the epilogue; of a B read MN-major
// always 128 columns a CTA), measured like BN2 more columns or twice that.  Single call / sustained under the power cap, 256
// columns -> fewer, us:
//   taken      K-major B: 2048 x 3072 over 2048 34.8 -> 30.7 / 28.7 -> 26.3 (192), 2560 x 2048 over 4096 56.3 -> 47.1 / 47.1 -> 40.7 (160),
//              4096 x 5120 over 4096 134 -> 120 / 145 -> 141 (224), 12544 x 640 64.4 -> 60.3 / 67.5 -> 62.8 (224: a sixth was padding);
//              MN-major: 2560 x 4096 over 4096 82.9 -> 72.7 / 79.1 -> 75.8 (192), fp32 and added to 91.0 -> 82.9 / 90.1 -> 89.2
//   not taken  8192 x 2560 over 2048 72.7 -> 76.8 / 75.8 -> 79.8 (160: seven rounds for five), 16384 x 1536 MN-major over 4096 216 -> 194 /
//              174 -> 178 (192: seven for six), 2048 x 8192 MN-major fp32 over 4096 136 -> 116 / 130 -> 134 (224: more tiles, no padding)
//   short      reductions end before a tile's epilogue does: 4096 x 5120 over 512 28.6 -> 29.1 sustained, 2048 x 10240 28.7 -> 29.3
// `more_tiles`: whether there may be more tiles than of 256 columns.  Rows off 128 bytes and an MN-major B: more tiles cost more than
// they save (3064 x 1984 over 4096 57.4 -> 65.3 with 192 columns, 3072 rows 54.3 -> 53.1); of a product as many do, too (12536 x 640 fp32
// over 4096 73.5 -> 77.9), of an input gradient they do not (3 x 3, 16 x 56 x 56 of 272 channels 120 -> 112 / 113 -> 97.5 with 160, 8 x 56 x
// 56 of 560 165 -> 144 / 144 -> 130, 64 x 28 x 28 of 264 133 -> 144 / 142 -> 133), and more do not inside one round (4 x 28 x 28 of 784
// 56.3 -> 48.1 / 47.1 -> 42.9; two rounds: 4 x 56 x 56 of 392 67.6 -> 70.6 / 61.4 -> 65.6).
// Convolutions 3 x 3: 16 x 28 x 28 of 640 channels, 224 columns, forward 67.6 -> 62.0, input gradient 68.5 -> 64.4; forward of 16 x 56 x 56
// of 320, 160 columns, 124 -> 85 / 104 -> 82, of 64 x 28 x 28 of 392, 224 columns, 200 -> 194 / 190 -> 183 (160: 218 / 205).
int tile_columns(int M, int N, int K, bool b_mn, bool more_tiles, int num_sms) {
  const long long pairs = num_sms / 2, m = (M + 255LL) / 256;
  auto n = [&](int bn) { return (N + bn - 1LL) / bn; };
  auto rounds = [&](int bn) { return (m * n(bn) + pairs - 1) / pairs; };
  auto cost = [&](int bn) { return rounds(bn) * (bn + (b_mn ? 2 * BN2 : BN2)); };
  int best = BN2;
  for (int bn = BN2 - 32; bn >= 160; bn -= 32)
    if (cost(bn) < cost(best) && (more_tiles || n(bn) == n(BN2))) best = bn;
  const bool less_padding = 10 * n(best) * best <= 9 * n(BN2) * BN2;
  const int percent = K < 1024 && rounds(BN2) > 2 ? 90 : !b_mn ? 95 : less_padding ? 96 : 93;
  return 100 * cost(best) <= percent * cost(BN2) ? best : BN2;
}
bool whole_lines(int lda, int ldb) { return lda % 64 == 0 && ldb % 64 == 0; }

template <bool A_MN, bool B_MN, bool GATHER>
int launch_pair(const void* A, int lda, const void* B, int ldb, const GemmParams& p, const GemmAgComm& cm, int num_sms,
                cudaStream_t stream) {
  CUtensorMap ta, ta2, tb;
  int rc;
  if (GATHER) {  // A = this rank's rows [M / tp][K]; the gather buffer holds all M rows
    rc = make_tma_2d_bf16(&ta, A, p.M / cm.tp, p.K, lda, BM2, BK2);
    if (rc != 0) return rc;
    rc = make_tma_2d_bf16(&ta2, cm.gather_ptrs_host_local, p.M, p.K, p.K, BM2, BK2);
  } else {
    rc = !A_MN ? make_tma_2d_bf16(&ta, A, p.M, p.K, lda, BM2, BK2) : make_tma_2d_bf16(&ta, A, p.K, p.M, lda, BK2, 64);
    ta2 = ta;
  }
  if (rc != 0) return rc;
  const bool wide = !GATHER && wide_tile(p.M, p.N, p.K, p.out_fp32, num_sms);
  const int bn = GATHER || wide || (B_MN && !whole_lines(lda, ldb)) ? BN2 : tile_columns(p.M, p.N, p.K, B_MN, true, num_sms);
  rc = !B_MN ? make_tma_2d_bf16(&tb, B, p.N, p.K, ldb, bn / 2, BK2) : make_tma_2d_bf16(&tb, B, p.K, p.N, ldb, BK2, 64);
  if (rc != 0) return rc;
  auto launch = [&](auto kernel_for) { return kernel_for(ta, ta2, tb, p, cm, ConvLoad{}, bn, num_sms, stream); };
  if constexpr (GATHER) {
    return launch(launch_maps<A_MN, B_MN, true, kConvNone, 1, false, false>);
  } else if (p.out_fp32) {
    if (wide) return launch(launch_maps<A_MN, B_MN, false, kConvNone, 2, false, true>);
    if (bn != BN2) return launch(launch_maps<A_MN, B_MN, false, kConvNone, 1, true, true>);
    return launch(launch_maps<A_MN, B_MN, false, kConvNone, 1, false, true>);
  } else {
    if (wide) return launch(launch_maps<A_MN, B_MN, false, kConvNone, 2, false, false>);
    if (bn != BN2) return launch(launch_maps<A_MN, B_MN, false, kConvNone, 1, true, false>);
    return launch(launch_maps<A_MN, B_MN, false, kConvNone, 1, false, false>);
  }
}

}  // namespace

// Columns of the output tile for a product that this kernel takes.
int gemm2_tile_columns(int M, int N, int K, bool b_mn, bool whole_lines, bool out_fp32, int num_sms) {
  if (wide_tile(M, N, K, out_fp32, num_sms)) return 2 * BN2;
  return b_mn && !whole_lines ? BN2 : tile_columns(M, N, K, b_mn, true, num_sms);
}

// Same contract as gemm_bf16_launch; callers pick this variant for outputs of at least 256 x 256.
int gemm2_bf16_launch(const void* A, int lda, int a_mn_major, const void* B, int ldb, int b_mn_major,
                      const GemmParams& p, int num_sms, cudaStream_t stream) {
  const GemmAgComm none{};
  if (!a_mn_major && !b_mn_major) return launch_pair<false, false, false>(A, lda, B, ldb, p, none, num_sms, stream);
  if (!a_mn_major && b_mn_major) return launch_pair<false, true, false>(A, lda, B, ldb, p, none, num_sms, stream);
  if (a_mn_major && b_mn_major) return launch_pair<true, true, false>(A, lda, B, ldb, p, none, num_sms, stream);
  return launch_pair<true, false, false>(A, lda, B, ldb, p, none, num_sms, stream);
}

// All-gather fused into the GEMM on the two-SM kernel.  Returns -100 when the shape does not fit this variant
// (rows per rank not a multiple of 256, narrow output): the caller then uses the one-CTA kernel of gemm_ag_sm100.cu.
int gemm2_ag_launch(const void* W, int ldw, const GemmParams& p, const GemmAgComm& cm, int num_sms, cudaStream_t stream) {
  const int rows_local = p.M / cm.tp;
  if (rows_local % (2 * BM2) || p.N < BN2 || (static_cast<size_t>(BM2) * p.K * 2) % kPushChunk2) return -100;
  return launch_pair<false, false, true>(cm.x_local, p.K, W, ldw, p, cm, num_sms, stream);
}

// Whether the implicit convolution takes this GEMM view of a k x k convolution: the two-SM tile must be worth it (the rule of
// gemm_bf16_launch), channel blocks of 64 may waste at most a fifth of the reduction (kConvA), and the limits of an
// im2col map hold (offsets below 256, corners within a signed byte).
bool conv_implicit_ok(long long M, int N, int C, int KH, int KW, int stride, int pad, bool columns_are_patches, int num_sms) {
  if (C % 8 || KH > 16 || KW > 16 || stride > 8 || pad < 0 || pad >= KH || pad >= KW || M > 0x7fffff00LL) return false;
  if (columns_are_patches ? C % 64 != 0 : (C % 64 != 0 && C < 256)) return false;
  const long long tiles = ((M + 255) / 256) * ((N + 255) / 256);
  return M >= 256 && N >= 256 && tiles >= num_sms / 4;
}

// y[N, Ho, Wo, K] = conv(x[N, H, W, C], w[K, KH * KW * C]); p describes the GEMM [N Ho Wo, K] with K = KH * KW * C.
int conv_fprop_launch(const void* x, int N, int H, int W, int C, const void* w, int ldw, int KH, int KW, int stride, int pad,
                      const GemmParams& p, int num_sms, cudaStream_t stream) {
  CUtensorMap ta, tb;
  int rc;
  if ((rc = make_tma_im2col_bf16(&ta, x, N, H, W, C, -pad, -pad, pad - (KH - 1), pad - (KW - 1), stride, BM2))) return rc;
  const int bn = tile_columns(p.M, p.N, p.K, false, true, num_sms);
  if ((rc = make_tma_2d_bf16(&tb, w, p.N, p.K, ldw, bn / 2, BK2))) return rc;
  ConvLoad cv{C, KH, KW, stride, -pad, -pad, (H + 2 * pad - KH) / stride + 1, (W + 2 * pad - KW) / stride + 1, 0, C};
  auto launch = bn == BN2 ? launch_maps<false, false, false, kConvA, 1, false, false> : launch_maps<false, false, false, kConvA, 1, true, false>;
  return launch(ta, ta, tb, p, GemmAgComm{}, cv, bn, num_sms, stream);
}

// dx[N, H, W, C] of a stride-1 convolution from dy[N, Ho, Wo, K]; p describes the GEMM [N H W, C] with K = KH * KW * K.
int conv_dgrad_launch(const void* dy, int N, int H, int W, int Kout, const void* w, int ldw, int C, int KH, int KW, int pad,
                      const GemmParams& p, int num_sms, cudaStream_t stream) {
  CUtensorMap ta, tb;
  int rc;
  const int Ho = H + 2 * pad - KH + 1, Wo = W + 2 * pad - KW + 1;
  const int lh = pad - (KH - 1), lw = pad - (KW - 1);
  if ((rc = make_tma_im2col_bf16(&ta, dy, N, Ho, Wo, Kout, lh, lw, -pad, -pad, 1, BM2))) return rc;
  if ((rc = make_tma_2d_bf16(&tb, w, Kout, static_cast<uint64_t>(KH) * KW * C, ldw, BK2, 64))) return rc;
  ConvLoad cv{Kout, KH, KW, 1, lh, lw, H, W, 1, C};
  const bool one_round = (p.M + 255LL) / 256 * ((p.N + 255LL) / 256) <= num_sms / 2;
  const int bn = tile_columns(p.M, p.N, p.K, true, whole_lines(Kout, ldw) || one_round, num_sms);
  auto launch = bn == BN2 ? launch_maps<false, true, false, kConvA, 1, false, false> : launch_maps<false, true, false, kConvA, 1, true, false>;
  return launch(ta, ta, tb, p, GemmAgComm{}, cv, bn, num_sms, stream);
}

// dw[K, KH * KW * C] from dy[N Ho Wo, K] and x; p describes the GEMM [K, KH * KW * C] with K = N Ho Wo.
int conv_wgrad_launch(const void* dy, int lddy, const void* x, int N, int H, int W, int C, int KH, int KW, int stride, int pad,
                      const GemmParams& p, int num_sms, cudaStream_t stream) {
  CUtensorMap ta, tb;
  int rc;
  if ((rc = make_tma_2d_bf16(&ta, dy, p.K, p.M, lddy, BK2, 64))) return rc;
  if ((rc = make_tma_im2col_bf16(&tb, x, N, H, W, C, -pad, -pad, pad - (KH - 1), pad - (KW - 1), stride, BK2))) return rc;
  ConvLoad cv{C, KH, KW, stride, -pad, -pad, (H + 2 * pad - KH) / stride + 1, (W + 2 * pad - KW) / stride + 1, 0, C};
  return launch_maps<true, true, false, kConvB, 1, false, true>(ta, ta, tb, p, GemmAgComm{}, cv, BN2, num_sms, stream);
}

}  // namespace ssb
