// bf16 GEMM for outputs of few tiles (at most one per SM; gemm_cluster_plan says which): a cluster of S CTAs shares an output tile of 128 x BN, each reduces
// its slice of K on its own SM, and the partial tiles meet in the epilogue over distributed shared memory.  Same operands
// and the same operations in the epilogue as the other GEMM kernels (gemm_sm100.cuh).
//
// A small output is a matter of latency: a chain of K / 64 steps on each of a few SMs, then an epilogue in which one thread
// walks one row.  Here the chain is cut by S and by narrower tiles (BN 64), and the epilogue goes through shared memory: CTA r of
// the cluster takes rows [128 r / S, 128 (r + 1) / S) of the tile, adds the S partial sums in slice order (deterministic),
// and its eight warps read operands and write results as whole row segments.  What the epilogue reads (old output, residual,
// derivative input) is fetched while the products still run.
//
// Measured against one CTA per tile of 128 x 128 (forward with dropout and residual / weight gradient into an fp32 buffer, us):
// 512 x 1024 x 1024 12.7 -> 9.1 / 15.0 -> 8.6, 512 x 1024 x 4096 23.0 -> 12.0, 512 x 4096 x 1024 13.1 -> 11.4, its input gradient
// 19.3 -> 11.6, 64 x 2048 x 512 9.9 -> 7.6 / 13.5 -> 6.0, 128 x 128 x 8192 36.1 -> 9.4.
//
// Threads: warp 0 = TMA, warp 1 = TMEM + MMA, warps 2..9 epilogue (TMEM lane quarter warp % 4, column half (warp - 2) / 4).
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "gemm_sm100.cuh"

namespace ssb {

int make_tma_2d_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
                     uint32_t box_cols);

namespace {

constexpr int BM = 128, BK = 64;
constexpr int kEpiThreads = 256, kThreads = 64 + kEpiThreads;
constexpr int kMaxCluster = 8;

template <int BN>
struct Cfg {
  static constexpr int kStages = BN == 128 ? 4 : 6;
  static constexpr int kABytes = BM * BK * 2, kBBytes = BN * BK * 2, kStageBytes = kABytes + kBBytes;
  static constexpr int kPitch = BN + 4;                      // floats a row of the partial tile: 16-byte pieces, odd count
  static constexpr int kOpBytes = BM * BN * 2, kOldBytes = BM * BN * 4;  // row operand (bf16) and old output of the rows
  static constexpr int kSmem = kStages * kStageBytes + kOpBytes + kOldBytes + 1024 + 256;
  static constexpr int kItems = BM * BN / 4 / kEpiThreads;   // groups of four columns per thread without a cluster
  static_assert(BM * kPitch * 4 <= kStages * kStageBytes, "the partial tile takes the place of the operand stages");
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ void unpack4(uint2 q, float (&f)[4]) {
  const float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
// four bf16 values from column n0 on, zeros behind column N
__device__ __forceinline__ uint2 load4(const void* base, size_t at, int left) {
  const __nv_bfloat16* s = reinterpret_cast<const __nv_bfloat16*>(base) + at;
  if (left >= 4) return *reinterpret_cast<const uint2*>(s);
  uint32_t h[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (i < left) h[i] = *reinterpret_cast<const unsigned short*>(s + i);
  return make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
}
__device__ __forceinline__ void store4(void* base, size_t at, const float (&v)[4], int left) {
  __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(base) + at;
  if (left >= 4) {
    *reinterpret_cast<uint2*>(d) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i < left) d[i] = __float2bfloat16(v[i]);
  }
}

// Copies rows [row0, row0 + rows) x columns [n0, min(n0 + BN, N)) of a matrix with E-byte elements to shared memory, [rows][BN].
template <int BN, int E>
__device__ __forceinline__ void fetch_rows(uint8_t* dst, const void* base, int ld, size_t row0, int rows, int n0, int N, int e) {
  constexpr int PER = 16 / E, PIECES = BN / PER;  // elements of a 16-byte piece, pieces of a row
#pragma unroll 1
  for (int i = e; i < rows * PIECES; i += kEpiThreads) {
    const int r = i / PIECES, c = (i % PIECES) * PER;
    const uint8_t* src = reinterpret_cast<const uint8_t*>(base) + ((row0 + r) * ld + n0 + c) * E;
    uint8_t* to = dst + (r * BN + c) * E;
    if (n0 + c + PER <= N) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to)), "l"(src) : "memory");
    } else {
#pragma unroll 1
      for (int j = 0; j < PER && n0 + c + j < N; ++j) {
        if (E == 4) reinterpret_cast<uint32_t*>(to)[j] = reinterpret_cast<const uint32_t*>(src)[j];
        else reinterpret_cast<unsigned short*>(to)[j] = reinterpret_cast<const unsigned short*>(src)[j];
      }
    }
  }
}

// Partial sums of the first N of U places from the S CTAs of the cluster, added in slice order; all loads are under way together.
template <int S, int N, int U>
__device__ __forceinline__ void sum_slices(const float* const (&mine)[U], float (&v)[U][4]) {
  static_assert(N <= U, "places");
  float4 t[S][N];
#pragma unroll
  for (int k = 0; k < S; ++k)
#pragma unroll
    for (int u = 0; u < N; ++u) t[k][u] = ld_cluster_v4(smem_u32(mine[u]), k);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (u >= N) {
      v[u][0] = v[u][1] = v[u][2] = v[u][3] = 0.f;
      continue;
    }
    float4 s = t[0][u < N ? u : 0];
#pragma unroll
    for (int k = 1; k < S; ++k) {
      const float4 x = t[k][u < N ? u : 0];
      s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
    }
    v[u][0] = s.x; v[u][1] = s.y; v[u][2] = s.z; v[u][3] = s.w;
  }
}

template <int BN, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmParams p,
                    const int slices) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + C::kStages * C::kABytes;
  float* part = reinterpret_cast<float*>(smem);   // after the last product: this CTA's partial tile, [128][kPitch]
  uint8_t* s_op = smem + C::kStages * C::kStageBytes;        // [128 / S][BN]
  uint8_t* s_old = s_op + C::kOpBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(s_old + C::kOldBytes);
  uint64_t* empty_bar = full_bar + C::kStages;
  uint64_t* acc_bar = empty_bar + C::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = slices > 1 ? static_cast<int>(cluster_rank()) : 0;
  const int tile = blockIdx.x / slices;
  const int num_m = (p.M + BM - 1) / BM;
  const int m0 = (tile % num_m) * BM, n0 = (tile / num_m) * BN;
  const int num_kb = (p.K + BK - 1) / BK, per = (num_kb + slices - 1) / slices;
  const int kb0 = rank * per, kb1 = min(num_kb, kb0 + per);

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  const bool derivative = p.act == kActDGelu || p.act == kActDRelu, has_operand = p.residual != nullptr || derivative;
  constexpr int LPR = BN / 4;                               // threads per row in the second half of the epilogue
  const int e = static_cast<int>(threadIdx.x) - 64;
  const int col = (e % LPR) * 4, left = p.N - n0 - col;     // first of this thread's four columns
  const int items = C::kItems / slices;
  bool ok = true;

  if (warp == 0) {
    if (elect_one()) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int n = kb - kb0, stage = n % C::kStages;
        if (!mbar_wait(&empty_bar[stage], ((n / C::kStages) & 1) ^ 1, abort_flag)) {
          for (int i = max(n - C::kStages, 0); i < n; ++i)  // let the copies in flight land before the CTA leaves
            for (uint32_t it = 0; it < (1u << 20); ++it)
              if (mbar_try_wait(&full_bar[i % C::kStages], (i / C::kStages) & 1)) break;
          break;
        }
        mbar_arrive_expect_tx(&full_bar[stage], C::kStageBytes);
        uint8_t* sa = smem_a + stage * C::kABytes;
        uint8_t* sb = smem_b + stage * C::kBBytes;
        if (!A_MN) {
          tma_load_2d(sa, &tma_a, &full_bar[stage], kb * BK, m0);
        } else {
#pragma unroll
          for (int c = 0; c < BM / 64; ++c) tma_load_2d(sa + c * (64 * BK * 2), &tma_a, &full_bar[stage], m0 + c * 64, kb * BK);
        }
        if (!B_MN) {
          tma_load_2d(sb, &tma_b, &full_bar[stage], kb * BK, n0);
        } else {
#pragma unroll
          for (int c = 0; c < BN / 64; ++c) tma_load_2d(sb + c * (64 * BK * 2), &tma_b, &full_bar[stage], n0 + c * 64, kb * BK);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(BM, BN, A_MN, B_MN);
      bool fine = true;
      for (int kb = kb0; kb < kb1 && fine; ++kb) {
        const int n = kb - kb0, stage = n % C::kStages;
        if (!(fine = mbar_wait(&full_bar[stage], (n / C::kStages) & 1, abort_flag))) break;
        tc_fence_after_sync();
        const uint32_t sa = smem_u32(smem_a + stage * C::kABytes), sb = smem_u32(smem_b + stage * C::kBBytes);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          const uint64_t da = A_MN ? umma_desc_sw128(sa + k * 2048, 64 * BK * 2, 1024) : umma_desc_sw128(sa + k * 32, 16, 1024);
          const uint64_t db = B_MN ? umma_desc_sw128(sb + k * 2048, 64 * BK * 2, 1024) : umma_desc_sw128(sb + k * 32, 16, 1024);
          umma_f16_ss(tmem_base, da, db, idesc, (n | k) != 0 ? 1u : 0u);
        }
        umma_commit(&empty_bar[stage]);
      }
      if (fine) umma_commit(acc_bar);
    }
  } else {
    // what the epilogue reads, under the products
    const int rows = min(BM / slices, p.M - m0 - rank * (BM / slices));
    const size_t row0 = static_cast<size_t>(m0 + rank * (BM / slices));
    if (has_operand) fetch_rows<BN, 2>(s_op, p.residual != nullptr ? p.residual : p.aux, p.residual != nullptr ? p.ldres : p.ldaux, row0, rows, n0, p.N, e);
    if (p.accumulate) {
      if (p.out_fp32) fetch_rows<BN, 4>(s_old, p.D, p.ldd, row0, rows, n0, p.N, e);
      else fetch_rows<BN, 2>(s_old, p.D, p.ldd, row0, rows, n0, p.N, e);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    ok = __all_sync(0xffffffffu, mbar_wait(acc_bar, 0, abort_flag));
    if (ok) {
      tc_fence_after_sync();
      const int quarter = warp & 3, c0 = ((warp - 2) >> 2) * (BN / 2);
      float* dst = part + (quarter * 32 + lane) * C::kPitch + c0;
#pragma unroll
      for (int c = 0; c < BN / 2; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c0 + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
      }
    }
  }
  tc_fence_before_sync();
  __syncwarp();
  if (slices > 1) cluster_barrier();  // (also the CTA's own barrier)
  else __syncthreads();

  if (warp >= 2 && ok) {
    const uint32_t keep16 = dropout_keep16(p.dropout_p);
    const float drop_scale = p.dropout_p > 0.f ? 65536.0f / static_cast<float>(keep16) : 1.0f;
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.bias != nullptr && left > 0) {
      if (p.bias_fp32) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < left) bias[i] = __ldg(reinterpret_cast<const float*>(p.bias) + n0 + col + i);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < left) bias[i] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[n0 + col + i]);
      }
    }
    // Four rows at a time in a rolled loop: fully unrolled, fetching the code took longer than the work (15000 cycles for a tile
    // of 128 x 128); one row at a time, the tests of the epilogue's options did (6000).
    constexpr int U = 4;
#pragma unroll 1
    for (int i = 0; i < items; i += U) {
      float v[U][4];
      bool valid[U];
      size_t row[U];
      int at_op[U];
      const float* mine[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int in_rows = e / LPR + (i + u) * (kEpiThreads / LPR), in_tile = rank * (BM / slices) + in_rows;
        row[u] = static_cast<size_t>(m0 + in_tile);
        at_op[u] = in_rows * BN + col;
        valid[u] = i + u < items && m0 + in_tile < p.M && left > 0;
        mine[u] = part + (i + u < items ? in_tile : 0) * C::kPitch + col;
      }
      if (slices == 1) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float4 t = *reinterpret_cast<const float4*>(mine[u]);
          v[u][0] = t.x; v[u][1] = t.y; v[u][2] = t.z; v[u][3] = t.w;
        }
      } else if (slices == 2) {
        sum_slices<2, U>(mine, v);
      } else if (slices == 4) {
        sum_slices<4, U>(mine, v);
      } else {
        sum_slices<8, C::kItems / 8>(mine, v);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[u][j] = v[u][j] * p.alpha + bias[j];
      if (p.preact_out != nullptr) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (valid[u]) store4(p.preact_out, row[u] * p.ldpre + n0 + col, v[u], left);
      }
      if (p.act == kActGelu) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int j = 0; j < 4; ++j) v[u][j] = gelu_tanh(v[u][j]);
      } else if (p.act == kActRelu) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int j = 0; j < 4; ++j) v[u][j] = fmaxf(v[u][j], 0.f);
      } else if (derivative) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!valid[u]) continue;
          float x[4];
          unpack4(p.residual == nullptr ? *reinterpret_cast<const uint2*>(s_op + at_op[u] * 2)
                                        : load4(p.aux, row[u] * p.ldaux + n0 + col, left), x);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[u][j] = p.act == kActDGelu ? v[u][j] * gelu_tanh_grad(x[j]) : (x[j] > 0.f ? v[u][j] : 0.f);
        }
      }
      if (p.dropout_p > 0.f) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint64_t g = (static_cast<uint64_t>(row[u]) * static_cast<uint64_t>(p.N) + n0 + col) >> 2;
          const uint32_t m = dropout_keep4(p.dropout_seed, g, keep16);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[u][j] = ((m >> j) & 1u) ? v[u][j] * drop_scale : 0.f;
        }
      }
      if (p.residual != nullptr) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!valid[u]) continue;
          float x[4];
          unpack4(*reinterpret_cast<const uint2*>(s_op + at_op[u] * 2), x);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[u][j] += x[j];
        }
      }
      if (p.accumulate) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!valid[u]) continue;
          float x[4];
          if (p.out_fp32) {
            const float4 t = *reinterpret_cast<const float4*>(s_old + at_op[u] * 4);
            x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
          } else {
            unpack4(*reinterpret_cast<const uint2*>(s_old + at_op[u] * 2), x);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) v[u][j] += x[j];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!valid[u]) continue;
        const size_t at = row[u] * p.ldd + n0 + col;
        if (!p.out_fp32) {
          store4(p.D, at, v[u], left);
        } else {
          float* d = reinterpret_cast<float*>(p.D) + at;
          if (left >= 4) {
            *reinterpret_cast<float4*>(d) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (j < left) d[j] = v[u][j];
          }
        }
      }
    }
  }
  __syncwarp();
  if (slices > 1) cluster_barrier();  // no CTA leaves while others read its partial tile
  else __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && p.status != nullptr) atomicMax(p.status, static_cast<int>(kStatusMbarTimeout));
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, BN);
  }
}

template <int BN, bool A_MN, bool B_MN>
int launch(const void* A, int lda, const void* B, int ldb, const GemmParams& p, int slices, cudaStream_t stream) {
  using C = Cfg<BN>;
  CUtensorMap ta, tb;
  int rc = A_MN ? make_tma_2d_bf16(&ta, A, p.K, p.M, lda, BK, 64) : make_tma_2d_bf16(&ta, A, p.M, p.K, lda, BM, BK);
  if (rc == 0) rc = B_MN ? make_tma_2d_bf16(&tb, B, p.K, p.N, ldb, BK, 64) : make_tma_2d_bf16(&tb, B, p.N, p.K, ldb, BN, BK);
  if (rc != 0) return rc;
  auto kernel = gemm_cluster_kernel<BN, A_MN, B_MN>;
  rc = static_cast<int>(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
  if (rc != 0) return rc;
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * slices);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = slices;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = slices > 1 ? 1 : 0;
  rc = static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, ta, tb, p, slices));
  return rc != 0 ? rc : static_cast<int>(cudaGetLastError());
}

}  // namespace

// Tile width and slices for an output, or slices = 0 where the kernel with one thread per output row is the better one.
//
// That kernel takes 220 ns a K block and its epilogue goes by chunks of 32 columns: 470 ns each for a plain bf16 result, more with
// operands, a column of a chunk that is not whole 60; with a single warp of rows 0.6 of it.  Here the chain is shorter by the
// slices and the epilogue does not grow with the columns, but the whole starts 2000 ns later (the partial tile, the operands),
// and the meeting costs 500 to 1700.  So outputs of few columns and short reductions stay there: 2048 x 8 x 200 5.4 us, here 6.4;
// 64 x 4096 x 512 plain 7.1, here 8.4; 1000 x 32 x 64 with GeLU and pre-activation 5.5, here 6.4.  Reductions that are long and not
// split are fed by four stages instead of six, 64 ns a K block beyond the 32nd: 512 x 4096 x 16384 with GeLU 68.7, here 89.9.
// Over 8447 calls (2 to 8192 in each size, nine epilogues) 29 are slower by more than 3 % than with that kernel alone; with a rule
// that only asked for few tiles 534 were.
void gemm_cluster_plan(const GemmParams& p, int num_sms, int* bn_out, int* slices_out) {
  const int M = p.M, N = p.N, num_m = (M + BM - 1) / BM, num_kb = (p.K + BK - 1) / BK;
  *slices_out = 0;
  *bn_out = 128;
  if (static_cast<long long>(num_m) * ((N + 127) / 128) > num_sms) return;
  int best = 0, bn = 128, slices = 0;
  for (int width = 64; width <= 128; width += 64) {
    const long long tiles = static_cast<long long>(num_m) * ((N + width - 1) / width);
    for (int s = 1; s <= kMaxCluster; s *= 2) {
      const int per = (num_kb + s - 1) / s;
      // clusters of four and more do not fill every last SM of a GPC
      if (tiles * s > (s == 8 ? num_sms * 2 / 3 : s == 4 ? num_sms * 7 / 8 : num_sms) || (s > 1 && (per < 2 || (s - 1) * per >= num_kb))) continue;
      // cycles: the operands of a K block (an SM receives 70 to 80 bytes a clock: 24 KB 345, 32 KB 462), the meeting over
      // distributed shared memory, the epilogue
      const int cost = per * (width == 64 ? 345 : 462) + (s > 1 ? 800 : 0) + 2400 * width / 128 / s;
      if (slices == 0 || cost < best) {
        best = cost;
        bn = width;
        slices = s;
      }
    }
  }
  if (slices == 0) return;
  const bool row_operand = p.residual != nullptr || p.aux != nullptr;
  // nothing to gain but the epilogue, and that one is simple
  if (slices == 1 && !p.out_fp32 && !p.accumulate && p.preact_out == nullptr && !row_operand && p.dropout_p == 0.f) return;
  const int chunk = 470 + (p.bias != nullptr ? 300 : 0) + (p.preact_out != nullptr ? 230 : 0) + (row_operand ? 540 : 0) +
                    (p.out_fp32 ? 250 : 0) + (p.accumulate ? (p.out_fp32 ? 1350 : 900) : 0);
  int epilogue = chunk * (((N < 128 ? N : 128) + 31) / 32) + (N < 128 ? 60 * (N % 32) : 0);
  if (M <= 32) epilogue = epilogue * 6 / 10;
  const int per = (num_kb + slices - 1) / slices;
  int late = 2000;
  if (slices == 1) late += num_kb > 32 ? 64 * (num_kb - 32) : 0;
  else if (bn == 64) late += slices == 2 ? 500 : 1100;
  else late += slices == 4 ? 1700 : 1000;
  if (epilogue + 220 * (num_kb - per) + (bn == 64 ? 40 * per : 0) <= late) return;
  *bn_out = bn;
  *slices_out = slices;
}

int gemm_cluster_launch(const void* A, int lda, int a_mn, const void* B, int ldb, int b_mn, const GemmParams& p, int bn, int slices,
                        cudaStream_t stream) {
#define SSB_GEMM(BN)                                                                                                        \
  (a_mn ? (b_mn ? launch<BN, true, true>(A, lda, B, ldb, p, slices, stream) : launch<BN, true, false>(A, lda, B, ldb, p, slices, stream)) \
        : (b_mn ? launch<BN, false, true>(A, lda, B, ldb, p, slices, stream) : launch<BN, false, false>(A, lda, B, ldb, p, slices, stream)))
  return bn == 64 ? SSB_GEMM(64) : SSB_GEMM(128);
#undef SSB_GEMM
}

}  // namespace ssb
