// LayerNorm forward / backward for bf16 activations with fp32 statistics, one to eight warps per row.
// Covers the role of the reference's mixed-precision fused LayerNorm extension
// (runtime/megatron/fused_kernels/layer_norm_cuda_kernel.cu:290-334 forward,
// :415-651 backward): y = (x - mean) * rstd * gamma + beta, saving mean and rstd;
// backward produces dx and per-column partial sums for dgamma / dbeta that a
// second small kernel folds (deterministic, no atomics).
//
// HBM-bound.  The one-pass backward streams rows through a ring of shared-memory stages filled by bulk asynchronous
// copies, so that the bytes in flight (about 100 KB per SM) do not depend on how many registers a warp can spare; the
// other kernels move 16 bytes per lane per access.
#include "common.cuh"

namespace ssb {

constexpr int kColsumTickets = 4096;   // column blocks of 256 that one column-sum call may cover in one pass
int colsum_tickets() { return kColsumTickets; }
namespace {

constexpr int kLnWarpsPerBlock = 4;

// Rows with a residual, and rows of 513 to 768 and of more than 2048 columns, that fit in the registers of a warp, read once: up to VPL
// vectors of 8 bf16 per lane; FULL = false: the last one, or for VPL > 8 the last few, are not there for every lane.  Values are
// kept as fp32 up to VPL 8, packed beyond that.  Lengths that are not 512, 1024, 2048 or 4096 used to take the kernel for any
// length: 512 rows of 704 4.1 -> 2.8 us.  What bounds it is the latency of the loads with few warps an SM (125 registers for
// 2048 columns: 15 warps).  Two rows at a time leave too few of them; fp32 arithmetic two values per instruction is slower, too.
template <int VPL, bool FULL>
__global__ void __launch_bounds__(kLnWarpsPerBlock * 32)
ln_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
              const float* __restrict__ gamma, const float* __restrict__ beta, __nv_bfloat16* __restrict__ y,
              __nv_bfloat16* __restrict__ sum_out, float* __restrict__ mean_out, float* __restrict__ rstd_out,
              int rows, int H, float eps) {
  const int lane = threadIdx.x & 31;
  const int warp_global = blockIdx.x * kLnWarpsPerBlock + (threadIdx.x >> 5);
  const int warps_total = gridDim.x * kLnWarpsPerBlock;
  const int nvec = H / 8;
  const bool last = (VPL - 1) * 32 + lane < nvec;
  auto mine = [&](int i) { return FULL || (VPL > 8 ? i * 32 + lane < nvec : i < VPL - 1 || last); };
  auto unpack = [](const uint4& q, float2 (&f)[4]) {
    f[0] = unpack_bf16x2(q.x); f[1] = unpack_bf16x2(q.y); f[2] = unpack_bf16x2(q.z); f[3] = unpack_bf16x2(q.w);
  };
  for (int row = warp_global; row < rows; row += warps_total) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * H);
    const uint4* rr = residual ? reinterpret_cast<const uint4*>(residual + static_cast<size_t>(row) * H) : nullptr;
    uint4* sr = sum_out ? reinterpret_cast<uint4*>(sum_out + static_cast<size_t>(row) * H) : nullptr;
    constexpr bool kPacked = VPL > 8;
    float2 f[kPacked ? 1 : VPL][4];
    uint4 q[kPacked ? VPL : 1];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      uint4 x0 = mine(i) ? xr[i * 32 + lane] : make_uint4(0u, 0u, 0u, 0u);
      float2(&v)[4] = f[kPacked ? 0 : i];
      unpack(x0, v);
      if (rr != nullptr && mine(i)) {
        float2 g[4];
        unpack(rr[i * 32 + lane], g);
        uint4 o;
        uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          w[j] = pack_bf16x2(v[j].x + g[j].x, v[j].y + g[j].y);
        }
        if (sr) sr[i * 32 + lane] = o;
        unpack(o, v);  // statistics are taken on the rounded sum so that forward and backward see the same x
        x0 = o;
      }
      if constexpr (kPacked) q[i] = x0;
#pragma unroll
      for (int j = 0; j < 4; ++j) s += v[j].x + v[j].y;
    }
    const float mean = warp_sum(s) / static_cast<float>(H);
    s = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (!mine(i)) continue;
      float2(&v)[4] = f[kPacked ? 0 : i];
      if constexpr (kPacked) unpack(q[i], v);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j].x -= mean;
        v[j].y -= mean;
        s += v[j].x * v[j].x + v[j].y * v[j].y;
      }
    }
    const float rstd = rsqrtf(warp_sum(s) / static_cast<float>(H) + eps);
    if (lane == 0) {
      mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
    uint4* yr = reinterpret_cast<uint4*>(y + static_cast<size_t>(row) * H);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = i * 32 + lane;
      if (!mine(i)) continue;
      const float4 g0 = reinterpret_cast<const float4*>(gamma)[2 * v], g1 = reinterpret_cast<const float4*>(gamma)[2 * v + 1];
      const float4 b0 = reinterpret_cast<const float4*>(beta)[2 * v], b1 = reinterpret_cast<const float4*>(beta)[2 * v + 1];
      const float2 g[4] = {make_float2(g0.x, g0.y), make_float2(g0.z, g0.w), make_float2(g1.x, g1.y), make_float2(g1.z, g1.w)};
      const float2 b[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w), make_float2(b1.x, b1.y), make_float2(b1.z, b1.w)};
      float2(&d)[4] = f[kPacked ? 0 : i];
      if constexpr (kPacked) {
        unpack(q[i], d);
#pragma unroll
        for (int j = 0; j < 4; ++j) d[j] = make_float2(d[j].x - mean, d[j].y - mean);
      }
      uint4 o;
      uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        w[j] = pack_bf16x2(d[j].x * rstd * g[j].x + b[j].x, d[j].y * rstd * g[j].y + b[j].y);
      }
      yr[v] = o;
    }
  }
}

// Rows without a residual of up to 512 and of 769 to 2048 columns are taken by two kernels, few of them by ln_fwd_parts_kernel, many by
// ln_fwd_group_kernel.  A row has the same bits in either, so its result does not depend on how many there are: vector 32 j + lane
// belongs to part j % parts of the row; a part has its sum and the sum of its squares about (nearly) its own mean, which are brought
// together about the row's.  The pieces, with every rounding spelled out:
__device__ __forceinline__ float ln_add8(float sum, const float (&v)[8]) {
  return sum + (((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
}
__device__ __forceinline__ float ln_add_squares8(float sum, const float (&v)[8], float m) {
  float u = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) u = fmaf(v[j] - m, v[j] - m, u);
  return sum + u;
}
__device__ __forceinline__ float ln_part_mean(float sum, float inv_columns) { return __fmul_rn(sum, inv_columns); }
// Squares about the row's mean from those about m, the value of ln_part_mean: sum (v - mean)^2 = squares + 2 (m - mean) sum (v - m) +
// columns (m - mean)^2.  The middle term is what the rounding of m leaves; with it a row of parts is as exact as one summed whole
// (rows of 1000 columns about 300, 1 / std: 5.8e-8 whole, 1.5e-7 without it, 4.3e-8 with it).
__device__ __forceinline__ float ln_part_squares(float sum, float squares, float columns, float inv_columns, float mean) {
  const float m = ln_part_mean(sum, inv_columns), d = m - mean, rest = fmaf(-m, columns, sum);
  return fmaf(d, fmaf(columns, d, rest + rest), squares);
}
// a / n for n > 0 and inv near 1 / n: the product, and once its residual (Newton's method), which is left out of infinities.  The
// products alone put the means of rows that are no power of two off by half as much again as a division does.
__device__ __forceinline__ float ln_quotient(float a, float n, float inv) {
  const float q = __fmul_rn(a, inv), rest = fmaf(-q, n, a);
  return rest - rest == 0.f ? fmaf(rest, inv, q) : q;
}
__device__ __forceinline__ uint4 ln_values8(const float (&v)[8], float mean, float rstd, const float (&g)[8], const float (&b)[8]) {
  float o[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = fmaf((v[j] - mean) * rstd, g[j], b[j]);
  return pack8(o);
}

// A warp per row, up to VPL vectors per lane.  FULL, WIDE: every lane has all of them, gamma and beta start on 16 bytes.  HOLD: gamma and
// beta are fetched in front of the row, where all rows are on the chip at once anyway; otherwise where they are used.
template <int VPL, bool FULL, bool WIDE, bool HOLD>
__global__ void __launch_bounds__(kLnWarpsPerBlock * 32)
ln_fwd_parts_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                    __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int H,
                    float eps) {
  constexpr int kParts = (VPL + 1) / 2;
  const int lane = threadIdx.x & 31, nvec = H / 8;
  auto mine = [&](int i) { return FULL || i < VPL - 1 || i * 32 + lane < nvec; };
  const float h = static_cast<float>(H), inv_h = 1.0f / h;
  float columns[kParts], inv_columns[kParts];
#pragma unroll
  for (int p = 0; p < kParts; ++p) {
    int n = 0;
#pragma unroll
    for (int i = p; i < VPL; i += kParts) n += FULL || i < VPL - 1 ? 256 : 8 * min(32, nvec - i * 32);
    columns[p] = static_cast<float>(n);
    inv_columns[p] = 1.0f / columns[p];
  }
  auto parameters = [&](const float* from, int i, float (&v)[8]) {
    const int at = i * 32 + lane;
    if constexpr (WIDE) {
      const float4 a = reinterpret_cast<const float4*>(from)[2 * at], c = reinterpret_cast<const float4*>(from)[2 * at + 1];
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = from[8 * at + j];
    }
  };
  float g[HOLD ? VPL : 1][8], b[HOLD ? VPL : 1][8];
  if constexpr (HOLD) {
#pragma unroll
    for (int i = 0; i < VPL; ++i)
      if (mine(i)) {
        parameters(gamma, i, g[i]);
        parameters(beta, i, b[i]);
      }
  }
  for (int row = blockIdx.x * kLnWarpsPerBlock + (threadIdx.x >> 5); row < rows; row += gridDim.x * kLnWarpsPerBlock) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * H);
    float f[VPL][8], m[kParts] = {}, s2[kParts] = {};  // m: sums
#pragma unroll
    for (int i = 0; i < VPL; ++i) unpack8(mine(i) ? xr[i * 32 + lane] : make_uint4(0u, 0u, 0u, 0u), f[i]);
#pragma unroll
    for (int i = 0; i < VPL; ++i) m[i % kParts] = ln_add8(m[i % kParts], f[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int p = 0; p < kParts; ++p) m[p] += __shfl_xor_sync(0xffffffffu, m[p], o);
    float mean = kParts == 1 ? ln_quotient(m[0], h, inv_h) : 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int p = i % kParts;
      if (mine(i)) s2[p] = ln_add_squares8(s2[p], f[i], kParts == 1 ? mean : ln_part_mean(m[p], inv_columns[p]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int p = 0; p < kParts; ++p) s2[p] += __shfl_xor_sync(0xffffffffu, s2[p], o);
    float squares = s2[0];
    if constexpr (kParts > 1) {
      squares = 0.f;
#pragma unroll
      for (int p = 0; p < kParts; ++p) mean += m[p];
      mean = ln_quotient(mean, h, inv_h);
#pragma unroll
      for (int p = 0; p < kParts; ++p) squares += ln_part_squares(m[p], s2[p], columns[p], inv_columns[p], mean);
    }
    const float rstd = rsqrtf(ln_quotient(squares, h, inv_h) + eps);
    if (lane == 0) {
      mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
    uint4* yr = reinterpret_cast<uint4*>(y + static_cast<size_t>(row) * H);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (!mine(i)) continue;
      if constexpr (!HOLD) {
        parameters(gamma, i, g[0]);
        parameters(beta, i, b[0]);
      }
      yr[i * 32 + lane] = ln_values8(f[i], mean, rstd, g[HOLD ? i : 0], b[HOLD ? i : 0]);
    }
  }
}

// Many rows of up to 2048: WPR warps share a row and take R rows at a time, the next R on their way meanwhile.  gamma and beta stay in
// registers; a warp per row read them from the L1 for every row, and its loads, sums and stores came one after the other
// (warps an SM and loads in flight were what bounded it: DRAM 47 %, issue slots 35 %).  The warps of a row exchange their sums and sums
// of squares once per R rows.  Three rows: with four the unpacked values spill (32768 x 2048 57 us), two have less in flight (50.4).
// What is done once per row is done by a lane per row, not by every lane for all of them (issue slots 74 -> 64 % busy, DRAM 50 -> 61 %;
// 47.6 -> 45.2 us, x 1800 46.0 -> 43.3, x 512 12.3 -> 12.0).  Measured, a warp per row -> this: 32768 x 2048 55.7 -> 45.2 us, x 1536 49.1 -> 36.5, 4096 x 2048
// 11.6 -> 8.7; a copy takes 42.0, 32.4, 7.3.  32768 x 1024 28.4 -> 24.6, x 896 27.6 -> 23.5, x 1280 36.8 -> 33.6, 8192 x 1024 10.2 -> 9.2.
// Rows of 513 to 768 columns stay with a warp each (x 640 20.0 -> 20.7, x 768 22.3 -> 22.0: the second warp is idle in part), and so do 4096 x
// 1024 (6.3 -> 6.6: the last groups have none).
template <int WPR>
struct LnGroup {
  static constexpr int kRows = 3, kGroups = WPR == 1 ? 4 : 1, kThreads = 32 * WPR * kGroups, kBlocks = 512 / kThreads;  // per SM
};
bool ln_fwd_in_parts(int H) { return H > 0 && (H <= 512 || (H > 768 && H <= 2048)); }
bool ln_fwd_grouped(int rows, int H, int num_sms) {  // every group has all of its rows at least once, of 769 to 1280 columns twice
  const int groups = num_sms * (H <= 512 ? LnGroup<1>::kBlocks * 4 : H <= 1024 ? LnGroup<2>::kBlocks : H <= 1536 ? LnGroup<3>::kBlocks : LnGroup<4>::kBlocks);
  return rows >= groups * 3 * (H > 768 && H <= 1280 ? 2 : 1);
}
template <int WPR>
__global__ void __launch_bounds__(LnGroup<WPR>::kThreads, LnGroup<WPR>::kBlocks)
ln_fwd_group_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                    __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int H,
                    float eps) {
  constexpr int VPL = 2, G = LnGroup<WPR>::kGroups, R = LnGroup<WPR>::kRows;
  __shared__ float2 xch[2][G][WPR][R];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slot = warp / WPR, part = warp % WPR;
  const int nvec = H / 8;
  float g[VPL][8], b[VPL][8];
  bool mine[VPL];
  int at[VPL], count = 0;  // this lane's vectors; columns of this warp
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    at[i] = (i * WPR + part) * 32 + lane;
    mine[i] = at[i] < nvec;
    count += 8 * max(0, min(32, nvec - (i * WPR + part) * 32));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      g[i][j] = mine[i] ? __ldg(gamma + at[i] * 8 + j) : 0.f;  // once: any alignment
      b[i][j] = mine[i] ? __ldg(beta + at[i] * 8 + j) : 0.f;
    }
  }
  const float n = static_cast<float>(count), inv_n = 1.0f / n, h = static_cast<float>(H), inv_h = 1.0f / h;
  __shared__ float2 columns[WPR];  // of every warp of a row, and their reciprocal
  if (WPR > 1 && lane == 0) columns[part] = make_float2(n, inv_n);
  if (WPR > 1) __syncthreads();
  uint4 next[R][VPL];
  auto fetch = [&](int row0) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int i = 0; i < VPL; ++i)
        if (mine[i] && row0 + r < rows) next[r][i] = __ldg(reinterpret_cast<const uint4*>(x + static_cast<size_t>(row0 + r) * H) + at[i]);
  };
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < VPL; ++i) next[r][i] = make_uint4(0u, 0u, 0u, 0u);
  const int step = gridDim.x * G * R;
  int row0 = (blockIdx.x * G + slot) * R, turn = 0;
  fetch(row0);
  for (; row0 < rows; row0 += step, turn ^= 1) {
    uint4 q[R][VPL];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int i = 0; i < VPL; ++i) q[r][i] = next[r][i];
    fetch(row0 + step);
    // The rows stay packed: each of the three uses unpacks them again (kept as fp32 they would not fit and be spilled).
    auto packed = [&]() {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < VPL; ++i) asm volatile("" : "+r"(q[r][i].x), "+r"(q[r][i].y), "+r"(q[r][i].z), "+r"(q[r][i].w));
    };
    float m[R], s2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float t = 0.f;
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        float v[8];
        unpack8(q[r][i], v);
        t = ln_add8(t, v);
      }
      m[r] = t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) m[r] += __shfl_xor_sync(0xffffffffu, m[r], o);
    packed();
    // What is done per row is done by the lane of its number, for all R at once.
    auto of_lane = [&](const float (&v)[R]) { return lane == 1 ? v[1] : lane == 2 ? v[2] : v[0]; };
    auto to_all = [&](float v, float (&all)[R]) {
#pragma unroll
      for (int r = 0; r < R; ++r) all[r] = __shfl_sync(0xffffffffu, v, r);
    };
    static_assert(R == 3, "rows at a time");
    float centre[R], rs[R], mean;
    if constexpr (WPR == 1) {
      mean = ln_quotient(of_lane(m), h, inv_h);
      to_all(mean, centre);
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) centre[r] = ln_part_mean(m[r], inv_n);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float t = 0.f;
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        float v[8];
        unpack8(q[r][i], v);
        const float with = ln_add_squares8(t, v, centre[r]);
        if (mine[i]) t = with;
      }
      s2[r] = t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) s2[r] += __shfl_xor_sync(0xffffffffu, s2[r], o);
    packed();
    float squares;
    if constexpr (WPR == 1) {
      squares = of_lane(s2);
    } else {
      float2(&slots)[WPR][R] = xch[turn][slot];
      if (lane == 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) slots[part][r] = make_float2(m[r], s2[r]);
      }
      __syncthreads();  // (one row slot per block: all warps have the same rows)
      const int r = lane < R ? lane : 0;
      mean = squares = 0.f;
#pragma unroll
      for (int w = 0; w < WPR; ++w) mean += slots[w][r].x;
      mean = ln_quotient(mean, h, inv_h);
#pragma unroll
      for (int w = 0; w < WPR; ++w) squares += ln_part_squares(slots[w][r].x, slots[w][r].y, columns[w].x, columns[w].y, mean);
      to_all(mean, centre);
    }
    const float rstd = rsqrtf(ln_quotient(squares, h, inv_h) + eps);
    to_all(rstd, rs);
    if (part == 0 && lane < R && row0 + lane < rows) {
      mean_out[row0 + lane] = mean;
      rstd_out[row0 + lane] = rstd;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = row0 + r;
      if (row >= rows) break;
      uint4* yr = reinterpret_cast<uint4*>(y + static_cast<size_t>(row) * H);
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        if (!mine[i]) continue;
        float v[8];
        unpack8(q[r][i], v);
        yr[at[i]] = ln_values8(v, centre[r], rs[r], g[i], b[i]);
      }
    }
  }
}

// Any row length that is a multiple of 8, parameters at any address: the row is read three times.
__global__ void __launch_bounds__(kLnWarpsPerBlock * 32)
ln_fwd_long_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                   const float* __restrict__ gamma, const float* __restrict__ beta, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ sum_out, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                   int rows, int H, float eps) {
  const int lane = threadIdx.x & 31;
  const int warp_global = blockIdx.x * kLnWarpsPerBlock + (threadIdx.x >> 5);
  const int warps_total = gridDim.x * kLnWarpsPerBlock;
  const int nvec = H / 8;
  for (int row = warp_global; row < rows; row += warps_total) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * H);
    const uint4* rr = residual ? reinterpret_cast<const uint4*>(residual + static_cast<size_t>(row) * H) : nullptr;
    uint4* sr = sum_out ? reinterpret_cast<uint4*>(sum_out + static_cast<size_t>(row) * H) : nullptr;
    float s = 0.f;
    for (int v = lane; v < nvec; v += 32) {
      uint4 q = xr[v];
      float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z), f3 = unpack_bf16x2(q.w);
      float e[8] = {f0.x, f0.y, f1.x, f1.y, f2.x, f2.y, f3.x, f3.y};
      if (rr) {
        uint4 r = rr[v];
        float2 g0 = unpack_bf16x2(r.x), g1 = unpack_bf16x2(r.y), g2 = unpack_bf16x2(r.z), g3 = unpack_bf16x2(r.w);
        e[0] += g0.x; e[1] += g0.y; e[2] += g1.x; e[3] += g1.y; e[4] += g2.x; e[5] += g2.y; e[6] += g3.x; e[7] += g3.y;
        uint4 o;
        o.x = pack_bf16x2(e[0], e[1]); o.y = pack_bf16x2(e[2], e[3]);
        o.z = pack_bf16x2(e[4], e[5]); o.w = pack_bf16x2(e[6], e[7]);
        if (sr) sr[v] = o;
        float2 h0 = unpack_bf16x2(o.x), h1 = unpack_bf16x2(o.y), h2 = unpack_bf16x2(o.z), h3 = unpack_bf16x2(o.w);
        e[0] = h0.x; e[1] = h0.y; e[2] = h1.x; e[3] = h1.y; e[4] = h2.x; e[5] = h2.y; e[6] = h3.x; e[7] = h3.y;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s += e[j];
    }
    const float mean = warp_sum(s) / static_cast<float>(H);
    float sq = 0.f;
    // reads the (just written) sum back; make the stores visible to the warp
    const uint4* src = (rr && sr) ? reinterpret_cast<const uint4*>(sr) : xr;
    if (rr && sr) __syncwarp();
    for (int v = lane; v < nvec; v += 32) {
      uint4 q = src[v];
      float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z), f3 = unpack_bf16x2(q.w);
      float e[8] = {f0.x, f0.y, f1.x, f1.y, f2.x, f2.y, f3.x, f3.y};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = e[j] - mean;
        sq += d * d;
      }
    }
    const float var = warp_sum(sq) / static_cast<float>(H);
    const float rstd = rsqrtf(var + eps);
    if (lane == 0) {
      mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
    uint4* yr = reinterpret_cast<uint4*>(y + static_cast<size_t>(row) * H);
    for (int v = lane; v < nvec; v += 32) {
      uint4 q = src[v];
      float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z), f3 = unpack_bf16x2(q.w);
      float e[8] = {f0.x, f0.y, f1.x, f1.y, f2.x, f2.y, f3.x, f3.y};
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = (e[j] - mean) * rstd * gamma[v * 8 + j] + beta[v * 8 + j];
      uint4 w;
      w.x = pack_bf16x2(o[0], o[1]); w.y = pack_bf16x2(o[2], o[3]);
      w.z = pack_bf16x2(o[4], o[5]); w.w = pack_bf16x2(o[6], o[7]);
      yr[v] = w;
    }
  }
}

// dx = rstd * (dy*gamma - mean_H(dy*gamma) - xhat * mean_H(dy*gamma*xhat)) (+ dresidual)
__global__ void __launch_bounds__(kLnWarpsPerBlock * 32)
ln_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                 const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ rstd,
                 const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx, int rows, int H) {
  const int lane = threadIdx.x & 31;
  const int warp_global = blockIdx.x * kLnWarpsPerBlock + (threadIdx.x >> 5);
  const int warps_total = gridDim.x * kLnWarpsPerBlock;
  const int nvec = H / 8;
  for (int row = warp_global; row < rows; row += warps_total) {
    const uint4* dyr = reinterpret_cast<const uint4*>(dy + static_cast<size_t>(row) * H);
    const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * H);
    const float mu = mean[row], rs = rstd[row];
    float s1 = 0.f, s2 = 0.f;
    for (int v = lane; v < nvec; v += 32) {
      const uint4 qd = dyr[v], qx = xr[v];
      const float2 d0 = unpack_bf16x2(qd.x), d1 = unpack_bf16x2(qd.y), d2 = unpack_bf16x2(qd.z), d3 = unpack_bf16x2(qd.w);
      const float2 x0 = unpack_bf16x2(qx.x), x1 = unpack_bf16x2(qx.y), x2 = unpack_bf16x2(qx.z), x3 = unpack_bf16x2(qx.w);
      const float d[8] = {d0.x, d0.y, d1.x, d1.y, d2.x, d2.y, d3.x, d3.y};
      const float xv[8] = {x0.x, x0.y, x1.x, x1.y, x2.x, x2.y, x3.x, x3.y};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float dg = d[j] * gamma[v * 8 + j];
        s1 += dg;
        s2 += dg * (xv[j] - mu) * rs;
      }
    }
    s1 = warp_sum(s1) / static_cast<float>(H);
    s2 = warp_sum(s2) / static_cast<float>(H);
    uint4* dxr = reinterpret_cast<uint4*>(dx + static_cast<size_t>(row) * H);
    const uint4* drr = dres ? reinterpret_cast<const uint4*>(dres + static_cast<size_t>(row) * H) : nullptr;
    for (int v = lane; v < nvec; v += 32) {
      const uint4 qd = dyr[v], qx = xr[v];
      const float2 d0 = unpack_bf16x2(qd.x), d1 = unpack_bf16x2(qd.y), d2 = unpack_bf16x2(qd.z), d3 = unpack_bf16x2(qd.w);
      const float2 x0 = unpack_bf16x2(qx.x), x1 = unpack_bf16x2(qx.y), x2 = unpack_bf16x2(qx.z), x3 = unpack_bf16x2(qx.w);
      const float d[8] = {d0.x, d0.y, d1.x, d1.y, d2.x, d2.y, d3.x, d3.y};
      const float xv[8] = {x0.x, x0.y, x1.x, x1.y, x2.x, x2.y, x3.x, x3.y};
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = (xv[j] - mu) * rs;
        o[j] = rs * (d[j] * gamma[v * 8 + j] - s1 - xhat * s2);
      }
      if (drr) {
        const uint4 qr = drr[v];
        const float2 r0 = unpack_bf16x2(qr.x), r1 = unpack_bf16x2(qr.y), r2 = unpack_bf16x2(qr.z), r3 = unpack_bf16x2(qr.w);
        o[0] += r0.x; o[1] += r0.y; o[2] += r1.x; o[3] += r1.y; o[4] += r2.x; o[5] += r2.y; o[6] += r3.x; o[7] += r3.y;
      }
      uint4 w;
      w.x = pack_bf16x2(o[0], o[1]); w.y = pack_bf16x2(o[2], o[3]);
      w.z = pack_bf16x2(o[4], o[5]); w.w = pack_bf16x2(o[6], o[7]);
      dxr[v] = w;
    }
  }
}

constexpr int kLnStages = 3;

// Ring of stages filled by one thread; `chunk` c of this block sits in stage c % kLnStages.
struct LnRing {
  uint64_t* full;
  uint64_t* empty;
  volatile int* abort_flag;
  __device__ __forceinline__ bool wait_full(int c) const {
    return mbar_wait_one(&full[c % kLnStages], (c / kLnStages) & 1);
  }
  __device__ __forceinline__ bool wait_empty(int c) const {
    return mbar_wait_one(&empty[c % kLnStages], ((c / kLnStages) & 1) ^ 1);
  }
  __device__ __forceinline__ bool mbar_wait_one(uint64_t* bar, uint32_t parity) const {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
  }
  __device__ __forceinline__ void release(int c, int lane) const {  // one arrival per computing warp
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[c % kLnStages]);
  }
};

// One pass over dy, x and dres for any H <= 512 * WPR: dx, and in the same sweep every lane keeps running sums of
// dy * xhat and dy for its 16 columns over all rows its warp visits (their gamma stays in registers).  A chunk is
// NW / WPR consecutive rows of the three matrices; WPR warps share a row (each owns 512 columns) and exchange their two
// row sums through shared memory.  The warps of a block fold their column sums through shared memory in a fixed order
// and the block writes ONE row of partials (part_g[block][h], part_b[block][h]); fold_partials2_kernel adds the blocks.
// The result does not depend on the order of execution.  dy and x are kept packed over the warps' meeting and unpacked again behind it:
// fewer registers, less spilled.  What bounds it is the chain of a chunk (copies, sums, meeting, stores), two blocks an SM; more
// stages, more and smaller blocks, or two rows of a warp at a time are slower.  Three warps a row up to 1536 columns, where four
// were idle in part.  32768 rows with residual gradient, this kernel and the fold, before -> now: x 2048 100 -> 93 us, x 1536 87 -> 68,
// x 1152 82 -> 65, x 1024 55 -> 50, x 512 33 -> 29 (a copy of two such matrices: 84, 65, 50, 45, 24).
// NW warps compute, WPR of them on a row; one more issues the copies.  Two blocks an SM.
template <int WPR_, int NW_>
struct LnBwd {
  static constexpr int WPR = WPR_, NW = NW_, kRows = NW / WPR, kThreads = (NW + 1) * 32;  // kRows: of a chunk
  static constexpr bool kStatsAhead = WPR <= 3;
};
template <class Cfg>
__global__ void __launch_bounds__(Cfg::kThreads, 2)
ln_bwd_stream_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                     const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ rstd,
                     const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                     float* __restrict__ part_g, float* __restrict__ part_b, int rows, int H, int* __restrict__ status) {
  constexpr int WPR = Cfg::WPR, kLnWarps = Cfg::NW, RPB = Cfg::kRows;
  constexpr int VPL = 2;       // vectors per lane
  extern __shared__ __align__(128) uint8_t ring_smem[];
  __shared__ float2 xch[2][RPB][WPR];
  __shared__ uint64_t bars[2 * kLnStages];
  __shared__ int aborted;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row_bytes = H * 2, part_bytes = RPB * row_bytes, stage_bytes = 3 * part_bytes, nvec = H / 8;
  const int chunks = (rows + RPB - 1) / RPB;
  // From the last rows to the first: the kernel that wrote dy ended with them, so they are still in the L2 (32768 x 2048 behind the
  // forward, whose x it is there, 92.0 -> 89.4 us).
  auto place = [&](int ch) { return chunks - 1 - ch; };
  if (threadIdx.x == 0) {
    for (int i = 0; i < kLnStages; ++i) {
      mbar_init(&bars[i], 1);
      mbar_init(&bars[kLnStages + i], kLnWarps);
    }
    aborted = 0;
    fence_mbar_init();
  }
  __syncthreads();
  const LnRing ring{bars, bars + kLnStages, &aborted};
  float ag[VPL][8], ab[VPL][8];
  const int rslot = warp / WPR, part = warp % WPR;
  if (warp == kLnWarps) {
    int c = 0;
    for (int ch = blockIdx.x; ch < chunks; ch += gridDim.x, ++c) {
      if (!ring.wait_empty(c)) break;
      if (lane == 0) {
        const int st = c % kLnStages, bytes = min(RPB, rows - place(ch) * RPB) * row_bytes;
        const size_t at = static_cast<size_t>(place(ch)) * RPB * H;
        uint8_t* dst = ring_smem + st * stage_bytes;
        mbar_arrive_expect_tx(&bars[st], bytes * (dres ? 3 : 2));
        bulk_load(dst, dy + at, bytes, &bars[st]);
        bulk_load(dst + part_bytes, x + at, bytes, &bars[st]);
        if (dres) bulk_load(dst + 2 * part_bytes, dres + at, bytes, &bars[st]);
      }
      __syncwarp();
    }
    // The last copies land before the block may end, also where the computing warps have given up on them.
    if (lane == 0)
      for (int i = max(c - kLnStages, 0); i < c; ++i)
        for (uint32_t it = 0; it < (1u << 20); ++it)
          if (mbar_try_wait(&bars[i % kLnStages], (i / kLnStages) & 1)) break;
    __syncwarp();
  } else {
    const float inv_h = 1.0f / static_cast<float>(H);
    float g[VPL][8];
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = (part * VPL + i) * 32 + lane;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        g[i][j] = v < nvec ? __ldg(gamma + v * 8 + j) : 0.f;  // once: any alignment
        ag[i][j] = ab[i][j] = 0.f;
      }
    }
    // The warps of a row meet once per chunk.  One whose bounded wait ran out at chunk `ch` still comes to the meetings ahead: the
    // others may pass the same wait a moment later and must not be left waiting.
    auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + rslot), "r"(32 * WPR) : "memory"); };
    auto meet_to_the_end = [&](int ch) {
      if (WPR > 1)
        for (; ch < chunks; ch += gridDim.x)
          if (place(ch) * RPB + rslot < rows) meet();
    };
    int c = 0;
    // Statistics of the row: loaded a chunk ahead, like the row itself (32768 x 512 33.0 -> 29.8 us, x 1024 55.4 -> 53.4, x 1536 72.8 ->
    // 67.7; with four warps a row 93.0 -> 96.3).
    float mu_next = 0.f, rs_next = 0.f;
    auto fetch_stats = [&](int ch) {
      const int row = place(ch) * RPB + rslot;
      const bool have = ch < chunks && row < rows;
      mu_next = have ? __ldg(mean + row) : 0.f;
      rs_next = have ? __ldg(rstd + row) : 0.f;
    };
    if (Cfg::kStatsAhead) fetch_stats(blockIdx.x);
    for (int ch = blockIdx.x; ch < chunks; ch += gridDim.x, ++c) {
      const int row = place(ch) * RPB + rslot;              // the same for all warps of a row slot
      if (!Cfg::kStatsAhead) fetch_stats(ch);
      const float mu = mu_next, rs = rs_next;
      if (Cfg::kStatsAhead) fetch_stats(ch + gridDim.x);
      if (!ring.wait_full(c)) {
        meet_to_the_end(ch);
        break;
      }
      if (row < rows) {
        const uint8_t* base = ring_smem + (c % kLnStages) * stage_bytes + rslot * row_bytes;
        const uint4* pd = reinterpret_cast<const uint4*>(base);
        const uint4* px = reinterpret_cast<const uint4*>(base + part_bytes);
        const uint4* pr = reinterpret_cast<const uint4*>(base + 2 * part_bytes);
        uint4 qd[VPL], qx[VPL];
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
          const int v = (part * VPL + i) * 32 + lane;
          const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
          float d[8], xv[8];
          qd[i] = v < nvec ? pd[v] : zero;
          qx[i] = v < nvec ? px[v] : zero;
          unpack8(qd[i], d);
          unpack8(qx[i], xv);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xh = (xv[j] - mu) * rs, dg = d[j] * g[i][j];
            s1 += dg;
            s2 += dg * xh;
            ag[i][j] += d[j] * xh;
            ab[i][j] += d[j];
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          s1 += __shfl_xor_sync(0xffffffffu, s1, o);
          s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        }
        if constexpr (WPR > 1) {
          float2(&slot)[WPR] = xch[c & 1][rslot];
          if (lane == 0) slot[part] = make_float2(s1, s2);
          meet();
          s1 = s2 = 0.f;
#pragma unroll
          for (int w = 0; w < WPR; ++w) {
            const float2 e = slot[w];
            s1 += e.x;
            s2 += e.y;
          }
        }
        s1 *= inv_h;
        s2 *= inv_h;
        uint4* dxr = reinterpret_cast<uint4*>(dx) + static_cast<size_t>(row) * nvec;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
          const int v = (part * VPL + i) * 32 + lane;
          if (v >= nvec) break;
          float d[8], xv[8], o[8];
          unpack8(qd[i], d);
          unpack8(qx[i], xv);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xh = (xv[j] - mu) * rs;
            o[j] = rs * (d[j] * g[i][j] - s1 - xh * s2);
          }
          if (dres) {
            float t[8];
            unpack8(pr[v], t);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] += t[j];
          }
          dxr[v] = pack8(o);
        }
      }
      ring.release(c, lane);
    }
  }
  __syncthreads();
  // Every copy has landed and been read: the ring takes the sums of the row slots, [2][RPB][H], which are then added in the order
  // 0, 1, ...  (One slot after the other into one row of sums took eight rounds at one warp per row: 16 x 512 9.5 us instead of 5.5.)
  float* slots = reinterpret_cast<float*>(ring_smem);
  if (warp < kLnWarps) {
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int v = (part * VPL + i) * 32 + lane;
      if (v >= nvec) break;
      float4* pg = reinterpret_cast<float4*>(slots + rslot * H + v * 8);
      float4* pb = reinterpret_cast<float4*>(slots + (RPB + rslot) * H + v * 8);
      pg[0] = make_float4(ag[i][0], ag[i][1], ag[i][2], ag[i][3]);
      pg[1] = make_float4(ag[i][4], ag[i][5], ag[i][6], ag[i][7]);
      pb[0] = make_float4(ab[i][0], ab[i][1], ab[i][2], ab[i][3]);
      pb[1] = make_float4(ab[i][4], ab[i][5], ab[i][6], ab[i][7]);
    }
  }
  __syncthreads();
  for (int col = threadIdx.x; col < H; col += blockDim.x) {
    float g = slots[col], b = slots[RPB * H + col];
#pragma unroll
    for (int sl = 1; sl < RPB; ++sl) {
      g += slots[sl * H + col];
      b += slots[(RPB + sl) * H + col];
    }
    part_g[static_cast<size_t>(blockIdx.x) * H + col] = g;
    part_b[static_cast<size_t>(blockIdx.x) * H + col] = b;
  }
  if (threadIdx.x == 0 && aborted && status != nullptr) atomicMax(status, static_cast<int>(kStatusMbarTimeout));
}

// Partial column sums over a slice of rows: part_g[slice][h] = sum dy*xhat, part_b[slice][h] = sum dy.
// Block = 32 columns-pairs x 8 row lanes: thread (tx, ty) owns columns 2*(bx*32+tx), +1 and rows ty, ty+8, ...
__global__ void __launch_bounds__(256)
ln_bwd_gb_partial_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                         const float* __restrict__ mean, const float* __restrict__ rstd, float* __restrict__ part_g,
                         float* __restrict__ part_b, int rows, int H, int rows_per_slice) {
  __shared__ float sg[8][64], sb[8][64];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int col = (blockIdx.x * 32 + tx) * 2;
  const int r0 = blockIdx.y * rows_per_slice;
  const int r1 = min(rows, r0 + rows_per_slice);
  float g0 = 0.f, g1 = 0.f, b0 = 0.f, b1 = 0.f;
  if (col < H) {
    for (int r = r0 + ty; r < r1; r += 8) {
      const uint32_t qd = *reinterpret_cast<const uint32_t*>(dy + static_cast<size_t>(r) * H + col);
      const uint32_t qx = *reinterpret_cast<const uint32_t*>(x + static_cast<size_t>(r) * H + col);
      const float2 d = unpack_bf16x2(qd), xv = unpack_bf16x2(qx);
      const float mu = mean[r], rs = rstd[r];
      g0 += d.x * (xv.x - mu) * rs;
      g1 += d.y * (xv.y - mu) * rs;
      b0 += d.x;
      b1 += d.y;
    }
  }
  sg[ty][tx * 2] = g0; sg[ty][tx * 2 + 1] = g1;
  sb[ty][tx * 2] = b0; sb[ty][tx * 2 + 1] = b1;
  __syncthreads();
  if (ty == 0 && col < H) {
    float a0 = 0.f, a1 = 0.f, c0 = 0.f, c1 = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      a0 += sg[k][tx * 2]; a1 += sg[k][tx * 2 + 1];
      c0 += sb[k][tx * 2]; c1 += sb[k][tx * 2 + 1];
    }
    part_g[static_cast<size_t>(blockIdx.y) * H + col] = a0;
    part_g[static_cast<size_t>(blockIdx.y) * H + col + 1] = a1;
    part_b[static_cast<size_t>(blockIdx.y) * H + col] = c0;
    part_b[static_cast<size_t>(blockIdx.y) * H + col + 1] = c1;
  }
}

// out[h] (+)= sum_slices part[slice][h]
__global__ void fold_partials_kernel(const float* __restrict__ part, float* __restrict__ out, int slices, int H,
                                     int accumulate) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= H) return;
  float s = 0.f;
  for (int k = 0; k < slices; ++k) s += part[static_cast<size_t>(k) * H + h];
  out[h] = accumulate ? out[h] + s : s;
}

// Both LayerNorm weight gradients in one launch: block (x, which) folds 32 columns of part_g (which = 0) or part_b
// (which = 1); its threads are 32 columns x G groups of slices, added in a fixed order.  G 32 for the many partials of the
// one-pass kernel (with four groups a chain of 74 loads, 11 us for 296 slices), 4 for few (2 slices of 5120 columns: 1.9 us
// instead of 2.9).
template <int G>
__global__ void __launch_bounds__(32 * G)
fold_partials2_kernel(const float* __restrict__ part_g, const float* __restrict__ part_b, float* __restrict__ dgamma,
                      float* __restrict__ dbeta, int slices, int H, int accumulate) {
  __shared__ float sm[G][33];
  const float* part = blockIdx.y == 0 ? part_g : part_b;
  float* out = blockIdx.y == 0 ? dgamma : dbeta;
  const int c = threadIdx.x & 31, sg = threadIdx.x >> 5, h = blockIdx.x * 32 + c;
  float s = 0.f;
  if (h < H)
    for (int k = sg; k < slices; k += G) s += part[static_cast<size_t>(k) * H + h];
  sm[sg][c] = s;
  __syncthreads();
  static_assert(G == 4 || G == 32, "groups");
  if constexpr (G == 32) {  // warp w adds column w's groups by a butterfly: the same order every time
    const float t = warp_sum(sm[c][sg]);
    const int hw = blockIdx.x * 32 + sg;
    if (c == 0 && hw < H) out[hw] = accumulate ? out[hw] + t : t;
  } else if (sg == 0 && h < H) {
    const float t = (sm[0][c] + sm[1][c]) + (sm[2][c] + sm[3][c]);
    out[h] = accumulate ? out[h] + t : t;
  }
}

void fold_partials2(const float* part_g, const float* part_b, float* dgamma, float* dbeta, int slices, int H, int accumulate,
                    cudaStream_t stream) {
  const dim3 grid((H + 31) / 32, 2);
  if (slices > 64) fold_partials2_kernel<32><<<grid, 1024, 0, stream>>>(part_g, part_b, dgamma, dbeta, slices, H, accumulate);
  else fold_partials2_kernel<4><<<grid, 128, 0, stream>>>(part_g, part_b, dgamma, dbeta, slices, H, accumulate);
}

// Column sum of a bf16 matrix [rows, N] (bias gradients) in ONE launch, for 16-byte aligned rows (N, lda multiples
// of 8).  A warp covers 512 contiguous bytes of a row (eight columns per lane), the eight warps of a block take
// every eighth row of the block's slice, and the block writes one row of partials for its 256 columns.  The block
// that finishes LAST for a column block (a ticket counter per column block, which it sets back to zero) adds the
// partials of all slices, every warp an eighth of them and then the eight sums in order, so the result does not depend on which
// block that is.  The counters are shared by all calls on a device: calls must be ordered on one stream.
//
// As many slices as give every SM kColsumBlocks blocks, but no more than colsum_slices: with a slice per 256 rows and a thread that added
// the partials of a column one after the other, before -> now: 8192 x 8192 31.8 -> 23.9 us, 32768 x 6144 75.0 -> 61.3 (6.6 TB/s), 32768 x
// 2048 35.7 -> 25.6, 512 x 512 6.6 -> 4.1.  Short ones wait for loads, the partials and the ticket, one after the other; with the matrix
// still in the L2: 8192 x 2048 8.8 -> 8.1 in 64 slices (9.6 in 111), 4096 x 4096 8.0 -> 7.4 with four blocks an SM (8.4 with six),
// 8192 x 3072 9.2 -> 8.8 (9.7); from memory 32768 x 768 19.4 -> 15.6 in 128 slices (17.6 in 64).
constexpr int kColsumBlocks = 4, kColsumMaxSlices = 128;
__global__ void __launch_bounds__(256, 6)
colsum_onepass_kernel(const __nv_bfloat16* __restrict__ a, int lda, float* __restrict__ part, float* __restrict__ out,
                      int* __restrict__ tickets, int rows, int N, int rows_per_slice, int accumulate) {
  __shared__ __align__(16) float red[8][256];
  __shared__ int is_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = blockIdx.x * 256 + lane * 8;
  const int r0 = blockIdx.y * rows_per_slice;
  const int r1 = min(rows, r0 + rows_per_slice);
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = 0.f;
  auto add = [&](const uint4& q) {
    const float2 v0 = unpack_bf16x2(q.x), v1 = unpack_bf16x2(q.y), v2 = unpack_bf16x2(q.z), v3 = unpack_bf16x2(q.w);
    s[0] += v0.x; s[1] += v0.y; s[2] += v1.x; s[3] += v1.y; s[4] += v2.x; s[5] += v2.y; s[6] += v3.x; s[7] += v3.y;
  };
  // This warp's sums for 256 columns -> the block's, a column per thread (added in the order of the warps).
  auto block_sum = [&]() {
    *reinterpret_cast<float4*>(&red[warp][lane * 8]) = make_float4(s[0], s[1], s[2], s[3]);
    *reinterpret_cast<float4*>(&red[warp][lane * 8 + 4]) = make_float4(s[4], s[5], s[6], s[7]);
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += red[k][threadIdx.x];
    return t;
  };
  if (c0 < N) {
    int r = r0 + warp;
    for (; r + 24 < r1; r += 32) {                   // four independent rows in flight per thread
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = *reinterpret_cast<const uint4*>(a + static_cast<size_t>(r + 8 * u) * lda + c0);
#pragma unroll
      for (int u = 0; u < 4; ++u) add(q[u]);
    }
    for (; r < r1; r += 8) add(*reinterpret_cast<const uint4*>(a + static_cast<size_t>(r) * lda + c0));
  }
  const int col = blockIdx.x * 256 + threadIdx.x;
  float t = block_sum();
  if (gridDim.y > 1) {
    if (col < N) {
      part[static_cast<size_t>(blockIdx.y) * N + col] = t;
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(&tickets[blockIdx.x], 1) == static_cast<int>(gridDim.y) - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = 0.f;
    if (c0 < N) {
      const float* src = part + c0;
#pragma unroll 4
      for (int k = warp; k < static_cast<int>(gridDim.y); k += 8) {
        const float4 lo = __ldcg(reinterpret_cast<const float4*>(src + static_cast<size_t>(k) * N));
        const float4 hi = __ldcg(reinterpret_cast<const float4*>(src + static_cast<size_t>(k) * N + 4));
        s[0] += lo.x; s[1] += lo.y; s[2] += lo.z; s[3] += lo.w;
        s[4] += hi.x; s[5] += hi.y; s[6] += hi.z; s[7] += hi.w;
      }
    }
    t = block_sum();
    if (threadIdx.x == 0) tickets[blockIdx.x] = 0;
  }
  if (col < N) out[col] = accumulate ? out[col] + t : t;
}

// Column sum of a bf16 matrix [rows, N] into partials[slice][N] (bias gradients).
__global__ void __launch_bounds__(256)
colsum_partial_kernel(const __nv_bfloat16* __restrict__ a, int lda, float* __restrict__ part, int rows, int N,
                      int rows_per_slice) {
  __shared__ float sm[8][64];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int col = (blockIdx.x * 32 + tx) * 2;
  const int r0 = blockIdx.y * rows_per_slice;
  const int r1 = min(rows, r0 + rows_per_slice);
  float s0 = 0.f, s1 = 0.f;
  if (col < N) {
    for (int r = r0 + ty; r < r1; r += 8) {
      const float2 d = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(a + static_cast<size_t>(r) * lda + col));
      s0 += d.x;
      s1 += d.y;
    }
  }
  sm[ty][tx * 2] = s0;
  sm[ty][tx * 2 + 1] = s1;
  __syncthreads();
  if (ty == 0 && col < N) {
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      a0 += sm[k][tx * 2];
      a1 += sm[k][tx * 2 + 1];
    }
    part[static_cast<size_t>(blockIdx.y) * N + col] = a0;
    part[static_cast<size_t>(blockIdx.y) * N + col + 1] = a1;
  }
}

}  // namespace

constexpr int kLnStreamMaxH = 4096;

static bool misaligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }

int layernorm_fwd_launch(const void* x, const void* residual, const float* gamma, const float* beta, void* y,
                         void* sum_out, float* mean, float* rstd, int rows, int H, float eps, int num_sms,
                         cudaStream_t stream) {
  if (H % 8 || misaligned(x) || misaligned(residual) || misaligned(y) || misaligned(sum_out)) return -3;
  const int blocks = min((rows + kLnWarpsPerBlock - 1) / kLnWarpsPerBlock, num_sms * 16);
  const dim3 grid(blocks), block(kLnWarpsPerBlock * 32);
  const auto* xb = reinterpret_cast<const __nv_bfloat16*>(x);
  const auto* rb = reinterpret_cast<const __nv_bfloat16*>(residual);
  auto* yb = reinterpret_cast<__nv_bfloat16*>(y);
  auto* sb = reinterpret_cast<__nv_bfloat16*>(sum_out);
  const bool wide = !misaligned(gamma) && !misaligned(beta);  // 16-byte loads of both
  if (residual == nullptr && ln_fwd_in_parts(H)) {
    if (ln_fwd_grouped(rows, H, num_sms)) {
      auto launch = [&](auto kernel, auto cfg) {
        using Cfg = decltype(cfg);
        kernel<<<num_sms * Cfg::kBlocks, Cfg::kThreads, 0, stream>>>(xb, gamma, beta, yb, mean, rstd, rows, H, eps);
      };
      if (H <= 512) launch(ln_fwd_group_kernel<1>, LnGroup<1>{});
      else if (H <= 1024) launch(ln_fwd_group_kernel<2>, LnGroup<2>{});
      else if (H <= 1536) launch(ln_fwd_group_kernel<3>, LnGroup<3>{});
      else launch(ln_fwd_group_kernel<4>, LnGroup<4>{});
      return static_cast<int>(cudaGetLastError());
    }
    // HOLD takes three times the registers.  592 rows of 1024 2.86 -> 2.29 us, of 2048 3.48 -> 2.92, one row of 1536 3.14 -> 2.04; where
    // the rows then wait for one another it loses: 4096 of 1024 4.9 -> 5.8, 1700 of 1280 3.9 -> 4.05, of 2048 5.0 -> 6.4.
    const bool hold = rows <= num_sms * (H <= 1024 ? 16 : 4);
    auto launch = [&](auto full, auto any, auto any_hold, auto full_hold, auto off) {
      auto kernel = !wide ? off : H % 256 ? (hold ? any_hold : any) : hold ? full_hold : full;
      kernel<<<grid, block, 0, stream>>>(xb, gamma, beta, yb, mean, rstd, rows, H, eps);
    };
#define SSB_LN_CASE(V)                                                                                                       \
  case V:                                                                                                                    \
    launch(ln_fwd_parts_kernel<V, true, true, false>, ln_fwd_parts_kernel<V, false, true, false>,                            \
           ln_fwd_parts_kernel<V, false, true, true>, ln_fwd_parts_kernel<V, true, true, true>,                              \
           ln_fwd_parts_kernel<V, false, false, false>);                                                                     \
    break
    switch ((H + 255) / 256) {
      SSB_LN_CASE(1);
      SSB_LN_CASE(2);
      SSB_LN_CASE(4);
      SSB_LN_CASE(5);
      SSB_LN_CASE(6);
      SSB_LN_CASE(7);
      SSB_LN_CASE(8);
    }
#undef SSB_LN_CASE
    return static_cast<int>(cudaGetLastError());
  }
#define SSB_LN_ARGS <<<grid, block, 0, stream>>>(xb, rb, gamma, beta, yb, sb, mean, rstd, rows, H, eps)
#define SSB_LN_CASE(V)                                          \
  case V:                                                       \
    if (H == V * 256) ln_fwd_kernel<V, true> SSB_LN_ARGS;       \
    else ln_fwd_kernel<V, false> SSB_LN_ARGS;                   \
    break
  // parameters that start elsewhere take the kernel for any address
  switch (wide ? (H + 255) / 256 : 0) {
    SSB_LN_CASE(1);
    SSB_LN_CASE(2);
    SSB_LN_CASE(3);
    SSB_LN_CASE(4);
    SSB_LN_CASE(5);
    SSB_LN_CASE(6);
    SSB_LN_CASE(7);
    SSB_LN_CASE(8);
    case 9: case 10: case 11: case 12: ln_fwd_kernel<12, false> SSB_LN_ARGS; break;
    case 13: case 14: case 15: ln_fwd_kernel<16, false> SSB_LN_ARGS; break;
    SSB_LN_CASE(16);
    default: ln_fwd_long_kernel SSB_LN_ARGS; break;
  }
#undef SSB_LN_CASE
#undef SSB_LN_ARGS
  return static_cast<int>(cudaGetLastError());
}

// part_g / part_b: scratch of `slices` x H floats each (slices = ln_bwd_slices(rows)).
int ln_bwd_slices(int rows) {
  int s = (rows + 255) / 256;
  return s < 1 ? 1 : (s > 128 ? 128 : s);
}

// Calls fn with the form of the one-pass backward for rows of H.
template <class Fn>
static auto ln_bwd_form(int H, Fn fn) {
  if (H <= 512) return fn(LnBwd<1, 8>{});
  if (H <= 1024) return fn(LnBwd<2, 8>{});
  if (H <= 1536) return fn(LnBwd<3, 6>{});
  if (H <= 2048) return fn(LnBwd<4, 8>{});
  return fn(LnBwd<8, 8>{});
}

// Rows of partial sums the backward needs in each of part_g / part_b (then H floats per row).
int ln_bwd_part_rows(int rows, int H, int num_sms) {
  if (H <= kLnStreamMaxH)  // one-pass kernel: one row of partials per block
    return ln_bwd_form(H, [&](auto cfg) {
      using Cfg = decltype(cfg);
      const int want = (rows + Cfg::kRows - 1) / Cfg::kRows;
      return want < num_sms * 2 ? want : num_sms * 2;
    });
  return ln_bwd_slices(rows);
}

int layernorm_bwd_launch(const void* dy, const void* x, const float* gamma, const float* mean, const float* rstd,
                         const void* dres, void* dx, float* dgamma, float* dbeta, float* part_g, float* part_b,
                         int accumulate_wgrad, int rows, int H, int* status, int num_sms, cudaStream_t stream) {
  if (H % 8) return -3;
  const auto* dyb = reinterpret_cast<const __nv_bfloat16*>(dy);
  const auto* xb = reinterpret_cast<const __nv_bfloat16*>(x);
  const auto* drb = reinterpret_cast<const __nv_bfloat16*>(dres);
  auto* dxb = reinterpret_cast<__nv_bfloat16*>(dx);
  if (misaligned(dy) || misaligned(x) || misaligned(dres) || misaligned(dx)) return -3;  // every kernel moves 16 bytes a lane
  if (H <= kLnStreamMaxH) {
    // dy and x are read once: dx and the per-column sums come out of the same sweep
    const int nb = ln_bwd_part_rows(rows, H, num_sms);
    const int rc = ln_bwd_form(H, [&](auto cfg) {
      using Cfg = decltype(cfg);
      const int smem = kLnStages * 3 * Cfg::kRows * H * 2;
      const int e = static_cast<int>(cudaFuncSetAttribute(ln_bwd_stream_kernel<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      if (e == 0)
        ln_bwd_stream_kernel<Cfg><<<nb, Cfg::kThreads, smem, stream>>>(dyb, xb, gamma, mean, rstd, drb, dxb, part_g, part_b, rows, H, status);
      return e;
    });
    if (rc) return rc;
    fold_partials2(part_g, part_b, dgamma, dbeta, nb, H, accumulate_wgrad, stream);
    return static_cast<int>(cudaGetLastError());
  }
  const int blocks = min((rows + kLnWarpsPerBlock - 1) / kLnWarpsPerBlock, num_sms * 16);
  const dim3 g(blocks), b(kLnWarpsPerBlock * 32);
  ln_bwd_dx_kernel<<<g, b, 0, stream>>>(dyb, xb, gamma, mean, rstd, drb, dxb, rows, H);
  const int slices = ln_bwd_slices(rows);
  const int rps = (rows + slices - 1) / slices;
  dim3 grid((H / 2 + 31) / 32, slices);
  ln_bwd_gb_partial_kernel<<<grid, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(dy),
                                                     reinterpret_cast<const __nv_bfloat16*>(x), mean, rstd, part_g,
                                                     part_b, rows, H, rps);
  fold_partials2(part_g, part_b, dgamma, dbeta, slices, H, accumulate_wgrad, stream);
  return static_cast<int>(cudaGetLastError());
}

// Slices that the one-pass column sum takes at most: of 64 rows at least up to 64 of them, of 256 beyond.
static int colsum_slices(int rows) {
  const int few = (rows + 63) / 64, many = rows / 256;
  const int slices = few < 64 ? few : many > 64 ? many : 64;
  return slices < kColsumMaxSlices ? slices : kColsumMaxSlices;
}

// Rows of N partial sums that a call of colsum_launch needs as scratch, whichever of its kernels takes it.
int colsum_part_rows(int rows) {
  const int one_pass = colsum_slices(rows), two_pass = ln_bwd_slices(rows);
  return one_pass > two_pass ? one_pass : two_pass;
}

// out[N] (+)= column sums of a[rows, N]; `part` is scratch of colsum_part_rows(rows) x N floats, 16-byte aligned; `tickets` holds
// kColsumTickets zero-initialised counters that every call leaves at zero.
int colsum_launch(const void* a, int lda, float* out, float* part, int* tickets, int accumulate, int rows, int N, int num_sms,
                  cudaStream_t stream) {
  if (N % 2 || lda % 2) return -3;
  const int slices = ln_bwd_slices(rows);
  const int rps = (rows + slices - 1) / slices;
  const int colblocks = (N + 255) / 256;
  if (N % 8 == 0 && lda % 8 == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0 && colblocks <= kColsumTickets &&
      tickets != nullptr) {
    int sl = num_sms * kColsumBlocks / colblocks;
    const int most = colsum_slices(rows);
    sl = sl > most ? most : sl;
    sl = sl < 1 ? 1 : sl;
    const int rows_per = rows > sl ? (rows + sl - 1) / sl : 1;
    sl = rows > 0 ? (rows + rows_per - 1) / rows_per : 1;
    colsum_onepass_kernel<<<dim3(colblocks, sl), 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(a), lda, part,
                                                                   out, tickets, rows, N, rows_per, accumulate);
    return static_cast<int>(cudaGetLastError());
  }
  dim3 grid((N / 2 + 31) / 32, slices);
  colsum_partial_kernel<<<grid, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(a), lda, part, rows, N, rps);
  fold_partials_kernel<<<(N + 255) / 256, 256, 0, stream>>>(part, out, slices, N, accumulate);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ssb
