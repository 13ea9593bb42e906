// Embedding gradient without a sort: dW[id - v0] += g, dP[pos] += g, every row summed by one block in token order with plain
// stores, so repeated runs give bitwise equal results (reference: runtime/megatron/mpu/layers.py:185-205 backward,
// runtime/megatron/model/flex_ops.py:356-376).
//
// The sum needs the tokens of each row together and in order, but not the rows in any order.  One kernel groups them: a
// cluster of eight CTAs per table (words, positions) counts the tokens of every row it meets, hands each row a stretch of a
// list and puts its tokens there, as they come, with a cluster barrier between the phases.  Nothing is cleared or scanned over
// the table: only the counters of rows that occur are touched.  The second kernel has a block for every row that occurs (the
// grid covers as many as there are tokens or rows); it puts the row's tokens in order (by rank for up to kRankMax of them, by a bitmap
// over the batch beyond) and sums their rows of g.
//
// The radix sort it replaces (a library call on 16- or 32-bit keys, two tables one after the other) took ten launches and as
// many clears a table.  16384 tokens x 2048, V 51200: grouping 12.5 us where the sorts took 82; the pass 302 -> 200 us.
#include "common.cuh"

#include <utility>

namespace ssb {
namespace {

constexpr int kGroupCtas = 8, kGroupThreads = 1024;
constexpr int kMaxTokens = 65536;                                   // bitmap of a batch: 8 KB of shared memory
constexpr int kPerThread = kMaxTokens / (kGroupCtas * kGroupThreads);
constexpr int kRankMax = 256;
constexpr int kSumBlocks = 5;  // per SM: with the 63 registers the compiler likes there were four, with six it spills

struct GroupTable {
  const long long* ids;
  long long k0;          // id of row 0
  long long n;           // rows
  float* dst;            // fp32 [n, H]
  int *cnt, *base;       // [n] tokens of a row, start of its stretch (rows that occur only)
  int *list, *order;     // [tokens] the stretches; ordered copies of long ones
  int4* runs;            // [tokens] rows that occur: {row, start of its stretch, tokens, one of them}
  int* totals;           // {rows that occur, tokens in the lists}
};
struct GroupArgs {
  GroupTable t[2];
  int blocks0;  // of the summing kernel for the first table, in front of those for the second
};

__global__ void __cluster_dims__(kGroupCtas, 1, 1) __launch_bounds__(kGroupThreads)
embedding_group_kernel(const GroupArgs args, int tokens) {
  const GroupTable& a = args.t[blockIdx.x / kGroupCtas];
  const int first = (blockIdx.x % kGroupCtas) * kGroupThreads + threadIdx.x;
  int key[kPerThread], slot[kPerThread];
#pragma unroll
  for (int i = 0; i < kPerThread; ++i) {
    const int t = first + i * (kGroupCtas * kGroupThreads);
    key[i] = -1;
    if (t < tokens) {
      const long long id = a.ids[t];
      if (id >= a.k0 && id - a.k0 < a.n) {
        key[i] = static_cast<int>(id - a.k0);
        __stcg(a.cnt + key[i], 0);
      }
    }
  }
  if (first < 2) __stcg(a.totals + first, 0);
  __threadfence();
  cluster_barrier();
#pragma unroll
  for (int i = 0; i < kPerThread; ++i) slot[i] = key[i] >= 0 ? atomicAdd(a.cnt + key[i], 1) : -1;
  __threadfence();
  cluster_barrier();
  // One reservation per warp: thousands of additions to one address would go one by one.
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < kPerThread; ++i) {
    const bool head = slot[i] == 0;
    const uint32_t heads = __ballot_sync(0xffffffffu, head);
    if (heads == 0u) continue;
    const int n = head ? __ldcg(a.cnt + key[i]) : 0;
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += up;
    }
    int run0 = 0, base0 = 0;
    if (lane == 31) {
      run0 = atomicAdd(a.totals, __popc(heads));
      base0 = atomicAdd(a.totals + 1, incl);
    }
    run0 = __shfl_sync(0xffffffffu, run0, 31);
    base0 = __shfl_sync(0xffffffffu, base0, 31);
    if (head) {
      const int base = base0 + incl - n;
      __stcg(a.base + key[i], base);
      a.runs[run0 + __popc(heads & ((1u << lane) - 1u))] = make_int4(key[i], base, n, first + i * (kGroupCtas * kGroupThreads));
    }
  }
  __threadfence();
  cluster_barrier();
#pragma unroll
  for (int i = 0; i < kPerThread; ++i)
    if (slot[i] >= 0) a.list[__ldcg(a.base + key[i]) + slot[i]] = first + i * (kGroupCtas * kGroupThreads);
}

// What a block does is a chain of loads (row, its tokens, their gradients); the values that are added to are fetched in front of it,
// four gradients at a time.  16384 tokens x 2048, V 51200, with positions: 84 -> 70 us (78 with four blocks an SM, 85 with six),
// V 2048 52 -> 35; x 576 29 -> 20.
__global__ void __launch_bounds__(256, kSumBlocks)
embedding_sum_kernel(const GroupArgs args, const __nv_bfloat16* __restrict__ g, int tokens, int H, float dropout_p,
                     unsigned long long seed) {
  __shared__ uint32_t bits[kMaxTokens / 32];   // kRankMax or fewer tokens: [unordered | ordered]
  __shared__ int warp_total[8];
  const bool second = static_cast<int>(blockIdx.x) >= args.blocks0;
  const GroupTable& a = args.t[second];
  const int index = static_cast<int>(blockIdx.x) - (second ? args.blocks0 : 0);
  const int4 run = a.runs[index];
  if (index >= a.totals[0]) return;
  const int key = run.x, base = run.y, n = run.z, t = run.w;
  const int* list = a.list + base;
  const int nvec = H / 8;
  const uint4* gradients = reinterpret_cast<const uint4*>(g);
  float4* out = reinterpret_cast<float4*>(a.dst + static_cast<size_t>(key) * H);
  float4 lo, hi;  // what is there already: on its way while the tokens are put in order
  if (static_cast<int>(threadIdx.x) < nvec) {
    lo = out[2 * threadIdx.x];
    hi = out[2 * threadIdx.x + 1];
  }
  int* sorted = reinterpret_cast<int*>(bits) + kRankMax;
  if (n > 1 && n <= kRankMax) {
    int* raw = reinterpret_cast<int*>(bits);
    for (int i = threadIdx.x; i < n; i += blockDim.x) raw[i] = list[i];
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int mine = raw[i];
      int rank = 0;
      for (int j = 0; j < n; ++j) rank += raw[j] < mine;
      sorted[rank] = mine;
    }
    __syncthreads();
  } else if (n > kRankMax) {
    const int words = (tokens + 31) / 32, per = (words + blockDim.x - 1) / blockDim.x;
    for (int i = threadIdx.x; i < words; i += blockDim.x) bits[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) atomicOr(&bits[list[i] >> 5], 1u << (list[i] & 31));
    __syncthreads();
    const int w0 = min(words, static_cast<int>(threadIdx.x) * per), w1 = min(words, w0 + per);
    int mine = 0;
    for (int i = w0; i < w1; ++i) mine += __popc(bits[i]);
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, d);
      if ((threadIdx.x & 31) >= d) incl += up;
    }
    if ((threadIdx.x & 31) == 31) warp_total[threadIdx.x >> 5] = incl;
    __syncthreads();
    int at = base + incl - mine;
    for (int i = 0; i < static_cast<int>(threadIdx.x >> 5); ++i) at += warp_total[i];
    for (int i = w0; i < w1; ++i)
      for (uint32_t x = bits[i]; x != 0u; x &= x - 1) a.order[at++] = i * 32 + __ffs(x) - 1;
    __syncthreads();
    sorted = a.order + base;
  }
  const uint32_t keep16 = dropout_keep16(dropout_p);
  const float scale = dropout_p > 0.f ? 65536.0f / static_cast<float>(keep16) : 1.0f;
  for (int c = threadIdx.x; c < nvec; c += blockDim.x) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (c >= static_cast<int>(blockDim.x)) {
      lo = out[2 * c];
      hi = out[2 * c + 1];
    }
    auto at = [&](int token) { return static_cast<size_t>(token) * nvec + c; };
    auto add = [&](int token, const uint4& q) {
      const float2 x0 = unpack_bf16x2(q.x), x1 = unpack_bf16x2(q.y), x2 = unpack_bf16x2(q.z), x3 = unpack_bf16x2(q.w);
      float f[8] = {x0.x, x0.y, x1.x, x1.y, x2.x, x2.y, x3.x, x3.y};
      if (dropout_p > 0.f) {
        const uint64_t v = at(token);
        dropout_apply4(f, dropout_drop4(seed, v * 2, keep16), scale);
        dropout_apply4(f + 4, dropout_drop4(seed, v * 2 + 1, keep16), scale);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += f[i];
    };
    if (n == 1) {
      add(t, gradients[at(t)]);
    } else {
      for (int j = 0; j < n; j += 4) {           // four rows under way at a time, added in token order
        int token[4];
        uint4 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          token[i] = sorted[min(j + i, n - 1)];
          if (j + i < n) q[i] = gradients[at(token[i])];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (j + i < n) add(token[i], q[i]);
      }
    }
    lo.x += acc[0]; lo.y += acc[1]; lo.z += acc[2]; lo.w += acc[3];
    hi.x += acc[4]; hi.y += acc[5]; hi.z += acc[6]; hi.w += acc[7];
    out[2 * c] = lo;
    out[2 * c + 1] = hi;
  }
}

}  // namespace

int embedding_group_max_tokens() { return kMaxTokens; }

// ints of workspace for one table
long long embedding_group_ints(long long tokens, long long rows) { return (2 * rows + 6 * tokens + 4 + 3) / 4 * 4; }

// `ids[i]` null: no table i.  ws: embedding_group_ints() of every table that is there, one after the other.
int embedding_bwd_grouped_launch(const long long* const* ids, const long long* k0, const long long* rows, float* const* dst,
                                 int* ws, const void* g, long long tokens, int H, float dropout_p, unsigned long long seed,
                                 cudaStream_t stream) {
  if (H % 8) return -3;
  if (tokens < 1 || tokens > kMaxTokens) return -4;
  GroupArgs args{};
  int tables = 0;
  for (int i = 0; i < 2; ++i) {
    if (ids[i] == nullptr) continue;
    if (rows[i] < 0 || rows[i] >= 0x7fffffffLL) return -4;
    GroupTable& a = args.t[tables++];
    a.ids = ids[i];
    a.k0 = k0[i];
    a.n = rows[i];
    a.dst = dst[i];
    a.totals = ws;
    a.runs = reinterpret_cast<int4*>(ws + 4);
    a.list = ws + 4 + 4 * tokens;
    a.order = a.list + tokens;
    a.cnt = a.order + tokens;
    a.base = a.cnt + rows[i];
    ws += embedding_group_ints(tokens, rows[i]);
  }
  if (tables == 0) return 0;
  embedding_group_kernel<<<tables * kGroupCtas, kGroupThreads, 0, stream>>>(args, static_cast<int>(tokens));
  const int want = (H / 8 + 31) / 32 * 32, threads = want < 64 ? 64 : (want > 256 ? 256 : want);
  // A block for every row that may occur: as many as there are tokens, for either table, left 14000 of 32000 blocks that only looked
  // that they were not wanted (16384 tokens in 2048 positions).  Positions come first where they have more than a token each, the
  // longest chains then (4096 x 512 14.7 us, 15.1 behind the words), words otherwise (1024 x 1024 of 2048 rows 11.6, 12.3).
  auto most = [&](const GroupTable& a) { return static_cast<int>(a.n < tokens ? a.n : tokens); };
  if (tables > 1 && args.t[1].n < tokens && args.t[1].n < args.t[0].n) std::swap(args.t[0], args.t[1]);
  args.blocks0 = most(args.t[0]);
  const int sum_blocks = args.blocks0 + (tables > 1 ? most(args.t[1]) : 0);
  if (sum_blocks == 0) return static_cast<int>(cudaGetLastError());
  embedding_sum_kernel<<<static_cast<unsigned>(sum_blocks), threads, 0, stream>>>(
      args, reinterpret_cast<const __nv_bfloat16*>(g), static_cast<int>(tokens), H, dropout_p, seed);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ssb
