// Embedding and vocab-parallel cross-entropy kernels.
//
// embedding fwd : out[t,:] = dropout( W[id[t]-v0,:] (0 if id outside [v0,v1)) + P[pos[t],:] )
//                 (reference: runtime/megatron/mpu/layers.py:185-205 masked lookup,
//                  runtime/megatron/model/flex_ops.py:356-376 position add + dropout)
// embedding bwd : dW[id-v0,:] += g, dP[pos,:] += g with fp32 atomics into the main-grad buffers.
// cross entropy : two phases so that a tensor-parallel group can all-reduce the row statistics
//                 between them (reference: runtime/megatron/mpu/cross_entropy.py:36-115):
//   stats    : per row local max, sum exp(x - local max), and the target logit if it is local
//   finalize : loss = log(sum) + max - target; logits overwritten in place by
//              (softmax - onehot) * grad_scale  (the backward of the mean loss)
// One CTA per row; rows are V_local bf16 logits.
#include "common.cuh"

namespace ssb {
namespace {

constexpr int kEmbedBlocks = 6;  // of 256 threads, per SM; more of the shorter ones that take one token at a time

// A row of threads per token (`tpr`: 1 to 16 in powers of two, or a multiple of 32), the next token's id and position on their way while
// this one's rows are.  Bounded by the latency of id -> row and by the hashes of the dropout mask.  A thread per eight columns of
// the whole output, which divided by the row length and read the id as it went, before -> now: 16384 tokens x 2048 of 51200 rows 29.2
// -> 25.8 us (with dropout 34.0 -> 32.2), of 2048 rows 25.4 -> 19.5, x 64 3.05 -> 2.55 (4.2 with 32 threads a token), x 2560 33.9 -> 31.5 (36.6
// with six blocks of 160 threads), 512 x 1024 2.6 -> 2.1.  Blocks of 192 threads for two tokens of 768 columns: 8192 tokens 7.7 -> 5.2 with six,
// 5.3 with eight.  Eight blocks of 256 spill (20.3 of 2048 rows); four tokens at a time leave too few threads (53 instead of 37 us, a
// cold pass with dropout).
__global__ void __launch_bounds__(256, kEmbedBlocks)
embedding_fwd_kernel(const long long* __restrict__ ids, const long long* __restrict__ pos,
                     const __nv_bfloat16* __restrict__ W, const __nv_bfloat16* __restrict__ P,
                     __nv_bfloat16* __restrict__ out, long long tokens, int H, long long v0, long long v1,
                     float dropout_p, unsigned long long seed, int tpr) {
  const uint32_t keep16 = dropout_keep16(dropout_p);
  const float scale = dropout_p > 0.f ? 65536.0f / static_cast<float>(keep16) : 1.0f;
  const int nvec = H / 8, slots = blockDim.x / tpr;
  const uint4* table = reinterpret_cast<const uint4*>(W);
  const uint4* places = reinterpret_cast<const uint4*>(P);
  const int step = gridDim.x * slots, col0 = threadIdx.x % tpr;
  long long t = static_cast<long long>(blockIdx.x) * slots + threadIdx.x / tpr;
  if (t >= tokens) return;
  long long id = ids[t], at = P != nullptr ? pos[t] : 0;
  while (t < tokens) {
    const bool have = id >= v0 && id < v1;
    const uint4* row = table + (have ? id - v0 : 0) * nvec;
    const uint4* place = places + at * nvec;
    const long long next = t + step;
    if (next < tokens) {
      id = ids[next];
      if (P != nullptr) at = pos[next];
    }
    for (int c = col0; c < nvec; c += tpr) {
      uint4 q = make_uint4(0u, 0u, 0u, 0u), r = q;
      if (have) q = row[c];
      if (P != nullptr) r = place[c];
      const float2 a0 = unpack_bf16x2(q.x), a1 = unpack_bf16x2(q.y), a2 = unpack_bf16x2(q.z), a3 = unpack_bf16x2(q.w);
      float f[8] = {a0.x, a0.y, a1.x, a1.y, a2.x, a2.y, a3.x, a3.y};
      if (P != nullptr) {
        const float2 b0 = unpack_bf16x2(r.x), b1 = unpack_bf16x2(r.y), b2 = unpack_bf16x2(r.z), b3 = unpack_bf16x2(r.w);
        f[0] += b0.x; f[1] += b0.y; f[2] += b1.x; f[3] += b1.y; f[4] += b2.x; f[5] += b2.y; f[6] += b3.x; f[7] += b3.y;
      }
      const long long v = t * nvec + c;
      if (dropout_p > 0.f) {
        dropout_apply4(f, dropout_drop4(seed, static_cast<uint64_t>(v) * 2, keep16), scale);
        dropout_apply4(f + 4, dropout_drop4(seed, static_cast<uint64_t>(v) * 2 + 1, keep16), scale);
      }
      uint4 o;
      o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
      o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
      reinterpret_cast<uint4*>(out)[v] = o;
    }
    t = next;
  }
}

// g is the gradient w.r.t. the embedding OUTPUT (after dropout); the mask is regenerated here.
__global__ void __launch_bounds__(256)
embedding_bwd_kernel(const long long* __restrict__ ids, const long long* __restrict__ pos,
                     const __nv_bfloat16* __restrict__ g, float* __restrict__ dW, float* __restrict__ dP,
                     long long tokens, int H, long long v0, long long v1, float dropout_p, unsigned long long seed) {
  const uint32_t keep16 = dropout_keep16(dropout_p);
  const float scale = dropout_p > 0.f ? 65536.0f / static_cast<float>(keep16) : 1.0f;
  const int nvec = H / 8;
  for (long long v = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; v < tokens * nvec;
       v += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long t = v / nvec;
    const int c = static_cast<int>(v % nvec);
    const uint4 q = *reinterpret_cast<const uint4*>(g + v * 8);
    float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), cc = unpack_bf16x2(q.z), d = unpack_bf16x2(q.w);
    float f[8] = {a.x, a.y, b.x, b.y, cc.x, cc.y, d.x, d.y};
    if (dropout_p > 0.f) {
      dropout_apply4(f, dropout_drop4(seed, static_cast<uint64_t>(v) * 2, keep16), scale);
      dropout_apply4(f + 4, dropout_drop4(seed, static_cast<uint64_t>(v) * 2 + 1, keep16), scale);
    }
    const long long id = ids[t];
    if (dW != nullptr && id >= v0 && id < v1) {
      float* dst = dW + (id - v0) * H + c * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) atomicAdd(dst + j, f[j]);
    }
    if (dP != nullptr) {
      float* dst = dP + pos[t] * H + c * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) atomicAdd(dst + j, f[j]);
    }
  }
}

// Order-independent variant of the scatter above: `keys` are the row indices (token ids, or positions) in
// ascending order and `order[p]` is the token that holds keys[p].  Block p works only if it is the first of its
// run of equal keys; it then sums the run's rows in the order given and adds the total to row keys[p] - k0 of dst
// with plain stores (no other block touches that row), so repeated runs give bitwise equal results.
template <typename Key>
__global__ void __launch_bounds__(256)
embedding_bwd_sorted_kernel(const Key* __restrict__ keys, const long long* __restrict__ order,
                            const __nv_bfloat16* __restrict__ g, float* __restrict__ dst, long long tokens, int H,
                            long long k0, long long k1, float dropout_p, unsigned long long seed) {
  const long long p = blockIdx.x;
  const long long key = keys[p];
  if (key < k0 || key >= k1) return;
  if (p > 0 && keys[p - 1] == key) return;
  const uint32_t keep16 = dropout_keep16(dropout_p);
  const float scale = dropout_p > 0.f ? 65536.0f / static_cast<float>(keep16) : 1.0f;
  const int nvec = H / 8;
  for (int c = threadIdx.x; c < nvec; c += blockDim.x) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (long long j = p; j < tokens && keys[j] == key; ++j) {
      const long long v = order[j] * nvec + c;
      const uint4 q = *reinterpret_cast<const uint4*>(g + v * 8);
      float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), cc = unpack_bf16x2(q.z), d = unpack_bf16x2(q.w);
      float f[8] = {a.x, a.y, b.x, b.y, cc.x, cc.y, d.x, d.y};
      if (dropout_p > 0.f) {
        dropout_apply4(f, dropout_drop4(seed, static_cast<uint64_t>(v) * 2, keep16), scale);
        dropout_apply4(f + 4, dropout_drop4(seed, static_cast<uint64_t>(v) * 2 + 1, keep16), scale);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += f[i];
    }
    float4* out = reinterpret_cast<float4*>(dst + (key - k0) * H + c * 8);
    float4 lo = out[0], hi = out[1];
    lo.x += acc[0]; lo.y += acc[1]; lo.z += acc[2]; lo.w += acc[3];
    hi.x += acc[4]; hi.y += acc[5]; hi.z += acc[6]; hi.w += acc[7];
    out[0] = lo;
    out[1] = hi;
  }
}

// Sort keys of the rows a table holds: ids of [k0, k0 + n) as 0 .. n - 1, every other id as n.  In 16 or 32 bits the radix sort
// makes two or four passes over the tokens instead of the eight that 64-bit ids take (9 us each for 16384 tokens).
template <typename Key>
__global__ void __launch_bounds__(256)
embedding_keys_kernel(const long long* __restrict__ ids, Key* __restrict__ keys, long long tokens, long long k0, long long n) {
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < tokens; i += gridDim.x * 256LL) {
    const long long id = ids[i];
    keys[i] = static_cast<Key>(id >= k0 && id - k0 < n ? id - k0 : n);
  }
}

constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float block_reduce(float v, bool is_max, float* sm) {
  v = is_max ? warp_max(v) : warp_sum(v);
  __syncthreads();  // protects `sm` between successive calls
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  float t = (threadIdx.x & 31) < nw ? sm[threadIdx.x & 31] : (is_max ? -INFINITY : 0.f);
  return is_max ? warp_max(t) : warp_sum(t);
}

// stats[row] = {local max, sum exp(x - local max), target logit or 0}
__global__ void __launch_bounds__(256)
ce_stats_kernel(const __nv_bfloat16* __restrict__ logits, int ld, const long long* __restrict__ targets,
                float* __restrict__ row_max, float* __restrict__ row_sum, float* __restrict__ row_tgt, int V,
                long long v0) {
  __shared__ float sm[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* x = logits + row * ld;
  const int nvec = V / 8;
  float mx = -INFINITY;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const uint4 q = reinterpret_cast<const uint4*>(x)[v];
    float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), c = unpack_bf16x2(q.z), d = unpack_bf16x2(q.w);
    mx = fmaxf(mx, fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(b.x, b.y)), fmaxf(fmaxf(c.x, c.y), fmaxf(d.x, d.y))));
  }
  for (int k = nvec * 8 + threadIdx.x; k < V; k += blockDim.x) mx = fmaxf(mx, __bfloat162float(x[k]));
  mx = block_reduce(mx, true, sm);
  float s = 0.f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const uint4 q = reinterpret_cast<const uint4*>(x)[v];
    float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), c = unpack_bf16x2(q.z), d = unpack_bf16x2(q.w);
    s += __expf(a.x - mx) + __expf(a.y - mx) + __expf(b.x - mx) + __expf(b.y - mx) + __expf(c.x - mx) +
         __expf(c.y - mx) + __expf(d.x - mx) + __expf(d.y - mx);
  }
  for (int k = nvec * 8 + threadIdx.x; k < V; k += blockDim.x) s += __expf(__bfloat162float(x[k]) - mx);
  s = block_reduce(s, false, sm);
  if (threadIdx.x == 0) {
    row_max[row] = mx;
    row_sum[row] = s;
    const long long t = targets[row] - v0;
    row_tgt[row] = (t >= 0 && t < V) ? __bfloat162float(x[t]) : 0.f;
  }
}

// gmax / gsum / gtgt are the group-reduced statistics (gsum already rescaled to gmax by the caller for
// tensor parallel runs; for a single rank they are the outputs of ce_stats_kernel).
// loss_mask: optional fp32 [rows] weights (0 drops the token); grad_scale multiplies the gradient.
__global__ void __launch_bounds__(256)
ce_finalize_kernel(__nv_bfloat16* __restrict__ logits, int ld, const long long* __restrict__ targets,
                   const float* __restrict__ gmax, const float* __restrict__ gsum, const float* __restrict__ gtgt,
                   const float* __restrict__ loss_mask, float* __restrict__ loss, int V, long long v0,
                   float grad_scale, int write_grad) {
  const long long row = blockIdx.x;
  __nv_bfloat16* x = logits + row * ld;
  const float mx = gmax[row], sum = gsum[row];
  const float w = loss_mask ? loss_mask[row] : 1.0f;
  if (threadIdx.x == 0) loss[row] = (logf(sum) + mx - gtgt[row]) * w;
  if (!write_grad) return;
  const float inv = 1.0f / sum;
  const float gs = grad_scale * w;
  const long long t = targets[row] - v0;
  const int nvec = V / 8;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const uint4 q = reinterpret_cast<const uint4*>(x)[v];
    float2 a = unpack_bf16x2(q.x), b = unpack_bf16x2(q.y), c = unpack_bf16x2(q.z), d = unpack_bf16x2(q.w);
    float f[8] = {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float pr = __expf(f[j] - mx) * inv;
      if (static_cast<long long>(v) * 8 + j == t) pr -= 1.0f;
      f[j] = pr * gs;
    }
    uint4 o;
    o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
    o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
    reinterpret_cast<uint4*>(x)[v] = o;
  }
  for (int k = nvec * 8 + threadIdx.x; k < V; k += blockDim.x) {
    float pr = __expf(__bfloat162float(x[k]) - mx) * inv;
    if (k == t) pr -= 1.0f;
    x[k] = __float2bfloat16(pr * gs);
  }
}

// exp(x - off) = 2^((x - off) log2 e) of two packed logits, two differences and two products per instruction.  kTiny: results
// below 2^-126 are kept (a gradient is scaled afterwards); in a sum next to a term of one they are nothing, and zero will do.
template <bool kTiny>
__device__ __forceinline__ float2 exp_pair(uint32_t two, float off) {
  const float2 d = mul_f32x2(add_f32x2(unpack_bf16x2(two), make_float2(-off, -off)), make_float2(kLog2e, kLog2e));
  float2 e;
  if constexpr (kTiny) {
    asm("ex2.approx.f32 %0, %1;" : "=f"(e.x) : "f"(d.x));
    asm("ex2.approx.f32 %0, %1;" : "=f"(e.y) : "f"(d.y));
  } else {
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(d.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(d.y));
  }
  return e;
}

// Loss and gradient of whole rows in one pass over memory, for logits that no other rank shares.  The row is read once, into
// shared memory; every thread keeps a running maximum and the sum of exponentials relative to it on the way, so that the
// special-function unit works under the loads, and only the gradient is left for a second pass.  Same quantities as
// ce_stats + ce_finalize, which read the row three times.  T threads a row, 1024 per SM: one CTA loads while others write.
// 4096 rows x 51200: 177 us (4.7 TB/s, two exponentials an element) against 263 for the two kernels; results below the normal
// range are 6 us of it.
constexpr int kCeMaxCols = 56 * 1024;  // 112 KB of shared memory: two rows per SM

// AHEAD: the next four loads of a thread are under way while it works on the last four.  4096 rows x 51200 191 -> 176 us, x 40000 148 -> 133,
// x 32000 115 -> 106, x 20480 71 -> 66 (eight loads at a time instead: x 51200 201).  With one round of loads or two it is slower (4096 x 2048
// 12.3 -> 13.1, x 15000 52.2 -> 53.1), and where the logits are still in the L2: 2048 x 20480 30.6 -> 31.4, 1024 x 20480 16.2 -> 16.9, 400 x
// 32000 11.9 -> 12.3, 200 x 51200 12.3 -> 12.8; 700 x 32000 18.8 -> 18.5, 1500 x 32000 42.3 -> 38.9.
template <int T, bool AHEAD>
__global__ void __launch_bounds__(T, 1024 / T)
ce_fused_kernel(__nv_bfloat16* __restrict__ logits, int ld, const long long* __restrict__ targets,
                const float* __restrict__ loss_mask, float* __restrict__ loss, int V, long long v0, float grad_scale) {
  extern __shared__ uint4 row_smem[];
  __shared__ float sm[32];
  const long long row = blockIdx.x;
  __nv_bfloat16* x = logits + row * ld;
  uint4* xv = reinterpret_cast<uint4*>(x);
  const int nvec = V / 8;
  const int k0 = nvec * 8 + threadIdx.x;           // at most seven columns behind the last whole vector
  const float tail = k0 < V ? __bfloat162float(x[k0]) : -INFINITY;
  const long long t = targets[row] - v0;
  // read by every thread before the barriers of the reductions, so before any thread overwrites the row
  const float tgt = (t >= 0 && t < V) ? __bfloat162float(x[t]) : 0.f;
  float tmax = tail, tsum = tail != -INFINITY ? __expf(tail - tail) : 0.f;  // this thread's maximum and sum exp(x - maximum)
  uint4 next[4];
  auto fetch = [&](int v, uint4 (&q)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v + u * T < nvec) q[u] = __ldcs(xv + v + u * T);
  };
  if (AHEAD) fetch(threadIdx.x, next);
  for (int v = threadIdx.x; v < nvec; v += 4 * T) {
    uint4 q[4];
    if constexpr (AHEAD) {
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = next[u];
      fetch(v + 4 * T, next);
    } else {
      fetch(v, q);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (v + u * T < nvec) {
        row_smem[v + u * T] = q[u];       // each thread reads back what it wrote: no barrier needed
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q[u]);
        const float2 m2 = __bfloat1622float2(__hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
        const float m8 = fmaxf(m2.x, m2.y);
        if (m8 > tmax) {
          tsum *= __expf(tmax - m8);               // tmax = -inf: 0
          tmax = m8;
        }
        const float off = tmax == -INFINITY ? 0.f : tmax;
        const float2 s2 = add_f32x2(add_f32x2(exp_pair<false>(q[u].x, off), exp_pair<false>(q[u].y, off)),
                                    add_f32x2(exp_pair<false>(q[u].z, off), exp_pair<false>(q[u].w, off)));
        tsum += s2.x + s2.y;
      }
    }
  }
  const float mx = block_reduce(tmax, true, sm);
  float s = block_reduce(tmax == -INFINITY ? tsum : tsum * __expf(tmax - mx), false, sm);
  if (mx == -INFINITY) s = NAN;                    // no finite logit: no distribution, whatever the target (as in ce_stats)
  const float w = loss_mask ? loss_mask[row] : 1.0f;
  if (threadIdx.x == 0) loss[row] = (logf(s) + mx - tgt) * w;
  const float inv = 1.0f / s, gs = grad_scale * w;
  const float2 inv2 = make_float2(inv, inv), gs2 = make_float2(gs, gs);
  const int tv = t >= 0 && t < V ? static_cast<int>(t >> 3) : -1;  // vector of the target
  for (int v = threadIdx.x; v < nvec; v += T) {
    const uint4 q = row_smem[v];
    float2 f[4] = {mul_f32x2(exp_pair<true>(q.x, mx), inv2), mul_f32x2(exp_pair<true>(q.y, mx), inv2),
                   mul_f32x2(exp_pair<true>(q.z, mx), inv2), mul_f32x2(exp_pair<true>(q.w, mx), inv2)};
    if (v == tv) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if ((t & 7) == 2 * j) f[j].x -= 1.0f;
        if ((t & 7) == 2 * j + 1) f[j].y -= 1.0f;
      }
    }
    uint4 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f[j] = mul_f32x2(f[j], gs2);
      reinterpret_cast<uint32_t*>(&o)[j] = pack_bf16x2(f[j].x, f[j].y);
    }
    xv[v] = o;
  }
  if (k0 < V) {
    float pr = __expf(tail - mx) * inv;
    if (k0 == t) pr -= 1.0f;
    x[k0] = __float2bfloat16(pr * gs);
  }
}

}  // namespace

bool ce_fused_ok(int V) { return V <= kCeMaxCols; }

int ce_fused_launch(void* logits, int ld, const long long* targets, const float* loss_mask, float* loss, long long rows, int V,
                    long long v0, float grad_scale, int num_sms, cudaStream_t stream) {
  if (ld % 8) return -3;
  auto launch = [&](auto kernel, int threads) {
    const int rc = static_cast<int>(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCeMaxCols * 2));
    if (rc) return rc;
    kernel<<<static_cast<unsigned>(rows), threads, (V / 8) * 16, stream>>>(reinterpret_cast<__nv_bfloat16*>(logits), ld, targets,
                                                                           loss_mask, loss, V, v0, grad_scale);
    return static_cast<int>(cudaGetLastError());
  };
  // Threads of a row, 4096 rows: 128 and 256 threads take 49 and 53 us at 12288 columns, 69 and 67 at 16384; 256 and 512 take
  // 138 and 145 at 32000, 201 and 181 at 40960 (512 throughout: 27 us at 1024 columns, where the two kernels take 15 and 128
  // threads 9.5).  Rows that all fit on the chip at once are a matter of latency: 16 rows of 8192 take 4.6 us with 128 threads
  // and 3.8 with 512.
  const bool few = rows <= 2LL * num_sms;
  // Loads ahead: where a thread has at least two rounds of them and the logits have left the L2 since the product that made them.
  const long long bytes = rows * V * 2;
  const bool ahead = V > 16 * 1024 && bytes > (V > 24 * 1024 ? 40LL << 20 : 96LL << 20);
  if (few || V > 36 * 1024) return ahead ? launch(ce_fused_kernel<512, true>, 512) : launch(ce_fused_kernel<512, false>, 512);
  if (V > 14 * 1024) return ahead ? launch(ce_fused_kernel<256, true>, 256) : launch(ce_fused_kernel<256, false>, 256);
  return launch(ce_fused_kernel<128, false>, 128);
}

int embedding_fwd_launch(const long long* ids, const long long* pos, const void* W, const void* P, void* out,
                         long long tokens, int H, long long v0, long long v1, float dropout_p,
                         unsigned long long seed, int num_sms, cudaStream_t stream) {
  if (H % 8) return -3;
  if (H == 0) return 0;  // rows of no columns: nothing to look up
  const int nvec = H / 8, passes = (nvec + 255) / 256;
  int tpr = ((nvec + passes - 1) / passes + 31) / 32 * 32;
  while (tpr <= 32 && tpr / 2 >= nvec) tpr /= 2;
  const int slots = 256 / tpr, per_sm = slots > 1 ? kEmbedBlocks : kEmbedBlocks * 256 / tpr;
  const long long want = (tokens + slots - 1) / slots, most = static_cast<long long>(num_sms) * per_sm;
  const int blocks = static_cast<int>(want < 1 ? 1 : (want > most ? most : want));
  embedding_fwd_kernel<<<blocks, slots * tpr, 0, stream>>>(ids, pos, reinterpret_cast<const __nv_bfloat16*>(W),
                                                           reinterpret_cast<const __nv_bfloat16*>(P),
                                                           reinterpret_cast<__nv_bfloat16*>(out), tokens, H, v0, v1,
                                                           dropout_p, seed, tpr);
  return static_cast<int>(cudaGetLastError());
}

int embedding_bwd_launch(const long long* ids, const long long* pos, const void* g, float* dW, float* dP,
                         long long tokens, int H, long long v0, long long v1, float dropout_p,
                         unsigned long long seed, int num_sms, cudaStream_t stream) {
  if (H % 8) return -3;
  long long want = (tokens * (H / 8) + 255) / 256;
  const int blocks = static_cast<int>(want < 1 ? 1 : (want > num_sms * 32LL ? num_sms * 32LL : want));
  embedding_bwd_kernel<<<blocks, 256, 0, stream>>>(ids, pos, reinterpret_cast<const __nv_bfloat16*>(g), dW, dP,
                                                   tokens, H, v0, v1, dropout_p, seed);
  return static_cast<int>(cudaGetLastError());
}

// key_bytes: 2, 4 or 8 (short, int, long long)
int embedding_keys_launch(const long long* ids, void* keys, int key_bytes, long long tokens, long long k0, long long n,
                          cudaStream_t stream) {
  if (tokens < 1) return -4;
  const long long want = (tokens + 255) / 256;
  const unsigned blocks = static_cast<unsigned>(want < 1184 ? want : 1184);
  if (key_bytes == 2)
    embedding_keys_kernel<<<blocks, 256, 0, stream>>>(ids, reinterpret_cast<short*>(keys), tokens, k0, n);
  else if (key_bytes == 4)
    embedding_keys_kernel<<<blocks, 256, 0, stream>>>(ids, reinterpret_cast<int*>(keys), tokens, k0, n);
  else
    return -2;
  return static_cast<int>(cudaGetLastError());
}

int embedding_bwd_sorted_launch(const void* keys, int key_bytes, const long long* order, const void* g, float* dst,
                                long long tokens, int H, long long k0, long long k1, float dropout_p,
                                unsigned long long seed, cudaStream_t stream) {
  if (H % 8) return -3;
  if (tokens < 1 || tokens > 0x7fffffffLL) return -4;
  const auto* gb = reinterpret_cast<const __nv_bfloat16*>(g);
  const unsigned blocks = static_cast<unsigned>(tokens);
  if (key_bytes == 2)
    embedding_bwd_sorted_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const short*>(keys), order, gb, dst, tokens, H, k0, k1, dropout_p, seed);
  else if (key_bytes == 4)
    embedding_bwd_sorted_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const int*>(keys), order, gb, dst, tokens, H, k0, k1, dropout_p, seed);
  else
    embedding_bwd_sorted_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const long long*>(keys), order, gb, dst, tokens, H, k0, k1, dropout_p, seed);
  return static_cast<int>(cudaGetLastError());
}

int ce_stats_launch(const void* logits, int ld, const long long* targets, float* row_max, float* row_sum,
                    float* row_tgt, long long rows, int V, long long v0, cudaStream_t stream) {
  if (ld % 8) return -3;
  ce_stats_kernel<<<static_cast<unsigned>(rows), 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(logits), ld,
                                                                   targets, row_max, row_sum, row_tgt, V, v0);
  return static_cast<int>(cudaGetLastError());
}

int ce_finalize_launch(void* logits, int ld, const long long* targets, const float* gmax, const float* gsum,
                       const float* gtgt, const float* loss_mask, float* loss, long long rows, int V, long long v0,
                       float grad_scale, int write_grad, cudaStream_t stream) {
  if (ld % 8) return -3;
  ce_finalize_kernel<<<static_cast<unsigned>(rows), 256, 0, stream>>>(reinterpret_cast<__nv_bfloat16*>(logits), ld,
                                                                      targets, gmax, gsum, gtgt, loss_mask, loss, V,
                                                                      v0, grad_scale, write_grad);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ssb
