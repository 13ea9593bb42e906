// Fused optimizer kernels over FLAT buffers: every parameter of a pipeline stage lives in one
// contiguous fp32 master buffer, with matching fp32 gradient, Adam moment and bf16 model buffers.
// One launch replaces the reference's chain of apex multi-tensor kernels: copy model grads to main
// grads, unscale + inf check, l2 norm, clip, FusedAdam, copy main params back to half
// (runtime/megatron/optimizer/optimizer.py:348-390,404-443,
//  runtime/megatron/optimizer/clip_grads.py:29-120).
//
//   sumsq  : sum of squares of the gradient buffer (two-stage, deterministic)
//   adam   : p, m, v update with the clip coefficient and the inf/nan skip decided ON DEVICE from the
//            reduced sum of squares (no host synchronisation), bf16 copy-out of the new parameters,
//            optional zeroing of the gradient buffer for the next iteration.
//   sgd    : momentum SGD with the same plumbing (the reference uses apex FusedSGD for --optimizer sgd).
#include "common.cuh"

namespace ssb {
namespace {

__global__ void __launch_bounds__(256)
sumsq_partial_kernel(const float* __restrict__ g, long long n, float* __restrict__ partials) {
  __shared__ float sm[8];
  float s = 0.f;
  const long long n4 = n / 4;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float4 f = reinterpret_cast<const float4*>(g)[i];
    s += f.x * f.x + f.y * f.y + f.z * f.z + f.w * f.w;
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const float f = g[n4 * 4 + threadIdx.x];
    s += f * f;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < 8 ? sm[threadIdx.x] : 0.f;
    t = warp_sum(t);
    if (threadIdx.x == 0) partials[blockIdx.x] = t;
  }
}

__global__ void sumsq_fold_kernel(const float* __restrict__ partials, int n, float* __restrict__ out, int accumulate) {
  __shared__ float sm[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partials[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.f;
    t = warp_sum(t);
    if (threadIdx.x == 0) out[0] = accumulate ? out[0] + t : t;
  }
}

struct AdamArgs {
  float lr, beta1, beta2, eps, weight_decay;
  float bias_corr1, bias_corr2;  // 1 - beta^t
  float grad_scale;              // gradients are multiplied by this first (1/num_microbatches, 1/loss_scale)
  float max_norm;                // <= 0: no clipping
  long long wd_end;              // elements [0, wd_end) get weight decay, the rest none
  int zero_grad;
};

// One element.  The fused multiply-adds are written out, so that the vector body and the scalar remainder round alike.
__device__ __forceinline__ void adam_element(float& p, float& m, float& v, float g, const AdamArgs& a, float gs, float inv_bc1,
                                             float inv_sqrt_bc2, float wd) {
  const float gi = __fmul_rn(g, gs);
  m = __fmaf_rn(a.beta1, m, __fmul_rn(1.0f - a.beta1, gi));
  v = __fmaf_rn(a.beta2, v, __fmul_rn(__fmul_rn(1.0f - a.beta2, gi), gi));
  const float denom = __fmaf_rn(sqrtf(v), inv_sqrt_bc2, a.eps);
  p = __fmaf_rn(-a.lr, __fmaf_rn(wd, p, __fdiv_rn(__fmul_rn(m, inv_bc1), denom)), p);
}

// Bound by HBM (30 bytes an element, 34 with the gradient cleared).  A thread works on 2 x 4 consecutive elements with
// 16-byte accesses, all eight loads before the first use: norm + update of 400 M elements 2784 -> 2153 us (4-byte accesses
// left the memory system waiting, 4.3 TB/s).  VEC: every buffer 16-byte aligned (8 bytes for the bf16 copy); parts of
// a flat buffer that start elsewhere take the scalar loop.
template <bool VEC>
__global__ void __launch_bounds__(256)
adam_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v, float* __restrict__ g,
            __nv_bfloat16* __restrict__ p16, long long n, const float* __restrict__ sumsq, int* __restrict__ skipped,
            AdamArgs a) {
  const long long tid = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const long long threads = static_cast<long long>(gridDim.x) * blockDim.x;
  float clip = 1.0f;
  if (sumsq != nullptr) {
    const float ss = sumsq[0];
    if (!isfinite(ss)) {  // inf / nan gradients: leave the parameters alone, report, still clear the grads
      if (blockIdx.x == 0 && threadIdx.x == 0 && skipped != nullptr) atomicAdd(skipped, 1);
      if (a.zero_grad)
        for (long long i = tid; i < n; i += threads) g[i] = 0.f;
      return;
    }
    if (a.max_norm > 0.f) {
      const float norm = sqrtf(ss) * a.grad_scale;
      clip = fminf(1.0f, a.max_norm / (norm + 1.0e-6f));
    }
  }
  const float gs = a.grad_scale * clip;
  const float inv_bc1 = 1.0f / a.bias_corr1;
  const float inv_sqrt_bc2 = rsqrtf(a.bias_corr2);
  const long long n4 = VEC ? n / 4 : 0;
  if constexpr (VEC) {
    constexpr int U = 2;
    for (long long base = (blockIdx.x * static_cast<long long>(blockDim.x)) * U + threadIdx.x; base < n4; base += threads * U) {
      float4 pv[U], mv[U], vv[U], gv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long i = base + u * blockDim.x;
        if (i < n4) {
          pv[u] = reinterpret_cast<const float4*>(p)[i];
          mv[u] = reinterpret_cast<const float4*>(m)[i];
          vv[u] = reinterpret_cast<const float4*>(v)[i];
          gv[u] = reinterpret_cast<const float4*>(g)[i];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long i = base + u * blockDim.x;
        if (i >= n4) break;
        const long long left = a.wd_end - 4 * i;  // the decayed part may end inside the vector
        adam_element(pv[u].x, mv[u].x, vv[u].x, gv[u].x, a, gs, inv_bc1, inv_sqrt_bc2, left > 0 ? a.weight_decay : 0.f);
        adam_element(pv[u].y, mv[u].y, vv[u].y, gv[u].y, a, gs, inv_bc1, inv_sqrt_bc2, left > 1 ? a.weight_decay : 0.f);
        adam_element(pv[u].z, mv[u].z, vv[u].z, gv[u].z, a, gs, inv_bc1, inv_sqrt_bc2, left > 2 ? a.weight_decay : 0.f);
        adam_element(pv[u].w, mv[u].w, vv[u].w, gv[u].w, a, gs, inv_bc1, inv_sqrt_bc2, left > 3 ? a.weight_decay : 0.f);
        reinterpret_cast<float4*>(p)[i] = pv[u];
        reinterpret_cast<float4*>(m)[i] = mv[u];
        reinterpret_cast<float4*>(v)[i] = vv[u];
        reinterpret_cast<uint2*>(p16)[i] = make_uint2(pack_bf16x2(pv[u].x, pv[u].y), pack_bf16x2(pv[u].z, pv[u].w));
        if (a.zero_grad) reinterpret_cast<float4*>(g)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  }
  for (long long i = 4 * n4 + tid; i < n; i += threads) {
    float pi = p[i], mi = m[i], vi = v[i];
    adam_element(pi, mi, vi, g[i], a, gs, inv_bc1, inv_sqrt_bc2, i < a.wd_end ? a.weight_decay : 0.f);
    p[i] = pi;
    m[i] = mi;
    v[i] = vi;
    p16[i] = __float2bfloat16(pi);
    if (a.zero_grad) g[i] = 0.f;
  }
}

struct SgdArgs {
  float lr, momentum, weight_decay, grad_scale, max_norm;
  long long wd_end;
  int zero_grad, first_step;
};

__global__ void __launch_bounds__(256)
sgd_kernel(float* __restrict__ p, float* __restrict__ mom, float* __restrict__ g, __nv_bfloat16* __restrict__ p16,
           long long n, const float* __restrict__ sumsq, int* __restrict__ skipped, SgdArgs a) {
  float clip = 1.0f;
  if (sumsq != nullptr) {
    const float ss = sumsq[0];
    if (!isfinite(ss)) {
      if (blockIdx.x == 0 && threadIdx.x == 0 && skipped != nullptr) atomicAdd(skipped, 1);
      if (a.zero_grad)
        for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
             i += static_cast<long long>(gridDim.x) * blockDim.x)
          g[i] = 0.f;
      return;
    }
    if (a.max_norm > 0.f) clip = fminf(1.0f, a.max_norm / (sqrtf(ss) * a.grad_scale + 1.0e-6f));
  }
  const float gs = a.grad_scale * clip;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float pi = p[i];
    float gi = g[i] * gs + (i < a.wd_end ? a.weight_decay : 0.f) * pi;
    float bi = a.first_step ? gi : a.momentum * mom[i] + gi;
    mom[i] = bi;
    pi -= a.lr * bi;
    p[i] = pi;
    p16[i] = __float2bfloat16(pi);
    if (a.zero_grad) g[i] = 0.f;
  }
}

}  // namespace

constexpr int kSumsqBlocks = 1024;

// partials: scratch of kSumsqBlocks floats.  out[0] (+)= sum g^2.
int sumsq_launch(const float* g, long long n, float* partials, float* out, int accumulate, cudaStream_t stream) {
  long long want = (n / 4 + 255) / 256;
  const int blocks = static_cast<int>(want < 1 ? 1 : (want > kSumsqBlocks ? kSumsqBlocks : want));
  sumsq_partial_kernel<<<blocks, 256, 0, stream>>>(g, n, partials);
  sumsq_fold_kernel<<<1, 256, 0, stream>>>(partials, blocks, out, accumulate);
  return static_cast<int>(cudaGetLastError());
}

int adam_launch(float* p, float* m, float* v, float* g, void* p16, long long n, const float* sumsq, int* skipped,
                float lr, float beta1, float beta2, float eps, float weight_decay, int step, float grad_scale,
                float max_norm, long long wd_end, int zero_grad, int num_sms, cudaStream_t stream) {
  AdamArgs a;
  a.lr = lr; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.weight_decay = weight_decay;
  a.bias_corr1 = 1.0f - powf(beta1, static_cast<float>(step));
  a.bias_corr2 = 1.0f - powf(beta2, static_cast<float>(step));
  a.grad_scale = grad_scale; a.max_norm = max_norm; a.wd_end = wd_end; a.zero_grad = zero_grad;
  auto* out16 = reinterpret_cast<__nv_bfloat16*>(p16);
  const uintptr_t low = reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v) |
                        reinterpret_cast<uintptr_t>(g) | (reinterpret_cast<uintptr_t>(p16) * 2);
  // Small buffers are a matter of latency: an element a thread, 16384 elements 2.3 us against 3.0 with vectors, 100000 2.9
  // against 3.3, 200000 3.3 against 3.2.
  const bool vec = (low & 15) == 0 && n > num_sms * 1024LL;
  const long long per_block = vec ? 2048 : 256;   // elements of one block's pass
  const long long want = (n + per_block - 1) / per_block;
  // Eight vector blocks are resident on an SM: no more of them while most of the data fits the L2, 4 M elements 16.0 us against
  // 17.2 with sixteen (an element a thread 16.4), 5 M 24.5 against 26.3; at 400 M sixteen are the better ones by 0.2 %.
  const long long cap = num_sms * (vec && n <= (1 << 24) ? 8LL : 16LL);
  const int blocks = static_cast<int>(want < 1 ? 1 : (want > cap ? cap : want));
  if (vec)
    adam_kernel<true><<<blocks, 256, 0, stream>>>(p, m, v, g, out16, n, sumsq, skipped, a);
  else
    adam_kernel<false><<<blocks, 256, 0, stream>>>(p, m, v, g, out16, n, sumsq, skipped, a);
  return static_cast<int>(cudaGetLastError());
}

int sgd_launch(float* p, float* mom, float* g, void* p16, long long n, const float* sumsq, int* skipped, float lr,
               float momentum, float weight_decay, float grad_scale, float max_norm, long long wd_end, int zero_grad,
               int first_step, int num_sms, cudaStream_t stream) {
  SgdArgs a;
  a.lr = lr; a.momentum = momentum; a.weight_decay = weight_decay; a.grad_scale = grad_scale; a.max_norm = max_norm;
  a.wd_end = wd_end; a.zero_grad = zero_grad; a.first_step = first_step;
  long long want = (n + 255) / 256;
  const int blocks = static_cast<int>(want < 1 ? 1 : (want > num_sms * 16LL ? num_sms * 16LL : want));
  sgd_kernel<<<blocks, 256, 0, stream>>>(p, mom, g, reinterpret_cast<__nv_bfloat16*>(p16), n, sumsq, skipped, a);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ssb
