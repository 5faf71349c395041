// Flat-buffer AdamW and gradient-norm kernels for the sharded optimizer.
// Replaces torch.optim.AdamW + clip_grad_norm_ of the reference (siirl/engine/fsdp_workers.py:1022-1088,
// siirl/engine/actor/dp_actor.py:265-283).  All parameters of a model live in one flat bf16 buffer with an fp32
// gradient buffer beside it; each rank owns a contiguous shard of fp32 master weights and Adam moments.
//   sumsq_kernel    partial sum of squares of an fp32 range -> one float (atomicAdd), for the global grad norm
//   adamw_kernel    p_master, m, v update on the owned shard with the clip factor read from device memory
//                   (no host sync), writes the bf16 working copy; a non-finite norm skips the update,
//                   as the reference does.
#include "common.cuh"
#include "launchers.h"

namespace sb {

__global__ void sumsq_kernel(const float* __restrict__ g, long long n, float* __restrict__ out) {
  float s = 0.f;
  const long long n4 = n / 4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const float4 v = reinterpret_cast<const float4*>(g)[i];
    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const float v = g[n4 * 4 + threadIdx.x];
    s += v * v;
  }
  __shared__ float red[32];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    t = warp_sum(t);
    if (threadIdx.x == 0) atomicAdd(out, t);
  }
}

struct AdamParams {
  float* master;           // fp32 [n] owned shard
  float* m;
  float* v;
  const float* grad;       // fp32 [n] (already reduced over data-parallel ranks)
  __nv_bfloat16* param;    // bf16 [n] working copy of the shard
  const float* sumsq;      // device scalar: global sum of squared gradients (before grad_scale)
  float* grad_norm_out;    // optional device scalar receiving the norm
  long long n;
  float lr, beta1, beta2, eps, weight_decay, bc1, bc2, max_norm, grad_scale;
};

__device__ __forceinline__ void adamw_element(const AdamParams& p, float gs, float g, float& w, float& m, float& v) {
  g *= gs;
  m = p.beta1 * m + (1.f - p.beta1) * g;
  v = p.beta2 * v + (1.f - p.beta2) * g * g;
  w -= p.lr * p.weight_decay * w;
  w -= p.lr * (m / p.bc1) / (sqrtf(v / p.bc2) + p.eps);
}

// Bound by HBM: 16 bytes read and 14 written per parameter.  VEC = 4 moves 16 bytes per load (64 in flight per thread)
// and marks them as read once, so that they do not push the weights out of L2; one element per thread kept only 32 KB
// per SM in flight.  A block's piece is contiguous and small (64 blocks per SM): eight streams at distances that change with
// every block spread better over the memory than in lockstep sweeps.  512 M parameters: one element per thread 5.28 ms (3.0
// TB/s); 16 bytes in sweeps of 8 blocks per SM 3.55 ms, of 64 3.24 ms; in pieces 3.21 ms (5.0 TB/s).
// VEC = 1 serves shards whose start is no multiple of four elements, and the last n % 4 elements.
template <int VEC>
__global__ void __launch_bounds__(256) adamw_kernel(AdamParams p) {
  float clip = 1.f;
  bool skip = false;
  if (p.sumsq) {
    const float norm = sqrtf(*p.sumsq) * p.grad_scale;
    if (!isfinite(norm)) skip = true;
    else if (p.max_norm > 0.f) clip = fminf(1.f, p.max_norm / (norm + 1e-6f));
    if (p.grad_norm_out && blockIdx.x == 0 && threadIdx.x == 0) *p.grad_norm_out = norm;
  }
  if (skip) return;
  const float gs = p.grad_scale * clip;
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  const long long nv = VEC == 4 ? p.n / 4 : 0;
  const long long piece = ((nv + gridDim.x - 1) / gridDim.x + 255) / 256 * 256;
  const long long end = min(nv, piece * (blockIdx.x + 1));
  for (long long i = piece * blockIdx.x + threadIdx.x; i < end; i += 256) {
    const float4 g = __ldcs(reinterpret_cast<const float4*>(p.grad) + i);
    float4 w = __ldcs(reinterpret_cast<const float4*>(p.master) + i);
    float4 m = __ldcs(reinterpret_cast<const float4*>(p.m) + i);
    float4 v = __ldcs(reinterpret_cast<const float4*>(p.v) + i);
    adamw_element(p, gs, g.x, w.x, m.x, v.x);
    adamw_element(p, gs, g.y, w.y, m.y, v.y);
    adamw_element(p, gs, g.z, w.z, m.z, v.z);
    adamw_element(p, gs, g.w, w.w, m.w, v.w);
    __stcs(reinterpret_cast<float4*>(p.m) + i, m);
    __stcs(reinterpret_cast<float4*>(p.v) + i, v);
    __stcs(reinterpret_cast<float4*>(p.master) + i, w);
    reinterpret_cast<uint2*>(p.param)[i] = make_uint2(pack_bf16x2(w.x, w.y), pack_bf16x2(w.z, w.w));
  }
  for (long long i = nv * 4 + first; i < p.n; i += step) {
    float w = p.master[i], m = p.m[i], v = p.v[i];
    adamw_element(p, gs, p.grad[i], w, m, v);
    p.m[i] = m;
    p.v[i] = v;
    p.master[i] = w;
    p.param[i] = __float2bfloat16(w);
  }
}

__global__ void cast_f32_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16(src[i]);
}

}  // namespace sb

using namespace sb;

static int grid_cap(long long work, int threads, int per_sm) {
  long long b = (work + threads - 1) / threads;
  const long long cap = (long long)num_sms() * per_sm;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

extern "C" int sb_sumsq_accumulate(const float* g, long long n, float* out, cudaStream_t stream) {
  if (n == 0) return 0;
  sumsq_kernel<<<grid_cap(n / 4 + 1, 256, 8), 256, 0, stream>>>(g, n, out);
  return (int)cudaGetLastError();
}

extern "C" int sb_adamw_step(float* master, float* m, float* v, const float* grad, void* param_bf16,
                             const float* sumsq, float* grad_norm_out, long long n, float lr, float beta1,
                             float beta2, float eps, float weight_decay, int step, float max_norm, float grad_scale,
                             cudaStream_t stream) {
  if (n == 0) return 0;
  AdamParams p;
  p.master = master; p.m = m; p.v = v; p.grad = grad; p.param = (__nv_bfloat16*)param_bf16;
  p.sumsq = sumsq; p.grad_norm_out = grad_norm_out; p.n = n;
  p.lr = lr; p.beta1 = beta1; p.beta2 = beta2; p.eps = eps; p.weight_decay = weight_decay;
  p.bc1 = 1.f - powf(beta1, (float)step);
  p.bc2 = 1.f - powf(beta2, (float)step);
  p.max_norm = max_norm; p.grad_scale = grad_scale;
  const uintptr_t all = (uintptr_t)master | (uintptr_t)m | (uintptr_t)v | (uintptr_t)grad | ((uintptr_t)param_bf16 << 1);
  if ((all & 15) == 0) adamw_kernel<4><<<grid_cap(n / 4 + 1, 256, 64), 256, 0, stream>>>(p);
  else adamw_kernel<1><<<grid_cap(n, 256, 8), 256, 0, stream>>>(p);
  return (int)cudaGetLastError();
}

extern "C" int sb_cast_f32_bf16(const float* src, void* dst, long long n, cudaStream_t stream) {
  if (n == 0) return 0;
  cast_f32_bf16_kernel<<<grid_cap(n, 256, 8), 256, 0, stream>>>(src, (__nv_bfloat16*)dst, n);
  return (int)cudaGetLastError();
}
