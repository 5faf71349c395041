// Memory-bound transformer ops for packed [tokens, hidden] bf16 activations:
// RMSNorm (+residual) fwd/bwd, RoPE / mrope, SwiGLU fwd/bwd, embedding gather / scatter-add,
// dtype casts.  They replace apex fused_rms_norm_affine, flash-attn's rotary and the eager HF
// activation code the reference runs (siirl/models/llama/megatron/layers/parallel_rmsnorm.py:18-48,
// siirl/models/transformers/qwen2.py).  All loads/stores are 16-byte vectors; fp32 math.
#include "common.cuh"
#include "launchers.h"

namespace sb {

__device__ __forceinline__ void bf16x8_to_float(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 float_to_bf16x8(const float (&f)[8]) {
  uint4 o;
  o.x = pack_bf16x2(f[0], f[1]);
  o.y = pack_bf16x2(f[2], f[3]);
  o.z = pack_bf16x2(f[4], f[5]);
  o.w = pack_bf16x2(f[6], f[7]);
  return o;
}

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < THREADS / 32) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}

// ---------------------------------------------------------------------------------------
// RMSNorm forward:  h = x (+ residual);  y = h * rsqrt(mean(h^2) + eps) * w
// x may also be the fp32 partial sums of a split contraction (`slabs`), added up here: a pass of their own over so few
// rows costs a launch (2.9 us against some 0.3 us of memory time for 8 x 896) and a rounding.
// Bound by memory.  All of a row's loads come before its first store, and the weights before the rows: the compiler may not
// move them across a store by itself (9600 x 3584: 66 us with the stores of the sum in between, 46 us so).  Rows of up to
// 2048 columns: eight blocks on an SM, as many as the grid has (9600 x 1024 with six: 17.7 us, with eight 14.7).  Partial sums
// have at most 512 rows, for which four blocks are enough, and want the registers for loads in flight (8 x 896, 8 slabs:
// 3.1 us with eight blocks, 2.3 with three; 500 x 896, 3 slabs, 3.4 and 3.6, the rows beyond three blocks coming last).
// ---------------------------------------------------------------------------------------
constexpr int kNormThreads = 256;
constexpr int kNormMaxChunks = 4;  // hidden <= 256 * 8 * 4 = 8192

template <int CH, bool SLABS>
__global__ void __launch_bounds__(kNormThreads, CH == 1 ? (SLABS ? 4 : 8) : CH == 2 && !SLABS ? 4 : 2)
rmsnorm_fwd_kernel(const __nv_bfloat16* x, const float* slabs, long long slab_stride, int splits,
                   const __nv_bfloat16* residual, const __nv_bfloat16* w, __nv_bfloat16* y, __nv_bfloat16* h_out,
                   float* rstd_out, int T, int H, float eps) {
  __shared__ float red[32];
  chain_sync();
  const int nvec = H / 8;
  uint4 w4[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int vi = threadIdx.x + c * kNormThreads;
    if (vi < nvec) w4[c] = reinterpret_cast<const uint4*>(w)[vi];
  }
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    float hv[CH][8];
    uint4 x4[CH], r4[CH];
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int vi = threadIdx.x + c * kNormThreads;
      if (vi < nvec) {
        if (SLABS) slab_sum8(slabs + (size_t)row * H + vi * 8, slab_stride, splits, hv[c]);
        else x4[c] = reinterpret_cast<const uint4*>(x + (size_t)row * H)[vi];
        if (residual) r4[c] = reinterpret_cast<const uint4*>(residual + (size_t)row * H)[vi];
      }
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int vi = threadIdx.x + c * kNormThreads;
      if (vi < nvec) {
        if (!SLABS) bf16x8_to_float(x4[c], hv[c]);
        if (residual) {
          float rv[8];
          bf16x8_to_float(r4[c], rv);
#pragma unroll
          for (int i = 0; i < 8; ++i) hv[c][i] += rv[i];
          if (h_out) {
            uint4 o = float_to_bf16x8(hv[c]);
            reinterpret_cast<uint4*>(h_out + (size_t)row * H)[vi] = o;
            // keep the math consistent with what backward will re-read
            bf16x8_to_float(o, hv[c]);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += hv[c][i] * hv[c][i];
      }
    }
    const float tot = block_sum<kNormThreads>(ss, red);
    const float rstd = rsqrtf(tot / (float)H + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int vi = threadIdx.x + c * kNormThreads;
      if (vi < nvec) {
        float wv[8], o[8];
        bf16x8_to_float(w4[c], wv);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = hv[c][i] * rstd * wv[i];
        reinterpret_cast<uint4*>(y + (size_t)row * H)[vi] = float_to_bf16x8(o);
      }
    }
  }
}

// RMSNorm backward.  dx = rstd * (g - xhat * mean(g * xhat)),  g = dy * w,  xhat = h * rstd.
// dx is optionally added to `dres` (gradient arriving through the residual branch).
// Per-block partial dw rows go to dw_partial[gridDim.x, H]; a second kernel folds them into fp32 dw.
// THREADS 128: rows of at most 1024 columns, four blocks per SM (9600 x 896: 256 threads, two blocks, 38 us).
template <int THREADS, int CH>
__global__ void __launch_bounds__(THREADS)
rmsnorm_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* h, const __nv_bfloat16* w, const float* rstd,
                   const __nv_bfloat16* dres, __nv_bfloat16* dx, float* dw_partial, int T, int H) {
  __shared__ float red[32];
  chain_sync();
  const int nvec = H / 8;
  float dwacc[CH][8];
  float wv[CH][8];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int vi = threadIdx.x + c * THREADS;
#pragma unroll
    for (int i = 0; i < 8; ++i) dwacc[c][i] = 0.f;
    if (vi < nvec) bf16x8_to_float(reinterpret_cast<const uint4*>(w)[vi], wv[c]);
  }
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    const float rs = rstd[row];
    float g[CH][8], xh[CH][8];
    float dot = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int vi = threadIdx.x + c * THREADS;
      if (vi < nvec) {
        float dyv[8], hv[8];
        bf16x8_to_float(reinterpret_cast<const uint4*>(dy + (size_t)row * H)[vi], dyv);
        bf16x8_to_float(reinterpret_cast<const uint4*>(h + (size_t)row * H)[vi], hv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          xh[c][i] = hv[i] * rs;
          g[c][i] = dyv[i] * wv[c][i];
          dot += g[c][i] * xh[c][i];
          dwacc[c][i] += dyv[i] * xh[c][i];
        }
      }
    }
    const float mean = block_sum<THREADS>(dot, red) / (float)H;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int vi = threadIdx.x + c * THREADS;
      if (vi < nvec) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = rs * (g[c][i] - xh[c][i] * mean);
        if (dres) {
          float rv[8];
          bf16x8_to_float(reinterpret_cast<const uint4*>(dres + (size_t)row * H)[vi], rv);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += rv[i];
        }
        reinterpret_cast<uint4*>(dx + (size_t)row * H)[vi] = float_to_bf16x8(o);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int vi = threadIdx.x + c * THREADS;
    if (vi < nvec) {
      float4* dst = reinterpret_cast<float4*>(dw_partial + (size_t)blockIdx.x * H + (size_t)vi * 8);
      dst[0] = make_float4(dwacc[c][0], dwacc[c][1], dwacc[c][2], dwacc[c][3]);
      dst[1] = make_float4(dwacc[c][4], dwacc[c][5], dwacc[c][6], dwacc[c][7]);
    }
  }
}

// out[col] (+)= sum of `rows` partial rows.  32 columns and 8 groups of rows per block: with one thread per column the chain
// of 296 dependent additions took 11.5 us for 896 columns.
__global__ void __launch_bounds__(256) colsum_accumulate_kernel(const float* partial, float* out, int rows, int H,
                                                                int accumulate) {
  chain_sync();
  __shared__ float red[8][33];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, col = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (col < H) {
#pragma unroll 4
    for (int r = grp; r < rows; r += 8) s += partial[(size_t)r * H + col];
  }
  red[grp][lane] = s;
  __syncthreads();
  if (grp == 0 && col < H) {
#pragma unroll
    for (int i = 1; i < 8; ++i) s += red[i][lane];
    out[col] = accumulate ? out[col] + s : s;
  }
}

// partial[block, :] = column sums of this block's rows of a bf16 matrix [T, N] (bias gradients); eight columns per thread
__global__ void __launch_bounds__(128) colsum_rows_kernel(const __nv_bfloat16* x, float* partial, int T, int N) {
  chain_sync();
  const int v = blockIdx.x * 128 + threadIdx.x;
  if (v >= N / 8) return;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
  for (int t = blockIdx.y; t < T; t += gridDim.y) {
    float f[8];
    bf16x8_to_float(reinterpret_cast<const uint4*>(x + (size_t)t * N)[v], f);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += f[i];
  }
  float4* dst = reinterpret_cast<float4*>(partial + (size_t)blockIdx.y * N + (size_t)v * 8);
  dst[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
  dst[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

// out += sum over `splits` slabs (weight gradients of split contractions)
__global__ void __launch_bounds__(256) slab_accumulate_kernel(const float* slabs, long long slab_stride, int splits, float* out,
                                                              long long n4) {
  chain_sync();
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n4; i += gridDim.x * 256ll) {
    float4 a = reinterpret_cast<const float4*>(out)[i];
#pragma unroll 4
    for (int s = 0; s < splits; ++s) {
      const float4 b = reinterpret_cast<const float4*>(slabs + s * slab_stride)[i];
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    reinterpret_cast<float4*>(out)[i] = a;
  }
}

// ---------------------------------------------------------------------------------------
// RoPE (rotate-half / "neox" layout) applied in place to the q and k parts of a packed qkv row.
// cos/sin come from a [max_pos, D/2] fp32 table.  `pos` is [rows_of_pos, T]; with 3 rows
// (t, h, w — Qwen2-VL mrope) frequency index i uses row 0 below sec0, row 1 below sec1, else row 2.
// `sign` = +1 forward, -1 backward (inverse rotation = gradient).
// ---------------------------------------------------------------------------------------
__global__ void rope_kernel(__nv_bfloat16* __restrict__ qkv, const int* __restrict__ pos,
                            const float* __restrict__ cos_tab, const float* __restrict__ sin_tab, int T,
                            int row_stride, int n_heads_rot, int D, int pos_rows, int sec0, int sec1,
                            float sign) {
  const int half = D / 2;
  const int pairs_per_tok = n_heads_rot * half;
  const long long total = (long long)T * pairs_per_tok;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / pairs_per_tok);
    const int r = (int)(idx % pairs_per_tok);
    const int head = r / half, i = r % half;
    int prow = 0;
    if (pos_rows == 3) prow = (i < sec0) ? 0 : (i < sec1 ? 1 : 2);
    const int pidx = pos[(size_t)prow * T + t];
    const float c = cos_tab[(size_t)pidx * half + i];
    const float s = sign * sin_tab[(size_t)pidx * half + i];
    __nv_bfloat16* base = qkv + (size_t)t * row_stride + (size_t)head * D;
    const float a = __bfloat162float(base[i]);
    const float b = __bfloat162float(base[i + half]);
    base[i] = __float2bfloat16(a * c - b * s);
    base[i + half] = __float2bfloat16(b * c + a * s);
  }
}

// The same from one buffer to another, whole rows: a copy followed by rotation in place read and wrote every row twice, and
// the scalar form spent its time on 64-bit divisions: 18400 rows of 28 + 4 + 4 heads of 128 took 243 us, now 68 (5.0 TB/s);
// 9600 rows of 14 + 2 + 2 heads of 64 40 us, now 15.  One thread takes 8 pairs of a rotated head, or 16 columns that are copied.  D % 16 == 0, 16-byte rows.
__global__ void __launch_bounds__(256) rope_rows_kernel(const __nv_bfloat16* in, __nv_bfloat16* out, const int* pos,
                                                        const float* cos_tab, const float* sin_tab, int T, int row_stride,
                                                        int n_heads_rot, int D, int pos_rows, int sec0, int sec1, float sign) {
  chain_sync();
  const int half = D / 2;
  const unsigned units = row_stride / 16, total = (unsigned)T * units;  // below 2^31: checked by the caller
  for (unsigned idx = blockIdx.x * 256 + threadIdx.x; idx < total; idx += gridDim.x * 256) {
    const unsigned t = idx / units, u = idx % units;
    const __nv_bfloat16* src = in + (size_t)t * row_stride;
    __nv_bfloat16* dst = out + (size_t)t * row_stride;
    const int head = u * 16 / D, i0 = (u * 16 % D) / 2;
    const bool rot = head < n_heads_rot;
    const int lo = rot ? head * D + i0 : u * 16, hi = rot ? lo + half : lo + 8;
    uint4 a4 = *reinterpret_cast<const uint4*>(src + lo), b4 = *reinterpret_cast<const uint4*>(src + hi);
    if (rot) {
      float a[8], b[8], c[8], s[8];
      bf16x8_to_float(a4, a);
      bf16x8_to_float(b4, b);
      if (pos_rows == 3) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int i = i0 + k, prow = i < sec0 ? 0 : (i < sec1 ? 1 : 2);
          const size_t at = (size_t)pos[(size_t)prow * T + t] * half + i;
          c[k] = cos_tab[at];
          s[k] = sin_tab[at];
        }
      } else {
        const size_t at = (size_t)pos[t] * half + i0;
#pragma unroll
        for (int k = 0; k < 8; k += 4) {
          const float4 cv = *reinterpret_cast<const float4*>(cos_tab + at + k);
          const float4 sv = *reinterpret_cast<const float4*>(sin_tab + at + k);
          c[k] = cv.x; c[k + 1] = cv.y; c[k + 2] = cv.z; c[k + 3] = cv.w;
          s[k] = sv.x; s[k + 1] = sv.y; s[k + 2] = sv.z; s[k + 3] = sv.w;
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float sk = sign * s[k], x = a[k];
        a[k] = x * c[k] - b[k] * sk;
        b[k] = b[k] * c[k] + x * sk;
      }
      a4 = float_to_bf16x8(a);
      b4 = float_to_bf16x8(b);
    }
    *reinterpret_cast<uint4*>(dst + lo) = a4;
    *reinterpret_cast<uint4*>(dst + hi) = b4;
  }
}

// ---------------------------------------------------------------------------------------
// SwiGLU on a fused gate|up projection: gu is [T, 2*I] with gate in columns [0,I), up in [I,2I).
// ---------------------------------------------------------------------------------------
// Bound by memory.  Two-dimensional grids (a flat one pays a 64-bit division per vector) and two rows in flight per thread:
// 24000 x 2 * 18944 forward 569 -> 488 us (5.6 TB/s), backward 800 -> 711 us (6.4 TB/s); 9600 x 2 * 4864: 65 -> 61, 91 -> 81.
constexpr int kSwigluThreads = 128;

// First row, step between rows and column of a thread.  NARROW: rows whose columns would leave a quarter of whole blocks idle
// are divided evenly over blocks, and short ones share a block (9600 x 2 * 264: forward 6.9 -> 4.8 us, backward 7.9 -> 5.3).
struct SwigluAt {
  int t, step, v;
};
template <bool NARROW>
__device__ __forceinline__ SwigluAt swiglu_at(int width) {
  if (!NARROW) return {(int)blockIdx.y, (int)gridDim.y, (int)(blockIdx.x * kSwigluThreads + threadIdx.x)};
  const int rows = blockDim.x / width, row = threadIdx.x / width;
  return {(int)blockIdx.y * rows + row, (int)gridDim.y * rows, (int)blockIdx.x * width + (int)threadIdx.x - row * width};
}

__device__ __forceinline__ void swiglu_vec(const uint4& gv, const uint4& uv, uint4* dst) {
  float g[8], u[8], o[8];
  bf16x8_to_float(gv, g);
  bf16x8_to_float(uv, u);
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = g[i] / (1.f + __expf(-g[i])) * u[i];
  *dst = float_to_bf16x8(o);
}

template <bool NARROW>
__global__ void __launch_bounds__(kSwigluThreads) swiglu_fwd_kernel(const __nv_bfloat16* gu, __nv_bfloat16* out, int T, int I,
                                                                    int width) {
  chain_sync();
  const SwigluAt at = swiglu_at<NARROW>(width);
  const int nvec = I / 8, v = at.v;
  if (v >= nvec) return;
  const uint4* src = reinterpret_cast<const uint4*>(gu) + v;
  uint4* dst = reinterpret_cast<uint4*>(out) + v;
  const size_t pitch = 2 * (size_t)nvec;
  for (int t = at.t; t < T; t += 2 * at.step) {
    const int t1 = t + at.step;
    const bool two = t1 < T;
    const uint4 g0 = src[t * pitch], u0 = src[t * pitch + nvec];
    uint4 g1 = g0, u1 = u0;
    if (two) {
      g1 = src[t1 * pitch];
      u1 = src[t1 * pitch + nvec];
    }
    swiglu_vec(g0, u0, dst + (size_t)t * nvec);
    if (two) swiglu_vec(g1, u1, dst + (size_t)t1 * nvec);
  }
}

// the same of a split contraction's partial sums: fp32 slabs [T, 2*I]
__global__ void swiglu_slabs_kernel(const float* slabs, long long slab_stride, int splits, __nv_bfloat16* out, int T, int I) {
  chain_sync();
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= I / 8) return;
  for (int t = blockIdx.y; t < T; t += gridDim.y) {
    float g[8], u[8], o[8];
    slab_sum8(slabs + (size_t)t * 2 * I + v * 8, slab_stride, splits, g);
    slab_sum8(slabs + (size_t)t * 2 * I + I + v * 8, slab_stride, splits, u);
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = g[i] / (1.f + __expf(-g[i])) * u[i];
    reinterpret_cast<uint4*>(out + (size_t)t * I)[v] = float_to_bf16x8(o);
  }
}

__device__ __forceinline__ void swiglu_grad_vec(const uint4& gv, const uint4& uv, const uint4& dv, uint4* dg_dst, uint4* du_dst) {
  float g[8], u[8], d[8], dg[8], du[8];
  bf16x8_to_float(gv, g);
  bf16x8_to_float(uv, u);
  bf16x8_to_float(dv, d);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float sig = 1.f / (1.f + __expf(-g[i]));
    const float silu = g[i] * sig;
    dg[i] = d[i] * u[i] * (sig + silu * (1.f - sig));
    du[i] = d[i] * silu;
  }
  *dg_dst = float_to_bf16x8(dg);
  *du_dst = float_to_bf16x8(du);
}

template <bool NARROW>
__global__ void __launch_bounds__(kSwigluThreads) swiglu_bwd_kernel(const __nv_bfloat16* gu, const __nv_bfloat16* dout,
                                                                    __nv_bfloat16* dgu, int T, int I, int width) {
  chain_sync();
  const SwigluAt at = swiglu_at<NARROW>(width);
  const int nvec = I / 8, v = at.v;
  if (v >= nvec) return;
  const uint4 *src = reinterpret_cast<const uint4*>(gu) + v, *d = reinterpret_cast<const uint4*>(dout) + v;
  uint4* dst = reinterpret_cast<uint4*>(dgu) + v;
  const size_t pitch = 2 * (size_t)nvec;
  for (int t = at.t; t < T; t += 2 * at.step) {
    const int t1 = t + at.step;
    const bool two = t1 < T;
    const uint4 g0 = src[t * pitch], u0 = src[t * pitch + nvec], d0 = d[(size_t)t * nvec];
    uint4 g1 = g0, u1 = u0, d1 = d0;
    if (two) {
      g1 = src[t1 * pitch];
      u1 = src[t1 * pitch + nvec];
      d1 = d[(size_t)t1 * nvec];
    }
    swiglu_grad_vec(g0, u0, d0, dst + t * pitch, dst + t * pitch + nvec);
    if (two) swiglu_grad_vec(g1, u1, d1, dst + t1 * pitch, dst + t1 * pitch + nvec);
  }
}

// ---------------------------------------------------------------------------------------
// Embedding gather and its gradient (fp32 scatter-add into the main-grad buffer).
// ---------------------------------------------------------------------------------------
SB_BOUNDS_WORD_DEFINE(elementwise)

__global__ void embedding_fwd_kernel(const long long* ids, const __nv_bfloat16* table, __nv_bfloat16* out, int T, int H,
                                     int V) {
  chain_sync();
  const int nvec = H / 8;
  const long long total = (long long)T * nvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / nvec), v = (int)(idx % nvec);
    long long id = ids[t];
    SB_CHECK_INDEX(id, V, 1);
    id = id < 0 ? 0 : (id >= V ? V - 1 : id);
    reinterpret_cast<uint4*>(out + (size_t)t * H)[v] = reinterpret_cast<const uint4*>(table + (size_t)id * H)[v];
  }
}

__global__ void embedding_bwd_kernel(const long long* __restrict__ ids, const __nv_bfloat16* __restrict__ dout,
                                     float* __restrict__ dtable, int T, int H, int V) {
  const int nvec = H / 8;
  const long long total = (long long)T * nvec;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / nvec), v = (int)(idx % nvec);
    long long id = ids[t];
    SB_CHECK_INDEX(id, V, 2);
    if (id < 0 || id >= V) continue;
    float d[8];
    bf16x8_to_float(reinterpret_cast<const uint4*>(dout + (size_t)t * H)[v], d);
    float* dst = dtable + (size_t)id * H + (size_t)v * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) atomicAdd(dst + i, d[i]);
  }
}

// out[i] = bf16(a[i] + b[i])  (residual adds outside the norm kernels)
__global__ void add_bf16_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                __nv_bfloat16* __restrict__ out, long long nvec) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < nvec;
       idx += (long long)gridDim.x * blockDim.x) {
    float x[8], y[8];
    bf16x8_to_float(reinterpret_cast<const uint4*>(a)[idx], x);
    bf16x8_to_float(reinterpret_cast<const uint4*>(b)[idx], y);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] += y[i];
    reinterpret_cast<uint4*>(out)[idx] = float_to_bf16x8(x);
  }
}

static inline int grid_for(long long work, int threads, int per_sm = 8) {
  long long blocks = (work + threads - 1) / threads;
  long long cap = (long long)num_sms() * per_sm;
  return (int)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

}  // namespace sb

using namespace sb;

static int rmsnorm_fwd(const void* x, const float* slabs, long long slab_stride, int splits, const void* residual,
                       const void* w, void* y, void* h_out, float* rstd, int T, int H, float eps, cudaStream_t stream) {
  if (H % 8 || H > kNormThreads * 8 * kNormMaxChunks) return -3;
  if (T == 0) return 0;
  const int ch = (H / 8 + kNormThreads - 1) / kNormThreads;
  const int grid = T < num_sms() * 8 ? T : num_sms() * 8;
#define SB_LAUNCH(CH)                                                                                     \
  return launch_chained(slabs ? rmsnorm_fwd_kernel<CH, true> : rmsnorm_fwd_kernel<CH, false>, grid, kNormThreads, 0, stream, \
      (const __nv_bfloat16*)x, slabs, slab_stride, splits, (const __nv_bfloat16*)residual,                  \
      (const __nv_bfloat16*)w, (__nv_bfloat16*)y, (__nv_bfloat16*)h_out, rstd, T, H, eps)
  switch (ch) {
    case 1: SB_LAUNCH(1);
    case 2: SB_LAUNCH(2);
    case 3: SB_LAUNCH(3);
    default: SB_LAUNCH(4);
  }
#undef SB_LAUNCH
}

extern "C" int sb_rmsnorm_fwd(const void* x, const void* residual, const void* w, void* y, void* h_out,
                              float* rstd, int T, int H, float eps, cudaStream_t stream) {
  return rmsnorm_fwd(x, nullptr, 0, 0, residual, w, y, h_out, rstd, T, H, eps, stream);
}

// x = sum of `splits` fp32 slabs [T, H], slab_stride floats apart
extern "C" int sb_rmsnorm_slabs_fwd(const float* slabs, long long slab_stride, int splits, const void* residual,
                                    const void* w, void* y, void* h_out, int T, int H, float eps, cudaStream_t stream) {
  if (splits < 1 || slab_stride % 4) return -3;
  return rmsnorm_fwd(nullptr, slabs, slab_stride, splits, residual, w, y, h_out, nullptr, T, H, eps, stream);
}

// rows of dw_partial that sb_rmsnorm_bwd writes for T rows of H columns
extern "C" int sb_rmsnorm_bwd_blocks(int T, int H) {
  const int cap = num_sms() * (H <= 1024 ? 4 : 2);
  return T < cap ? (T > 0 ? T : 1) : cap;
}

static int colsum_accumulate(const float* partial, float* out, int rows, int H, int accumulate, cudaStream_t stream) {
  return launch_chained(colsum_accumulate_kernel, (H + 31) / 32, 256, 0, stream, partial, out, rows, H, accumulate);
}

extern "C" int sb_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const void* dres,
                              void* dx, float* dw_partial, float* dw, int dw_accumulate, int T, int H,
                              cudaStream_t stream) {
  if (H % 8 || H > kNormThreads * 8 * kNormMaxChunks) return -3;
  if (T == 0) return 0;
  const int ch = (H / 8 + kNormThreads - 1) / kNormThreads;
  const int grid = sb_rmsnorm_bwd_blocks(T, H);
  int rc;
#define SB_LAUNCH(THREADS, CH)                                                                              \
  rc = launch_chained(rmsnorm_bwd_kernel<THREADS, CH>, grid, THREADS, 0, stream, (const __nv_bfloat16*)dy,  \
                      (const __nv_bfloat16*)h, (const __nv_bfloat16*)w, rstd, (const __nv_bfloat16*)dres,   \
                      (__nv_bfloat16*)dx, dw_partial, T, H)
  if (H <= 1024) SB_LAUNCH(128, 1);
  else if (ch == 1) SB_LAUNCH(kNormThreads, 1);
  else if (ch == 2) SB_LAUNCH(kNormThreads, 2);
  else if (ch == 3) SB_LAUNCH(kNormThreads, 3);
  else SB_LAUNCH(kNormThreads, 4);
#undef SB_LAUNCH
  return rc ? rc : colsum_accumulate(dw_partial, dw, grid, H, dw_accumulate, stream);
}

extern "C" int sb_colsum_blocks(int T) {
  const int rows = (T + 31) / 32;
  return rows < 128 ? (rows > 0 ? rows : 1) : 128;
}

// out[N] (+)= column sums of x [T, N] bf16; partial: fp32 [sb_colsum_blocks(T), N]
extern "C" int sb_colsum_bf16(const void* x, float* partial, float* out, int T, int N, int accumulate, cudaStream_t stream) {
  if (N % 8 || ((uintptr_t)x & 15)) return -3;
  if (N == 0) return 0;
  const int gy = sb_colsum_blocks(T);
  const int rc = launch_chained(colsum_rows_kernel, dim3((N / 8 + 127) / 128, gy), 128, 0, stream, (const __nv_bfloat16*)x,
                                partial, T, N);
  return rc ? rc : colsum_accumulate(partial, out, gy, N, accumulate, stream);
}

// out[n] += sum of `splits` slabs of n floats, slab_stride apart
extern "C" int sb_slab_accumulate(const float* slabs, long long slab_stride, int splits, float* out, long long n,
                                  cudaStream_t stream) {
  if (n % 4 || slab_stride % 4 || ((uintptr_t)out & 15)) return -3;
  if (n == 0) return 0;
  return launch_chained(slab_accumulate_kernel, grid_for(n / 4, 256, 16), 256, 0, stream, slabs, slab_stride, splits, out,
                        n / 4);
}

extern "C" int sb_rope(void* qkv, const int* pos, const float* cos_tab, const float* sin_tab, int T,
                       int row_stride, int n_heads_rot, int D, int pos_rows, int sec0, int sec1, float sign,
                       cudaStream_t stream) {
  if (T == 0) return 0;
  const long long total = (long long)T * n_heads_rot * (D / 2);
  rope_kernel<<<grid_for(total, 256), 256, 0, stream>>>((__nv_bfloat16*)qkv, pos, cos_tab, sin_tab, T, row_stride,
                                                        n_heads_rot, D, pos_rows, sec0, sec1, sign);
  return (int)cudaGetLastError();
}

// all columns; rows in pairs, or as many of them as fill the SMs twice over, or single rows where pairs are too few blocks
struct SwigluGrid {
  dim3 grid;
  int threads, width;  // width 0: the wide form
};
static SwigluGrid swiglu_grid(int T, int I) {
  const int nvec = I / 8, gx = (nvec + kSwigluThreads - 1) / kSwigluThreads;
  const bool narrow = nvec * 4 < gx * kSwigluThreads * 3;
  const int width = (nvec + gx - 1) / gx, rows = narrow ? kSwigluThreads / width : 1;
  const int cap = (num_sms() * 32 + gx - 1) / gx, blocks = (T + rows - 1) / rows, pairs = (blocks + 1) / 2;
  int gy = (long long)gx * pairs < 4 * num_sms() ? blocks : pairs < cap ? pairs : cap;
  if (gy > 65535) gy = 65535;
  return {dim3(gx, gy), narrow ? rows * width : kSwigluThreads, narrow ? width : 0};
}

extern "C" int sb_swiglu_fwd(const void* gu, void* out, int T, int I, cudaStream_t stream) {
  if (I % 8) return -3;
  if (T == 0 || I == 0) return 0;
  const SwigluGrid g = swiglu_grid(T, I);
  return launch_chained(g.width ? swiglu_fwd_kernel<true> : swiglu_fwd_kernel<false>, g.grid, g.threads, 0, stream,
                        (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, T, I, g.width);
}

// out of place, whole rows; -2: a shape for a copy and sb_rope instead
extern "C" int sb_rope_rows(const void* in, void* out, const int* pos, const float* cos_tab, const float* sin_tab, int T,
                            int row_stride, int n_heads_rot, int D, int pos_rows, int sec0, int sec1, float sign,
                            cudaStream_t stream) {
  if (T == 0) return 0;
  const uintptr_t all = (uintptr_t)in | (uintptr_t)out | (uintptr_t)cos_tab | (uintptr_t)sin_tab;
  if (D % 16 || row_stride % 16 || (all & 15) || (long long)n_heads_rot * D > row_stride ||
      (long long)T * (row_stride / 16) >= (1ll << 31) - 1024 * 256 * 8)
    return -2;
  return launch_chained(rope_rows_kernel, grid_for((long long)T * (row_stride / 16), 256), 256, 0, stream,
                        (const __nv_bfloat16*)in, (__nv_bfloat16*)out, pos, cos_tab, sin_tab, T, row_stride, n_heads_rot, D,
                        pos_rows, sec0, sec1, sign);
}

extern "C" int sb_swiglu_slabs_fwd(const float* slabs, long long slab_stride, int splits, void* out, int T, int I,
                                   cudaStream_t stream) {
  if (I % 8 || splits < 1 || slab_stride % 4) return -3;
  if (T == 0) return 0;
  return launch_chained(swiglu_slabs_kernel, dim3((I / 8 + 127) / 128, T < 65535 ? T : 65535), 128, 0, stream, slabs,
                        slab_stride, splits, (__nv_bfloat16*)out, T, I);
}

extern "C" int sb_swiglu_bwd(const void* gu, const void* dout, void* dgu, int T, int I, cudaStream_t stream) {
  if (I % 8) return -3;
  if (T == 0 || I == 0) return 0;
  const SwigluGrid g = swiglu_grid(T, I);
  return launch_chained(g.width ? swiglu_bwd_kernel<true> : swiglu_bwd_kernel<false>, g.grid, g.threads, 0, stream,
                        (const __nv_bfloat16*)gu, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dgu, T, I, g.width);
}

extern "C" int sb_embedding_fwd(const long long* ids, const void* table, void* out, int T, int H, int V,
                                cudaStream_t stream) {
  if (H % 8) return -3;
  if (T == 0) return 0;
  return launch_chained(embedding_fwd_kernel, grid_for((long long)T * (H / 8), 256), 256, 0, stream, ids,
                        (const __nv_bfloat16*)table, (__nv_bfloat16*)out, T, H, V);
}

extern "C" int sb_embedding_bwd(const long long* ids, const void* dout, float* dtable, int T, int H, int V,
                                cudaStream_t stream) {
  if (H % 8) return -3;
  if (T == 0) return 0;
  embedding_bwd_kernel<<<grid_for((long long)T * (H / 8), 256), 256, 0, stream>>>(
      ids, (const __nv_bfloat16*)dout, dtable, T, H, V);
  return (int)cudaGetLastError();
}

extern "C" int sb_add_bf16(const void* a, const void* b, void* out, long long n, cudaStream_t stream) {
  if (n % 8) return -3;
  if (n == 0) return 0;
  add_bf16_kernel<<<grid_for(n / 8, 256), 256, 0, stream>>>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b,
                                                           (__nv_bfloat16*)out, n / 8);
  return (int)cudaGetLastError();
}
