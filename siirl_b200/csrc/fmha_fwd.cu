// Packed variable-length attention forward (causal or full, GQA) on tcgen05 tensor cores.
// Replaces flash-attn's varlen forward that the reference reaches through HF
// `attn_implementation="flash_attention_2"` (siirl/engine/fsdp_workers.py:631-744,
// siirl/models/transformers/monkey_patch.py:51-109).
//
// Layout: one packed buffer qkv[T, (Hq + 2*Hkv) * D] (q heads, then k heads, then v heads per row);
// sequences are row ranges given by cu_seqlens.  One CTA = 256 query rows (two 128-row tiles) of one q head, or 128:
//   S_w = Q_w K_j^T     tcgen05.mma 128 x KV x D    -> TMEM, w = 0, 1
//   softmax             one warpgroup per query tile, thread = row; the weights (bf16) replace the scores in TMEM
//   O_w += P_w V_j      tcgen05.mma 128 x D x KV, P from TMEM, V through an MN-major descriptor (no transpose copy)
// Outputs: O[T, Hq*D] bf16 and LSE[Hq, T] fp32 (natural log) for the backward pass.
//
// What bounds it: with D = 128 the MMAs (1024 cycles per 128 x 128 tile) and the exponentials (16 a cycle and SM: 1024
// cycles as well), with D = 64 the exponentials.  The two query tiles take turns: while one warpgroup does its softmax the
// tensor cores work for the other one.  K and V are fetched once for 256 rows (at 128 rows the L2 traffic, 7.8 TB/s at
// 1 PFLOP/s, is a bound of its own).  D = 128 takes 128 keys at a time: S and O of both tiles fill all 512 TMEM columns.
// D = 64 takes 64, so that two CTAs fit an SM and one of them always has exponentials to do: 1.15 ms against 1.30 ms
// for 128 keys and one CTA (14 / 2 heads, sequences of 14900 and 15400).  Causal, before (one 128-row tile per CTA, each step
// waiting for the one before) and now: D = 128, 28 / 4 heads, 1 x 16384: 3.47 ms (554 TFLOP/s), 1.85 ms (1045); 8 x 2048:
// 0.56 ms, 0.37 ms; D = 64, 14 / 2 heads, the sequences above: 1.95 ms (423), 1.14 ms (720).  Short sequences are bound by
// the latency of a CTA's first loads, softmax and stores, some 7 us: 32 x 256-1000 tokens, D = 128: 0.36 ms, 0.32 ms.  With
// one tile and 64 keys at a time two CTAs (D = 128) or three fit an SM: 128 x 128 tokens, 28 / 4 heads, D = 128: 133 us
// (one tile per CTA, each step waiting for the one before), 188 (two tiles), 119; D = 64, 14 / 2: 38, 43, 35.
#include "common.cuh"
#include "launchers.h"

namespace sb {

struct FmhaFwdParams {
  const int* tile_seq_start;  // [num_tiles] first token row of the tile's sequence
  const int* tile_seq_len;    // [num_tiles]
  const int* tile_q0;         // [num_tiles] first query position (within the sequence) of the tile
  __nv_bfloat16* out;         // [T, Hq*D]
  float* lse;                 // [Hq, T]
  int T, Hq, Hkv, causal, negate;
  float scale_log2;  // |softmax scale| * log2(e); `negate` says that the scale is negative
  int* status;
};

template <int D, int KV, int QT>
struct FwdSmem {
  static constexpr int kQBytes = 128 * D * 2;   // one query tile
  static constexpr int kKvBytes = KV * D * 2;   // one K or V tile
  static constexpr int kStages = QT == 1 ? 4 : D == 128 ? 5 : 6;
  static constexpr int kRingOff = QT * kQBytes;
  static constexpr int kBarOff = kRingOff + kStages * kKvBytes;  // q[2], s_full[2], p_full[2], o_full[2], full[], empty[]
  static constexpr int kTotal = kBarOff + (8 + 2 * kStages) * 8 + 16;
};

// KV: keys of a tile; QT: query tiles; CTAS: blocks of an SM.
// Four warps for the softmax of each query tile (thread = row), then one for TMA and the MMA issuer.
template <int D, int KV, int QT, int CTAS>
__global__ void __launch_bounds__(QT * 128 + 64, CTAS)
fmha_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                FmhaFwdParams p) {
  using L = FwdSmem<D, KV, QT>;
  constexpr int kDChunks = D / 64, kStages = L::kStages, kTmaWarp = QT * 4, kMmaWarp = QT * 4 + 1;
  // S (P over it) and O of every query tile
  constexpr uint32_t kTmemCols = QT * (KV + D) <= 128 ? 128 : QT * (KV + D) <= 256 ? 256 : 512;
  // 1024-byte alignment is required by the 128-byte swizzle
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) atomicCAS(p.status, 0, (int)kStatusBadArgument);
    return;
  }
  uint8_t* sQ = smem;
  uint8_t* ring = smem + L::kRingOff;
  uint64_t* bar_q = reinterpret_cast<uint64_t*>(smem + L::kBarOff);  // [2]
  uint64_t* s_full = bar_q + 2;                                      // [2] scores are in TMEM
  uint64_t* p_full = bar_q + 4;                                      // [2] weights have replaced the scores
  uint64_t* o_full = bar_q + 6;                                      // [2] the output is complete
  uint64_t* full = bar_q + 8;                                        // [kStages] ring of K and V tiles
  uint64_t* empty = full + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty + kStages);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_kv);
    for (int i = 0; i < 8; ++i) mbar_init(&bar_q[i], (i == 4 || i == 5) ? 128 : 1);
    for (int i = 0; i < 2 * kStages; ++i) mbar_init(&full[i], 1);
    fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_sync();
  const int h = (int)(blockIdx.x % p.Hq), tile = (int)(blockIdx.x / p.Hq);
  const int seq_start = p.tile_seq_start[tile], seq_len = p.tile_seq_len[tile], q0 = p.tile_q0[tile];
  const int kvh = h / (p.Hq / p.Hkv);
  // key tiles that query tile w walks over
  auto key_tiles = [&](int w) {
    const int first = q0 + w * 128;
    if (first >= seq_len) return 0;
    return ((p.causal ? min(first + 128, seq_len) : seq_len) + KV - 1) / KV;
  };
  const int n0 = key_tiles(0), n1 = QT == 2 ? key_tiles(1) : 0;
  const int n_max = max(n0, n1);

  if (warp == kTmaWarp) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      const int qcol = h * D, kcol = (p.Hq + kvh) * D, vcol = (p.Hq + p.Hkv + kvh) * D;
      auto load_q = [&](int w) {
        mbar_arrive_expect_tx(&bar_q[w], L::kQBytes);
#pragma unroll
        for (int c = 0; c < kDChunks; ++c)
          tma_load_2d(sQ + w * L::kQBytes + c * 16384, &map_q, &bar_q[w], qcol + c * 64, seq_start + q0 + w * 128);
      };
      load_q(0);
      int i = 0;
      for (; i < 2 * n_max; ++i) {  // K0 V0 K1 V1 ...
        const int st = i % kStages;
        if (!mbar_wait(&empty[st], ((i / kStages) & 1) ^ 1, p.status, kStatusTimeoutProducer)) break;
        uint8_t* dst = ring + st * L::kKvBytes;
        const int col = (i & 1) ? vcol : kcol, row = seq_start + (i >> 1) * KV;
        mbar_arrive_expect_tx(&full[st], L::kKvBytes);
#pragma unroll
        for (int c = 0; c < kDChunks; ++c) tma_load_2d(dst + c * (KV * 128), &map_kv, &full[st], col + c * 64, row);
        if (i == 0 && n1 > 0) load_q(1);
      }
      if (i < 2 * n_max) {  // gave up: no copy may land in shared memory that has been handed on
        mbar_wait(&bar_q[0], 0, nullptr, 0);
        if (n1 > 0 && i > 0) mbar_wait(&bar_q[1], 0, nullptr, 0);
        for (int k = max(0, i - kStages); k < i; ++k) mbar_wait(&full[k % kStages], (k / kStages) & 1, nullptr, 0);
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------ MMA issuer (converged; lane 0 issues) ------------------------------
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, KV, 0, 0);
    constexpr uint32_t idesc_o = umma_idesc_bf16(128, D, 0, 1);
    const uint32_t leader = lane == 0;
    const uint32_t aq = smem_u32(sQ), ar = smem_u32(ring);
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      const bool ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, p.status, kStatusTimeoutMma));
      tc_fence_after();
      return ok;
    };
    auto wait_ring = [&](int i) { return wait(&full[i % kStages], (i / kStages) & 1); };
    auto scores = [&](int w, int j) {
      const uint32_t bk = ar + ((2 * j) % kStages) * L::kKvBytes;
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)
        umma_bf16_ss_if(leader, tmem_base + w * KV,
                        umma_smem_desc(aq + w * L::kQBytes + (kk / 4) * 16384 + (kk % 4) * 32, 16, 1024),
                        umma_smem_desc(bk + (kk / 4) * (KV * 128) + (kk % 4) * 32, 16, 1024), idesc_s, kk ? 1u : 0u);
      umma_commit_if(leader, &s_full[w]);
    };
    bool ok = wait(&bar_q[0], 0) && wait_ring(0);
    if (ok) {
      scores(0, 0);
      if (n1 > 0) {
        ok = wait(&bar_q[1], 0);
        if (ok) scores(1, 0);
      }
      umma_commit_if(leader, &empty[0]);
    }
    for (int j = 0; j < n_max && ok; ++j) {
      ok = wait_ring(2 * j + 1);
#pragma unroll
      for (int w = 0; w < QT; ++w) {
        const int n = w ? n1 : n0;
        if (ok && j < n) {
          ok = wait(&p_full[w], j & 1);
          if (ok) {
            const uint32_t bv = ar + ((2 * j + 1) % kStages) * L::kKvBytes;
#pragma unroll
            for (int kk = 0; kk < KV / 16; ++kk)
              umma_bf16_ts_if(leader, tmem_base + QT * KV + w * D, tmem_base + w * KV + kk * 8,
                              umma_smem_desc(bv + kk * 2048, KV * 128, 1024), idesc_o, (j | kk) ? 1u : 0u);
            if (j + 1 == n) umma_commit_if(leader, &o_full[w]);
          }
        }
        if (w == QT - 1) umma_commit_if(leader, &empty[(2 * j + 1) % kStages]);
        if (ok && j + 1 < n) {
          ok = wait_ring(2 * j + 2);
          if (ok) scores(w, j + 1);
        }
      }
      if (j + 1 < n_max) umma_commit_if(leader, &empty[(2 * j + 2) % kStages]);
    }
  } else {
    // ------------------------------ softmax and output: thread = query row ------------------------------
    const int w = warp >> 2;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tmem_s = tmem_base + lane_off + w * KV;
    const uint32_t tmem_o = tmem_base + lane_off + QT * KV + w * D;
    const int first = q0 + w * 128;
    const int qpos = first + (warp & 3) * 32 + lane;  // position within the sequence
    const int n = w ? n1 : n0;
    const float sc = p.scale_log2;
    float m_used = -INFINITY;  // running maximum, scaled
    float2 l_run = make_float2(0.f, 0.f);
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait(&s_full[w], j & 1, p.status, kStatusTimeoutEpilogue));
      if (!ok) break;
      tc_fence_after();
      uint32_t s[KV / 32][32];
#pragma unroll
      for (int c = 0; c < KV / 32; ++c) tmem_ld_32x32(tmem_s + c * 32, s[c]);
      tmem_ld_wait();
      if (p.negate) {
#pragma unroll
        for (int i = 0; i < KV; ++i) s[i / 32][i % 32] ^= 0x80000000u;
      }
      const int kv0 = j * KV;
      if (kv0 + KV > seq_len || (p.causal && kv0 + KV - 1 > first)) {
        const int visible = min(p.causal ? qpos + 1 : seq_len, seq_len) - kv0;
#pragma unroll
        for (int i = 0; i < KV; ++i)
          if (i >= visible) s[i / 32][i % 32] = 0xff800000u;  // -inf
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < KV; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(s[i / 32][i % 32]));
      const float row_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc;
      const float m_new = fmaxf(m_used, row_max);
      const float alpha = fast_exp2(m_used - (m_new == -INFINITY ? 0.f : m_new));
      const bool grows = __any_sync(0xffffffffu, m_new > m_used);
      m_used = m_new;
      l_run.x *= alpha;
      l_run.y *= alpha;
      const float m_ref = m_used == -INFINITY ? 0.f : m_used;
      const float2 sc2 = make_float2(sc, sc), neg = make_float2(-m_ref, -m_ref);
#pragma unroll
      for (int c = 0; c < KV / 32; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float2 x = make_float2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
          x = fma_f32x2(x, sc2, neg);
          x.x = fast_exp2(x.x);
          x.y = fast_exp2(x.y);
          l_run = add_f32x2(l_run, x);
          pk[i / 2] = pack_bf16x2(x.x, x.y);
        }
        tmem_st_32x16(tmem_s + c * 16, pk);
      }
      // A row maximum has grown: the output so far is scaled.  The barrier of the scores also said that P V of the
      // previous tile is done; by now the scores' registers are free, and all of the row's loads can be in flight.
      if (j > 0 && grows) {
        constexpr int kBatch = KV / 32;
#pragma unroll 1
        for (int c0 = 0; c0 < D / 32; c0 += kBatch) {
          uint32_t r[kBatch][32];
#pragma unroll
          for (int c = 0; c < kBatch; ++c) tmem_ld_32x32(tmem_o + (c0 + c) * 32, r[c]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < kBatch; ++c) {
#pragma unroll
            for (int i = 0; i < 32; ++i) r[c][i] = __float_as_uint(__uint_as_float(r[c][i]) * alpha);
            tmem_st_32x32(tmem_o + (c0 + c) * 32, r[c]);
          }
        }
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[w]);
    }
    if (ok && n > 0) ok = __all_sync(0xffffffffu, mbar_wait(&o_full[w], 0, p.status, kStatusTimeoutEpilogue));
    // ---- O / l -> bf16, LSE (TMEM loads are warp-collective; only the stores are predicated) ----
    if (ok && n > 0) {
      tc_fence_after();
      const bool row_valid = qpos < seq_len;
      const float l = l_run.x + l_run.y;
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      const size_t row = (size_t)(seq_start + (row_valid ? qpos : 0));
      __nv_bfloat16* orow = p.out + row * (size_t)(p.Hq * D) + (size_t)h * D;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_o + c * 32, r);
        tmem_ld_wait();
        if (row_valid) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(r[g * 8 + 0]) * inv_l, __uint_as_float(r[g * 8 + 1]) * inv_l);
            o.y = pack_bf16x2(__uint_as_float(r[g * 8 + 2]) * inv_l, __uint_as_float(r[g * 8 + 3]) * inv_l);
            o.z = pack_bf16x2(__uint_as_float(r[g * 8 + 4]) * inv_l, __uint_as_float(r[g * 8 + 5]) * inv_l);
            o.w = pack_bf16x2(__uint_as_float(r[g * 8 + 6]) * inv_l, __uint_as_float(r[g * 8 + 7]) * inv_l);
            *reinterpret_cast<uint4*>(orow + c * 32 + g * 8) = o;
          }
        }
      }
      if (row_valid)
        p.lse[(size_t)h * p.T + row] = (m_used == -INFINITY) ? -INFINITY : (m_used + log2f(l)) * 0.6931471805599453f;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int D, int KV, int QT, int CTAS>
static int launch_fwd(const CUtensorMap& mq, const CUtensorMap& mkv, const FmhaFwdParams& p, int num_tiles,
                      cudaStream_t stream) {
  using L = FwdSmem<D, KV, QT>;
  auto kernel = fmha_fwd_kernel<D, KV, QT, CTAS>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const long long blocks = (long long)num_tiles * p.Hq;
  if (blocks > 0x7fffffffll) return -4;
  return launch_chained(kernel, (unsigned)blocks, QT * 128 + 64, L::kTotal, stream, mq, mkv, p);
}

}  // namespace sb

using namespace sb;

// Entry i of the tile lists covers tile_rows (128 or 256) query rows from tile_q0[i] on, as far as they exist, of its
// sequence.
extern "C" int sb_fmha_fwd(const void* qkv, void* out, float* lse, const int* tile_seq_start,
                           const int* tile_seq_len, const int* tile_q0, int num_tiles, int tile_rows, int T, int Hq, int Hkv,
                           int D, int causal, float scale, int* status, cudaStream_t stream) {
  if (num_tiles == 0 || T == 0) return 0;
  if (D != 64 && D != 128) return -2;
  if (tile_rows != 128 && tile_rows != 256) return -3;
  static thread_local bool tl_context_bound = false;
  if (!tl_context_bound) {
    cudaFree(0);
    tl_context_bound = true;
  }
  const long long width = (long long)(Hq + 2 * Hkv) * D;
  CUtensorMap mq, mkv;
  int r = make_tensor_map_bf16_2d(&mq, qkv, width, T, width, 64, 128);
  if (r) return r;
  r = make_tensor_map_bf16_2d(&mkv, qkv, width, T, width, 64, D == 128 && tile_rows == 256 ? 128 : 64);
  if (r) return r;
  FmhaFwdParams p;
  p.tile_seq_start = tile_seq_start; p.tile_seq_len = tile_seq_len; p.tile_q0 = tile_q0;
  p.out = reinterpret_cast<__nv_bfloat16*>(out); p.lse = lse;
  p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal;
  p.negate = scale < 0.f;
  p.scale_log2 = fmaxf(fabsf(scale) * 1.4426950408889634f, 1e-30f);  // 0 times a hidden score would not be a number
  p.status = status;
  if (tile_rows == 128)
    return D == 128 ? launch_fwd<128, 64, 1, 2>(mq, mkv, p, num_tiles, stream)
                    : launch_fwd<64, 64, 1, 3>(mq, mkv, p, num_tiles, stream);
  return D == 128 ? launch_fwd<128, 128, 2, 1>(mq, mkv, p, num_tiles, stream)
                  : launch_fwd<64, 64, 2, 2>(mq, mkv, p, num_tiles, stream);
}
