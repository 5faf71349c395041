// Packed variable-length attention backward (causal or full, GQA) on tcgen05 tensor cores.
// Counterpart of fmha_fwd.cu; replaces flash-attn's varlen backward used by the reference's training path
// (siirl/engine/actor/dp_actor.py:87-263 through HF flash_attention_2).
//
// One CTA owns one 128-row K/V tile of one kv head and walks over (a share of) the q heads of its GQA group and the query
// tiles that can attend to it.  TMEM lane = kv row.  Per step i:
//   S^T = K Q^T,  dP^T = V dO^T             128 x 128 x D each
//   P^T = exp2(S^T*c - LSE) -> bf16, over S^T in TMEM;   dS^T = P^T (dP^T - Delta) -> bf16, swizzled smem
//   dV += P^T dO (A from TMEM)   dK += dS^T Q   dQ_i = dS K (A = dS^T read MN-major)
//   dQ_i is added to an fp32 buffer by vector reductions of whole 128-byte lines
// The softmax scale is applied once, to dK and dQ at the end.
//
// Blocks that share a group's heads keep dK and dV apart for the pass that converts them, which adds them in order.  dQ comes
// from all K/V tiles of a sequence.  ORDERED: they add to it one after the other, tile 0 first (it stores, nothing is
// zeroed), so that equal inputs give equal gradients.  Tiles then walk over the query tiles from the last to the first and
// take their work by ticket, tile 0 first: no block waits for one that may not have started, and the one it waits for is
// ahead unless both start at once.  Else tiles start on the diagonal and add as they come: tiles that run together are then
// always at different rows, and none waits until its predecessor's additions have reached memory.  Microseconds ordered /
// not, causal: 8 x 568-1232, 14 / 2 heads, D = 64: 144 / 142; 4 x 1024, 28 / 4, D = 128: 230 / 206; 8 x 2048: 1088 / 873;
// 1 x 4096: 551 / 398; 1 x 16384: 7430 / 5500; 1 x 9900, 14 / 2, D = 64: 955 / 713.
//
// What bounds it: the five products take 2560 cycles a step with D = 128 (1536 with D = 64, whose operands come from shared
// memory at its full rate), the exponentials 1024 and the rest of the element-wise work about as much.  All of it is in
// flight at once: while the math warps take step i + 1 from scores to weights the tensor cores run dQ, dK and dP behind
// step i, and while they go from dP to dS, dV and the next scores.  Lane = kv row because P^T is then an operand in TMEM
// (no shared memory, which is full with D = 128); the row statistics become columns, staged by a warp of their own.
// Blocks are listed by their number of steps.  One block per kv head leaves SMs idle when a sequence is long and kv heads
// are few: its first K/V tile has twice the average work, times the heads of the group.  The caller then splits the group
// (bwd_head_splits).  Causal, before (256 threads, one step after the other) and now: 28 / 4 heads, D = 128, 1 x 16384:
// 9.99 ms (482 TFLOP/s), 5.50 ms (875); 8 x 2048: 1.50 ms, 1.09 ms; 14 / 2 heads, D = 64, 1 x 9900: 2.15 ms (204), 0.71 ms
// (617; unsplit 1.21 ms); 8 x 568-1232: 0.31 ms, 0.14 ms (unsplit 0.24 ms).
#include "common.cuh"
#include "launchers.h"

namespace sb {

struct FmhaBwdParams {
  const int* tile_seq_start;  // per kv tile
  const int* tile_seq_len;
  const int* tile_k0;         // first kv position of the tile inside its sequence
  const float* lse;           // [Hq, T]
  const float* delta;         // [Hq, T]  rowsum(dO * O)
  float* dq_accum;            // [T, Hq*D] fp32, zero-initialised when the tiles are not ordered
  float* dkv_accum;           // [head_splits, T, 2*Hkv*D] fp32 when the q heads of a group are split (else unused)
  int* turn;                  // ordered: [Hq, T + 1] zero-initialised: at the first of each 32 query rows of a sequence the
                              // number of K/V tiles that have added their dQ; at row T of head 0 the next block's ticket
  __nv_bfloat16* dqkv;        // [T, (Hq+2Hkv)*D]; this kernel writes the k and v parts when they are not split
  int T, Hq, Hkv, causal, head_splits;
  float scale, scale_log2;
  int* status;
};

constexpr int kBwdStagePitch = 32 * 4 + 16;  // a row of 32 dQ columns; the pad spreads the rows over the banks

template <int D>
struct BwdSmem {
  static constexpr int kTile = 128 * D * 2;      // K, V, Q, dO tiles
  static constexpr int kSq = 128 * 128 * 2;      // dS^T
  static constexpr int kDoStages = D == 128 ? 1 : 2;
  static constexpr int kAccPitch = D * 4 + 16;   // a row of dK / dV on its way to the fp32 buffer
  static constexpr int kKOff = 0;
  static constexpr int kVOff = kKOff + kTile;
  static constexpr int kQOff = kVOff + kTile;               // 2 stages
  static constexpr int kDoOff = kQOff + 2 * kTile;
  static constexpr int kDsOff = kDoOff + kDoStages * kTile;
  static constexpr int kStageOff = kDsOff + kSq;
  static constexpr int kStatOff = kStageOff + 128 * kBwdStagePitch;  // 2 x (128 of -lse * log2e, 128 of -delta)
  static constexpr int kBarOff = kStatOff + 2 * 1024;
  static constexpr int kTotal = kBarOff + 20 * 8 + 16;  // barriers, TMEM address, ticket
  static_assert(2 * 128 * kAccPitch <= kStageOff, "dK and dV rows are staged over the operand tiles");
};

__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}

// copies `bytes` bytes from shared memory to global memory (both 16-byte aligned)
__device__ __forceinline__ void bulk_store(float* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {  // returns at once
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait until *turn, written by other blocks of this kernel, is at least `n`.
__device__ __forceinline__ bool wait_turn(const int* turn, int n, int* status) {
  auto arrived = [&] {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(turn) : "memory");
    return v >= n;
  };
  if (arrived()) return true;
  const uint64_t t0 = global_timer_ns();
  while (true) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i)
      if (arrived()) return true;
    if (global_timer_ns() - t0 > SB_WAIT_LIMIT_NS) {
      atomicCAS(status, 0, (int)kStatusTimeoutFlag);
      return false;
    }
  }
}

template <int N>
__device__ __forceinline__ void regs_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regs_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

__device__ __forceinline__ float2 add_mul_f32x2(float2 a, float2 b, float2 f) {  // (a + b) * f
  uint64_t d;
  asm("{\n\t.reg .b64 t;\n\t"
      "add.rn.f32x2 t, %1, %2;\n\t"
      "mul.rn.f32x2 %0, t, %3;\n\t}"
      : "=l"(d)
      : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&f)));
  return *reinterpret_cast<float2*>(&d);
}

// 16 warps: 0-7 P and dS (thread = kv row and one half of the query columns), 8-11 dQ, 12 TMA, 13 MMA issuer, 14 row
// statistics.  The launch's 128 registers a thread are shared out as 144, 144, 152 and 72 to the four warpgroups.  __maxnreg__
// and not __launch_bounds__: it is the directive from which setmaxnreg takes the count at launch, while launch bounds only
// limit what the compiler may use.
constexpr int kBwdThreads = 512, kBwdRegs = 128;
constexpr int kRegsMath = 144, kRegsDq = 152, kRegsIssue = 72;
static_assert(2 * kRegsMath + kRegsDq + kRegsIssue <= 4 * kBwdRegs, "more registers than the launch has");
static_assert(kBwdThreads * kBwdRegs <= 65536, "more registers than an SM has");

template <int D, bool ORDERED>
__global__ void __maxnreg__(kBwdRegs)
fmha_bwd_kernel(const __grid_constant__ CUtensorMap map_qkv, const __grid_constant__ CUtensorMap map_do,
                FmhaBwdParams p) {
  using L = BwdSmem<D>;
  constexpr int kDChunks = D / 64, kDo = L::kDoStages;
  constexpr bool kDqOverDp = D == 128;  // TMEM is full: dQ takes the columns of dP
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) atomicCAS(p.status, 0, (int)kStatusBadArgument);
    return;
  }
  uint8_t* sK = smem + L::kKOff;
  uint8_t* sV = smem + L::kVOff;
  uint8_t* sQ = smem + L::kQOff;
  uint8_t* sDo = smem + L::kDoOff;
  uint8_t* sDs = smem + L::kDsOff;  // dS^T [kv rows][q columns], bf16, 128-byte swizzle, two 64-column chunks
  uint64_t* bar_kv = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* q_full = bar_kv + 1;     // [2]
  uint64_t* q_empty = bar_kv + 3;    // [2]
  uint64_t* do_full = bar_kv + 5;    // [2]
  uint64_t* do_empty = bar_kv + 7;   // [2]
  uint64_t* st_full = bar_kv + 9;    // [2] row statistics
  uint64_t* st_empty = bar_kv + 11;  // [2]
  uint64_t* s_full = bar_kv + 13;
  uint64_t* dp_full = bar_kv + 14;
  uint64_t* p_ready = bar_kv + 15;
  uint64_t* ds_ready = bar_kv + 16;
  uint64_t* dq_full = bar_kv + 17;
  uint64_t* dq_read = bar_kv + 18;
  uint64_t* done = bar_kv + 19;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_kv + 20);
  int* ticket_slot = reinterpret_cast<int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_tile = p.Hkv * p.head_splits;
  int ticket = (int)blockIdx.x, seq_start, seq_len, k0;
  auto take_tile = [&] {
    const int tile = ticket / per_tile;
    seq_start = p.tile_seq_start[tile];
    seq_len = p.tile_seq_len[tile];
    k0 = p.tile_k0[tile];
  };
  if (ORDERED) {
    if (tid == 32) *ticket_slot = atomicAdd(p.turn + p.T, 1);
  } else {
    take_tile();
  }
  if (tid == 0) {
    tma_prefetch_desc(&map_qkv);
    tma_prefetch_desc(&map_do);
    for (int i = 0; i < 20; ++i) {
      const int count = (i == 9 || i == 10) ? 32 : (i == 11 || i == 12 || i == 15 || i == 16) ? 256 : i == 18 ? 128 : 1;
      mbar_init(&bar_kv[i], count);
    }
    fence_barrier_init();
  }
  if (warp == 13) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 128, tm_dv = tmem_base + 256, tm_dk = tm_dv + D;
  const uint32_t tm_dq = kDqOverDp ? tm_dp : tm_dk + D;
  const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;

  if (ORDERED) {
    ticket = *ticket_slot;
    take_tile();
  }
  const int kvh = ticket % per_tile / p.head_splits, share = ticket % per_tile % p.head_splits;
  const int rep = p.Hq / p.Hkv;
  const int h_first = kvh * rep + rep * share / p.head_splits, h_end = kvh * rep + rep * (share + 1) / p.head_splits;
  const int i_low = p.causal ? k0 / 128 : 0, i_high = (seq_len + 127) / 128 - 1, per_head = i_high + 1 - i_low;
  const int i_first = ORDERED ? i_high : i_low;  // query tiles of every head: from here down, or up
  constexpr int kDir = ORDERED ? -1 : 1;
  const int steps = per_head * (h_end - h_first);
  const int kcol = (p.Hq + kvh) * D, vcol = (p.Hq + p.Hkv + kvh) * D;

  if (warp < 8) {
    // ------------------------------ P and dS, then dK and dV ------------------------------
    regs_inc<kRegsMath>();
    const int half = warp >> 2, r = (warp & 3) * 32 + lane;
    const int kp = k0 + r;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    bool ok = true;
    int q0 = i_first * 128, left = per_head;
    for (int i = 0; i < steps; ++i) {
      const float4* stat = reinterpret_cast<const float4*>(smem + L::kStatOff + (i & 1) * 1024) + half * 16;
      ok = __all_sync(0xffffffffu, mbar_wait(&st_full[i & 1], (i >> 1) & 1, p.status, kStatusTimeoutEpilogue) &&
                                       mbar_wait(s_full, i & 1, p.status, kStatusTimeoutEpilogue));
      if (!ok) break;
      tc_fence_after();
      uint32_t rs[2][32];
      float2 pr[32];  // this row's weights of the 64 query columns
      tmem_ld_32x32(tm_s + lane_off + half * 64, rs[0]);
      tmem_ld_32x32(tm_s + lane_off + half * 64 + 32, rs[1]);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < 16; ++g) {
        const float4 l = stat[g];
        const uint32_t* x = &rs[g / 8][(g % 8) * 4];
        float2 a = fma_f32x2(make_float2(__uint_as_float(x[0]), __uint_as_float(x[1])), sc2, make_float2(l.x, l.y));
        float2 b = fma_f32x2(make_float2(__uint_as_float(x[2]), __uint_as_float(x[3])), sc2, make_float2(l.z, l.w));
        pr[2 * g] = make_float2(fast_exp2(a.x), fast_exp2(a.y));
        pr[2 * g + 1] = make_float2(fast_exp2(b.x), fast_exp2(b.y));
      }
      // only the diagonal tile (causal) and tiles that stick out of the sequence have hidden entries
      if ((p.causal && q0 < k0 + 128) || q0 + 128 > seq_len || k0 + 128 > seq_len) {
        const int lo = (p.causal ? kp - q0 : 0) - half * 64, hi = (kp < seq_len ? seq_len - q0 : 0) - half * 64;
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          if (2 * c < lo || 2 * c >= hi) pr[c].x = 0.f;
          if (2 * c + 1 < lo || 2 * c + 1 >= hi) pr[c].y = 0.f;
        }
      }
      {
        uint32_t pk[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) pk[c] = pack_bf16x2(pr[c].x, pr[c].y);
        tmem_st_32x32(tm_s + lane_off + half * 64, pk);  // over this warp's own scores
        tmem_st_wait();
      }
      tc_fence_before();
      mbar_arrive(p_ready);
      ok = __all_sync(0xffffffffu, mbar_wait(dp_full, i & 1, p.status, kStatusTimeoutEpilogue));
      if (!ok) break;
      tc_fence_after();
      // dP(i) was issued behind the MMAs that read dS(i - 1): the buffer is free
      uint8_t* drow = sDs + half * 16384 + r * 128;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        tmem_ld_32x32(tm_dp + lane_off + half * 64 + c * 32, rs[0]);
        tmem_ld_wait();
        uint32_t dd[16];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const float4 dl = stat[32 + c * 8 + g];
          const uint32_t* x = &rs[0][g * 4];
          const float2 a = add_mul_f32x2(make_float2(__uint_as_float(x[0]), __uint_as_float(x[1])), make_float2(dl.x, dl.y),
                                    pr[c * 16 + 2 * g]);
          const float2 b = add_mul_f32x2(make_float2(__uint_as_float(x[2]), __uint_as_float(x[3])), make_float2(dl.z, dl.w),
                                    pr[c * 16 + 2 * g + 1]);
          dd[2 * g] = pack_bf16x2(a.x, a.y);
          dd[2 * g + 1] = pack_bf16x2(b.x, b.y);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4*>(drow + (((c * 4 + q) ^ (r & 7)) << 4)) =
              make_uint4(dd[q * 4], dd[q * 4 + 1], dd[q * 4 + 2], dd[q * 4 + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(ds_ready);
      mbar_arrive(&st_empty[i & 1]);
      q0 += kDir * 128;
      if (--left == 0) {
        left = per_head;
        q0 = i_first * 128;
      }
    }
    // ---- dK, dV (lane = kv row, this warp's half of the D columns) ----
    ok = ok && __all_sync(0xffffffffu, mbar_wait(done, 0, p.status, kStatusTimeoutEpilogue));
    if (ok) {
      tc_fence_after();
      const bool row_valid = kp < seq_len;
      const size_t row = (size_t)(seq_start + (row_valid ? kp : 0));
#pragma unroll 1
      for (int x = 0; x < D / 32; ++x) {
        const bool is_v = x >= D / 64;
        const int col = (half * (D / 64) + x % (D / 64)) * 32;
        const float f = is_v ? 1.f : p.scale;
        uint32_t ra[32];
        tmem_ld_32x32((is_v ? tm_dv : tm_dk) + lane_off + col, ra);
        tmem_ld_wait();
        if (p.head_splits > 1) {
          // every MMA has read its operands: their tiles hold the rows on the way to this share's fp32 sums
          float* stage = reinterpret_cast<float*>(smem + (is_v * 128 + r) * L::kAccPitch) + col;
#pragma unroll
          for (int g = 0; g < 8; ++g)
            *reinterpret_cast<float4*>(stage + g * 4) =
                make_float4(__uint_as_float(ra[g * 4]) * f, __uint_as_float(ra[g * 4 + 1]) * f,
                            __uint_as_float(ra[g * 4 + 2]) * f, __uint_as_float(ra[g * 4 + 3]) * f);
          fence_proxy_async_smem();
          if (row_valid)
            bulk_store(p.dkv_accum + ((size_t)share * p.T + row) * (size_t)(2 * p.Hkv * D) +
                           (size_t)((is_v ? p.Hkv : 0) + kvh) * D + col, stage, 128);
          tma_store_commit();
        } else if (row_valid) {
          __nv_bfloat16* dst = p.dqkv + row * (size_t)((p.Hq + 2 * p.Hkv) * D) + (is_v ? vcol : kcol) + col;
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 a;
            a.x = pack_bf16x2(__uint_as_float(ra[g * 8 + 0]) * f, __uint_as_float(ra[g * 8 + 1]) * f);
            a.y = pack_bf16x2(__uint_as_float(ra[g * 8 + 2]) * f, __uint_as_float(ra[g * 8 + 3]) * f);
            a.z = pack_bf16x2(__uint_as_float(ra[g * 8 + 4]) * f, __uint_as_float(ra[g * 8 + 5]) * f);
            a.w = pack_bf16x2(__uint_as_float(ra[g * 8 + 6]) * f, __uint_as_float(ra[g * 8 + 7]) * f);
            *reinterpret_cast<uint4*>(dst + g * 8) = a;
          }
        }
      }
      tma_store_wait_read<0>();  // shared memory is given back below
    }
  } else if (warp < 12) {
    // ------------------------------ dQ -> fp32 sums (lane = query row) ------------------------------
    regs_inc<kRegsDq>();
    uint8_t* stage = smem + L::kStageOff + (warp & 3) * (32 * kBwdStagePitch);
    const int order = k0 / 128;   // of this tile among those that add to a query tile
    int* next = nullptr;          // where the tile behind this one waits for the previous step's rows
    auto hand_on = [&] {
      if (next == nullptr) return;
      __syncwarp();
      if (lane == 0) asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(next), "r"(order + 1) : "memory");
      next = nullptr;
    };
    int q0 = i_first * 128, left = per_head, h = h_first;
    for (int i = 0; i < steps; ++i) {
      if (!__all_sync(0xffffffffu, mbar_wait(dq_full, i & 1, p.status, kStatusTimeoutEpilogue))) break;
      tc_fence_after();
      uint32_t rq[D / 32][32];
#pragma unroll
      for (int c = 0; c < D / 32; ++c) tmem_ld_32x32(tm_dq + lane_off + c * 32, rq[c]);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(dq_read);
      if (ORDERED) hand_on();
      const int first = q0 + (warp & 3) * 32;
      int* turn = ORDERED ? p.turn + (size_t)h * (p.T + 1) + seq_start + first : nullptr;
      if (ORDERED && first < seq_len && order > 0) {
        bool mine = true;
        if (lane == 0) mine = wait_turn(turn, order, p.status);
        if (!__all_sync(0xffffffffu, mine)) break;
      }
      // TMEM hands every thread one query row; turned through shared memory, each warp instruction adds four lines of
      // 128 bytes instead of 32 pieces of 16
      float* dst = p.dq_accum + (size_t)(seq_start + first) * (size_t)(p.Hq * D) + (size_t)h * D + (lane & 7) * 4;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
#pragma unroll
        for (int g = 0; g < 8; ++g)
          *reinterpret_cast<uint4*>(stage + lane * kBwdStagePitch + g * 16) =
              make_uint4(rq[c][g * 4], rq[c][g * 4 + 1], rq[c][g * 4 + 2], rq[c][g * 4 + 3]);
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const int row = g * 4 + (lane >> 3);
          const float4 v = *reinterpret_cast<const float4*>(stage + row * kBwdStagePitch + (lane & 7) * 16);
          float* at = dst + (size_t)row * (size_t)(p.Hq * D) + c * 32;
          if (first + row < seq_len) {
            if (ORDERED && order == 0) *reinterpret_cast<float4*>(at) = v;
            else red_add_v4(at, v.x, v.y, v.z, v.w);
          }
        }
        __syncwarp();
      }
      if (ORDERED) {
        // Rows are handed on at once while there is nothing else to do, else behind the next step's loads: by then the
        // additions are done, and the release does not wait for them.
        if (first < seq_len && order < (p.causal ? q0 / 128 : i_high)) next = turn;
        if (i + 1 == steps || !__all_sync(0xffffffffu, mbar_test(dq_full, (i + 1) & 1))) hand_on();
      }
      q0 += kDir * 128;
      if (--left == 0) {
        left = per_head;
        q0 = i_first * 128;
        ++h;
      }
    }
  } else {
    regs_dec<kRegsIssue>();
    if (warp == 12) {
      // ------------------------------ TMA producer ------------------------------
      if (lane == 0) {
        mbar_arrive_expect_tx(bar_kv, 2 * L::kTile);
#pragma unroll
        for (int c = 0; c < kDChunks; ++c) {
          tma_load_2d(sK + c * 16384, &map_qkv, bar_kv, kcol + c * 64, seq_start + k0);
          tma_load_2d(sV + c * 16384, &map_qkv, bar_kv, vcol + c * 64, seq_start + k0);
        }
        int n_q = 0, n_do = 0;  // loads issued
        int qi = i_first, left = per_head, h = h_first;
        for (int i = 0; i < steps; ++i) {
          const int row = seq_start + qi * 128;
          if (!mbar_wait(&q_empty[i & 1], ((i >> 1) & 1) ^ 1, p.status, kStatusTimeoutProducer)) break;
          mbar_arrive_expect_tx(&q_full[i & 1], L::kTile);
#pragma unroll
          for (int c = 0; c < kDChunks; ++c)
            tma_load_2d(sQ + (i & 1) * L::kTile + c * 16384, &map_qkv, &q_full[i & 1], h * D + c * 64, row);
          n_q = i + 1;
          if (!mbar_wait(&do_empty[i % kDo], ((i / kDo) & 1) ^ 1, p.status, kStatusTimeoutProducer)) break;
          mbar_arrive_expect_tx(&do_full[i % kDo], L::kTile);
#pragma unroll
          for (int c = 0; c < kDChunks; ++c)
            tma_load_2d(sDo + (i % kDo) * L::kTile + c * 16384, &map_do, &do_full[i % kDo], h * D + c * 64, row);
          n_do = i + 1;
          qi += kDir;
          if (--left == 0) {
            left = per_head;
            qi = i_first;
            ++h;
          }
        }
        if (n_do < steps) {  // gave up: no copy may land in shared memory that has been handed on
          mbar_wait(bar_kv, 0, nullptr, 0);
          for (int k = max(0, n_q - 2); k < n_q; ++k) mbar_wait(&q_full[k & 1], (k >> 1) & 1, nullptr, 0);
          for (int k = max(0, n_do - kDo); k < n_do; ++k) mbar_wait(&do_full[k % kDo], (k / kDo) & 1, nullptr, 0);
        }
      }
    } else if (warp == 13) {
      // ------------------------------ MMA issuer (converged; lane 0 issues) ------------------------------
      constexpr uint32_t idesc_kk = umma_idesc_bf16(128, 128, 0, 0);  // both operands K-major, N = 128
      constexpr uint32_t idesc_kmn = umma_idesc_bf16(128, D, 0, 1);   // A K-major (or in TMEM), B MN-major, N = D
      constexpr uint32_t idesc_mnmn = umma_idesc_bf16(128, D, 1, 1);  // both MN-major, N = D
      const uint32_t leader = lane == 0;
      const uint32_t ak = smem_u32(sK), av = smem_u32(sV), aq = smem_u32(sQ), ado = smem_u32(sDo), ads = smem_u32(sDs);
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        const bool ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, p.status, kStatusTimeoutMma));
        tc_fence_after();
        return ok;
      };
      auto products = [&](uint32_t d, uint32_t a, uint32_t b) {  // [128 x 128] = a b^T over D
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * 16384 + (kk % 4) * 32;
          umma_bf16_ss_if(leader, d, umma_smem_desc(a + off, 16, 1024), umma_smem_desc(b + off, 16, 1024), idesc_kk,
                          kk ? 1u : 0u);
        }
      };
      bool ok = wait(bar_kv, 0) && wait(&q_full[0], 0);
      if (ok) {
        products(tm_s, ak, aq);
        umma_commit_if(leader, s_full);
        ok = wait(&do_full[0], 0);
      }
      if (ok) {
        products(tm_dp, av, ado);
        umma_commit_if(leader, dp_full);
      }
      for (int i = 0; i < steps && ok; ++i) {
        const uint32_t q = aq + (i & 1) * L::kTile, d_o = ado + (i % kDo) * L::kTile;
        ok = wait(p_ready, i & 1);
        if (!ok) break;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)  // dV += P^T dO; each half of the query columns starts at its half of the scores
          umma_bf16_ts_if(leader, tm_dv, tm_s + (kk / 4) * 64 + (kk % 4) * 8, umma_smem_desc(d_o + kk * 2048, 16384, 1024),
                          idesc_kmn, (i | kk) ? 1u : 0u);
        umma_commit_if(leader, &do_empty[i % kDo]);
        if (i + 1 < steps) {
          ok = wait(&q_full[(i + 1) & 1], ((i + 1) >> 1) & 1);
          if (!ok) break;
          products(tm_s, ak, aq + ((i + 1) & 1) * L::kTile);
          umma_commit_if(leader, s_full);
        }
        ok = wait(ds_ready, i & 1) && (kDqOverDp || i == 0 || wait(dq_read, (i - 1) & 1));
        if (!ok) break;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)  // dQ = dS K, contraction over the kv rows
          umma_bf16_ss_if(leader, tm_dq, umma_smem_desc(ads + kk * 2048, 16384, 1024),
                          umma_smem_desc(ak + kk * 2048, 16384, 1024), idesc_mnmn, kk ? 1u : 0u);
        umma_commit_if(leader, dq_full);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)  // dK += dS^T Q, contraction over the query rows
          umma_bf16_ss_if(leader, tm_dk, umma_smem_desc(ads + (kk / 4) * 16384 + (kk % 4) * 32, 16, 1024),
                          umma_smem_desc(q + kk * 2048, 16384, 1024), idesc_kmn, (i | kk) ? 1u : 0u);
        umma_commit_if(leader, &q_empty[i & 1]);
        if (i + 1 < steps) {
          ok = wait(&do_full[(i + 1) % kDo], ((i + 1) / kDo) & 1) && (!kDqOverDp || wait(dq_read, i & 1));
          if (!ok) break;
          products(tm_dp, av, ado + ((i + 1) % kDo) * L::kTile);
          umma_commit_if(leader, dp_full);
        }
      }
      umma_commit_if(leader, done);
    } else if (warp == 14) {
      // ------------------------------ row statistics: -lse * log2(e), -delta ------------------------------
      int q0 = i_first * 128, left = per_head, h = h_first;
      for (int i = 0; i < steps; ++i) {
        if (!__all_sync(0xffffffffu, mbar_wait(&st_empty[i & 1], ((i >> 1) & 1) ^ 1, p.status, kStatusTimeoutProducer))) break;
        float* dst = reinterpret_cast<float*>(smem + L::kStatOff + (i & 1) * 1024);
        const size_t at = (size_t)h * p.T + seq_start + q0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int q = e * 32 + lane;
          const bool in = q0 + q < seq_len;
          dst[q] = in ? p.lse[at + q] * -1.4426950408889634f : -INFINITY;
          dst[128 + q] = in ? -p.delta[at + q] : 0.f;
        }
        mbar_arrive(&st_full[i & 1]);
        q0 += kDir * 128;
        if (--left == 0) {
          left = per_head;
          q0 = i_first * 128;
          ++h;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]; one warp per (t, h).  Clears `turn` as well (if not null).
__global__ void fmha_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                  float* __restrict__ delta, int* __restrict__ turn, int T, int Hq, int D) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (long long)T * Hq) return;
  const int t = (int)(w / Hq), h = (int)(w % Hq);
  const __nv_bfloat16* a = o + ((size_t)t * Hq + h) * D;
  const __nv_bfloat16* b = d_o + ((size_t)t * Hq + h) * D;
  float s = 0.f;
  for (int i = lane * 2; i < D; i += 64) {
    const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(a + i));
    const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(b + i));
    s += x.x * y.x + x.y * y.y;
  }
  s = warp_sum(s);
  if (lane == 0) {
    delta[(size_t)h * T + t] = s;
    if (turn) {
      turn[(size_t)h * (T + 1) + t] = 0;
      if (t == 0) turn[(size_t)h * (T + 1) + T] = 0;
    }
  }
}

// dqkv[t, col + c] = bf16(scale * acc[t, c]) for `cols` columns; SUM: of the sum of `slabs` such buffers
template <bool SUM>
__global__ void fmha_cast_kernel(const float* __restrict__ acc, int slabs, __nv_bfloat16* __restrict__ dqkv, int T, int cols,
                                 int col, int width, float scale) {
  const long long total = (long long)T * (cols / 4);
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(idx / (cols / 4)), c = (int)(idx % (cols / 4)) * 4;
    float4 v = *reinterpret_cast<const float4*>(acc + (size_t)t * cols + c);
    for (int s = 1; SUM && s < slabs; ++s) {
      const float4 b = *reinterpret_cast<const float4*>(acc + ((size_t)s * T + t) * cols + c);
      v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
    }
    uint2 o;
    o.x = pack_bf16x2(v.x * scale, v.y * scale);
    o.y = pack_bf16x2(v.z * scale, v.w * scale);
    *reinterpret_cast<uint2*>(dqkv + (size_t)t * width + col + c) = o;
  }
}

static void launch_cast(const float* acc, int slabs, __nv_bfloat16* dqkv, int T, int cols, int col, int width, float scale,
                        cudaStream_t stream) {
  const long long total = (long long)T * (cols / 4), cap = (long long)num_sms() * 8;
  const long long blocks = (total + 255) / 256;
  auto kernel = slabs > 1 ? fmha_cast_kernel<true> : fmha_cast_kernel<false>;
  kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, stream>>>(acc, slabs, dqkv, T, cols, col, width, scale);
}

template <int D, bool ORDERED>
static int launch_bwd(const CUtensorMap& mqkv, const CUtensorMap& mdo, const FmhaBwdParams& p, int num_tiles,
                      cudaStream_t stream) {
  using L = BwdSmem<D>;
  auto kernel = fmha_bwd_kernel<D, ORDERED>;
  static bool configured = false;
  if (!configured) {
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, kernel);
    if (e != cudaSuccess) return (int)e;
    // the warpgroups' shares are drawn from the registers that the block is launched with: with fewer they would wait for good
    if (attr.numRegs * 4 < 2 * kRegsMath + kRegsDq + kRegsIssue) return -6;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const long long blocks = (long long)num_tiles * p.Hkv * p.head_splits;
  if (blocks > 0x7fffffffll) return -4;
  kernel<<<(unsigned)blocks, kBwdThreads, L::kTotal, stream>>>(mqkv, mdo, p);
  return (int)cudaGetLastError();
}

}  // namespace sb

using namespace sb;

// qkv: packed forward input; out/d_out: [T, Hq*D]; dq_accum: fp32 scratch [T, Hq*D]; delta: fp32 scratch [Hq, T]; dqkv: packed
// gradient output.  head_splits > 1 divides the q heads of each group over that many blocks, whose dK and dV go to dkv_accum:
// fp32 scratch [head_splits, T, 2*Hkv*D].  turn: int scratch [Hq, T + 1] for ordered sums, or null.  For these all tiles of a
// sequence stand in the lists, tile_k0 ascending, and rows outside the sequences get what dq_accum holds as their q gradient.
extern "C" int sb_fmha_bwd(const void* qkv, const void* out, const void* d_out, const float* lse, float* delta,
                           float* dq_accum, float* dkv_accum, int* turn, void* dqkv, const int* tile_seq_start,
                           const int* tile_seq_len, const int* tile_k0, int num_tiles, int T, int Hq, int Hkv, int D,
                           int causal, int head_splits, float scale, int* status, cudaStream_t stream) {
  if (num_tiles == 0 || T == 0) return 0;
  if (D != 64 && D != 128) return -2;
  if (head_splits < 1 || head_splits > Hq / Hkv || (head_splits > 1 && !dkv_accum)) return -3;
  static thread_local bool tl_context_bound = false;
  if (!tl_context_bound) {
    cudaFree(0);
    tl_context_bound = true;
  }
  const long long width = (long long)(Hq + 2 * Hkv) * D;
  const long long qwidth = (long long)Hq * D;
  CUtensorMap mqkv, mdo;
  int r = make_tensor_map_bf16_2d(&mqkv, qkv, width, T, width, 64, 128);
  if (r) return r;
  r = make_tensor_map_bf16_2d(&mdo, d_out, qwidth, T, qwidth, 64, 128);
  if (r) return r;
  if (!turn) cudaMemsetAsync(dq_accum, 0, sizeof(float) * (size_t)T * qwidth, stream);
  {
    const long long warps = (long long)T * Hq;
    const int threads = 256;
    const long long blocks = (warps * 32 + threads - 1) / threads;
    fmha_delta_kernel<<<(unsigned)blocks, threads, 0, stream>>>((const __nv_bfloat16*)out, (const __nv_bfloat16*)d_out,
                                                                delta, turn, T, Hq, D);
  }
  FmhaBwdParams p;
  p.tile_seq_start = tile_seq_start; p.tile_seq_len = tile_seq_len; p.tile_k0 = tile_k0;
  p.lse = lse; p.delta = delta; p.dq_accum = dq_accum; p.dkv_accum = dkv_accum; p.turn = turn;
  p.dqkv = reinterpret_cast<__nv_bfloat16*>(dqkv);
  p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal; p.head_splits = head_splits;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  if (turn) r = D == 128 ? launch_bwd<128, true>(mqkv, mdo, p, num_tiles, stream) : launch_bwd<64, true>(mqkv, mdo, p, num_tiles, stream);
  else r = D == 128 ? launch_bwd<128, false>(mqkv, mdo, p, num_tiles, stream) : launch_bwd<64, false>(mqkv, mdo, p, num_tiles, stream);
  if (r) return r;
  launch_cast(dq_accum, 1, p.dqkv, T, (int)qwidth, 0, (int)width, scale, stream);
  if (head_splits > 1) launch_cast(dkv_accum, head_splits, p.dqkv, T, 2 * Hkv * D, (int)qwidth, (int)width, 1.f, stream);
  return (int)cudaGetLastError();
}
