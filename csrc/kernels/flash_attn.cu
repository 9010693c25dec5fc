// Flash-style attention forward / backward for head dim 64 on tcgen05 tensor cores.
//
// Replaces `at::scaled_dot_product_attention` (flodl-sys/ops_nn.cpp:367-388) behind the encoder
// layers (flodl-hf/src/models/transformer_layer.rs:243-251) and the decomposed
// matmul / masked_fill / softmax / matmul chain of `MultiheadAttention`
// (flodl/src/nn/attention.rs:108-151): additive key mask [B,S], causal masking, attention-prob
// dropout, O(S) memory (only the log-sum-exp per row is saved).
//
// This file: a single key block (S <= 128), one CTA per (head, batch) in either pass; flash_attn_long.cu has more. 4 warps (one TMEM lane = one
// query row per thread) do the softmax arithmetic; a fifth warp issues every TMA load and every `tcgen05.mma` from one thread.
// Q, K, V, dO tiles arrive by TMA with 128-byte swizzle in their natural [row][64] layout; the
// same tile serves as a K-major operand (QK^T, dO V^T) or an MN-major operand (P V, P^T dO,
// dS^T Q, dS K) by flipping the major bit of the instruction descriptor, so nothing is transposed.
// P and dS are written to shared memory by the softmax threads in the swizzled layout the MMA
// expects. All accumulators (S, dP, O, dQ, dK, dV) live in TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../include/flodl_b200.h"
#include "flash_attn_common.cuh"

namespace fb {

// Per-CTA timeline of the single-block kernels (a tuning aid, compiled in only with -DFB_TIMELINE=1): 8 clock64
// stamps per CTA for the first 1024 CTAs of a launch (forward) / 16 per CTA (backward), read back with fb_attn_timeline.
#ifndef FB_TIMELINE
#define FB_TIMELINE 0
#endif
#if FB_TIMELINE
__device__ long long g_attn_ts[16 * 1024];
#define FB_ATTN_TS(slot) do { const int cta_ = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z); if (cta_ < 1024) { \
    long long v_ = clock64(); if ((slot) >= 14) { unsigned long long g_; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(g_)); v_ = static_cast<long long>(g_); } \
    g_attn_ts[cta_ * 16 + (slot)] = v_; } } while (0)
#else
#define FB_ATTN_TS(slot) do { } while (0)
#endif

// ===================================================================================== forward
// A single key block (S <= 128, the encoder shapes): Q and K are dead once S = Q K^T has completed, so the probabilities
// are written over them (49 KB); with the output accumulator taking over the TMEM columns of S as well (128 columns per
// CTA), four CTAs share an SM and hide one another's load / MMA / softmax latencies, which is what bounds a
// 128 x 128 x 64 problem. Keys are worked on by thirty-twos up to the sequence's end, two of them an instruction. us, without dropout, in brackets always all 128, one
// an instruction and a full-range power: batch x heads x length 32 x 12 x 128 10.2 (10.7), 64 x 12 x 16 8.4 (14.4), 32 x 4 x 64 causal 4.1 (5.4), 1 x 12 x 77 4.4 (5.2).
struct FwdSmem {
  static constexpr int Q = 0, K = 16384, V = 2 * 16384;
  static constexpr int P = 0;                    // 2 panels, over Q and K
  static constexpr int MASK = V + 16384;         // 128 floats
  static constexpr int BARS = MASK + 512;
  static constexpr int TOTAL = BARS + 256;
};

__global__ void __launch_bounds__(kAttnThreads, 4)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, __nv_bfloat16* __restrict__ o, float* __restrict__ lse,
                const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kTmemCols = 128;
  using L = FwdSmem;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t* in_full = bars + 0;
  uint64_t* s_full = bars + 1;
  uint64_t* p_ready = bars + 2;
  uint64_t* o_full = bars + 3;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* mask_s = reinterpret_cast<float*>(smem + L::MASK);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, b = blockIdx.y;
  if (threadIdx.x == 0) { FB_ATTN_TS(0); FB_ATTN_TS(14); }
  const unsigned long long seed = p.seed + (p.seed_dev ? *p.seed_dev : 0ull);

  if (threadIdx.x == 0) {
    mbar_init(in_full, 1);
    mbar_init(s_full, 1);
    mbar_init(p_ready, 4);
    mbar_init(o_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 4) {
    tmem_alloc<1>(tmem_slot, kTmemCols);
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base;
  pdl_entry();       // barriers, TMEM and descriptors are set up; everything below reads the predecessor's output
  if (threadIdx.x == 0) FB_ATTN_TS(1);
  // every softmax thread has read its row of S before P V is issued (p_ready), so O reuses S's columns
  const uint32_t tmem_O = tmem_base;
  const int keys = min(kBlk, (p.S + 31) & ~31);      // what is worked on: keys past these have no weight

  if (warp == 4) {
    if (lane == 0) {
      // ---------------------------------------------------------- loads + MMA issue (one thread)
      const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_o = make_idesc_bf16(128, kHD, 0, 1);
      const uint32_t sQ = smem_u32(smem + L::Q), sK = smem_u32(smem + L::K), sV = smem_u32(smem + L::V), sP = smem_u32(smem + L::P);
      mbar_expect_tx(in_full, 49152);
      tma_load_4d(smem + L::Q, &tmQ, in_full, 0, 0, h, b);
      tma_load_4d(smem + L::K, &tmK, in_full, 0, 0, h, b);
      tma_load_4d(smem + L::V, &tmV, in_full, 0, 0, h, b);
      bool ok = mbar_wait(in_full, 0, abort_flag, p.status, kStatusWaitFull);
      if (ok) {
        tc_fence_after_sync();
        FB_ATTN_TS(2);
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tmem_S, make_smem_desc(sQ + k4 * 32, 16, 1024), make_smem_desc(sK + k4 * 32, 16, 1024), idesc_s, k4 > 0);
        umma_commit(s_full);
        ok = mbar_wait(p_ready, 0, abort_flag, p.status, kStatusWaitEpi);
      }
      if (ok) {
        tc_fence_after_sync();
        // O = P V
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          if (k8 * 16 < keys) umma_bf16<1>(tmem_O, make_smem_desc(sP + (k8 >> 2) * 16384 + (k8 & 3) * 32, 16, 1024), make_smem_desc(sV + k8 * 2048, 8192, 1024), idesc_o, k8 > 0);
        umma_commit(o_full);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax threads
    const int t = threadIdx.x;            // query row == TMEM lane
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const uint32_t sP = smem_u32(smem + L::P);
    const F2 sc2 = f2_splat(p.scale * kLog2e);
    const float inv_keep = p.p_drop > 0.f ? 1.f / (1.f - p.p_drop) : 1.f;
    // the additive mask (mask * log2e; -inf beyond S)
    mask_s[t] = (t < p.S) ? (p.mask ? p.mask[static_cast<long long>(b) * p.S + t] * kLog2e : 0.f) : -INFINITY;
    asm volatile("bar.sync 1, 128;");
    bool ok = __all_sync(0xffffffffu, mbar_wait(s_full, 0, abort_flag, p.status, kStatusWaitAccum));
    if (ok) {
      tc_fence_after_sync();
      if (t == 0) FB_ATTN_TS(3);
      // pass 1: row maximum
      float m_blk = -INFINITY;
#pragma unroll 1
      for (int c = 0; c < keys; c += 32) {
        uint32_t v[32];
        tmem_ld32(tmem_S + lane_base + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int i4 = 0; i4 < 32; i4 += 4) {
          const float4 mk = *reinterpret_cast<const float4*>(mask_s + c + i4);     // one 16-byte shared load per 4 keys
          const F2 s01 = f2_fma(f2_make(__uint_as_float(v[i4]), __uint_as_float(v[i4 + 1])), sc2, f2_make(mk.x, mk.y));
          const F2 s23 = f2_fma(f2_make(__uint_as_float(v[i4 + 2]), __uint_as_float(v[i4 + 3])), sc2, f2_make(mk.z, mk.w));
          float s[4];
          f2_get(s01, s[0], s[1]);
          f2_get(s23, s[2], s[3]);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (p.causal && c + i4 + k > t) s[k] = -INFINITY;
            m_blk = fmaxf(m_blk, s[k]);
          }
        }
      }
      const float m_use = (m_blk == -INFINITY) ? 0.f : m_blk;
      float l = 0.f;
      const F2 minus_m = f2_splat(-m_use);
      // pass 2: probabilities -> shared memory (bf16, swizzled), row sum
#pragma unroll 1
      for (int c = 0; c < keys; c += 32) {
        uint32_t v[32];
        tmem_ld32(tmem_S + lane_base + c, v);
        tmem_ld_wait();
        float pr[32];
#pragma unroll
        for (int i4 = 0; i4 < 32; i4 += 4) {
          const float4 mk = *reinterpret_cast<const float4*>(mask_s + c + i4);
          // score - row maximum in one FMA, two keys an instruction
          const F2 s01 = f2_fma(f2_make(__uint_as_float(v[i4]), __uint_as_float(v[i4 + 1])), sc2, f2_add(f2_make(mk.x, mk.y), minus_m));
          const F2 s23 = f2_fma(f2_make(__uint_as_float(v[i4 + 2]), __uint_as_float(v[i4 + 3])), sc2, f2_add(f2_make(mk.z, mk.w), minus_m));
          float s[4];
          f2_get(s01, s[0], s[1]);
          f2_get(s23, s[2], s[3]);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (p.causal && c + i4 + k > t) s[k] = -INFINITY;
            pr[i4 + k] = ex2_approx(s[k]);
            l += pr[i4 + k];
          }
        }
        if (p.p_drop > 0.f) {
          const unsigned long long base = ((static_cast<unsigned long long>(b) * p.H + h) * p.S + t) * p.S + c;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float s4[4];
            dropout_scale4(seed, base + i, p.p_drop, inv_keep, s4);
#pragma unroll
            for (int k = 0; k < 4; ++k) pr[i + k] *= s4[k];
          }
        }
        const uint32_t panel = sP + (c >> 6) * 16384;
#pragma unroll
        for (int g = 0; g < 4; ++g) st_shared_v4(swz_chunk(panel, t, ((c & 63) >> 3) + g), pack8(pr + 8 * g));
      }
      tc_fence_before_sync();
      fence_proxy_async_smem();
      if (t == 0) FB_ATTN_TS(4);
      arrive_warp(p_ready, lane);
      ok = __all_sync(0xffffffffu, mbar_wait(o_full, 0, abort_flag, p.status, kStatusWaitAccum));   // warp-uniform: the staged stores below use __syncwarp
      if (ok) {
        tc_fence_after_sync();
        if (t == 0) FB_ATTN_TS(5);
        // normalise, then out through the warp's staging area (P is dead: P V has completed)
        const float inv_l = l > 0.f ? 1.f / l : 0.f;
        const uint32_t stage = sP + warp * 4096;
#pragma unroll
        for (int c = 0; c < kHD; c += 32) {
          uint32_t v[32];
          tmem_ld32(tmem_O + lane_base + c, v);
          tmem_ld_wait();
          float f[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]) * inv_l;
          stage_half(stage, lane, c, f);
        }
        flush_rows(stage, lane, o + static_cast<long long>(b) * p.osb + static_cast<long long>(h) * p.osh, p.oss, warp * 32, p.S);
        // natural-log LSE of the scaled, masked scores
        if (t < p.S) lse[(static_cast<long long>(b) * p.H + h) * p.S + t] = (l > 0.f) ? (m_blk + log2f(l)) / kLog2e : -INFINITY;
      }
    }
  }
  if (threadIdx.x == 0) FB_ATTN_TS(6);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, kTmemCols);
  }
  if (threadIdx.x == 0) { FB_ATTN_TS(7); FB_ATTN_TS(15); }
}

// ==================================================================================== backward
// A single key block (S <= 128): V is dead once dP = dO V^T has completed, so the first dS panel takes its place
// (112.75 KB), and dV / dK / dQ accumulate in the columns S and dP occupied until the softmax threads had read them
// (256 columns): two CTAs share an SM.
struct BwdSmem {
  static constexpr int Q = 0, DO = 16384, K = 2 * 16384;
  static constexpr int P = 3 * 16384;             // 2 panels
  static constexpr int V = 5 * 16384;
  static constexpr int DS = 5 * 16384;            // 2 panels, the first one over V
  static constexpr int MASK = 7 * 16384;
  static constexpr int BARS = MASK + 512;
  static constexpr int TOTAL = BARS + 256;
};

// kShort, for sequences of up to 96 keys: they are worked on by thirty-twos up to the sequence's end. us, in brackets always all 128: batch x heads x length
// 64 x 12 x 16 16.8 (22.7), 32 x 4 x 64 causal 6.6 (7.4), 8 x 12 x 33 with dropout 7.4 (9.3), 32 x 12 x 80 with dropout 20.0 (22.5); with nothing to leave out, loops whose
// ends are not known cost 32 x 12 x 128 20.3 (20.0), with dropout 27.4 (25.8).
template <bool kShort>
__global__ void __launch_bounds__(kAttnThreads, 2)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                const float* __restrict__ lse, __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk,
                __nv_bfloat16* __restrict__ dv, const AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // The layout leaves no room for alignment slack (two CTAs must fit in one SM): it relies on the 1024-byte alignment
  // of the dynamic shared-memory window and reports instead of computing if that does not hold.
  uint8_t* smem = smem_raw;
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, static_cast<int>(kStatusBadArg));
    return;
  }
  using L = BwdSmem;
  constexpr int kTmemCols = 256;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;
  uint64_t* sdp_full = bars + 2;
  uint64_t* pds_ready = bars + 3;
  uint64_t* grads_full = bars + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* mask_s = reinterpret_cast<float*>(smem + L::MASK);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, b = blockIdx.y;
  if (threadIdx.x == 0) FB_ATTN_TS(8);
  const unsigned long long seed = p.seed + (p.seed_dev ? *p.seed_dev : 0ull);

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(q_full, 1);
    mbar_init(sdp_full, 1);
    mbar_init(pds_ready, 4);
    mbar_init(grads_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == 4) {
    tmem_alloc<1>(tmem_slot, kTmemCols);
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tDP = tmem_base + 128;
  pdl_entry();
  if (threadIdx.x == 0) FB_ATTN_TS(7);
  // S and dP have been read by every softmax thread (pds_ready) before the gradient MMAs are issued
  const int keys = kShort ? (p.S + 31) & ~31 : kBlk;      // what is worked on: keys past these have no weight, and rows of dK and dV that are not stored
  const uint32_t tDV = tmem_base, tDK = tmem_base + 64, tDQ = tmem_base + 128;

  if (warp == 4) {
    if (lane == 0) {
      const uint32_t idesc_kk = make_idesc_bf16(128, 128, 0, 0);      // S, dP: both operands K-major
      const uint32_t idesc_mn = make_idesc_bf16(128, kHD, 1, 1);      // dV, dK: A^T (MN-major) x MN-major
      const uint32_t idesc_kn = make_idesc_bf16(128, kHD, 0, 1);      // dQ: K-major x MN-major
      const uint32_t sQ = smem_u32(smem + L::Q), sDO = smem_u32(smem + L::DO);
      const uint32_t sK = smem_u32(smem + L::K), sV = smem_u32(smem + L::V);
      const uint32_t sP = smem_u32(smem + L::P), sDS = smem_u32(smem + L::DS);
      mbar_expect_tx(kv_full, 32768);
      tma_load_4d(smem + L::K, &tmK, kv_full, 0, 0, h, b);
      tma_load_4d(smem + L::V, &tmV, kv_full, 0, 0, h, b);
      mbar_expect_tx(q_full, 32768);
      tma_load_4d(smem + L::Q, &tmQ, q_full, 0, 0, h, b);
      tma_load_4d(smem + L::DO, &tmDO, q_full, 0, 0, h, b);
      bool ok = mbar_wait(kv_full, 0, abort_flag, p.status, kStatusWaitFull) && mbar_wait(q_full, 0, abort_flag, p.status, kStatusWaitFull);
      if (ok) {
        tc_fence_after_sync();
        FB_ATTN_TS(5);
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tS, make_smem_desc(sQ + k4 * 32, 16, 1024), make_smem_desc(sK + k4 * 32, 16, 1024), idesc_kk, k4 > 0);
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tDP, make_smem_desc(sDO + k4 * 32, 16, 1024), make_smem_desc(sV + k4 * 32, 16, 1024), idesc_kk, k4 > 0);
        umma_commit(sdp_full);
        ok = mbar_wait(pds_ready, 0, abort_flag, p.status, kStatusWaitEpi);
      }
      if (ok) {
        tc_fence_after_sync();
        // dV = P^T dO ; dK = dS^T Q   (M = key index, K = query index: 8 steps of 16 rows)
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16<1>(tDV, make_smem_desc(sP + k8 * 2048, 16384, 1024), make_smem_desc(sDO + k8 * 2048, 8192, 1024), idesc_mn, k8 > 0);
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16<1>(tDK, make_smem_desc(sDS + k8 * 2048, 16384, 1024), make_smem_desc(sQ + k8 * 2048, 8192, 1024), idesc_mn, k8 > 0);
        // dQ = dS K   (M = query, K = key index)
        if constexpr (!kShort) {
#pragma unroll
          for (int k8 = 0; k8 < kBlk / 16; ++k8)
            umma_bf16<1>(tDQ, make_smem_desc(sDS + (k8 >> 2) * 16384 + (k8 & 3) * 32, 16, 1024), make_smem_desc(sK + k8 * 2048, 8192, 1024), idesc_kn, k8 > 0);
        } else {
#pragma unroll 1
          for (int k8 = 0; k8 < keys / 16; ++k8)
            umma_bf16<1>(tDQ, make_smem_desc(sDS + (k8 >> 2) * 16384 + (k8 & 3) * 32, 16, 1024), make_smem_desc(sK + k8 * 2048, 8192, 1024), idesc_kn, k8 > 0);
        }
        umma_commit(grads_full);
      }
    }
  } else {
    const int t = threadIdx.x;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const uint32_t sP = smem_u32(smem + L::P), sDS = smem_u32(smem + L::DS);
    const float sc = p.scale * kLog2e;
    const float inv_keep = p.p_drop > 0.f ? 1.f / (1.f - p.p_drop) : 1.f;
    const int q = t;
    const bool q_ok = q < p.S;
    // The mask and the row statistics are in flight together: the LSE of a query row and D = rowsum(dO * O) (eight lanes per row, coalesced). The four
    // warps start them at once, behind the tensor loads: 256 x 12 heads x 128 tokens 111 us, without the barrier 132.
    asm volatile("bar.sync 1, 128;");
    const float mraw = (t < p.S && p.mask) ? __ldg(p.mask + static_cast<long long>(b) * p.S + t) : 0.f;
    const float lse_q = q_ok ? __ldg(lse + (static_cast<long long>(b) * p.H + h) * p.S + q) * kLog2e : 0.f;
    const float Dq = row_dot64(o + static_cast<long long>(b) * p.osb + static_cast<long long>(h) * p.osh,
                               d_o + static_cast<long long>(b) * p.osb + static_cast<long long>(h) * p.osh, p.oss, warp * 32, p.S, lane);
    mask_s[t] = (t < p.S) ? mraw * kLog2e : -INFINITY;
    asm volatile("bar.sync 1, 128;");
    if (t == 0) FB_ATTN_TS(9);
    bool ok = mbar_wait(sdp_full, 0, abort_flag, p.status, kStatusWaitAccum);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after_sync();
      if (t == 0) FB_ATTN_TS(10);
#pragma unroll 1
      for (int c = 0; c < keys; c += 32) {
        uint32_t sv[32], dpv[32];
        tmem_ld32(tS + lane_base + c, sv);
        tmem_ld32(tDP + lane_base + c, dpv);
        tmem_ld_wait();
        float pr[32], ds[32];
        float z[32];
        if (p.p_drop > 0.f) {
          const unsigned long long base = ((static_cast<unsigned long long>(b) * p.H + h) * p.S + q) * p.S + c;
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            float s4[4];
            dropout_scale4(seed, base + e, p.p_drop, inv_keep, s4);
#pragma unroll
            for (int k = 0; k < 4; ++k) z[e + k] = s4[k];
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) z[e] = 1.f;
        }
        const bool row_live = q_ok && lse_q != -INFINITY;
#pragma unroll
        for (int e4 = 0; e4 < 32; e4 += 4) {
          const float4 mk = *reinterpret_cast<const float4*>(mask_s + c + e4);
          const float mk4[4] = {mk.x - lse_q, mk.y - lse_q, mk.z - lse_q, mk.w - lse_q};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int e = e4 + k;
            float s = __uint_as_float(sv[e]) * sc + mk4[k];   // score - log-sum-exp in one FMA
            if (p.causal && c + e > q) s = -INFINITY;
            const float pe = row_live ? exp2f(s) : 0.f;
            const float dpe = __uint_as_float(dpv[e]) * z[e];
            pr[e] = pe * z[e];
            ds[e] = pe * (dpe - Dq) * p.scale;
          }
        }
        const uint32_t pp = sP + (c >> 6) * 16384, dp = sDS + (c >> 6) * 16384;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          st_shared_v4(swz_chunk(pp, t, ((c & 63) >> 3) + g), pack8(pr + 8 * g));
          st_shared_v4(swz_chunk(dp, t, ((c & 63) >> 3) + g), pack8(ds + 8 * g));
        }
      }
      tc_fence_before_sync();
      fence_proxy_async_smem();
      if (t == 0) FB_ATTN_TS(11);
      arrive_warp(pds_ready, lane);
      ok = __all_sync(0xffffffffu, mbar_wait(grads_full, 0, abort_flag, p.status, kStatusWaitAccum));   // warp-uniform: staged stores below
    }
    if (ok) {
      tc_fence_after_sync();
      if (t == 0) FB_ATTN_TS(12);
      // dQ, dK, dV rows through the staging area (the P panels are dead: every MMA has completed)
      const uint32_t stage = sP + warp * 4096;
      __nv_bfloat16* const bases[3] = {dq, dk, dv};
      const uint32_t cols[3] = {tDQ, tDK, tDV};
#pragma unroll
      for (int which = 0; which < 3; ++which) {
#pragma unroll
        for (int c = 0; c < kHD; c += 32) {
          uint32_t v[32];
          tmem_ld32(cols[which] + lane_base + c, v);
          tmem_ld_wait();
          float f[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) f[e] = __uint_as_float(v[e]);
          stage_half(stage, lane, c, f);
        }
        flush_rows(stage, lane, bases[which] + static_cast<long long>(b) * p.gsb + static_cast<long long>(h) * p.gsh, p.gss, warp * 32, p.S);
      }
    }
  }
  if (threadIdx.x == 0) FB_ATTN_TS(13);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, kTmemCols);
  }
}

}  // namespace fb

#if FB_TIMELINE
extern "C" int fb_attn_timeline(long long* host_out, int count) {
  return static_cast<int>(cudaMemcpyFromSymbol(host_out, fb::g_attn_ts, sizeof(long long) * static_cast<size_t>(count)));
}
#endif

extern "C" int fb_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const float* mask, int B, int H,
                           int S, const long long* qkv_strides, const long long* o_strides, float scale, int causal,
                           float p_drop, unsigned long long seed, const unsigned long long* seed_dev, int* status,
                           void* stream) {
  using namespace fb;
  if (B <= 0 || H <= 0 || S <= 0) return 0;
  const long long sb = qkv_strides[0], ss = qkv_strides[1], sh = qkv_strides[2];
  if (!strides_ok(q, sb, ss, sh) || !strides_ok(k, sb, ss, sh) || !strides_ok(v, sb, ss, sh) ||
      !strides_ok(o, o_strides[0], o_strides[1], o_strides[2]))
    return -3;
  CUtensorMap tq, tk, tv;
  int r;
  if ((r = make_tmap_bshd(&tq, q, B, H, S, sb, ss, sh))) return r;
  if ((r = make_tmap_bshd(&tk, k, B, H, S, sb, ss, sh))) return r;
  if ((r = make_tmap_bshd(&tv, v, B, H, S, sb, ss, sh))) return r;
  const AttnParams p = make_params(B, H, S, qkv_strides, o_strides, o_strides, mask, scale, causal, p_drop, seed, seed_dev, status);
  if (S > kBlk) return attn_fwd_long(tq, tk, tv, o, lse, p, static_cast<cudaStream_t>(stream));
  if (const cudaError_t e = allow_smem<attn_fwd_kernel>(FwdSmem::TOTAL + 1024, true)) return static_cast<int>(e);
  const cudaError_t le = launch_pdl(attn_fwd_kernel, dim3(H, B), dim3(kAttnThreads), static_cast<size_t>(FwdSmem::TOTAL + 1024), static_cast<cudaStream_t>(stream), tq, tk, tv,
                                    static_cast<__nv_bfloat16*>(o), lse, p);
  return static_cast<int>(le != cudaSuccess ? le : cudaGetLastError());
}

// dq_accum: fp32 scratch of B * H * S * 64 values; only touched when there is more than one key block (S > 128), may be
// null otherwise.
extern "C" int fb_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                           const float* mask, void* dq, void* dk, void* dv, float* dq_accum, int B, int H, int S,
                           const long long* qkv_strides, const long long* o_strides, const long long* g_strides,
                           float scale, int causal, float p_drop, unsigned long long seed,
                           const unsigned long long* seed_dev, int* status, void* stream) {
  using namespace fb;
  if (B <= 0 || H <= 0 || S <= 0) return 0;
  if (S > kBlk && !dq_accum) return -4;
  const long long sb = qkv_strides[0], ss = qkv_strides[1], sh = qkv_strides[2];
  if (!strides_ok(q, sb, ss, sh) || !strides_ok(k, sb, ss, sh) || !strides_ok(v, sb, ss, sh)) return -3;
  if (!strides_ok(o, o_strides[0], o_strides[1], o_strides[2]) || !strides_ok(d_o, o_strides[0], o_strides[1], o_strides[2])) return -3;
  if (!strides_ok(dq, g_strides[0], g_strides[1], g_strides[2]) || !strides_ok(dk, g_strides[0], g_strides[1], g_strides[2]) ||
      !strides_ok(dv, g_strides[0], g_strides[1], g_strides[2]))
    return -3;
  CUtensorMap tq, tk, tv, tdo;
  int r;
  if ((r = make_tmap_bshd(&tq, q, B, H, S, sb, ss, sh))) return r;
  if ((r = make_tmap_bshd(&tk, k, B, H, S, sb, ss, sh))) return r;
  if ((r = make_tmap_bshd(&tv, v, B, H, S, sb, ss, sh))) return r;
  if ((r = make_tmap_bshd(&tdo, d_o, B, H, S, o_strides[0], o_strides[1], o_strides[2]))) return r;
  const AttnParams p = make_params(B, H, S, qkv_strides, o_strides, g_strides, mask, scale, causal, p_drop, seed, seed_dev, status);
  if (S > kBlk) return attn_bwd_long(tq, tk, tv, tdo, o, d_o, lse, dq, dk, dv, dq_accum, p, static_cast<cudaStream_t>(stream));
  const auto go = [&](auto is_short) -> int {
    constexpr bool kShort = decltype(is_short)::value;
    if (const cudaError_t e = allow_smem<attn_bwd_kernel<kShort>>(BwdSmem::TOTAL, true)) return static_cast<int>(e);
    const cudaError_t le = launch_pdl(attn_bwd_kernel<kShort>, dim3(H, B), dim3(kAttnThreads), static_cast<size_t>(BwdSmem::TOTAL), static_cast<cudaStream_t>(stream),
                                      tq, tk, tv, tdo, static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(d_o), lse,
                                      static_cast<__nv_bfloat16*>(dq), static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), p);
    return static_cast<int>(le != cudaSuccess ? le : cudaGetLastError());
  };
  return S <= 96 ? go(std::true_type()) : go(std::false_type());
}
