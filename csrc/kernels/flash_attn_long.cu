// Attention over several key blocks (S > 128), head dim 64, on tcgen05. The entry points and the kernels of a single
// key block are in flash_attn.cu.
//
// Backward: one CTA per (key block of 128 rows, head, batch) walks the query blocks that see it. K, V and the dK / dV
// accumulators stay put; Q and dO stream through a three-stage TMA ring. Roles: 8 softmax warps (thread = one query row x
// 64 keys), 4 warps that drain dQ, one MMA issuer, one TMA producer. S and dP of the next query block are issued as soon
// as the softmax warps have loaded this block's into registers, so the tensor cores work under the exponentials.
// A query block's dQ is a sum over key blocks, i.e. over CTAs: it is added into an fp32 scratch with 16-byte vector
// reductions. The scratch is not row-major: within the 32 rows a warp owns, 16-byte chunk c of row r sits at
// (c * rows + r) * 16, so the 32 lanes of a reduction (one row each) hit 512 contiguous bytes. A pass before zeroes the
// scratch and leaves D = rowsum(dO * O) in the first word of each dQ row; a pass after turns the scratch into bf16 rows.
// What bounds it: shared-memory bandwidth (P and dS are written once and read by three products) about level with the
// exponentials. One CTA per (head, batch) walking all key blocks in turn, which this replaces, left most of the chip idle.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../include/flodl_b200.h"
#include "flash_attn_common.cuh"

namespace fb {

// ==================================================================================== backward
namespace {

constexpr int kSMs = 148;
constexpr int kBwdSoftmaxWarps = 8;
constexpr int kBwdThreads = 32 * (kBwdSoftmaxWarps + 4 + 2);

// Every byte of it is needed (226.75 KB), so there is no slack for alignment: the kernel relies on the 1024-byte alignment of the
// dynamic shared-memory window and reports instead of computing if that does not hold.
struct BwdLong {
  static constexpr int Q = 0;                                   // 2 x 16 KB
  static constexpr int DO = Q + 2 * 16384;                      // 2 x 16 KB
  static constexpr int K = DO + 2 * 16384;
  static constexpr int V = K + 16384;
  static constexpr int P = V + 16384;                           // 2 x (2 panels of 16 KB)
  static constexpr int DS = P + 2 * 32768;                      // 2 x (2 panels of 16 KB)
  static constexpr int STATS = DS + 2 * 32768;                  // 2 x 128 x {lse, D}
  static constexpr int MASK = STATS + 2 * 128 * 8;              // 128 floats
  static constexpr int BARS = MASK + 512;
  static constexpr int TOTAL = BARS + 192;
};
static_assert(BwdLong::TOTAL <= 227 * 1024, "shared memory budget");

// CTA index -> (block, head, batch). Causal: every block of equal length before the next shorter one (the longest first, so
// the last wave is short). Otherwise all blocks of a head together, which keeps its K / V (or Q / dO) in L2.
__device__ __forceinline__ void decode_block(int lin, int nblk, int H, int B, bool causal, int& blk, int& h, int& b) {
  int hb;
  if (causal) {
    blk = lin / (H * B);
    hb = lin - blk * (H * B);
  } else {
    hb = lin / nblk;
    blk = lin - hb * nblk;
  }
  b = hb / H;
  h = hb - b * H;
}

// The (key block, query block) tiles of one CTA of the backward kernel, in order. Work items (key blocks) are dealt out in rounds of
// gridDim.x, every other round backwards: with the longest items first, that evens out the sums.
struct BwdTiles {
  const AttnParams& p;
  int nblk, round = 0, it = 0;      // `it` counts the query blocks of the current item
  int j = 0, h = 0, b = 0, i0 = 0, n = 0;
  bool valid = true;
  __device__ explicit BwdTiles(const AttnParams& p_) : p(p_), nblk((p_.S + kBlk - 1) / kBlk) { item(); }
  __device__ void item() {
    const long long lin = static_cast<long long>(round) * gridDim.x + ((round & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    valid = lin < static_cast<long long>(nblk) * p.H * p.B;
    if (!valid) return;
    decode_block(static_cast<int>(lin), nblk, p.H, p.B, p.causal != 0, j, h, b);
    i0 = p.causal ? j : 0;
    n = nblk - i0;
  }
  __device__ void next() {
    if (++it == n) {
      it = 0;
      ++round;
      item();
    }
  }
  __device__ bool last() const { return it == n - 1; }
};

// Per query row: D = dot(dO, O) into the first word of the row's dQ slot (overwritten by attn_dq_kernel at the end), and the
// row's share of the dQ scratch zeroed. Eight lanes per row, rows of one (batch, head) consecutive.
__global__ void __launch_bounds__(256) attn_bwd_pre_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                                           __nv_bfloat16* __restrict__ dq, float* __restrict__ dq_accum, const AttnParams p) {
  pdl_entry();
  const long long rows = static_cast<long long>(p.B) * p.H * p.S;
  const int ch = threadIdx.x & 7;
  for (long long r = blockIdx.x * 32ll + (threadIdx.x >> 3); r < rows; r += gridDim.x * 32ll) {
    const int s = static_cast<int>(r % p.S);
    const long long bh = r / p.S;
    const int h = static_cast<int>(bh % p.H), b = static_cast<int>(bh / p.H);
    const long long off = b * p.osb + h * p.osh + s * p.oss + ch * 8;
    const uint4 xa = __ldg(reinterpret_cast<const uint4*>(o + off)), xb = __ldg(reinterpret_cast<const uint4*>(d_o + off));
    const __nv_bfloat162* ha = reinterpret_cast<const __nv_bfloat162*>(&xa);
    const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&xb);
    float d = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 fa = __bfloat1622float2(ha[e]), fb2 = __bfloat1622float2(hb[e]);
      d += fa.x * fb2.x + fa.y * fb2.y;
    }
    const unsigned m = 0xffu << (threadIdx.x & 24);
    d += __shfl_xor_sync(m, d, 1);
    d += __shfl_xor_sync(m, d, 2);
    d += __shfl_xor_sync(m, d, 4);
    if (ch == 0) *reinterpret_cast<float*>(dq + b * p.gsb + h * p.gsh + s * p.gss) = d;
    float4* z = reinterpret_cast<float4*>(dq_accum + r * kHD + ch * 8);
    z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// dQ scratch (layout above) -> bf16 rows. Eight lanes per row.
__global__ void __launch_bounds__(256) attn_dq_kernel(const float* __restrict__ dq_accum, __nv_bfloat16* __restrict__ dq, const AttnParams p) {
  pdl_entry();
  const long long rows = static_cast<long long>(p.B) * p.H * p.S;
  const int ch = threadIdx.x & 7;
  for (long long r = blockIdx.x * 32ll + (threadIdx.x >> 3); r < rows; r += gridDim.x * 32ll) {
    const int s = static_cast<int>(r % p.S);
    const long long bh = r / p.S;
    const int h = static_cast<int>(bh % p.H), b = static_cast<int>(bh / p.H);
    const int row0 = s & ~31, nr = min(32, p.S - row0);
    const float4* base = reinterpret_cast<const float4*>(dq_accum + (bh * p.S + row0) * kHD) + (s - row0);
    const float4 x = __ldcs(base + (2 * ch) * nr), y = __ldcs(base + (2 * ch + 1) * nr);
    const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    *reinterpret_cast<uint4*>(dq + b * p.gsb + h * p.gsh + s * p.gss + ch * 8) = pack8(v);
  }
}

__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_long_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmDO, const float* __restrict__ lse, const __nv_bfloat16* __restrict__ dq,
                     __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, float* __restrict__ dq_accum, const AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) set_status(p.status, kStatusBadArg);
    return;
  }
  using L = BwdLong;
  // Tile g of the CTA (counted over all its items) uses buffer g & 1 of everything that has two: Q / dO, P / dS, dQ, statistics.
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t* kv_full = bars;            // K and V of an item have landed
  uint64_t* acc_free = bars + 1;       // dK and dV of an item have been read out of TMEM
  uint64_t* sdp_full = bars + 2;       // S and dP are in TMEM
  uint64_t* sdp_free = bars + 3;       // ... and in the softmax warps' registers
  uint64_t* pds_ready = bars + 4;      // P and dS are in shared memory
  uint64_t* q_full = bars + 5;         // [2] Q and dO have landed
  uint64_t* grads = bars + 7;          // [2] dV, dK, dQ of the tile have retired: its Q / dO, P / dS may be overwritten, its dQ read
  uint64_t* dq_free = bars + 9;        // [2] dQ has been read
  uint64_t* stat_full = bars + 11;     // [2] lse and D are in shared memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* mask_s = reinterpret_cast<float*>(smem + L::MASK);
  float2* stats = reinterpret_cast<float2*>(smem + L::STATS);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned long long seed = p.seed + (p.seed_dev ? *p.seed_dev : 0ull);

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(acc_free, 32 * kBwdSoftmaxWarps);
    mbar_init(sdp_full, 1);
    mbar_init(sdp_free, 32 * kBwdSoftmaxWarps);
    mbar_init(pds_ready, 32 * kBwdSoftmaxWarps);
    for (int s = 0; s < 2; ++s) { mbar_init(&q_full[s], 1); mbar_init(&grads[s], 1); mbar_init(&dq_free[s], 4); mbar_init(&stat_full[s], 128); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kBwdSoftmaxWarps + 4) {
    tmem_alloc<1>(tmem_slot, 512);
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tDP = tmem_base + 128, tDV = tmem_base + 256, tDK = tmem_base + 320, tDQ = tmem_base + 384;
  pdl_entry();

  BwdTiles w(p);
  if (warp == kBwdSoftmaxWarps + 5) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      for (int g = 0; w.valid; ++g, w.next()) {
        const int buf = g & 1;
        if (!mbar_wait(&grads[buf], ((g >> 1) & 1) ^ 1, abort_flag, p.status, kStatusWaitEmpty)) break;        // tile g - 2
        mbar_expect_tx(&q_full[buf], 32768);
        tma_load_4d(smem + L::Q + buf * 16384, &tmQ, &q_full[buf], 0, (w.i0 + w.it) * kBlk, w.h, w.b);
        tma_load_4d(smem + L::DO + buf * 16384, &tmDO, &q_full[buf], 0, (w.i0 + w.it) * kBlk, w.h, w.b);
        if (w.it == 0) {
          if (g > 0 && !mbar_wait(&grads[buf ^ 1], ((g - 1) >> 1) & 1, abort_flag, p.status, kStatusWaitEmpty)) break;     // the last tile of the item before
          mbar_expect_tx(kv_full, 32768);
          tma_load_4d(smem + L::K, &tmK, kv_full, 0, w.j * kBlk, w.h, w.b);
          tma_load_4d(smem + L::V, &tmV, kv_full, 0, w.j * kBlk, w.h, w.b);
        }
      }
    }
  } else if (warp == kBwdSoftmaxWarps + 4) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc_kk = make_idesc_bf16(128, 128, 0, 0);      // S, dP: both operands K-major
      const uint32_t idesc_mn = make_idesc_bf16(128, kHD, 1, 1);      // dV, dK: A^T (MN-major) x MN-major
      const uint32_t idesc_kn = make_idesc_bf16(128, kHD, 0, 1);      // dQ: K-major x MN-major
      const uint32_t sK = smem_u32(smem + L::K), sV = smem_u32(smem + L::V);
      auto scores = [&](int g) {
        const uint32_t sQ = smem_u32(smem + L::Q + (g & 1) * 16384), sDO = smem_u32(smem + L::DO + (g & 1) * 16384);
        if (!mbar_wait(&q_full[g & 1], (g >> 1) & 1, abort_flag, p.status, kStatusWaitFull)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tS, make_smem_desc(sQ + k4 * 32, 16, 1024), make_smem_desc(sK + k4 * 32, 16, 1024), idesc_kk, k4 > 0);
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tDP, make_smem_desc(sDO + k4 * 32, 16, 1024), make_smem_desc(sV + k4 * 32, 16, 1024), idesc_kk, k4 > 0);
        umma_commit(sdp_full);
        return true;
      };
      bool ok = true;
      for (int g = 0; w.valid; ++g, w.next()) {
        if (w.it == 0) {       // an item's first S overwrites the last S of the item before, whose readers have arrived
          ok = mbar_wait(kv_full, w.round & 1, abort_flag, p.status, kStatusWaitFull) &&
               (g == 0 || mbar_wait(sdp_free, (g - 1) & 1, abort_flag, p.status, kStatusWaitEpi)) && scores(g);
          if (!ok) break;
        }
        if (!w.last()) {
          ok = mbar_wait(sdp_free, g & 1, abort_flag, p.status, kStatusWaitEpi) && scores(g + 1);
          if (!ok) break;
        }
        const int buf = g & 1;
        const uint32_t sQ = smem_u32(smem + L::Q + buf * 16384), sDO = smem_u32(smem + L::DO + buf * 16384);
        const uint32_t sP = smem_u32(smem + L::P + buf * 32768), sDS = smem_u32(smem + L::DS + buf * 32768);
        ok = mbar_wait(pds_ready, g & 1, abort_flag, p.status, kStatusWaitEpi) && mbar_wait(&dq_free[buf], ((g >> 1) & 1) ^ 1, abort_flag, p.status, kStatusWaitEpi) &&
             (w.it > 0 || mbar_wait(acc_free, (w.round & 1) ^ 1, abort_flag, p.status, kStatusWaitEpi));
        if (!ok) break;
        tc_fence_after_sync();
        // dV += P^T dO ; dK += dS^T Q   (M = key index, K = query index: 8 steps of 16 rows)
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16<1>(tDV, make_smem_desc(sP + k8 * 2048, 16384, 1024), make_smem_desc(sDO + k8 * 2048, 8192, 1024), idesc_mn, w.it > 0 || k8 > 0);
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16<1>(tDK, make_smem_desc(sDS + k8 * 2048, 16384, 1024), make_smem_desc(sQ + k8 * 2048, 8192, 1024), idesc_mn, w.it > 0 || k8 > 0);
        // dQ_tile = dS K   (M = query, K = key index)
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16<1>(tDQ + buf * 64, make_smem_desc(sDS + (k8 >> 2) * 16384 + (k8 & 3) * 32, 16, 1024), make_smem_desc(sK + k8 * 2048, 8192, 1024),
                       idesc_kn, k8 > 0);
        umma_commit(&grads[buf]);
      }
    }
  } else if (warp >= kBwdSoftmaxWarps) {
    // ------------------------------------------------------------------ row statistics in, dQ out
    const int quarter = warp & 3, t = quarter * 32 + lane;
    BwdTiles ahead = w;        // the tile whose statistics are fetched: two in front
    auto load_stats = [&]() {
      const int q = (ahead.i0 + ahead.it) * kBlk + t;
      // a row beyond S, or one that no key takes part in, gets +inf: every probability of it is then 2^-inf = 0
      float l = INFINITY, D = 0.f;
      if (q < p.S) {
        l = __ldg(lse + (static_cast<long long>(ahead.b) * p.H + ahead.h) * p.S + q);
        l = l == -INFINITY ? INFINITY : l * kLog2e;
        D = *reinterpret_cast<const float*>(dq + ahead.b * p.gsb + ahead.h * p.gsh + q * p.gss);
      }
      return make_float2(l, D);
    };
    auto put_stats = [&](int buf, float2 ld) {
      stats[buf * 128 + t] = ld;
      mbar_arrive(&stat_full[buf]);
      ahead.next();
    };
    for (int g = 0; g < 2 && ahead.valid; ++g) put_stats(g, load_stats());
    for (int g = 0; w.valid; ++g, w.next()) {
      const int buf = g & 1;
      const float2 stat = ahead.valid ? load_stats() : make_float2(0.f, 0.f);
      if (!__all_sync(0xffffffffu, mbar_wait(&grads[buf], (g >> 1) & 1, abort_flag, p.status, kStatusWaitAccum))) break;
      tc_fence_after_sync();
      uint32_t v0[32], v1[32];
      tmem_ld32(tDQ + buf * 64 + (static_cast<uint32_t>(quarter * 32) << 16), v0);
      tmem_ld32(tDQ + buf * 64 + 32 + (static_cast<uint32_t>(quarter * 32) << 16), v1);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dq_free[buf]);
      if (ahead.valid) put_stats(buf, stat);      // every softmax thread has read this buffer: its P and dS went into the products
      const int row0 = (w.i0 + w.it) * kBlk + quarter * 32, nr = min(32, p.S - row0);
      if (lane < nr) {
        float* dst = dq_accum + ((static_cast<long long>(w.b) * p.H + w.h) * p.S + row0) * kHD + lane * 4;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          red_add_v4(dst + static_cast<long long>(c) * nr * 4, __uint_as_float(v0[4 * c]), __uint_as_float(v0[4 * c + 1]), __uint_as_float(v0[4 * c + 2]),
                     __uint_as_float(v0[4 * c + 3]));
          red_add_v4(dst + static_cast<long long>(c + 8) * nr * 4, __uint_as_float(v1[4 * c]), __uint_as_float(v1[4 * c + 1]), __uint_as_float(v1[4 * c + 2]),
                     __uint_as_float(v1[4 * c + 3]));
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax: thread = query row t x 64 keys
    const int quarter = warp & 3, half = warp >> 2, t = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const float sc = p.scale * kLog2e;
    const float inv_keep = p.p_drop > 0.f ? 1.f / (1.f - p.p_drop) : 1.f;
    bool ok = true;
    for (int g = 0; w.valid; ++g, w.next()) {
      const int buf = g & 1, kv0 = w.j * kBlk;
      const bool masked = p.mask != nullptr || kv0 + kBlk > p.S;
      if (w.it == 0 && masked) {      // the item's additive mask (mask * log2e; -inf beyond S)
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (threadIdx.x < kBlk) {
          const int kv = kv0 + threadIdx.x;
          mask_s[threadIdx.x] = kv < p.S ? (p.mask ? __ldg(p.mask + static_cast<long long>(w.b) * p.S + kv) * kLog2e : 0.f) : -INFINITY;
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
      }
      const int q = (w.i0 + w.it) * kBlk + t;
      const bool diagonal = p.causal && w.i0 + w.it == w.j;
      const uint32_t pp = smem_u32(smem + L::P + buf * 32768) + half * 16384, dp = smem_u32(smem + L::DS + buf * 32768) + half * 16384;
      ok = ok && mbar_wait(&stat_full[buf], (g >> 1) & 1, abort_flag, p.status, kStatusWaitFull);
      const float2 ld = stats[buf * 128 + t];
      ok = ok && mbar_wait(&grads[buf], ((g >> 1) & 1) ^ 1, abort_flag, p.status, kStatusWaitAccum);       // tile g - 2 has been read out of P and dS
      ok = __all_sync(0xffffffffu, ok && mbar_wait(sdp_full, g & 1, abort_flag, p.status, kStatusWaitAccum));
      if (!ok) continue;        // after a wait that gave up the loop runs out without work, so that no warp is missed at the barrier above
      tc_fence_after_sync();
#pragma unroll
      for (int cc = 0; cc < 64; cc += 32) {
        const int c = half * 64 + cc;
        uint32_t sv[32], dpv[32];
        tmem_ld32(tS + lane_base + c, sv);
        tmem_ld32(tDP + lane_base + c, dpv);
        tmem_ld_wait();
        if (cc == 32) {
          tc_fence_before_sync();
          mbar_arrive(sdp_free);
        }
        // P into sv
        if (masked) {
#pragma unroll
          for (int e4 = 0; e4 < 32; e4 += 4) {
            const float4 mk = *reinterpret_cast<const float4*>(mask_s + c + e4);
            const float mk4[4] = {mk.x - ld.x, mk.y - ld.x, mk.z - ld.x, mk.w - ld.x};
#pragma unroll
            for (int k = 0; k < 4; ++k) sv[e4 + k] = __float_as_uint(ex2_approx(__uint_as_float(sv[e4 + k]) * sc + mk4[k]));
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) sv[e] = __float_as_uint(ex2_approx(__uint_as_float(sv[e]) * sc - ld.x));
        }
        if (diagonal) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (kv0 + c + e > q) sv[e] = 0u;
        }
        float ds[32];
        if (p.p_drop > 0.f) {
          const unsigned long long base = ((static_cast<unsigned long long>(w.b) * p.H + w.h) * p.S + q) * p.S + kv0 + c;
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            float z[4];
            dropout_scale4(seed, base + e, p.p_drop, inv_keep, z);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float pe = __uint_as_float(sv[e + k]);
              ds[e + k] = pe * (__uint_as_float(dpv[e + k]) * z[k] - ld.y) * p.scale;
              sv[e + k] = __float_as_uint(pe * z[k]);
            }
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) ds[e] = __uint_as_float(sv[e]) * (__uint_as_float(dpv[e]) - ld.y) * p.scale;
        }
#pragma unroll
        for (int g8 = 0; g8 < 4; ++g8) {
          float pr[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) pr[e] = __uint_as_float(sv[8 * g8 + e]);
          st_shared_v4(swz_chunk(pp, t, (cc >> 3) + g8), pack8(pr));
          st_shared_v4(swz_chunk(dp, t, (cc >> 3) + g8), pack8(ds + 8 * g8));
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(pds_ready);
      if (w.last()) {
        // dK (warps 0..3) and dV (warps 4..7) out. Every product of the item has then retired, so the rows of P's first buffer that
        // this warp alone writes serve as its staging area.
        ok = __all_sync(0xffffffffu, mbar_wait(&grads[buf], (g >> 1) & 1, abort_flag, p.status, kStatusWaitAccum));
        if (!ok) continue;
        tc_fence_after_sync();
        const uint32_t stage = smem_u32(smem + L::P) + warp * 4096;
#pragma unroll
        for (int c = 0; c < kHD; c += 32) {
          uint32_t v[32];
          tmem_ld32((half == 0 ? tDK : tDV) + lane_base + c, v);
          tmem_ld_wait();
          if (c == 32) {
            tc_fence_before_sync();
            mbar_arrive(acc_free);
          }
          float f[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) f[e] = __uint_as_float(v[e]);
          stage_half(stage, lane, c, f);
        }
        flush_rows(stage, lane, (half == 0 ? dk : dv) + w.b * p.gsb + w.h * p.gsh, p.gss, kv0 + quarter * 32, p.S);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kBwdSoftmaxWarps + 4) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, 512);
  }
}

}  // namespace

int attn_bwd_long(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo, const void* o, const void* d_o,
                  const float* lse, void* dq, void* dk, void* dv, float* dq_accum, const AttnParams& p, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(attn_bwd_long_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdLong::TOTAL);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  const long long items = static_cast<long long>((p.S + kBlk - 1) / kBlk) * p.H * p.B;
  const long long rows = static_cast<long long>(p.B) * p.H * p.S;
  if (items > 0x7fffffffll) return -4;
  const int row_grid = static_cast<int>(rows / 32 + 1 < kSMs * 16 ? rows / 32 + 1 : kSMs * 16);
  auto* dq16 = static_cast<__nv_bfloat16*>(dq);
  launch_pdl(attn_bwd_pre_kernel, dim3(row_grid), dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(d_o), dq16, dq_accum, p);
  launch_pdl(attn_bwd_long_kernel, dim3(static_cast<unsigned>(items < kSMs ? items : kSMs)), dim3(kBwdThreads), static_cast<size_t>(BwdLong::TOTAL), stream, tq, tk, tv, tdo, lse,
             static_cast<const __nv_bfloat16*>(dq16), static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), dq_accum, p);
  launch_pdl(attn_dq_kernel, dim3(row_grid), dim3(256), 0, stream, static_cast<const float*>(dq_accum), dq16, p);
  return static_cast<int>(cudaGetLastError());
}

// ===================================================================================== forward
namespace {

constexpr int kFwdThreads = 32 * 6;
constexpr float kRescaleAt = 8.f;      // log2 of the factor by which a row maximum may grow before its accumulator is rescaled

struct FwdLong {
  static constexpr int Q = 0;
  static constexpr int K = 16384;                    // 2 x 16 KB
  static constexpr int V = K + 2 * 16384;            // 2 x 16 KB
  static constexpr int MASK = V + 2 * 16384;         // 2 x 128 floats
  static constexpr int BARS = MASK + 1024;
  static constexpr int TOTAL = BARS + 256;
};

template <bool kDrop>
__global__ void __launch_bounds__(kFwdThreads, 2)
attn_fwd_long_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     __nv_bfloat16* __restrict__ o, float* __restrict__ lse, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using L = FwdLong;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;     // [2]
  uint64_t* k_empty = bars + 3;    // [2]
  uint64_t* v_full = bars + 5;     // [2]
  uint64_t* v_empty = bars + 7;    // [2]
  uint64_t* s_full = bars + 9;     // the scores of a key block are in TMEM
  uint64_t* s_free = bars + 10;    // ... and in the softmax warps' registers
  uint64_t* p_ready = bars + 11;   // the probabilities are in TMEM and O has been rescaled where it had to be
  uint64_t* pv_done = bars + 12;   // P V has been added to O
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* mask_s = reinterpret_cast<float*>(smem + L::MASK);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = (p.S + kBlk - 1) / kBlk;
  int qb, h, b;
  decode_block(blockIdx.x, nblk, p.H, p.B, p.causal != 0, qb, h, b);
  if (p.causal) qb = nblk - 1 - qb;          // the last query block sees the most keys
  const int q0 = qb * kBlk;
  const int n = p.causal ? qb + 1 : nblk;
  const unsigned long long seed = p.seed + (p.seed_dev ? *p.seed_dev : 0ull);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    mbar_init(s_full, 1);
    mbar_init(s_free, 128);
    mbar_init(p_ready, 128);
    mbar_init(pv_done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4) {
    tmem_alloc<1>(tmem_slot, 256);
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tP = tmem_base + 128, tO = tmem_base + 192;
  pdl_entry();

  if (warp == 5) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      mbar_expect_tx(q_full, 16384);
      tma_load_4d(smem + L::Q, &tmQ, q_full, 0, q0, h, b);
      for (int j = 0; j < n; ++j) {
        const int st = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        if (!mbar_wait(&k_empty[st], ph, abort_flag, p.status, kStatusWaitEmpty)) break;
        mbar_expect_tx(&k_full[st], 16384);
        tma_load_4d(smem + L::K + st * 16384, &tmK, &k_full[st], 0, j * kBlk, h, b);
        if (!mbar_wait(&v_empty[st], ph, abort_flag, p.status, kStatusWaitEmpty)) break;
        mbar_expect_tx(&v_full[st], 16384);
        tma_load_4d(smem + L::V + st * 16384, &tmV, &v_full[st], 0, j * kBlk, h, b);
      }
    }
  } else if (warp == 4) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_o = make_idesc_bf16(128, kHD, 0, 1);
      const uint32_t sQ = smem_u32(smem + L::Q);
      auto scores = [&](int j) {
        const int st = j & 1;
        const uint32_t sK = smem_u32(smem + L::K + st * 16384);
        if (!mbar_wait(&k_full[st], (j >> 1) & 1, abort_flag, p.status, kStatusWaitFull)) return false;
        tc_fence_after_sync();
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tS, make_smem_desc(sQ + k4 * 32, 16, 1024), make_smem_desc(sK + k4 * 32, 16, 1024), idesc_s, k4 > 0);
        umma_commit(s_full);
        umma_commit(&k_empty[st]);
        return true;
      };
      bool ok = mbar_wait(q_full, 0, abort_flag, p.status, kStatusWaitFull) && scores(0);
      for (int j = 0; j < n && ok; ++j) {
        if (j + 1 < n) {
          ok = mbar_wait(s_free, j & 1, abort_flag, p.status, kStatusWaitEpi) && scores(j + 1);
          if (!ok) break;
        }
        const int st = j & 1;
        const uint32_t sV = smem_u32(smem + L::V + st * 16384);
        ok = mbar_wait(p_ready, j & 1, abort_flag, p.status, kStatusWaitEpi) && mbar_wait(&v_full[st], (j >> 1) & 1, abort_flag, p.status, kStatusWaitFull);
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16_ts(tO, tP + k8 * 8, make_smem_desc(sV + k8 * 2048, 8192, 1024), idesc_o, j > 0 || k8 > 0);
        umma_commit(pv_done);
        umma_commit(&v_empty[st]);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax: thread = query row
    const int t = threadIdx.x, q = q0 + t;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const float sc = p.scale * kLog2e;
    const float inv_keep = kDrop ? 1.f / (1.f - p.p_drop) : 1.f;
    float m_ref = -INFINITY, l_run = 0.f;       // the maximum the accumulator is relative to, and the row sum
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      const int kv0 = j * kBlk;
      const bool masked = p.mask != nullptr || kv0 + kBlk > p.S;
      const bool diagonal = p.causal && j == qb;
      const float* mk_s = mask_s + (j & 1) * kBlk;
      if (masked) {       // additive mask of this key block (mask * log2e; -inf beyond S); the other buffer may still be in use
        const int kv = kv0 + t;
        mask_s[(j & 1) * kBlk + t] = kv < p.S ? (p.mask ? __ldg(p.mask + static_cast<long long>(b) * p.S + kv) * kLog2e : 0.f) : -INFINITY;
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
      ok = __all_sync(0xffffffffu, ok && mbar_wait(s_full, j & 1, abort_flag, p.status, kStatusWaitAccum));
      if (!ok) continue;        // after a wait that gave up the loop runs out without work, so that no warp is missed at the barrier above
      tc_fence_after_sync();
      uint32_t sv[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tS + lane_base + 32 * c, sv[c]);
      tmem_ld_wait();
      tc_fence_before_sync();
      mbar_arrive(s_free);
      // row maximum; with a mask, on the diagonal or for a negative scale the scores are scaled here, otherwise in the exponent below
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      float mul = sc;
      if (masked || diagonal || sc < 0.f) {
        mul = 1.f;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i4 = 0; i4 < 32; i4 += 4) {
            const float4 mk = masked ? *reinterpret_cast<const float4*>(mk_s + 32 * c + i4) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float mk4[4] = {mk.x, mk.y, mk.z, mk.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              float s = __uint_as_float(sv[c][i4 + k]) * sc + mk4[k];
              if (diagonal && kv0 + 32 * c + i4 + k > q) s = -INFINITY;
              sv[c][i4 + k] = __float_as_uint(s);
              m4[k] = fmaxf(m4[k], s);
            }
          }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(sv[c][i]));
      }
      const float m_new = fmaxf(m_ref, fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * mul);
      if (j == 0) {
        m_ref = m_new;
      } else {
        ok = __all_sync(0xffffffffu, mbar_wait(pv_done, (j - 1) & 1, abort_flag, p.status, kStatusWaitAccum));     // P may be overwritten, O touched
        if (!ok) continue;
        tc_fence_after_sync();
        if (__any_sync(0xffffffffu, m_new > m_ref + kRescaleAt)) {
          const float alpha = m_new == -INFINITY ? 1.f : ex2_approx(m_ref - m_new);
          m_ref = m_new;
          l_run *= alpha;
#pragma unroll 1
          for (int c = 0; c < kHD; c += 16) {
            uint32_t v[16];
            tmem_ld16(tO + lane_base + c, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
            tmem_st16(tO + lane_base + c, v);
          }
        }
      }
      const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
      float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float pe = ex2_approx(fmaf(__uint_as_float(sv[c][i]), mul, neg_m));
          l4[i & 3] += pe;
          sv[c][i] = __float_as_uint(pe);
        }
        if constexpr (kDrop) {
          const unsigned long long base = ((static_cast<unsigned long long>(b) * p.H + h) * p.S + q) * p.S + kv0 + 32 * c;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float s4[4];
            dropout_scale4(seed, base + i, p.p_drop, inv_keep, s4);
#pragma unroll
            for (int k = 0; k < 4; ++k) sv[c][i + k] = __float_as_uint(__uint_as_float(sv[c][i + k]) * s4[k]);
          }
        }
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const __nv_bfloat162 two = __floats2bfloat162_rn(__uint_as_float(sv[c][2 * i]), __uint_as_float(sv[c][2 * i + 1]));
          pk[i] = *reinterpret_cast<const uint32_t*>(&two);
        }
        tmem_st16(tP + lane_base + 16 * c, pk);
      }
      l_run += (l4[0] + l4[1]) + (l4[2] + l4[3]);
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(p_ready);
    }
    ok = ok && mbar_wait(pv_done, (n - 1) & 1, abort_flag, p.status, kStatusWaitAccum);
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after_sync();
      const float inv_l = l_run > 0.f ? 1.f / l_run : 0.f;
      const uint32_t stage = smem_u32(smem + L::Q) + warp * 4096;        // every product that reads Q has retired
#pragma unroll
      for (int c = 0; c < kHD; c += 32) {
        uint32_t v[32];
        tmem_ld32(tO + lane_base + c, v);
        tmem_ld_wait();
        float f[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]) * inv_l;
        stage_half(stage, lane, c, f);
      }
      flush_rows(stage, lane, o + static_cast<long long>(b) * p.osb + static_cast<long long>(h) * p.osh, p.oss, q0 + warp * 32, p.S);
      // natural-log LSE of the scaled, masked scores
      if (q < p.S) lse[(static_cast<long long>(b) * p.H + h) * p.S + q] = (l_run > 0.f) ? (m_ref + log2f(l_run)) / kLog2e : -INFINITY;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, 256);
  }
}

}  // namespace

int attn_fwd_long(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, void* o, float* lse, const AttnParams& p, cudaStream_t stream) {
  const auto kern = p.p_drop > 0.f ? attn_fwd_long_kernel<true> : attn_fwd_long_kernel<false>;
  static bool configured = false;
  if (!configured) {
    for (auto k : {attn_fwd_long_kernel<true>, attn_fwd_long_kernel<false>}) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdLong::TOTAL + 1024);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    configured = true;
  }
  const long long ctas = static_cast<long long>((p.S + kBlk - 1) / kBlk) * p.H * p.B;
  if (ctas > 0x7fffffffll) return -4;
  const cudaError_t e = launch_pdl(kern, dim3(static_cast<unsigned>(ctas)), dim3(kFwdThreads), static_cast<size_t>(FwdLong::TOTAL + 1024), stream, tq, tk,
                                   tv, static_cast<__nv_bfloat16*>(o), lse, p);
  return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
}

}  // namespace fb
