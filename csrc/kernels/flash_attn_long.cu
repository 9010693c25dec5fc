// Attention over several key blocks (S > 128), head dim 64, on tcgen05. The entry points and the kernels of a single
// key block are in flash_attn.cu.
//
// Backward: one CTA per (key block of 128 rows, head, batch) walks the query blocks that see it. K, V and the dK / dV
// accumulators stay put; Q and dO stream through a three-stage TMA ring. Roles: 16 softmax warps (thread = one query row x
// 32 keys), 4 warps that drain dQ, two that add it to the scratch in turn, one MMA issuer, one producer (TMA and row statistics). S and dP of the next query
// block are issued as soon as the softmax warps have loaded this block's into registers, so the tensor cores work under the exponentials.
// A query block's dQ is a sum over key blocks, i.e. over CTAs: it is added into an fp32 scratch with bulk reductions, in the order of
// the key blocks, so that two calls give the same bits. The scratch is not row-major: within the 32 rows a warp owns, 16-byte chunk c of
// row r sits at (c * rows + r) * 16, so that the 32 lanes (one row each) write the staging area, which is copied as it is, without bank
// conflicts. A pass before zeroes the scratch and leaves D = rowsum(dO * O) in the first word of each dQ row; a pass after turns the
// scratch into bf16 rows.
// What bounds it: the chain scores -> exponentials -> P and dS in shared memory -> products of one tile, with the shared-memory
// pipe (P and dS are written once and read by three products) as its slowest part. The fixed order costs a causal head's first CTAs, which start
// together, about 4 us for each block between them (from the end of one's additions to the start of the next one's).
// Backward, bf16, us; in brackets with one adding thread, the row statistics behind the dQ staging area and one value per instruction: B 2 x H 12 x
// S 4096 causal 205 (276), full 358 (496), B 4 x H 8 x S 1024 causal 40 (47), B 6 x H 12 x S 509 with a mask 38 (43), B 32 x H 8 x S 256 causal 44 (47),
// B 64 x H 12 x S 384 with a mask 255 (280).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "../include/flodl_b200.h"
#include "flash_attn_common.cuh"

namespace fb {

namespace {
// Descriptor of the operand at `base` moved on by a constant number of bytes; K-major, or MN-major with `lbo` bytes between its 64-wide panels.
__device__ __forceinline__ uint64_t k_desc(uint32_t base, int bytes) { return desc_of(smem_desc_lo(base, 16) + (bytes >> 4), smem_desc_hi(1024)); }
__device__ __forceinline__ uint64_t mn_desc(uint32_t base, int bytes, int lbo) { return desc_of(smem_desc_lo(base, lbo) + (bytes >> 4), smem_desc_hi(1024)); }
}  // namespace

// ==================================================================================== backward
namespace {

constexpr int kBwdStages = 3;
constexpr int kBwdSoftmaxWarps = 16;
constexpr int kBwdThreads = 32 * (kBwdSoftmaxWarps + 4 + 4);

struct BwdLong {
  static constexpr int Q = 0;                                   // kBwdStages x 16 KB
  static constexpr int DO = Q + kBwdStages * 16384;             // kBwdStages x 16 KB
  static constexpr int K = DO + kBwdStages * 16384;
  static constexpr int V = K + 16384;
  static constexpr int P = V + 16384;                           // 2 panels of 16 KB
  static constexpr int DS = P + 2 * 16384;                      // 2 panels of 16 KB
  static constexpr int DQ = DS + 2 * 16384;                     // 4 warps x 8 KB: dQ on its way out
  static constexpr int STATS = DQ + 4 * 8192;                   // 2 x 128 x {lse, D}
  static constexpr int MASK = STATS + 2 * 128 * 8;              // 128 floats
  static constexpr int BARS = MASK + 512;
  static constexpr int TOTAL = BARS + 256;
};
static_assert(BwdLong::TOTAL <= 227 * 1024, "shared memory budget");

// Work item -> (block, head, batch). Causal: every block of equal length before the next shorter one (the longest first, so the last wave is
// short). Otherwise all blocks of a head together, which keeps its K / V (or Q / dO) in L2 (a group of 1), or one block of each of
// `group` heads after the other, so that blocks of one head, which add to dQ in turn, seldom run side by side (B 2 x H 12 x S 4096, all heads
// in one group 490 us, groups of 1 635).
__device__ __forceinline__ void decode_block(int lin, int nblk, int H, int B, bool causal, int group, int& blk, int& h, int& b) {
  const int heads = H * B;
  if (causal) group = heads;
  const int first = lin / (group * nblk) * group, size = min(group, heads - first), rest = lin - first * nblk;
  blk = rest / size;
  const int hb = first + rest - blk * size;
  b = hb / H;
  h = hb - b * H;
}

// Adds `bytes` of fp32 values to global memory (both sides 16-byte aligned), as a bulk copy: beside the LSU pipe, which the softmax
// warps' shared-memory traffic goes through.
__device__ __forceinline__ void bulk_add(float* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}

// What the first words of a dQ row hold until the row itself is written.
struct DqSlot {
  float D;
  unsigned int added;        // of a query block's first row: how many key blocks have been added to the block's scratch
  unsigned int ticket;       // of the very first row: work items handed out
  unsigned int unused;
};

// Waits until `want` key blocks have been added. Bounded like mbar_wait; a block that gave up never adds, which its status tells the others.
__device__ __forceinline__ bool wait_added(const unsigned int* added, unsigned int want, volatile int* abort_flag, int* status) {
  for (uint32_t it = 0; it < (1u << 20); ++it) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(added) : "memory");
    if (v >= want) {
      fence_proxy_async_global();
      return true;
    }
    if (*abort_flag || ((it & 4095) == 4095 && status && *reinterpret_cast<volatile int*>(status) != kStatusOk)) break;
    if (it > 16) __nanosleep(40);
  }
  *abort_flag = 1;
  set_status(status, kStatusWaitAccum);
  return false;
}

// Per query row: the first words of the row's dQ slot (overwritten by attn_dq_kernel at the end) take D = dot(dO, O) and two zeroed
// counters (DqSlot), and the row's share of the dQ scratch is zeroed. Eight lanes per row, rows of one (batch, head) consecutive.
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
    if (ch == 0) *reinterpret_cast<uint4*>(dq + b * p.gsb + h * p.gsh + s * p.gss) = make_uint4(__float_as_uint(d), 0u, 0u, 0u);
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
                     const __grid_constant__ CUtensorMap tmDO, const float* __restrict__ lse, __nv_bfloat16* dq,
                     __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, float* __restrict__ dq_accum, const AttnParams p) {
  // No room for alignment slack: the kernel relies on the 1024-byte alignment of the dynamic shared-memory window and reports instead of
  // computing if that does not hold.
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) set_status(p.status, kStatusBadArg);
    return;
  }
  using L = BwdLong;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;                    // [kBwdStages] Q and dO of a query block have landed
  uint64_t* q_empty = q_full + kBwdStages;        // [kBwdStages] ... and every product that reads them has retired
  uint64_t* sdp_full = q_empty + kBwdStages;      // S and dP are in TMEM
  uint64_t* sdp_free = sdp_full + 1;              // ... and in the softmax warps' registers
  uint64_t* pds_ready = sdp_free + 1;             // P and dS are in shared memory
  uint64_t* grads_full = pds_ready + 1;           // dV, dK, dQ of the block have retired (P, dS may be overwritten)
  uint64_t* dq_full = grads_full + 1;             // [2] the same event, per dQ buffer, for the draining warps
  uint64_t* dq_free = dq_full + 2;                // [2] the buffer has been read
  uint64_t* stat_full = dq_free + 2;              // [2] lse and D of a query block are in shared memory
  uint64_t* staged = stat_full + 2;               // [2] dQ of a query block is in shared memory
  uint64_t* stage_free = staged + 2;              // ... and has been read from there
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(stage_free + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* item = abort_flag + 1;            // key block, head, batch: reloaded where needed, the softmax warps have no registers to spare
  float* mask_s = reinterpret_cast<float*>(smem + L::MASK);
  float2* stats = reinterpret_cast<float2*>(smem + L::STATS);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int nblk = (p.S + kBlk - 1) / kBlk;
  // The key blocks of a head add to dQ in order (below), so a block may only wait for blocks that run already: the work is handed out by a
  // counter, in an order in which a head's earlier key blocks come first.
  const bool ordered = nblk > 2;
  if (ordered) pdl_entry();       // the counter is the previous kernel's
  if (warp == kBwdSoftmaxWarps + 5 && lane == 0) {
    const int lin = ordered ? static_cast<int>(atomicAdd(&reinterpret_cast<DqSlot*>(dq)->ticket, 1u)) : blockIdx.x;
    int j, h, b;
    decode_block(lin, nblk, p.H, p.B, p.causal != 0, ordered ? p.group : 1, j, h, b);
    item[0] = j; item[1] = h; item[2] = b;
  }
  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < kBwdStages; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); }
    mbar_init(sdp_full, 1);
    mbar_init(sdp_free, kBwdSoftmaxWarps);
    mbar_init(pds_ready, kBwdSoftmaxWarps);
    mbar_init(grads_full, 1);
    for (int s = 0; s < 2; ++s) { mbar_init(&dq_full[s], 1); mbar_init(&dq_free[s], 4); mbar_init(&stat_full[s], 1); mbar_init(&staged[s], 4); }
    mbar_init(stage_free, 1);
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
  if (!ordered) pdl_entry();
  // Query blocks from the last to the first that sees the keys: key blocks of a causal head that start together meet at their first query
  // block and then stay one hand-over apart; from the first to the last they would meet anew, one block later, at every step.
  const int n = p.causal ? nblk - item[0] : nblk;
  const auto query_block = [&](int it) { return nblk - 1 - it; };

  if (warp == kBwdSoftmaxWarps + 5) {
    // ------------------------------------------------------------------ TMA producer (this loop and the next one: the whole warp, one lane issues)
    const int j = item[0], h = item[1], b = item[2];
    if (elect_one()) {
      mbar_expect_tx(kv_full, 32768);
      tma_load_4d(smem + L::K, &tmK, kv_full, 0, j * kBlk, h, b);
      tma_load_4d(smem + L::V, &tmV, kv_full, 0, j * kBlk, h, b);
    }
    __syncwarp();
    // The row statistics go with them, a block later: their two buffers are free when the ring has a stage again, which block it - 3 left. (Where the
    // warps that drain dQ loaded them, behind the staging area that frees up with the additions, they reached the softmax warps 2000 cycles late.)
    const long long bh = static_cast<long long>(b) * p.H + h;
    float2 ahead[4];
    for (int it = 0; it <= n; ++it) {
      const int st = it % kBwdStages;
      if (!warp_wait(&q_empty[st], ((it / kBwdStages) & 1) ^ 1, abort_flag, p.status, kStatusWaitEmpty)) break;
      if (it < n && elect_one()) {
        mbar_expect_tx(&q_full[st], 32768);
        tma_load_4d(smem + L::Q + st * 16384, &tmQ, &q_full[st], 0, query_block(it) * kBlk, h, b);
        tma_load_4d(smem + L::DO + st * 16384, &tmDO, &q_full[st], 0, query_block(it) * kBlk, h, b);
      }
      __syncwarp();
      if (it > 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {      // (the arithmetic here: next to the loads it would wait for them)
          // a row beyond S, or one that no key takes part in, gets +inf: every probability of it is then 2^-inf = 0
          const float l = ahead[i].x == -INFINITY ? INFINITY : ahead[i].x * kLog2e;
          stats[((it - 1) & 1) * 128 + i * 32 + lane] = make_float2(l, ahead[i].y * p.scale);
        }
        arrive_warp(&stat_full[(it - 1) & 1], lane);
      }
      if (it == n) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = query_block(it) * kBlk + i * 32 + lane;
        ahead[i] = make_float2(-INFINITY, 0.f);
        if (q < p.S) {
          ahead[i].x = __ldg(lse + bh * p.S + q);
          ahead[i].y = __ldcg(&reinterpret_cast<const DqSlot*>(dq + b * p.gsb + h * p.gsh + q * p.gss)->D);
        }
      }
    }
  } else if (warp == kBwdSoftmaxWarps + 4) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t idesc_kk = make_idesc_bf16(128, 128, 0, 0);      // S, dP: both operands K-major
    const uint32_t idesc_mn = make_idesc_bf16(128, kHD, 1, 1);      // dV, dK: A^T (MN-major) x MN-major
    const uint32_t idesc_kn = make_idesc_bf16(128, kHD, 0, 1);      // dQ: K-major x MN-major
    const uint32_t sK = smem_u32(smem + L::K), sV = smem_u32(smem + L::V);
    const uint32_t sP = smem_u32(smem + L::P), sDS = smem_u32(smem + L::DS);
    auto scores = [&](int it) {
      const int st = it % kBwdStages;
      const uint32_t sQ = smem_u32(smem + L::Q + st * 16384), sDO = smem_u32(smem + L::DO + st * 16384);
      if (!warp_wait(&q_full[st], (it / kBwdStages) & 1, abort_flag, p.status, kStatusWaitFull)) return false;
      tc_fence_after_sync();
      if (elect_one()) {
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tS, k_desc(sQ, k4 * 32), k_desc(sK, k4 * 32), idesc_kk, k4 > 0);
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tDP, k_desc(sDO, k4 * 32), k_desc(sV, k4 * 32), idesc_kk, k4 > 0);
        umma_commit(sdp_full);
      }
      __syncwarp();
      return true;
    };
    bool ok = warp_wait(kv_full, 0, abort_flag, p.status, kStatusWaitFull) && scores(0);
    for (int it = 0; it < n && ok; ++it) {
      if (it + 1 < n) {
        ok = warp_wait(sdp_free, it & 1, abort_flag, p.status, kStatusWaitEpi) && scores(it + 1);
        if (!ok) break;
      }
      const int st = it % kBwdStages, qb = it & 1;
      const uint32_t sQ = smem_u32(smem + L::Q + st * 16384), sDO = smem_u32(smem + L::DO + st * 16384);
      ok = warp_wait(pds_ready, it & 1, abort_flag, p.status, kStatusWaitEpi) &&
           warp_wait(&dq_free[qb], ((it >> 1) & 1) ^ 1, abort_flag, p.status, kStatusWaitEpi);
      if (!ok) break;
      tc_fence_after_sync();
      if (elect_one()) {
        // dV += P^T dO ; dK += dS^T Q   (M = key index, K = query index: 8 steps of 16 rows)
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16<1>(tDV, mn_desc(sP, k8 * 2048, 16384), mn_desc(sDO, k8 * 2048, 8192), idesc_mn, it > 0 || k8 > 0);
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16<1>(tDK, mn_desc(sDS, k8 * 2048, 16384), mn_desc(sQ, k8 * 2048, 8192), idesc_mn, it > 0 || k8 > 0);
        // dQ_tile = dS K   (M = query, K = key index)
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16<1>(tDQ + qb * 64, k_desc(sDS, (k8 >> 2) * 16384 + (k8 & 3) * 32), mn_desc(sK, k8 * 2048, 8192),
                       idesc_kn, k8 > 0);
        umma_commit(grads_full);
        umma_commit(&dq_full[qb]);
        umma_commit(&q_empty[st]);
      }
      __syncwarp();
    }
  } else if (warp >= kBwdSoftmaxWarps + 6) {
    // ------------------------------------------------------------------ dQ into the scratch
    // One thread adds a query block's 128 rows at once; two of them take turns, so that one block's additions, which the next key block waits for the
    // end of, do not hold up the next block's. A sum of three or more depends on its order, so the third and later key blocks wait
    // for the ones before them; the first two may come either way round, 0 + a + b being 0 + b + a.
    if (lane == 0) {
      const int j = item[0], h = item[1], b = item[2];
      const uint32_t src = smem_u32(smem + L::DQ);
      for (int it = warp - kBwdSoftmaxWarps - 6; it < n; it += 2) {
        const int qblk = query_block(it), row0 = qblk * kBlk, adders = p.causal ? qblk + 1 : nblk;
        unsigned int* added = &reinterpret_cast<DqSlot*>(dq + b * p.gsb + h * p.gsh + row0 * p.gss)->added;
        if (j >= 2 && !wait_added(added, static_cast<unsigned int>(j), abort_flag, p.status)) break;
        if (!mbar_wait(&staged[it & 1], (it >> 1) & 1, abort_flag, p.status, kStatusWaitAccum)) break;
        bulk_add(dq_accum + ((static_cast<long long>(b) * p.H + h) * p.S + row0) * kHD, src, min(kBlk, p.S - row0) * kHD * 4);
        tma_store_commit();
        tma_store_wait_read();
        mbar_arrive(stage_free);
        if (adders > 2 && j + 1 < adders) {
          tma_store_wait_all();        // the additions are done, not only read
          fence_proxy_async_global();
          asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(added) : "memory");
        }
      }
    }
  } else if (warp >= kBwdSoftmaxWarps) {
    // ------------------------------------------------------------------ dQ out
    const int quarter = warp & 3;
    const uint32_t stage = smem_u32(smem + L::DQ) + quarter * 8192;
    for (int it = 0; it < n; ++it) {
      const int qb = it & 1;
      bool ok = mbar_wait(&dq_full[qb], (it >> 1) & 1, abort_flag, p.status, kStatusWaitAccum);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after_sync();
      // out of TMEM before the staging area is free: the next but one block's products need not wait for that
      uint32_t v[2][32];
      tmem_ld64_sync(tDQ + qb * 64 + (static_cast<uint32_t>(quarter * 32) << 16), v[0], v[1]);
      tc_fence_before_sync();
      arrive_warp(&dq_free[qb], lane);
      if (it > 0 && !warp_wait(stage_free, (it - 1) & 1, abort_flag, p.status, kStatusWaitEpi)) break;
      // 16-byte chunk c of this warp's row r at (c * rows + r) * 16, as in the scratch
      const int nr = min(32, p.S - query_block(it) * kBlk - quarter * 32);
      if (lane < nr) {
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
          for (int c = 0; c < 8; ++c)
            st_shared_v4(stage + ((half * 8 + c) * nr + lane) * 16, make_uint4(v[half][4 * c], v[half][4 * c + 1], v[half][4 * c + 2], v[half][4 * c + 3]));
      }
      fence_proxy_async_smem();
      arrive_warp(&staged[it & 1], lane);
    }
  } else {
    // ------------------------------------------------------------------ softmax: thread = query row t x 32 keys
    const int quarter = warp & 3, part = warp >> 2, t = quarter * 32 + lane, c = part * 32;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const float sc = p.scale * kLog2e;
    const float inv_keep = p.p_drop > 0.f ? 1.f / (1.f - p.p_drop) : 1.f;
    const int kv0 = item[0] * kBlk;
    if (threadIdx.x < kBlk) {      // the additive mask (mask * log2e; -inf beyond S)
      const int kv = kv0 + threadIdx.x;
      mask_s[threadIdx.x] = kv < p.S ? (p.mask ? __ldg(p.mask + static_cast<long long>(item[2]) * p.S + kv) * kLog2e : 0.f) : -INFINITY;
    }
    asm volatile("bar.sync 1, 512;" ::: "memory");
    const bool masked = p.mask != nullptr || kv0 + kBlk > p.S;
    const uint32_t pp = smem_u32(smem + L::P) + (part >> 1) * 16384, dp = smem_u32(smem + L::DS) + (part >> 1) * 16384;
    bool ok = true;
    for (int it = 0; it < n; ++it) {
      const bool diagonal = p.causal && it == n - 1;
      ok = mbar_wait(&stat_full[it & 1], (it >> 1) & 1, abort_flag, p.status, kStatusWaitFull);
      const float2 ld = stats[(it & 1) * 128 + t];
      ok = __all_sync(0xffffffffu, ok && mbar_wait(sdp_full, it & 1, abort_flag, p.status, kStatusWaitAccum));
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t sv[32], dpv[32];
      tmem_ld32(tS + lane_base + c, sv);
      tmem_ld32(tDP + lane_base + c, dpv);
      tmem_ld_wait();
      tc_fence_before_sync();
      arrive_warp(sdp_free, lane);
      // P into sv, dS into dpv
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
        for (int e = 0; e < 32; e += 2) {
          float lo, hi;
          f2_get(f2_fma(f2_make(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])), f2_splat(sc), f2_splat(-ld.x)), lo, hi);
          sv[e] = __float_as_uint(ex2_approx(lo));
          sv[e + 1] = __float_as_uint(ex2_approx(hi));
        }
      }
      if (diagonal) {
#pragma unroll
        for (int e = 0; e < 32; ++e)
          if (c + e > t) sv[e] = 0u;
      }
      if (p.p_drop > 0.f) {
        const unsigned long long base =
            ((static_cast<unsigned long long>(item[2]) * p.H + item[1]) * p.S + query_block(it) * kBlk + t) * p.S + item[0] * kBlk + c;
        const unsigned long long seed = p.seed + (p.seed_dev ? *p.seed_dev : 0ull);
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          float z[4];
          dropout_scale4(seed, base + e, p.p_drop, inv_keep, z);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float pe = __uint_as_float(sv[e + k]);
            dpv[e + k] = __float_as_uint(pe * fmaf(__uint_as_float(dpv[e + k]) * z[k], p.scale, -ld.y));
            sv[e + k] = __float_as_uint(pe * z[k]);
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const F2 d = f2_fma(f2_make(__uint_as_float(dpv[e]), __uint_as_float(dpv[e + 1])), f2_splat(p.scale), f2_splat(-ld.y));
          float lo, hi;
          f2_get(f2_mul(f2_make(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])), d), lo, hi);
          dpv[e] = __float_as_uint(lo);
          dpv[e + 1] = __float_as_uint(hi);
        }
      }
      // As they are stored, before the wait: the compiler would leave the arithmetic behind it, where nothing overlaps it.
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        sv[e] = pack2(__uint_as_float(sv[2 * e]), __uint_as_float(sv[2 * e + 1]));
        dpv[e] = pack2(__uint_as_float(dpv[2 * e]), __uint_as_float(dpv[2 * e + 1]));
        asm volatile("" : "+r"(sv[e]), "+r"(dpv[e]));
      }
      if (it > 0) {        // the previous block's products have read P and dS
        ok = __all_sync(0xffffffffu, mbar_wait(grads_full, (it - 1) & 1, abort_flag, p.status, kStatusWaitAccum));
        if (!ok) break;
      }
#pragma unroll
      for (int g8 = 0; g8 < 4; ++g8) {
        st_shared_v4(swz_chunk(pp, t, (part & 1) * 4 + g8), make_uint4(sv[4 * g8], sv[4 * g8 + 1], sv[4 * g8 + 2], sv[4 * g8 + 3]));
        st_shared_v4(swz_chunk(dp, t, (part & 1) * 4 + g8), make_uint4(dpv[4 * g8], dpv[4 * g8 + 1], dpv[4 * g8 + 2], dpv[4 * g8 + 3]));
      }
      fence_proxy_async_smem();
      arrive_warp(pds_ready, lane);
    }
    // dK (warps 0..3) and dV (warps 4..7) out, through the warp's 4 KB of the P panels, which every product has read
    ok = __all_sync(0xffffffffu, ok && part < 2 && mbar_wait(grads_full, (n - 1) & 1, abort_flag, p.status, kStatusWaitAccum));
    if (ok) {
      tc_fence_after_sync();
      const uint32_t stage = smem_u32(smem + L::P) + warp * 4096;
#pragma unroll
      for (int c2 = 0; c2 < kHD; c2 += 32) {
        uint32_t v[32];
        tmem_ld32((part == 0 ? tDK : tDV) + lane_base + c2, v);
        tmem_ld_wait();
        float f[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) f[e] = __uint_as_float(v[e]);
        stage_half(stage, lane, c2, f);
      }
      flush_rows(stage, lane, (part == 0 ? dk : dv) + item[2] * p.gsb + item[1] * p.gsh, p.gss, item[0] * kBlk + quarter * 32, p.S);
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
  if (const cudaError_t e = allow_smem<attn_bwd_long_kernel>(BwdLong::TOTAL)) return static_cast<int>(e);
  const long long items = static_cast<long long>((p.S + kBlk - 1) / kBlk) * p.H * p.B;
  const long long rows = static_cast<long long>(p.B) * p.H * p.S;
  if (items > 0x7fffffffll) return -4;
  const int row_grid = static_cast<int>(rows / 32 + 1 < p.group * 16 ? rows / 32 + 1 : p.group * 16);
  auto* dq16 = static_cast<__nv_bfloat16*>(dq);
  launch_pdl(attn_bwd_pre_kernel, dim3(row_grid), dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(d_o), dq16, dq_accum, p);
  launch_pdl(attn_bwd_long_kernel, dim3(static_cast<unsigned>(items)), dim3(kBwdThreads), static_cast<size_t>(BwdLong::TOTAL), stream, tq, tk, tv, tdo, lse,
             dq16, static_cast<__nv_bfloat16*>(dk), static_cast<__nv_bfloat16*>(dv), dq_accum, p);
  launch_pdl(attn_dq_kernel, dim3(row_grid), dim3(256), 0, stream, static_cast<const float*>(dq_accum), dq16, p);
  return static_cast<int>(cudaGetLastError());
}

// ===================================================================================== forward
namespace {

constexpr int kFwdSoftmaxWarps = 8;
constexpr int kFwdThreads = 32 * (kFwdSoftmaxWarps + 2);

struct FwdLong {
  static constexpr int Q = 0;
  static constexpr int K = 16384;                    // 2 x 16 KB
  static constexpr int V = K + 2 * 16384;            // 2 x 16 KB
  static constexpr int MASK = V + 2 * 16384;         // 2 x 128 floats
  static constexpr int XCHG = MASK + 1024;           // 2 x 2 x 128 floats: the half rows' maxima, and at the end their sums
  static constexpr int BARS = XCHG + 2048;
  static constexpr int TOTAL = BARS + 256;
};

// kMask: whether there is an additive mask. The last, ragged key block without one is cut off like the diagonal. Instances of their own, because
// the mask is needed twice, for the maximum and for the exponent: both forms in one kernel spilled (B 64 x H 12 x S 384 with a mask 118 us against
// 102, B 2 x H 12 x S 4096 causal without 120 against 100).
template <bool kDrop, bool kMask>
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

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int nblk = (p.S + kBlk - 1) / kBlk;
  int qb, h, b;
  decode_block(blockIdx.x, nblk, p.H, p.B, p.causal != 0, 1, qb, h, b);
  if (p.causal) qb = nblk - 1 - qb;          // the last query block sees the most keys
  const int q0 = qb * kBlk;
  const int n = p.causal ? qb + 1 : nblk;
  const unsigned long long seed = p.seed + (p.seed_dev ? *p.seed_dev : 0ull);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    mbar_init(s_full, 1);
    mbar_init(s_free, kFwdSoftmaxWarps);
    mbar_init(p_ready, kFwdSoftmaxWarps);
    mbar_init(pv_done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kFwdSoftmaxWarps) {
    tmem_alloc<1>(tmem_slot, 256);
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tP = tmem_base + 128, tO = tmem_base + 192;
  pdl_entry();

  if (warp == kFwdSoftmaxWarps + 1) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_expect_tx(q_full, 16384);
      tma_load_4d(smem + L::Q, &tmQ, q_full, 0, q0, h, b);
    }
    __syncwarp();
    for (int j = 0; j < n; ++j) {
      const int st = j & 1;
      const uint32_t ph = ((j >> 1) & 1) ^ 1;
      if (!warp_wait(&k_empty[st], ph, abort_flag, p.status, kStatusWaitEmpty)) break;
      if (elect_one()) {
        mbar_expect_tx(&k_full[st], 16384);
        tma_load_4d(smem + L::K + st * 16384, &tmK, &k_full[st], 0, j * kBlk, h, b);
      }
      __syncwarp();
      if (!warp_wait(&v_empty[st], ph, abort_flag, p.status, kStatusWaitEmpty)) break;
      if (elect_one()) {
        mbar_expect_tx(&v_full[st], 16384);
        tma_load_4d(smem + L::V + st * 16384, &tmV, &v_full[st], 0, j * kBlk, h, b);
      }
      __syncwarp();
    }
  } else if (warp == kFwdSoftmaxWarps) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
    const uint32_t idesc_o = make_idesc_bf16(128, kHD, 0, 1);
    const uint32_t sQ = smem_u32(smem + L::Q);
    auto scores = [&](int j) {
      const int st = j & 1;
      const uint32_t sK = smem_u32(smem + L::K + st * 16384);
      if (!warp_wait(&k_full[st], (j >> 1) & 1, abort_flag, p.status, kStatusWaitFull)) return false;
      tc_fence_after_sync();
      if (elect_one()) {
#pragma unroll
        for (int k4 = 0; k4 < kHD / 16; ++k4)
          umma_bf16<1>(tS, k_desc(sQ, k4 * 32), k_desc(sK, k4 * 32), idesc_s, k4 > 0);
        umma_commit(s_full);
        umma_commit(&k_empty[st]);
      }
      __syncwarp();
      return true;
    };
    bool ok = warp_wait(q_full, 0, abort_flag, p.status, kStatusWaitFull) && scores(0);
    for (int j = 0; j < n && ok; ++j) {
      if (j + 1 < n) {
        ok = warp_wait(s_free, j & 1, abort_flag, p.status, kStatusWaitEpi) && scores(j + 1);
        if (!ok) break;
      }
      const int st = j & 1;
      const uint32_t sV = smem_u32(smem + L::V + st * 16384);
      ok = warp_wait(p_ready, j & 1, abort_flag, p.status, kStatusWaitEpi) && warp_wait(&v_full[st], (j >> 1) & 1, abort_flag, p.status, kStatusWaitFull);
      if (!ok) break;
      tc_fence_after_sync();
      if (elect_one()) {
#pragma unroll
        for (int k8 = 0; k8 < kBlk / 16; ++k8)
          umma_bf16_ts(tO, tP + k8 * 8, mn_desc(sV, k8 * 2048, 8192), idesc_o, j > 0 || k8 > 0);
        umma_commit(pv_done);
        umma_commit(&v_empty[st]);
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------------ softmax: thread = query row t x 64 keys
    // (two warps share 32 rows: four warps a scheduler with two CTAs, which is what hides the TMEM loads and the exponentials' latency)
    const int quarter = warp & 3, half = warp >> 2, t = quarter * 32 + lane, q = q0 + t;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const float sc = p.scale == 0.f ? 1e-37f : p.scale * kLog2e;       // never 0: a score of -inf has to stay one
    const float inv_keep = kDrop ? 1.f / (1.f - p.p_drop) : 1.f;
    const float hidden = sc < 0.f ? INFINITY : -INFINITY;               // the score of a key that the row does not see
    float* xchg = reinterpret_cast<float*>(smem + L::XCHG);
    // the other half row's value; the two warps of a quarter meet, one of the two slots being free for the next exchange
    auto exchange = [&](int slot, float mine) {
      xchg[(slot * 2 + half) * kBlk + t] = mine;
      asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
      return xchg[(slot * 2 + (half ^ 1)) * kBlk + t];
    };
    float m_ref = -INFINITY, l_run = 0.f;       // the maximum the accumulator is relative to, and this half row's sum
    bool ok = true;
    // After a wait that gave up the loop runs out without work, so that no warp is missed at the barriers.
    for (int j = 0; j < n; ++j) {
      const int kv0 = j * kBlk, c0 = half * 64;
      const bool diagonal = p.causal && j == qb;
      const float* mk_s = mask_s + (j & 1) * kBlk + c0;
      if constexpr (kMask) {       // additive mask of this key block (mask * log2e; -inf beyond S); the other buffer may still be in use
        if (half == 0) {
          const int kv = kv0 + t;
          mask_s[(j & 1) * kBlk + t] = kv < p.S ? __ldg(p.mask + static_cast<long long>(b) * p.S + kv) * kLog2e : -INFINITY;
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
      }
      ok = __all_sync(0xffffffffu, ok && mbar_wait(s_full, j & 1, abort_flag, p.status, kStatusWaitAccum));
      uint32_t sv[2][32];
      float m_half = -INFINITY;
      if (ok) {
        tc_fence_after_sync();
        tmem_ld32(tS + lane_base + c0, sv[0]);
        tmem_ld32(tS + lane_base + c0 + 32, sv[1]);
        tmem_ld_wait();
        tc_fence_before_sync();
        arrive_warp(s_free, lane);
        // row maximum of score * scale (+ mask); the scores stay as they came for the exponent below
        if (kMask ? diagonal : diagonal || kv0 + kBlk > p.S) {
          const int seen = (p.causal ? min(q, p.S - 1) : p.S - 1) - kv0 - c0;
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (32 * c + i > seen) sv[c][i] = __float_as_uint(hidden);
        }
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if constexpr (kMask) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i4 = 0; i4 < 32; i4 += 4) {
              const float4 mk = *reinterpret_cast<const float4*>(mk_s + 32 * c + i4);
              const float mk4[4] = {mk.x, mk.y, mk.z, mk.w};
#pragma unroll
              for (int k = 0; k < 4; ++k) m4[k] = fmaxf(m4[k], fmaf(__uint_as_float(sv[c][i4 + k]), sc, mk4[k]));
            }
          m_half = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        } else if (sc < 0.f) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], -__uint_as_float(sv[c][i]));
          m_half = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * -sc;
        } else {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(sv[c][i]));
          m_half = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sc;
        }
      }
      const float m_new = fmaxf(m_ref, fmaxf(m_half, exchange(j & 1, m_half)));
      if (!ok) continue;
      if (j == 0) {
        m_ref = m_new;
      } else {
        ok = __all_sync(0xffffffffu, mbar_wait(pv_done, (j - 1) & 1, abort_flag, p.status, kStatusWaitAccum));     // P may be overwritten, O touched
        if (!ok) continue;
        tc_fence_after_sync();
        // At every growth, however small: relative to the true maximum a row's largest probability is exactly 1 and takes no rounding to bf16,
        // relative to an older one it is rounded like the rest (up to a fifth more error where few keys carry a row).
        // B 2 x H 12 x S 4096 causal: 100 us; 95 with rescaling at growths of 2^8 only.
        if (__any_sync(0xffffffffu, m_new > m_ref)) {       // the same for both warps of a row; each rescales half of O's columns
          const float alpha = m_new == -INFINITY ? 1.f : ex2_approx(m_ref - m_new);
          m_ref = m_new;
          l_run *= alpha;
#pragma unroll 1
          for (int c = half * 32; c < half * 32 + 32; c += 16) {
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
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int i4 = 0; i4 < 32; i4 += 4) {
          float off[4] = {neg_m, neg_m, neg_m, neg_m};
          if constexpr (kMask) {       // mask - maximum first, then one FMA: a large mask common to the row's keys costs the scores no bits
            const float4 mk = *reinterpret_cast<const float4*>(mk_s + 32 * c + i4);
            off[0] += mk.x; off[1] += mk.y; off[2] += mk.z; off[3] += mk.w;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float pe = ex2_approx(fmaf(__uint_as_float(sv[c][i4 + k]), sc, off[k]));
            l4[k] += pe;
            sv[c][i4 + k] = __float_as_uint(pe);
          }
        }
        if constexpr (kDrop) {
          const unsigned long long base = ((static_cast<unsigned long long>(b) * p.H + h) * p.S + q) * p.S + kv0 + c0 + 32 * c;
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
        tmem_st16(tP + lane_base + half * 32 + 16 * c, pk);
      }
      l_run += (l4[0] + l4[1]) + (l4[2] + l4[3]);
      tmem_st_wait();
      tc_fence_before_sync();
      arrive_warp(p_ready, lane);
    }
    l_run += exchange(n & 1, l_run);
    ok = ok && mbar_wait(pv_done, (n - 1) & 1, abort_flag, p.status, kStatusWaitAccum);
    ok = __all_sync(0xffffffffu, ok);
    const uint32_t stage = smem_u32(smem + L::Q) + quarter * 4096;        // every product that reads Q has retired
    if (ok) {
      tc_fence_after_sync();
      const float inv_l = l_run > 0.f ? 1.f / l_run : 0.f;
      uint32_t v[32];
      tmem_ld32(tO + lane_base + half * 32, v);
      tmem_ld_wait();
      float f[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]) * inv_l;
      stage_half(stage, lane, half * 32, f);
      // natural-log LSE of the scaled, masked scores
      if (half == 0 && q < p.S) lse[(static_cast<long long>(b) * p.H + h) * p.S + q] = (l_run > 0.f) ? (m_ref + log2f(l_run)) / kLog2e : -INFINITY;
    }
    asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
    if (ok) {         // both halves of the quarter's 32 rows are staged: each warp writes 16 of them, eight lanes per row
      __nv_bfloat16* base = o + static_cast<long long>(b) * p.osb + static_cast<long long>(h) * p.osh;
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        const int r = half * 16 + it * 4 + (lane >> 3), ch = lane & 7, row = q0 + quarter * 32 + r;
        const uint4 val = ld_shared_v4(stage + r * 128 + ((ch ^ (r & 7)) << 4));
        if (row < p.S) *reinterpret_cast<uint4*>(base + static_cast<long long>(row) * p.oss + ch * 8) = val;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kFwdSoftmaxWarps) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, 256);
  }
}

}  // namespace

int attn_fwd_long(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, void* o, float* lse, const AttnParams& p, cudaStream_t stream) {
  const long long ctas = static_cast<long long>((p.S + kBlk - 1) / kBlk) * p.H * p.B;
  if (ctas > 0x7fffffffll) return -4;
  const auto go = [&](auto drop, auto mask) {
    constexpr auto kern = attn_fwd_long_kernel<decltype(drop)::value, decltype(mask)::value>;
    constexpr int smem = FwdLong::TOTAL + 1024;
    if (const cudaError_t e = allow_smem<kern>(smem, true)) return static_cast<int>(e);
    const cudaError_t e = launch_pdl(kern, dim3(static_cast<unsigned>(ctas)), dim3(kFwdThreads), static_cast<size_t>(smem), stream, tq, tk, tv,
                                     static_cast<__nv_bfloat16*>(o), lse, p);
    return static_cast<int>(e != cudaSuccess ? e : cudaGetLastError());
  };
  constexpr std::true_type yes;
  constexpr std::false_type no;
  return p.p_drop > 0.f ? (p.mask ? go(yes, yes) : go(yes, no)) : (p.mask ? go(no, yes) : go(no, no));
}

}  // namespace fb
