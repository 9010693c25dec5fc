// bf16 GEMM for problems with few output tiles (a short text through an encoder, a small model's step): 128 x 64 tiles, the
// reduction of a tile split over the CTAs of a cluster.
//
// D[m,n] = sum_k A(m,k) * B(n,k), bf16 in and out, fp32 accumulate; A K-major, B K-major or MN-major; the epilogues of
// gemm_tcgen05.cu (bias, GELU with the pre-activation saved, GELU').
//
// What bounds such a product is not arithmetic but the latency of one CTA's chain (load, multiply, write out) and, because a dozen
// CTAs stream all of B, memory parallelism. So:
//   * up to eight CTAs of a cluster take a slice of K each, which shortens the chain and puts the whole chip on the loads; the fp32
//     partial tiles meet in shared memory, where each CTA sums and finishes its share of the rows through distributed shared memory;
//   * B's first tiles are prefetched into L2 before the wait for the previous kernel of the stream. That is allowed whoever wrote B:
//     a prefetch fills L2 only, where later writes and reads meet;
//   * 97 KB of shared memory and 64 TMEM columns, so that the next such kernel's CTAs fit beside this one's and run their set-up early.
// Back to back in one graph, against the persistent kernel's best tile: 77 x 768 x 768 6.7 -> 4.3 us, 77 x 768 x 3072 16.9 -> 5.2,
// 512 x 768 x 3072 17.5 -> 9.7, 1024 x 512 x 2048 12.8 -> 9.4.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../include/flodl_b200.h"
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace fb {

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld_elems,
                      uint32_t box_inner, uint32_t box_outer);  // gemm_tcgen05.cu

namespace {

constexpr int kTM = 128, kTN = 64, kTK = 64;
constexpr int kStages = 4;
constexpr int kABytes = kTM * kTK * 2, kStageBytes = kABytes + kTN * kTK * 2;
constexpr int kPitch = kTN + 4;                              // floats per row of the partial tile: 16-byte rows apart by four banks
constexpr int kThreads = 192;                                // TMA, MMA, 4 epilogue warps
constexpr int kSmem = kStages * kStageBytes + 1024 /*alignment*/ + 256 /*barriers*/;
static_assert(kTM * kPitch * 4 <= kStages * kStageBytes, "the partial tile takes the place of the operand stages");

// Up to three products of one A (the Q, K and V projections of a layer): their columns side by side in C, `group` apart.
struct BMaps { CUtensorMap b[3]; };
struct SmallGemm {
  int M, N, K, b_mn, kb_per;
  int group;                   // columns of one product, a multiple of the tile; N where there is but one
  const void* group_bias[3];
  __nv_bfloat16* C;
  long long ldc;
  int bias_fp32, epi;
  __nv_bfloat16* aux;
  long long ldaux;
  const float* alpha;
  int* status;
};

__device__ __forceinline__ void prefetch_2d(const void* tmap, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(tmap), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t cta) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(cta));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// For the end: "I have read the others' parts". Every value read has gone into a store by then, and nothing written has to be seen, so that the barrier
// doesn't wait for the stores, as one that releases them does: 512 x 512 x 512 4.8 -> 4.6 us, 77 x 768 x 3072 5.5 -> 5.2, 512 x 768 x 3072 10.1 -> 9.7.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void unpack4(const uint2& raw, float (&v)[4]) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&v)[4]) {
  const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
}

// grid = (CTAs per tile = cluster, column tiles, row tiles)
__global__ void __launch_bounds__(kThreads)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ BMaps maps, const __grid_constant__ SmallGemm p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  uint64_t* done = empty + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* part = reinterpret_cast<float*>(smem);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = gridDim.x, rank = blockIdx.x;            // the cluster spans x
  const int n0 = blockIdx.y * kTN, m0 = blockIdx.z * kTM;
  const int grp = n0 / p.group, b0 = n0 - grp * p.group;       // whose B, and the tile's first column in it
  const CUtensorMap& tmB = grp == 0 ? maps.b[0] : grp == 1 ? maps.b[1] : maps.b[2];
  const void* bias_of = grp == 0 ? p.group_bias[0] : grp == 1 ? p.group_bias[1] : p.group_bias[2];
  const int num_kb = (p.K + kTK - 1) / kTK;
  const int kb0 = rank * p.kb_per, kb1 = min(num_kb, kb0 + p.kb_per);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int kb = kb0; kb < min(kb1, kb0 + 2 * kStages); ++kb) p.b_mn ? prefetch_2d(&tmB, b0, kb * kTK) : prefetch_2d(&tmB, kb * kTK, b0);
  }
  if (warp == 1) {
    tmem_alloc<1>(tmem_slot, kTN);
    tmem_relinquish<1>();
  }
  // The bias as well: in an encoder whose weights outgrow L2 it comes from HBM.
  if (warp == 2 && lane < 2 && bias_of) prefetch_l2(static_cast<const char*>(bias_of) + (p.bias_fp32 ? 4 : 2) * min(b0 + lane * (kTN / 2), p.group - 1));
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_entry();

  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0, s = i % kStages;
        if (!mbar_wait(&empty[s], ((i / kStages) & 1) ^ 1, abort_flag, p.status, kStatusWaitEmpty)) break;
        uint8_t* sa = smem + s * kStageBytes;
        mbar_expect_tx(&full[s], kStageBytes);
        tma_load_2d(sa, &tmA, &full[s], kb * kTK, m0);
        if (p.b_mn) tma_load_2d(sa + kABytes, &tmB, &full[s], b0, kb * kTK);
        else tma_load_2d(sa + kABytes, &tmB, &full[s], kb * kTK, b0);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_bf16(kTM, kTN, 0, p.b_mn);
      const uint32_t b_lbo = p.b_mn ? 8192u : 16u, b_step = p.b_mn ? 2048u : 32u;
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        const int i = kb - kb0, s = i % kStages;
        ok = mbar_wait(&full[s], (i / kStages) & 1, abort_flag, p.status, kStatusWaitFull);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t sa = smem_u32(smem + s * kStageBytes), sb = sa + kABytes;
#pragma unroll
        for (int k4 = 0; k4 < kTK / 16; ++k4)
          umma_bf16<1>(tmem, make_smem_desc(sa + k4 * 32, 16, 1024), make_smem_desc(sb + k4 * b_step, b_lbo, 1024), idesc, i > 0 || k4 > 0);
        umma_commit(&empty[s]);
      }
      if (ok) umma_commit(done);
    }
  } else {
    // this CTA's partial tile: TMEM -> shared memory, over the operand stages, which every product has read
    const int q = warp & 3;
    ok = __all_sync(0xffffffffu, mbar_wait(done, 0, abort_flag, p.status, kStatusWaitAccum));
    if (ok) {
      tc_fence_after_sync();
      float* mine = part + (q * 32 + lane) * kPitch;
#pragma unroll
      for (int c = 0; c < kTN; c += 32) {
        uint32_t v[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(q * 32) << 16) + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          *reinterpret_cast<uint4*>(mine + c + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      }
      tc_fence_before_sync();
    }
  }
  __syncwarp();
  if (split > 1) cluster_barrier();
  else __syncthreads();

  // Rows are dealt out over the cluster; 16 threads finish a row, four columns each. After a wait that gave up there is nothing to
  // finish (the status says so), but every thread still meets the barriers.
  const int rows = min(kTM, p.M - m0), per = (rows + split - 1) / split;
  const int col = n0 + (threadIdx.x & 15) * 4;
  if (col < p.N && !*abort_flag) {
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if (bias_of) {
      const int bc = col - grp * p.group;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        bias[j] = p.bias_fp32 ? __ldg(static_cast<const float*>(bias_of) + bc + j) : __bfloat162float(static_cast<const __nv_bfloat16*>(bias_of)[bc + j]);
    }
    const float alpha = p.alpha ? __ldg(p.alpha) : 1.f;
    for (int r = rank * per + (threadIdx.x >> 4); r < min(rows, (rank + 1) * per); r += kThreads / 16) {
      const uint32_t at = smem_u32(part + r * kPitch + (threadIdx.x & 15) * 4);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (split == 1) {
        const float4 t = *reinterpret_cast<const float4*>(part + r * kPitch + (threadIdx.x & 15) * 4);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
      } else {
        float4 t[8];
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c < split) t[c] = ld_cluster_f4(at, c);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c < split) { v[0] += t[c].x; v[1] += t[c].y; v[2] += t[c].z; v[3] += t[c].w; }
      }
      const long long row = m0 + r;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = v[j] * alpha + bias[j];
      if (p.epi == FB_EPI_GELU_ERF || p.epi == FB_EPI_GELU_TANH) {
        if (p.aux) store4(p.aux + row * p.ldaux + col, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = p.epi == FB_EPI_GELU_ERF ? gelu_erf_fast(v[j]) : gelu_tanh_fast(v[j]);
      } else if (p.epi == FB_EPI_DGELU_ERF || p.epi == FB_EPI_DGELU_TANH) {
        float h[4];
        unpack4(*reinterpret_cast<const uint2*>(p.aux + row * p.ldaux + col), h);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] *= p.epi == FB_EPI_DGELU_ERF ? dgelu_erf_fast(h[j]) : dgelu_tanh_fast(h[j]);
      }
      store4(p.C + row * p.ldc + col, v);
    }
  }
  __syncwarp();
  if (split > 1) { cluster_arrive_relaxed(); cluster_wait(); }     // no CTA leaves while another reads its partial tile
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem, kTN);
  }
}

}  // namespace

// CTAs per tile, or 0 where this kernel does not apply. It is taken up to half as many tiles of 128 x 64 as SMs; with more the split has no SMs to spread
// over. The reduction has to be long enough for the split to pay for its hand-over, unless the tile is mostly padding, of which this kernel writes less:
// us against the persistent kernel, 1024 x 256 x 256 5.3 (4.6), 4096 x 128 x 512 6.3 (5.9), 512 x 512 x 512 5.0 (5.8), 512 x 768 x 768 6.4 (7.3), 32 x 128 x 128
// 2.9 (3.4), 128 x 128 x 128 4.0 (3.9). `several` products in one launch save launches as well and are taken with any reduction: six encoder layers of width
// 256 over 4 x 128 tokens 206 us, with Q, K and V one after the other 258. The reduction is split until every SM has a CTA or a CTA is down to two 64-wide steps: a step's products are over
// long before its loads are.
int gemm_small_split(int M, int N, int K, bool several) {
  const long long tiles = static_cast<long long>((M + kTM - 1) / kTM) * ((N + kTN - 1) / kTN);
  const int num_kb = (K + kTK - 1) / kTK, sms = sm_count();
  if (tiles > sms / 2) return 0;
  if (!several && M > 96 && K < 768 && (K < 512 || tiles > sms / 4)) return 0;
  int split = static_cast<int>(sms / tiles);
  if (split > 8) split = 8;
  if (split > num_kb / 2) split = num_kb / 2;
  if (split < 1) split = 1;
  const int per = (num_kb + split - 1) / split;
  return (num_kb + per - 1) / per;         // no CTA without a step
}

// Whether rows and pointers are aligned for four columns at a time.
bool gemm_small_aligned(int N, const void* C, long long ldc, const void* aux, long long ldaux) {
  return N % 4 == 0 && ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 7) == 0 && (!aux || (ldaux % 4 == 0 && (reinterpret_cast<uintptr_t>(aux) & 7) == 0));
}

int gemm_small(const void* A, const void* const* B, void* C, int M, int group, int groups, int K, long long lda, long long ldb, long long ldc, int b_mn,
               const void* const* bias, int bias_fp32, int epi, void* aux, long long ldaux, const float* alpha, int split, int* status, cudaStream_t stream) {
  const int N = group * groups;
  if (groups < 1 || groups > 3 || (groups > 1 && group % kTN)) return -2;
  CUtensorMap ta;
  BMaps tb;
  int r = make_tmap_bf16_2d(&ta, A, K, M, lda, kTK, kTM);
  for (int g = 0; g < 3 && !r; ++g) {
    const void* b = B[g < groups ? g : 0];
    r = b_mn ? make_tmap_bf16_2d(&tb.b[g], b, group, K, ldb, 64, kTK) : make_tmap_bf16_2d(&tb.b[g], b, K, group, ldb, kTK, kTN);
  }
  if (r) return r;
  if (const cudaError_t e = allow_smem<gemm_small_kernel>(kSmem, true)) return static_cast<int>(e);
  const int num_kb = (K + kTK - 1) / kTK;
  SmallGemm p{M, N, K, b_mn, (num_kb + split - 1) / split, group, {nullptr, nullptr, nullptr}, static_cast<__nv_bfloat16*>(C), ldc, bias_fp32, epi,
              static_cast<__nv_bfloat16*>(aux), ldaux, alpha, status};
  for (int g = 0; g < groups; ++g) p.group_bias[g] = bias[g];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(split, (N + kTN - 1) / kTN, (M + kTM - 1) / kTM);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (pdl_enabled()) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_small_kernel, ta, tb, p));
}

}  // namespace fb
