// What the attention kernels of one key block (flash_attn.cu) and of several (flash_attn_long.cu) share: the parameter
// block, the 4-D tensor maps over [B, S, H, 64] and the moves between row-per-thread registers and global rows.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "ptx_sm100.cuh"

namespace fb {

constexpr int kHD = 64;        // head dim
constexpr int kBlk = 128;      // rows per query / key block
constexpr int kAttnThreads = 160;
constexpr float kLog2e = 1.4426950408889634f;

void ensure_thread_context();                                    // gemm_tcgen05.cu

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

inline int make_tmap_bshd(CUtensorMap* out, const void* base, int B, int H, int S, long long sb, long long ss, long long sh) {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      return -1;
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  ensure_thread_context();
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(kHD), static_cast<cuuint64_t>(S), static_cast<cuuint64_t>(H), static_cast<cuuint64_t>(B)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(ss) * 2, static_cast<cuuint64_t>(sh) * 2, static_cast<cuuint64_t>(sb) * 2};
  cuuint32_t box[4] = {kHD, kBlk, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

__device__ __forceinline__ void tma_load_4d(void* smem_dst, const void* tmap, uint64_t* bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// One arrival for a warp whose lanes are all done. (An arrival is an atomic on the barrier's word; the tensor cores read their
// operands through the same shared-memory pipe.)
__device__ __forceinline__ void arrive_warp(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// Address of the 16-byte chunk holding columns [8*chunk, 8*chunk+8) of `row` in a [128][64] bf16
// tile stored with the 128-byte swizzle (tile base 1024-byte aligned).
__device__ __forceinline__ uint32_t swz_chunk(uint32_t tile_base, int row, int chunk) {
  return tile_base + row * 128 + ((chunk ^ (row & 7)) << 4);
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint4 pack8(const float* v) {
  uint4 r;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  return r;
}

__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// Row-per-thread data (the TMEM register layout: thread = row, 64 bf16 = 128 bytes per row) to and from global rows
// that are `row_stride` elements apart. A thread touching its own row would make every load / store instruction hit 32
// different 128-byte lines; instead each warp moves its 32 rows through a 4 KB staging area of shared memory
// (chunks XOR-swizzled by row, so both sides are free of bank conflicts) and eight lanes share one row in global
// memory. Only the warp's own rows are involved: __syncwarp is all the synchronisation needed.
//
// stage_half: thread `lane` deposits 32 consecutive columns [col0, col0 + 32) of its row.
__device__ __forceinline__ void stage_half(uint32_t stage, int lane, int col0, const float* v32) {
#pragma unroll
  for (int g = 0; g < 4; ++g) st_shared_v4(stage + lane * 128 + ((((col0 >> 3) + g) ^ (lane & 7)) << 4), pack8(v32 + 8 * g));
}
// flush_rows: after both halves were staged, writes rows [row0, row0 + 32) (those below `row_limit`) of a [*, 64] bf16 tensor.
__device__ __forceinline__ void flush_rows(uint32_t stage, int lane, __nv_bfloat16* base, long long row_stride, int row0, int row_limit) {
  __syncwarp();
  const int sub = lane >> 3, ch = lane & 7;
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int r = it * 4 + sub;
    const uint4 val = ld_shared_v4(stage + r * 128 + ((ch ^ (r & 7)) << 4));
    if (row0 + r < row_limit) *reinterpret_cast<uint4*>(base + static_cast<long long>(row0 + r) * row_stride + ch * 8) = val;
  }
  __syncwarp();
}
// D[row] = sum_c a[row][c] * b[row][c] over 64 columns for the warp's 32 rows, eight lanes per row; lane l gets row l's sum.
__device__ __forceinline__ float row_dot64(const __nv_bfloat16* a, const __nv_bfloat16* b, long long row_stride, int row0, int row_limit, int lane) {
  const int sub = lane >> 3, ch = lane & 7;
  float mine = 0.f;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    // all loads of four iterations first (the shuffles below would otherwise serialise one memory latency per iteration)
    uint4 xa[4], xb[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = (half * 4 + k) * 4 + sub;
      xa[k] = xb[k] = make_uint4(0u, 0u, 0u, 0u);
      if (row0 + r < row_limit) {
        xa[k] = __ldg(reinterpret_cast<const uint4*>(a + static_cast<long long>(row0 + r) * row_stride + ch * 8));
        xb[k] = __ldg(reinterpret_cast<const uint4*>(b + static_cast<long long>(row0 + r) * row_stride + ch * 8));
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int it = half * 4 + k;
      const __nv_bfloat162* ha = reinterpret_cast<const __nv_bfloat162*>(&xa[k]);
      const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&xb[k]);
      float d = 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 fa = __bfloat1622float2(ha[e]), fb2 = __bfloat1622float2(hb[e]);
        d += fa.x * fb2.x + fa.y * fb2.y;
      }
      d += __shfl_xor_sync(0xffffffffu, d, 1);
      d += __shfl_xor_sync(0xffffffffu, d, 2);
      d += __shfl_xor_sync(0xffffffffu, d, 4);
      // row it*4 + g now sits in lanes 8g .. 8g+7; lane l wants row l = it*4 + g  <=>  it == l / 4, g == l % 4
      const float got = __shfl_sync(0xffffffffu, d, (lane & 3) * 8);
      if ((lane >> 2) == it) mine = got;
    }
  }
  return mine;
}

struct AttnParams {
  int B, H, S;
  long long sb, ss, sh;      // element strides of q/k/v
  long long osb, oss, osh;   // ... of o / dO
  long long gsb, gss, gsh;   // ... of dq / dk / dv
  const float* mask;         // [B, S] additive, may be null
  float scale;
  int causal;
  float p_drop;
  unsigned long long seed;
  const unsigned long long* seed_dev;
  int* status;
  int group;                 // heads whose key blocks are handed out together in the backward pass: one for each SM
};

inline AttnParams make_params(int B, int H, int S, const long long* qs, const long long* os, const long long* gs, const float* mask,
                              float scale, int causal, float p_drop, unsigned long long seed,
                              const unsigned long long* seed_dev, int* status) {
  AttnParams p;
  p.B = B; p.H = H; p.S = S; p.sb = qs[0]; p.ss = qs[1]; p.sh = qs[2]; p.mask = mask;
  p.osb = os[0]; p.oss = os[1]; p.osh = os[2];
  p.gsb = gs[0]; p.gss = gs[1]; p.gsh = gs[2]; p.scale = scale; p.causal = causal;
  p.p_drop = p_drop; p.seed = seed; p.seed_dev = seed_dev; p.status = status;
  p.group = sm_count();
  return p;
}

inline bool strides_ok(const void* ptr, long long sb, long long ss, long long sh) {
  return (reinterpret_cast<uintptr_t>(ptr) % 16 == 0) && sb % 8 == 0 && ss % 8 == 0 && sh % 8 == 0;
}

// Forward and backward over several key blocks (flash_attn_long.cu); return a CUDA error code.
int attn_fwd_long(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, void* o, float* lse, const AttnParams& p, cudaStream_t stream);
int attn_bwd_long(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo, const void* o, const void* d_o,
                  const float* lse, void* dq, void* dk, void* dv, float* dq_accum, const AttnParams& p, cudaStream_t stream);

}  // namespace fb
