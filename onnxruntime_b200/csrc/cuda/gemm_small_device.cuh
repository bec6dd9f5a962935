// Device helpers shared by the decode-shaped GEMM kernels (gemm_smallm.cu, gemm_q4.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "gemm_internal.h"
#include "ptx_sm100.cuh"

namespace ortb200 {
namespace {

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// address of the same shared-memory location in CTA `cta` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_smem_addr, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(cta));
  return r;
}
__device__ __forceinline__ float ld_dsmem(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// four consecutive fp32 values of one location in the C partial tiles of a cluster, added in rank order
template <int C>
__device__ __forceinline__ void sum_partials(uint32_t local_smem_addr, float (&y)[4]) {
  float v[C][4];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const uint32_t a = C > 1 ? map_to_cta(local_smem_addr, static_cast<uint32_t>(c)) : local_smem_addr;
    if (C > 1) asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[c][0]), "=f"(v[c][1]), "=f"(v[c][2]), "=f"(v[c][3]) : "r"(a) : "memory");
    else asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[c][0]), "=f"(v[c][1]), "=f"(v[c][2]), "=f"(v[c][3]) : "r"(a) : "memory");
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    y[e] = 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c) y[e] += v[c][e];
  }
}
__device__ __forceinline__ float2 unpack16(uint32_t w, int dtype) {
  if (dtype == ORTB200_BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
__device__ __forceinline__ uint32_t pack16(float lo, float hi, int dtype) {
  if (dtype == ORTB200_BF16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float load16(const void* base, long long i, int dtype) {
  return unpack16(static_cast<const uint16_t*>(base)[i], dtype).x;
}

__device__ __forceinline__ float act_apply(int act, float v) {
  switch (act) {
    case ORTB200_ACT_GELU: return gelu_erf_fast(v);
    case ORTB200_ACT_FASTGELU: return 0.5f * v * (1.0f + tanhf(0.7978845608028654f * v * (1.0f + 0.044715f * v * v)));
    case ORTB200_ACT_RELU: return fmaxf(v, 0.0f);
    case ORTB200_ACT_SILU: return v / (1.0f + __expf(-v));
    case ORTB200_ACT_QUICKGELU: return v / (1.0f + __expf(-1.702f * v));
    default: return v;
  }
}

}  // namespace
}  // namespace ortb200
