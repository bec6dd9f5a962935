// Shared by the flash-attention kernels (attn_prefill.cu, attn_split.cu).
#pragma once
#include <cuda_runtime.h>
#include "ortb200_kernels.h"
#include "ptx_sm100.cuh"

namespace ortb200 {

struct AttnParams {
  const int* seqlens_k;
  const int* key_mask;
  const void* head_sink;
  void* out;
  int B, S, N, Nk, kv_len;
  long long o_strides[3];
  int first_prompt, causal, window;
  float scale_log2, softcap, scale;
  int bf16;
  int* status;
  // packed queries over a paged cache (block_table given)
  const int* block_table;
  const int* cu_seqlens;
  const int* past_seqlens;
  int block_size, max_blocks, num_blocks;
  int chunk;             // > 0: keys of the query's own chunk only
  int group_log2;        // attn_prefill.cu: log2 of the query heads of one key head that a CTA takes together
};

// Packed queries over a paged cache, softmax weights as the sum of two 16-bit terms (the caller has checked the arguments).
int launch_attn_split(const ortb200_attn_prefill_args* a, cudaStream_t stream);

#ifdef __CUDACC__
namespace {
__device__ uint4 g_zero_rows[63 * 8];
}
// What lies behind the last key in its value tile (BOXES boxes of 64 rows x 128 bytes, the first `live` of them of keys) may be
// anything, and 0 * NaN would reach the product.  The producer lane loads that tile on a barrier of its own (`loaded`), copies
// zeros over the other rows, and `full` then stands for both; the consumers know nothing of it.  (A condition around
// the products or in the softmax loop cost every causal prompt 6 - 13 %, those without such rows too; this costs 2 - 4 % of
// 8 x 1024, 122 -> 125 us here and 102 -> 106 with 32-bit weights, and 2 % of encoder batches, 114 -> 116.)
template <int BOXES, int BOX_BYTES>
__device__ __forceinline__ bool clear_stale_rows(uint8_t* tile, int live, uint64_t* loaded, uint64_t* full) {
  if (!mbar_wait(loaded, 0)) return false;
  const uint32_t bytes = static_cast<uint32_t>(64 - live) * 128;
  mbar_expect_tx(full, BOXES * bytes);
#pragma unroll
  for (int bx = 0; bx < BOXES; ++bx) bulk_load(tile + bx * BOX_BYTES + live * 128, g_zero_rows, bytes, full);
  return true;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
#endif

}  // namespace ortb200
