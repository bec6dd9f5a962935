// Shared by the two decode-attention kernels (CUDA-core split-KV kernel and the tcgen05 kernel): launch
// parameters and the tail that merges the splits and writes the output.
#pragma once
#include <cuda_runtime.h>
#include "ortb200_kernels.h"
#include "ptx_sm100.cuh"

namespace ortb200 {

struct DecodeParams {
  const void* q;
  const void* k_cache;
  const void* v_cache;
  const int* seqlens_k;
  const void* head_sink;
  void* out;
  float* ws;
  unsigned int* counters;
  int* status;
  int B, N, Nk, Smax, splits, window, gparts;
  int splits_last;         // (tcgen05 kernel) order of the grid: splits outermost instead of sequences
  int piece_tiles;         // > 0 (tcgen05 kernel): a sequence uses a split per this many tiles of its keys, at most `splits`
  float scale, softcap;
  // paged cache [num_blocks, block_size, Nk, H]: key j of sequence b lives in block block_table[b, j / block_size]
  const int* block_table;
  int block_size, max_blocks;
  // fused "unpack + rotary + append" (one new token per sequence): q, k and v are read from the packed projection
  // output qkv [B, (N + 2 Nk) H]; the CTA whose key range ends at the new position rotates the new key, writes
  // key and value into the cache and attends to them from registers
  const void* qkv;
  int cos_rows;
  const void* cos_cache;
  const void* sin_cache;
  int do_rotary, interleaved;
  // L2 prefetch of the next kernel's weights: CTA i asks for bytes [i, i + 1) * prefetch_per_cta of the range
  const unsigned char* prefetch;
  long long prefetch_bytes;
  int prefetch_per_cta;
  int chunk;               // > 0: keys of the new token's own chunk only
  long long q_ld, out_ld;  // elements between the rows of q and of out
};

// Running maxima start at a large negative finite value so that exp(m_old - m_new) never sees inf - inf.
constexpr float kNegBig = -1.0e30f;
__device__ __forceinline__ float safe_exp_diff(float a, float b) {
  return a <= kNegBig ? 0.f : __expf(a - b);
}


// Where the states of the splits lie behind the counters, and how many bytes there are: the merge reads 16-byte vectors, and a
// caller's workspace need only be aligned for floats.
inline float* decode_states(const ortb200_gqa_decode_args* a, int64_t* bytes) {
  const uintptr_t ws = reinterpret_cast<uintptr_t>(a->workspace), first = (ws + 65536 + 15) & ~uintptr_t(15);
  *bytes = ws ? a->workspace_bytes - static_cast<int64_t>(first - ws) : 0;
  return ws ? reinterpret_cast<float*>(first) : nullptr;
}

// tcgen05 decode kernel (gqa_decode_tc.cu)
bool gqa_decode_tc_supported(const ortb200_gqa_decode_args* a);
int launch_gqa_decode_tc(const ortb200_gqa_decode_args* a, cudaStream_t stream);

// Tail of a decode-attention CTA.  On entry thread tid < H holds, for each of the G query heads, its dim of the
// unnormalised output (fa), and every thread holds the running maximum (fm, natural-log domain) and the sum of
// exponentials (fl) of the CTA's key range.  With splits > 1 (of this sequence: at most p.splits) the state goes to the
// workspace and the CTA that arrives last on the tile's counter merges all splits; that CTA (or the only one) normalises and
// stores.
// `scratch`: 2 * splits * G floats of shared memory that nothing else needs any more.  In the merge a thread owns four dims of
// one head and fetches eight splits at a time, after all threads have fetched the maxima and sums: a dim per thread, head
// after head and load after load, was a chain of 2 * splits * G L2 round trips.
template <typename T, int H, int G>
__device__ __forceinline__ void decode_finish(const DecodeParams& p, int tile, int split, int splits, int b, int head0, int n_heads,
                                              int tid, float (&fm)[G], float (&fl)[G], float (&fa)[G],
                                              unsigned int* sm_last_ptr, float* scratch) {
  const bool owner = tid < H;
  unsigned int& sm_last = *sm_last_ptr;
  bool finalize = true;
  if (splits > 1) {
    // publish partial state: ws[tile][split][g][H + 4]
    constexpr int kState = H + 4;   // rows of 16-byte vectors
    float* my = p.ws + ((static_cast<size_t>(tile) * p.splits + split) * G) * kState;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (owner) my[g * kState + tid] = fa[g];
      if (tid == 0) {
        my[g * kState + H] = fm[g];
        my[g * kState + H + 1] = fl[g];
      }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      const unsigned int old = atomicAdd(&p.counters[tile], 1u);
      const unsigned int last = old == static_cast<unsigned int>(splits - 1) ? 1u : 0u;
      if (last) p.counters[tile] = 0;
      sm_last = last;
    }
    __syncthreads();
    finalize = false;   // the merge below stores the result itself
    if (sm_last != 0) {
      __threadfence();
      const float* base = p.ws + (static_cast<size_t>(tile) * p.splits * G) * kState;
      const int states = splits * G;
      for (int i = tid; i < states; i += blockDim.x) {
        scratch[i] = __ldcg(&base[i * kState + H]);
        scratch[states + i] = __ldcg(&base[i * kState + H + 1]);
      }
      __syncthreads();
      for (int i = tid; i < n_heads * (H / 4); i += blockDim.x) {
        const int g = i / (H / 4), d = i % (H / 4) * 4;
        float mm = kNegBig;
        for (int s = 0; s < splits; ++s) mm = fmaxf(mm, scratch[s * G + g]);
        float ll = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s0 = 0; s0 < splits; s0 += 8) {
          float4 v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            v[e] = s0 + e < splits ? __ldcg(reinterpret_cast<const float4*>(&base[((s0 + e) * G + g) * kState + d])) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (s0 + e >= splits) break;
            const float c = safe_exp_diff(scratch[(s0 + e) * G + g], mm);
            ll += scratch[states + (s0 + e) * G + g] * c;
            acc[0] += v[e].x * c;
            acc[1] += v[e].y * c;
            acc[2] += v[e].z * c;
            acc[3] += v[e].w * c;
          }
        }
        float scale = 1.f;
        if (p.head_sink) {
          const float sink = to_float<T>(static_cast<const T*>(p.head_sink)[head0 + g]);
          const float m2 = fmaxf(mm, sink);
          scale = safe_exp_diff(mm, m2);
          ll = ll * scale + __expf(sink - m2);
        }
        T* o = static_cast<T*>(p.out) + b * p.out_ld + static_cast<long long>(head0 + g) * H + d;
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = from_float<T>(ll > 0.f ? acc[e] * scale / ll : 0.f);
      }
    }
  }
  pdl_launch_dependents();
  if (finalize && owner) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (g >= n_heads) break;
      float ll = fl[g];
      if (p.head_sink) {
        const float sink = to_float<T>(static_cast<const T*>(p.head_sink)[head0 + g]);
        const float mm = fmaxf(fm[g], sink);
        const float c = safe_exp_diff(fm[g], mm);
        ll = ll * c + __expf(sink - mm);
        fa[g] *= c;
      }
      const float o = ll > 0.f ? fa[g] / ll : 0.f;
      static_cast<T*>(p.out)[b * p.out_ld + static_cast<long long>(head0 + g) * H + tid] = from_float<T>(o);
    }
  }
}

}  // namespace ortb200
