// Flash-attention forward for sm_100a on tcgen05: S = Q K^T and O_tile = P V run
// on the 5th-generation tensor cores with both accumulators in tensor memory.
//
// One CTA owns 128 query rows of one (batch, key head): 128 / G tokens of the G query heads that share the key head, so
// that a single token of a mixed batch costs one tile per key head and the diagonal of a prompt little masked work.
// Per 64-key tile:
//   MMA 1  S[128 q, 64 keys]   = Q[128, H] . K[64, H]^T       (both K-major)
//   softmax threads (one per query row) read their row of S from tensor memory, apply the mask and the online-softmax
//   update, and write P as packed bf16/fp16 pairs back over the scores
//   MMA 2  O[128 q, H]        += P[128, 64 keys] . V[64 keys, H]   (A from tensor memory, V MN-major)
// The bound is the exponentials (16 a clock and SM: 512 clocks a tile) and the latency of the chain S -> softmax -> P V.
// P takes no shared memory and S / P two buffers of 64 columns, so two CTAs share an SM (256 columns, at most 98 KB each):
// one's chain, prologue and epilogue hide behind the other's.
// 8 x 1024 causal, 32 / 8 heads of 128, takes 125 us so and 250 with one CTA per SM, 128-key tiles, P in shared memory and one
// query head per CTA; 64 x 384 masked, 16 heads of 64, 116 and 286; 2284 packed tokens of 25 sequences, 20 of them single
// tokens, 91 and 206.  2 x 4096 causal reaches 877 TFLOP/s; at 8 x 1024 (9 tiles a CTA) the special-function units are
// 31 % busy: what is left is the latency of a CTA's first loads and last stores.
// Value rows behind the last visible key (of a cache, or of a masked tail) may hold anything and never reach the product.  Rows
// that a key mask hides in front of that key take part with weight 0 and have to be finite.
// (attn_split.cu holds the form whose softmax weights stay 32-bit up to the product with V.)
//
// Replaces, for prompt processing and encoder self-attention, the FlashAttention-2
// (mma.sync) and CUTLASS FMHA kernels the reference dispatches to
// (onnxruntime/contrib_ops/cuda/bert/flash_attention/flash_fwd_kernel.h,
// bert/cutlass_fmha/kernel_forward.h) and its cuDNN SDPA path
// (bert/cudnn_fmha/cudnn_flash_attention.cc:105).
#include <cuda.h>
#include <cuda_runtime.h>
#include <math.h>
#include "attn_internal.h"
#include "ortb200_kernels.h"
#include "ptx_sm100.cuh"
#include "tensor_map.h"

namespace ortb200 {

namespace {

constexpr int kQT = 128;       // query rows per CTA
constexpr int kKT = 64;        // keys per tile
constexpr int kAttnThreads = 192;
constexpr int kTmemCols = 256; // two score buffers (2 x 64 columns) + O (HD columns)
constexpr int kMaskKeys = 8192;  // key masks up to this length are read once and kept as bits
constexpr int kBlockMultiple = 128;

template <int HD>
struct AttnSmem {
  static constexpr int kStages = HD == 64 ? 3 : 2;
  static constexpr int kBoxes = HD / 64;                // boxes of 64 elements per Q / K / V tile
  static constexpr int kQBox = kQT * 128, kBox = kKT * 128;
  static constexpr int kStageBytes = 2 * kBoxes * kBox;
  static constexpr int kOffKV = kBoxes * kQBox;
  static constexpr int kOffBar = kOffKV + kStages * kStageBytes;
  static constexpr int kOffMask = kOffBar + 256;        // uint32 bits[kMaskKeys / 32], then the last visible key per warp
  static constexpr int kTotal = kOffMask + kMaskKeys / 8 + 32 + 1024;
};

// Bit j of the result = key (key0 + j) of batch b may be attended to.  Called by all 32 lanes of a warp.
__device__ __forceinline__ unsigned key_keep_bits(const int* key_mask, int b, int kv_len, int key0, int lane) {
  const int key = key0 + lane;
  const bool keep = key < kv_len && key_mask[static_cast<long long>(b) * kv_len + key] != 0;
  return __ballot_sync(0xffffffffu, keep);
}

enum { BAR_Q = 0, BAR_K_FULL, BAR_K_EMPTY = BAR_K_FULL + 3, BAR_V_FULL = BAR_K_EMPTY + 3, BAR_V_EMPTY = BAR_V_FULL + 3, BAR_S = BAR_V_EMPTY + 3,
       BAR_P = BAR_S + 2, BAR_O = BAR_P + 2, BAR_END, BAR_V_LAST, BAR_COUNT };


template <int HD>
__global__ void __launch_bounds__(kAttnThreads, 2)
attn_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const AttnParams p) {
  using L = AttnSmem<HD>;
  constexpr int STAGES = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + BAR_COUNT);
  uint32_t* mask_bits = reinterpret_cast<uint32_t*>(smem + L::kOffMask);
  int* mask_end = reinterpret_cast<int*>(smem + L::kOffMask + kMaskKeys / 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tq_log2 = 7 - p.group_log2, tq = 1 << tq_log2;   // tokens per CTA
  const bool paged = p.block_table != nullptr;
  pdl_wait_prior_grids();
  // the last tokens have the most keys: their tiles start first
  int q0 = (static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x)) * tq, b = blockIdx.z, q_row0 = 0, S = p.S;
  if (paged) {
    // query tiles of all sequences are numbered from the last sequence's last tile on; the grid is an upper bound of their count
    int tile = blockIdx.x;
    for (b = p.B - 1; b >= 0; --b) {
      q_row0 = p.cu_seqlens[b];
      S = p.cu_seqlens[b + 1] - q_row0;
      const int tiles = (S + tq - 1) >> tq_log2;
      if (tile < tiles) {
        q0 = (tiles - 1 - tile) * tq;
        break;
      }
      tile -= tiles;
    }
    if (b < 0) return;
  }
  const int head0 = blockIdx.y << p.group_log2;
  const int kvh = head0 / (p.N / p.Nk);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    for (int i = 0; i < BAR_COUNT; ++i) mbar_init(&bars[i], i == BAR_P || i == BAR_P + 1 ? 128 : 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  const bool mask_kept = p.key_mask != nullptr && p.kv_len <= kMaskKeys;
  if (mask_kept) {
    int end = 0;
    for (int w = warp; w * 32 < (p.kv_len + 63) / 64 * 64; w += kAttnThreads / 32) {
      const unsigned keep = key_keep_bits(p.key_mask, b, p.kv_len, w * 32, lane);
      if (lane == 0) mask_bits[w] = keep;
      if (keep != 0) end = w * 32 + 32 - __clz(keep);
    }
    if (lane == 0) mask_end[warp] = end;
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_s = *tmem_slot;          // S / P: two buffers of 64 columns
  const uint32_t tmem_o = tmem_s + 2 * kKT;    // O, accumulated over all key tiles

  const int total = paged ? p.past_seqlens[b] + S : (p.seqlens_k ? p.seqlens_k[b] + 1 : p.kv_len);
  const int past = paged ? total - S : (p.first_prompt ? 0 : total - S);
  int visible_end = min(total, p.kv_len);
  if (mask_kept) {   // nothing is visible behind the last unmasked key
    int end = 0;
    for (int w = 0; w < kAttnThreads / 32; ++w) end = max(end, mask_end[w]);
    visible_end = min(visible_end, end);
  }
  // key range needed by this query tile
  const int kv_end = p.causal ? min(visible_end, past + q0 + tq) : visible_end;
  int kv_begin = 0;
  if (p.window > 0) kv_begin = max(0, past + q0 - p.window + 1) / kKT * kKT;
  if (p.chunk > 0) kv_begin = max(kv_begin, (past + q0) / p.chunk * p.chunk / kKT * kKT);
  const int n_tiles = kv_end > kv_begin ? (kv_end - kv_begin + kKT - 1) / kKT : 0;

  if (warp == 0) {
    if (lane == 0 && n_tiles > 0) {
      const int live = visible_end - kv_begin - (n_tiles - 1) * kKT;   // rows of the last value tile that belong to keys, when below 64
      mbar_expect_tx(&bars[BAR_Q], L::kBoxes * L::kQBox);
      for (int bx = 0; bx < L::kBoxes; ++bx)
        for (int h = 0; h < (1 << p.group_log2); ++h)   // rows of a head behind those of the head before it
          tma_load_4d(smem + bx * L::kQBox + h * tq * 128, &tm_q, &bars[BAR_Q], bx * 64, q_row0 + q0, head0 + h, paged ? 0 : b);
      const int cleared = live < kKT ? n_tiles - 1 : -1;   // the tile whose other rows are cleared
      bool ok = true;
      int s = 0;
      uint32_t parity = 1;   // the first round over the stages waits for nothing
      for (int t = 0; t < n_tiles; ++t) {
        const int key0 = kv_begin + t * kKT;
        // cache coordinates behind the head entry: (position, head, batch), or (position in block, head, block)
        int c1 = key0, c3 = b;
        if (paged) {
          const int bi = min(key0 / p.block_size, p.max_blocks - 1);
          c1 = key0 % p.block_size;
          c3 = min(max(p.block_table[static_cast<long long>(b) * p.max_blocks + bi], 0), p.num_blocks - 1);
        }
        uint8_t* st = smem + L::kOffKV + s * L::kStageBytes;
        if (!mbar_wait(&bars[BAR_K_EMPTY + s], parity)) { ok = false; break; }
        mbar_expect_tx(&bars[BAR_K_FULL + s], L::kBoxes * L::kBox);
        for (int bx = 0; bx < L::kBoxes; ++bx) tma_load_4d(st + bx * L::kBox, &tm_k, &bars[BAR_K_FULL + s], bx * 64, c1, kvh, c3);
        if (!mbar_wait(&bars[BAR_V_EMPTY + s], parity)) { ok = false; break; }
        uint64_t* v_bar = &bars[t == cleared ? BAR_V_LAST : BAR_V_FULL + s];
        mbar_expect_tx(v_bar, L::kBoxes * L::kBox);
        for (int bx = 0; bx < L::kBoxes; ++bx) tma_load_4d(st + (L::kBoxes + bx) * L::kBox, &tm_v, v_bar, bx * 64, c1, kvh, c3);
        if (t == cleared) ok = clear_stale_rows<L::kBoxes, L::kBox>(st + L::kBoxes * L::kBox, live, v_bar, &bars[BAR_V_FULL + s]);
        if (++s == STAGES) { s = 0; parity ^= 1u; }
      }
      if (!ok && p.status) atomicExch(p.status, kStatusTimeoutProducer);
    }
  } else if (warp == 1) {
    if (lane == 0 && n_tiles > 0) {
      const uint32_t idesc_s = umma_idesc_f16(p.bf16 != 0, kQT, kKT);
      const uint32_t idesc_o = umma_idesc_f16_bmn(p.bf16 != 0, kQT, HD);
      const uint32_t q_addr = smem_u32(smem);
      auto issue_s = [&](int t, int s) {
        const uint32_t k_addr = smem_u32(smem + L::kOffKV + s * L::kStageBytes);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk)
          umma_f16(tmem_s + (t & 1) * kKT, umma_desc_sw128(q_addr + (kk / 4) * L::kQBox + (kk % 4) * 32),
                   umma_desc_sw128(k_addr + (kk / 4) * L::kBox + (kk % 4) * 32), idesc_s, kk > 0 ? 1u : 0u);
        umma_commit(&bars[BAR_S + (t & 1)]);
        umma_commit(&bars[BAR_K_EMPTY + s]);
      };
      bool ok = mbar_wait(&bars[BAR_Q], 0) && mbar_wait(&bars[BAR_K_FULL], 0);
      if (ok) {
        tcgen05_fence_after();
        issue_s(0, 0);
      }
      int s = 0;
      uint32_t parity = 0;
      for (int t = 0; t < n_tiles && ok; ++t) {
        const int s1 = s + 1 == STAGES ? 0 : s + 1;
        const uint32_t parity1 = s1 == 0 ? parity ^ 1u : parity;
        if (t + 1 < n_tiles) {
          // S of the next tile goes over P of tile t - 1, whose product has to be finished
          if (t > 0 && !mbar_wait(&bars[BAR_O], (t - 1) & 1)) { ok = false; break; }
          if (!mbar_wait(&bars[BAR_K_FULL + s1], parity1)) { ok = false; break; }
          tcgen05_fence_after();
          issue_s(t + 1, s1);
        }
        if (!mbar_wait(&bars[BAR_V_FULL + s], parity) || !mbar_wait(&bars[BAR_P + (t & 1)], (t >> 1) & 1)) { ok = false; break; }
        tcgen05_fence_after();
        const uint32_t v_addr = smem_u32(smem + L::kOffKV + s * L::kStageBytes + L::kBoxes * L::kBox);
        const uint32_t tmem_p = tmem_s + (t & 1) * kKT;
#pragma unroll
        for (int kk = 0; kk < kKT / 16; ++kk)
          umma_f16_ts(tmem_o, tmem_p + kk * 8, umma_desc_mn_sw128(v_addr + kk * 2048, L::kBox, 1024), idesc_o, t > 0 || kk > 0 ? 1u : 0u);
        umma_commit(&bars[BAR_O]);
        umma_commit(&bars[BAR_V_EMPTY + s]);
        if (t == n_tiles - 1) umma_commit(&bars[BAR_END]);
        s = s1;
        parity = parity1;
      }
      if (!ok && p.status) atomicExch(p.status, kStatusTimeoutMma);
    }
  } else {
    // ------------------------------------------------ softmax (one thread per query row); O accumulates in TMEM
    const int qw = warp & 3;
    const int r = qw * 32 + lane;
    const int s_idx = q0 + (r & (tq - 1)), head = head0 + (r >> tq_log2);
    const int pos = past + s_idx;
    const uint32_t lane_addr = static_cast<uint32_t>(qw * 32) << 16;
    // The reference maximum of a row is raised only when a tile exceeds it by 2^8 (probabilities stay below 256),
    // so the accumulator in tensor memory is rescaled a few times per row instead of once per tile.
    constexpr float kRaise = 8.f;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int t = 0; t < n_tiles; ++t) {
      const int key0 = kv_begin + t * kKT;
      unsigned keep0 = 0xffffffffu, keep1 = 0xffffffffu;   // visible keys [key0, key0 + 32) and the 32 behind them
      if (mask_kept) {
        keep0 = mask_bits[key0 >> 5];
        keep1 = mask_bits[(key0 >> 5) + 1];
      } else if (p.key_mask != nullptr) {
        keep0 = key_keep_bits(p.key_mask, b, p.kv_len, key0, lane);
        keep1 = key_keep_bits(p.key_mask, b, p.kv_len, key0 + 32, lane);
      }
      // S of this tile was issued after the product of tile t - 2 had finished: BAR_O is at most one phase back below
      if (ok && !mbar_wait(&bars[BAR_S + (t & 1)], (t >> 1) & 1)) ok = false;
      tcgen05_fence_after();
      // Interior tiles (every key visible to every row of this query tile) skip the per-element mask logic.
      const bool need_mask = (key0 + kKT > total) || (key0 + kKT > p.kv_len) || (keep0 & keep1) != 0xffffffffu || (p.window > 0) ||
                             (p.causal && key0 + kKT - 1 > past + q0) || (p.softcap > 0.f) ||
                             (p.chunk > 0 && key0 < (past + q0 + tq - 1) / p.chunk * p.chunk);
      float sv[kKT];
      const uint32_t s_addr = tmem_s + (t & 1) * kKT + lane_addr;
      tmem_ld_x32(s_addr, sv);
      tmem_ld_x32(s_addr + 32, sv + 32);
      tmem_ld_wait();
      // Scores stay unscaled in registers: the scale is folded into the exponent's multiply-add.  Plain length /
      // causal masking is one compare and select per element against a per-row limit; soft-capping leaves final base-2
      // logits (scale 1).
      float fs = p.scale_log2;
      if (need_mask) {
        if (p.softcap > 0.f) {
          fs = 1.f;
#pragma unroll
          for (int j = 0; j < kKT; ++j) sv[j] = p.softcap * tanhf(sv[j] * p.scale / p.softcap) * 1.4426950408889634f;
        }
        // visible keys of this row within the tile: [lo, hi) and the tile's key-mask bits
        int hi = min(total, p.kv_len);
        if (p.causal) hi = min(hi, pos + 1);
        hi -= key0;
        int lo = p.window > 0 ? pos - p.window + 1 - key0 : -kKT;
        if (p.chunk > 0) lo = max(lo, pos / p.chunk * p.chunk - key0);
        if ((keep0 & keep1) == 0xffffffffu) {
#pragma unroll
          for (int j = 0; j < kKT; ++j) sv[j] = (j < hi && j >= lo) ? sv[j] : -INFINITY;
        } else {
#pragma unroll
          for (int j = 0; j < kKT; ++j) {
            const unsigned keep = j < 32 ? keep0 : keep1;
            sv[j] = (j < hi && j >= lo && ((keep >> (j & 31)) & 1u)) ? sv[j] : -INFINITY;
          }
        }
      }
      float m_raw = -INFINITY;
#pragma unroll
      for (int j = 0; j < kKT; j += 2) m_raw = fmax3(m_raw, sv[j], sv[j + 1]);
      const float m_tile = m_raw * fs;   // fs > 0: -inf stays -inf
      const bool raise = m_tile > m + kRaise;   // also the first finite maximum of a row (m = -inf)
      if (__any_sync(0xffffffffu, raise)) {
        // tensor-memory loads and stores are warp-wide: every lane takes part, rows that keep their maximum scale by 1
        const float corr = raise ? (m == -INFINITY ? 0.f : exp2f(m - m_tile)) : 1.f;
        if (t > 0) {
          if (ok && !mbar_wait(&bars[BAR_O], (t - 1) & 1)) ok = false;
          tcgen05_fence_after();
#pragma unroll 1
          for (int c = 0; c < HD; c += 32) {
            float v[32];
            tmem_ld_x32(tmem_o + lane_addr + c, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] *= corr;
            tmem_st_x32(tmem_o + lane_addr + c, v);
          }
        }
        l *= corr;
        if (raise) m = m_tile;
      }
      // masked scores are -inf and give 0; a row with no visible key so far (m = -inf) uses 0 as its reference
      const float neg_m = m == -INFINITY ? 0.f : -m;
      float row_sum = 0.f, row_sum1 = 0.f;
#pragma unroll
      for (int c = 0; c < kKT; c += 32) {
        uint32_t packed[16];
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float p0 = ex2_approx(fmaf(sv[c + j], fs, neg_m));
          const float p1 = ex2_approx(fmaf(sv[c + j + 1], fs, neg_m));
          row_sum += p0;
          row_sum1 += p1;
          if (p.bf16) {
            __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
            packed[j / 2] = *reinterpret_cast<uint32_t*>(&h);
          } else {
            __half2 h = __floats2half2_rn(p0, p1);
            packed[j / 2] = *reinterpret_cast<uint32_t*>(&h);
          }
        }
        tmem_st_x16_u32(s_addr + c / 2, packed);
      }
      l += row_sum + row_sum1;
      // publish P
      tmem_st_wait();
      tcgen05_fence_before();
      mbar_arrive(&bars[BAR_P + (t & 1)]);
    }
    // (BAR_O may still be two phases back here, where its parity would already read as done)
    if (n_tiles > 0 && ok && !mbar_wait(&bars[BAR_END], 0)) ok = false;
    tcgen05_fence_after();
    if (!ok && p.status) atomicExch(p.status, kStatusTimeoutEpilogue);
    pdl_launch_dependents();
    float denom = l;
    float rescale = 1.f;
    if (p.head_sink) {
      const float sink = (p.bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.head_sink)[head])
                                 : __half2float(static_cast<const __half*>(p.head_sink)[head])) * 1.4426950408889634f;
      const float mm = fmaxf(m, sink);
      rescale = m == -INFINITY ? 0.f : exp2f(m - mm);
      denom = l * rescale + exp2f(sink - mm);
    }
    const float inv = (denom > 0.f && n_tiles > 0) ? rescale / denom : 0.f;
    uint8_t* orow = static_cast<uint8_t*>(p.out) + 2 * ((paged ? 0 : b * p.o_strides[0]) + (q_row0 + s_idx) * p.o_strides[1] + head * p.o_strides[2]);
#pragma unroll 1
    for (int c0 = 0; c0 < HD; c0 += 32) {
      float v[32];
      if (n_tiles > 0) {   // uniform over the CTA
        tmem_ld_x32(tmem_o + lane_addr + c0, v);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
      }
      if (ok && s_idx < S) {
#pragma unroll
        for (int c = 0; c < 32; c += 8) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            if (p.bf16) {
              __nv_bfloat162 h = __floats2bfloat162_rn(v[c + j] * inv, v[c + j + 1] * inv);
              w[j / 2] = *reinterpret_cast<uint32_t*>(&h);
            } else {
              __half2 h = __floats2half2_rn(v[c + j] * inv, v[c + j + 1] * inv);
              w[j / 2] = *reinterpret_cast<uint32_t*>(&h);
            }
          }
          *reinterpret_cast<uint4*>(orow + (c0 + c) * 2) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_s, kTmemCols);
  }
}

template <int HD>
int launch_attn(const ortb200_attn_prefill_args* a, cudaStream_t stream) {
  using L = AttnSmem<HD>;
  const CUtensorMapDataType dt = a->dtype == ORTB200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const bool paged = a->block_table != nullptr;
  CUtensorMap tq, tk, tv;
  // Query heads per CTA: all that share a key head where they fill the 128 rows evenly (TMA places rows in groups of eight)
  const int group = a->N / a->Nk;
  int group_log2 = 0;
  if (group == 2 || group == 4 || group == 8 || group == 16) while ((1 << group_log2) < group) ++group_log2;
  const int tokens = kQT >> group_log2;
  {
    const int64_t dims[4] = {HD, paged ? a->T : a->S, a->N, paged ? 1 : a->B};
    const int64_t strides[3] = {a->q_strides[1] * 2, a->q_strides[2] * 2, paged ? a->T * a->q_strides[1] * 2 : a->q_strides[0] * 2};
    if (make_tensor_map_4d(&tq, a->q, dt, 2, dims, strides, 64, tokens) != 0) return -6;
  }
  {
    const int64_t row = static_cast<int64_t>(a->Nk) * HD * 2;
    const int64_t dims[4] = {HD, paged ? a->block_size : a->kv_len, a->Nk, paged ? a->num_blocks : a->B};
    const int64_t contiguous[3] = {a->kv_strides[2] * 2, a->kv_strides[1] * 2, a->kv_strides[0] * 2};
    const int64_t blocks[3] = {row, HD * 2, row * a->block_size};
    const int64_t* strides = paged ? blocks : contiguous;
    if (make_tensor_map_4d(&tk, a->k, dt, 2, dims, strides, 64, kKT) != 0) return -6;
    if (make_tensor_map_4d(&tv, a->v, dt, 2, dims, strides, 64, kKT) != 0) return -6;
  }
  AttnParams p{};
  p.seqlens_k = a->seqlens_k;
  p.key_mask = paged ? nullptr : a->key_mask;
  p.head_sink = a->head_sink;
  p.out = a->out;
  p.B = a->B; p.S = a->S; p.N = a->N; p.Nk = a->Nk; p.kv_len = paged ? (1 << 30) : a->kv_len;
  for (int i = 0; i < 3; ++i) p.o_strides[i] = a->o_strides[i];
  p.first_prompt = a->first_prompt; p.causal = a->causal; p.window = a->window;
  p.scale = a->scale != 0.f ? a->scale : 1.0f / sqrtf(static_cast<float>(HD));
  p.scale_log2 = p.scale * 1.4426950408889634f;
  p.softcap = a->softcap;
  p.bf16 = a->dtype == ORTB200_BF16 ? 1 : 0;
  p.status = a->status;
  p.block_table = a->block_table; p.cu_seqlens = a->cu_seqlens; p.past_seqlens = a->past_seqlens;
  p.block_size = a->block_size; p.max_blocks = a->max_blocks; p.num_blocks = a->num_blocks;
  p.chunk = a->chunk;
  p.group_log2 = group_log2;
  auto kern = attn_prefill_kernel<HD>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal) != cudaSuccess) return -10;
    attr_set = true;
  }
  // packed form: every sequence has at most one partly filled query tile
  const int tiles = paged ? a->T / tokens + (a->B < a->T ? a->B : a->T) : (a->S + tokens - 1) / tokens;
  dim3 grid(tiles, a->N >> group_log2, paged ? 1 : a->B);
  kern<<<grid, kAttnThreads, L::kTotal, stream>>>(tq, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // namespace

}  // namespace ortb200

using namespace ortb200;

extern "C" int ortb200_attn_prefill(const ortb200_attn_prefill_args* a, ortb200_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!a || !a->q || !a->k || !a->v || !a->out) return -1;
  const bool paged = a->block_table != nullptr;
  if (a->B <= 0 || a->N <= 0 || a->N > 65535 || a->Nk <= 0 || a->N % a->Nk != 0) return -1;
  if (!paged && (a->S <= 0 || a->kv_len <= 0)) return -1;
  if (paged && (!a->cu_seqlens || !a->past_seqlens || a->T <= 0 || a->block_size <= 0 || a->block_size % kBlockMultiple != 0 || a->max_blocks <= 0 ||
                a->num_blocks <= 0))
    return -1;
  if (a->H != 64 && a->H != 128) return -2;
  if (a->dtype != ORTB200_BF16 && a->dtype != ORTB200_F16) return -4;
  for (int i = paged ? 1 : 0; i < 3; ++i)
    if (a->q_strides[i] % 8 || a->o_strides[i] % 8 || (!paged && a->kv_strides[i] % 8)) return -3;
  if ((reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k) | reinterpret_cast<uintptr_t>(a->v) |
       reinterpret_cast<uintptr_t>(a->out)) & 15)
    return -3;
  if (a->chunk > 0 && !a->causal) return -2;
  if (a->split_weights) return paged ? launch_attn_split(a, stream) : -2;
  return a->H == 128 ? launch_attn<128>(a, stream) : launch_attn<64>(a, stream);
}
