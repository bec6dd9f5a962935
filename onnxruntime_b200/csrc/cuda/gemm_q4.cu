// Decode-shaped GEMM over packed 4-bit weights for sm_100a: weights go from the packed blob straight into the operand
// registers of warp-level tensor instructions.
//
//   out[M, N] = act(alpha * X[M, K] * dequant(W)[N, K]^T + bias) + residual
//
// The tcgen05 form (gemm_smallm.cu) expands a 128 x 64 block of weights into tensor memory, and that round trip costs the same
// for one token as for 64: 57344 x 8192 took 107 us, of which the 264 MB need 40.  Here a warp owns 32 weight rows.  A
// thread's share of a 16 x 16 operand tile is pairs of weights of two rows, which a shift, a mask, an exact subtraction and a
// multiplication make out of a packed word: nothing is stored in between.  Which k an operand slot stands for is free as
// long as both operands agree, so thread t of a quad takes k = 16 t .. 16 t + 15 of a 64-wide block: one 8-byte load of
// weights per row and two 16-byte loads of activations per token, all without bank conflicts.  The bound is the instruction
// stream (about 200 per warp and 32 x 64 weights at 8 tokens), not the bandwidth.
//
// The two forms, tcgen05 / this, us for one and for 16 tokens (fp16, event-timed alone, L2 cold, launch included): 57344 x 8192
// 118 / 86 and 123 / 100; 8192 x 28672 58 / 52 and 59 / 57; 10240 x 8192 38 / 27 and 40 / 31.6; 28672 x 4096 39 / 33 and 42 / 39;
// 4096 x 4096 15.5 / 13 and 15.5 / 15.  With 32 tokens the products cost more than the round trip saves (134 / 138 and
// 63 / 80 us), so the tcgen05 form keeps everything above 16.
//
// A cluster of C CTAs shares one 128-row tile over K and adds its partial tiles through distributed shared memory in rank
// order, as in gemm_smallm.cu.
#include <cuda.h>
#include <cuda_runtime.h>
#include "gemm_internal.h"
#include "gemm_small_device.cuh"
#include "ortb200_kernels.h"
#include "ptx_sm100.cuh"
#include "tensor_map.h"

namespace ortb200 {

namespace {

constexpr int kRows = 128;          // weight rows per CTA
constexpr int kBK = 64;
constexpr int kComputeWarps = 4;
constexpr int kThreads = (kComputeWarps + 1) * 32;
constexpr int kBlobBytes = 4864;    // of one k-block: [128][32] nibbles, [128][2] scales, [128][2] zero points
constexpr int kScaleOffset = 4096, kZeroOffset = 4608;
constexpr int kUnit = 2;            // k-blocks per pipeline stage: one barrier wait for 128 x 128 weights

template <int BN>
struct Q4Smem {
  static constexpr int kXBytes = BN * kBK * 2;         // activations of one k-block
  // Registers: 64 and, for 9 to 16 tokens, 72 in bf16.  In fp16 these spill, and four CTAs an SM (94 registers) are mostly faster
  // (57344 x 8192, 16 tokens: 104 -> 100 us, 8192 x 28672 61 -> 57, 8192 x 8192 27 -> 25, but 10240 x 8192 31 -> 31.6).
  static constexpr int ctas_per_sm(bool bf16) { return BN <= 8 ? 6 : bf16 ? 5 : 4; }
  static constexpr int kStages = 3;
  // activations first: their swizzle counts from 1 KiB boundaries
  static constexpr int kOffBlob = kUnit * kXBytes * kStages;
  static constexpr int kOffBar = kOffBlob + kUnit * kBlobBytes * kStages;
  static constexpr int kPartBytes = BN * kRows * 4;    // re-uses the drained stages
  static constexpr int kTotal = kOffBar + 16 * kStages + 1024;
  static_assert(kPartBytes <= kOffBar && kTotal * ctas_per_sm(true) <= 222 * 1024, "shared memory");
  static_assert(kOffBar % 8 == 0 && kOffBlob % 16 == 0, "alignment of barriers and bulk copies");
};

// Zero point and scale of a quantisation block, in both halves of a register.
struct BlockScale {
  uint32_t zero, zero16, scale;
};
template <bool BF16>
__device__ __forceinline__ BlockScale block_scale(uint32_t scale_bits, uint32_t zero_point) {
  BlockScale b;
  b.scale = scale_bits * 0x10001u;
  b.zero16 = 0;
  if (BF16) {
    const __nv_bfloat162 z = __float2bfloat162_rn(128.f + static_cast<float>(zero_point));   // exact up to 128, as in gemm_smallm.cu
    b.zero = *reinterpret_cast<const uint32_t*>(&z);
  } else {
    b.zero = (zero_point | 0x6400u) * 0x10001u;   // 1024 + z, exact
    const __half2 z = __hsub2(__float2half2_rn(960.f), *reinterpret_cast<const __half2*>(&b.zero));   // -(64 + z), exact
    b.zero16 = *reinterpret_cast<const uint32_t*>(&z);
  }
  return b;
}

// Weights 2 i and 2 i + 1 (i = 0 .. 3) of a packed word: (q - z) * s, the difference exact, the product rounded to 16 bits.
// fp16 takes the upper nibble of a byte where it lies, as 1024 + 16 q: one fused multiply-add by 1 / 16 gives q - z exactly,
// and a word needs one shift instead of three (bf16 has no bits for that).
template <bool BF16>
__device__ __forceinline__ uint32_t dequant(uint32_t w, int i, const BlockScale& b) {
  uint32_t q, r;
  if (BF16) {
    asm("lop3.b32 %0, %1, 0x000F000F, %2, 0xEA;" : "=r"(q) : "r"(w >> (4 * i)), "r"(0x43004300u));   // (a & b) | c
    const __nv_bfloat162 v = __hmul2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&q), *reinterpret_cast<const __nv_bfloat162*>(&b.zero)),
                                     *reinterpret_cast<const __nv_bfloat162*>(&b.scale));
    r = *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const uint32_t u = w >> (8 * (i >> 1));
    __half2 d;
    if (i & 1) {
      asm("lop3.b32 %0, %1, 0x00F000F0, %2, 0xEA;" : "=r"(q) : "r"(u), "r"(0x64006400u));
      d = __hfma2(*reinterpret_cast<const __half2*>(&q), __float2half2_rn(0.0625f), *reinterpret_cast<const __half2*>(&b.zero16));
    } else {
      asm("lop3.b32 %0, %1, 0x000F000F, %2, 0xEA;" : "=r"(q) : "r"(u), "r"(0x64006400u));
      d = __hsub2(*reinterpret_cast<const __half2*>(&q), *reinterpret_cast<const __half2*>(&b.zero));
    }
    d = __hmul2(d, *reinterpret_cast<const __half2*>(&b.scale));
    r = *reinterpret_cast<const uint32_t*>(&d);
  }
  return r;
}
template <bool BF16>
__device__ __forceinline__ void mma_16x8x16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int BN, bool BF16>
__global__ void __launch_bounds__(kThreads, Q4Smem<BN>::ctas_per_sm(BF16))
gemm_q4_kernel(const __grid_constant__ CUtensorMap tmap_x, const SmallGemmParams p) {
  using S = Q4Smem<BN>;
  constexpr int STAGES = S::kStages, NT = BN / 8;
  extern __shared__ uint8_t smem_raw[];
  // every CTA of the cluster applies the same rounding, so shared-memory offsets agree across the cluster
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* part = reinterpret_cast<float*>(smem);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::kOffBar);
  uint64_t* empty_bar = full_bar + STAGES;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int C = p.cluster;
  const int rank = C > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = blockIdx.x / C, n0 = tile * kRows, m0 = blockIdx.y * BN;
  const int units = (p.num_kb + kUnit - 1) / kUnit;
  const int u_begin = static_cast<int>(static_cast<long long>(rank) * units / C);
  const int nu = static_cast<int>(static_cast<long long>(rank + 1) * units / C) - u_begin;   // >= 1 (the host keeps C <= units)

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], kComputeWarps);
    }
    fence_mbar_init();
  }
  __syncthreads();
  pdl_launch_dependents();

  if (warp == kComputeWarps) {
    if (lane == 0) {
      const uint8_t* blob = static_cast<const uint8_t*>(p.nbits_blob) + (static_cast<long long>(tile) * p.num_kb + u_begin * kUnit) * kBlobBytes;
      auto blocks = [&](int i) { return min(kUnit, p.num_kb - (u_begin + i) * kUnit); };
      auto load_w = [&](int i, int s) {
        const int nb = blocks(i);
        mbar_expect_tx(&full_bar[s], nb * (kBlobBytes + S::kXBytes));
        bulk_load(smem + S::kOffBlob + s * kUnit * kBlobBytes, blob + static_cast<long long>(i) * kUnit * kBlobBytes, nb * kBlobBytes, &full_bar[s]);
      };
      auto load_x = [&](int i, int s) {
        const int nb = blocks(i);
        for (int k = 0; k < nb; ++k) tma_load_2d(smem + (s * kUnit + k) * S::kXBytes, &tmap_x, &full_bar[s], ((u_begin + i) * kUnit + k) * kBK, m0);
      };
      // weights do not depend on the previous kernel: their stream starts before its end is waited for
      const int pre = nu < STAGES ? nu : STAGES;
      for (int i = 0; i < pre; ++i) load_w(i, i);
      pdl_wait_prior_grids();
      for (int i = 0; i < pre; ++i) load_x(i, i);
      int s = 0, issued = pre;
      uint32_t parity = 0;
      for (; issued < nu; ++issued) {
        if (!mbar_wait(&empty_bar[s], parity)) {
          if (p.status) atomicExch(p.status, kStatusTimeoutProducer);
          break;
        }
        load_w(issued, s);
        load_x(issued, s);
        if (++s == STAGES) { s = 0; parity ^= 1u; }
      }
      // whoever gave up, no copy is in flight when this CTA leaves
      for (int i = max(issued - STAGES, 0); i < issued; ++i) mbar_wait(&full_bar[i % STAGES], (i / STAGES) & 1);
    }
    __syncwarp();
  } else {
    pdl_wait_prior_grids();   // no bounded wait may span the previous grid's run time
    const int g = lane >> 2, t = lane & 3;
    const int row0 = warp * 32 + g;    // rows row0, + 8, + 16, + 24 of the tile
    float acc[2][NT][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[mt][nt][e] = 0.f;
    bool ok = true;
    int s = 0;
    uint32_t parity = 0;
    for (int i = 0; i < nu; ++i) {
      if (ok && !mbar_wait(&full_bar[s], parity)) ok = false;
      __syncwarp();   // the products are warp-wide, also where only some lanes gave up
      const int nb = min(kUnit, p.num_kb - (u_begin + i) * kUnit);
#pragma unroll
      for (int k = 0; k < kUnit; ++k) {
        if (k >= nb) break;
        const uint8_t* blob = smem + S::kOffBlob + (s * kUnit + k) * kBlobBytes;
        const uint8_t* xs = smem + (s * kUnit + k) * S::kXBytes + g * 128;   // row g of every group of eight tokens
        uint2 w[4];
        BlockScale bs[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int row = row0 + 8 * r;
          w[r] = *reinterpret_cast<const uint2*>(blob + row * 32 + t * 8);
          bs[r] = block_scale<BF16>(*reinterpret_cast<const uint16_t*>(blob + kScaleOffset + row * 4 + (t >> 1) * 2), blob[kZeroOffset + row * 2 + (t >> 1)]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {     // two steps of 16 k per packed word
          uint4 x[NT];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) x[nt] = *reinterpret_cast<const uint4*>(xs + nt * 1024 + (((2 * t + h) ^ g) << 4));
#pragma unroll
          for (int st = 0; st < 2; ++st) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
              uint32_t a[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int r = 2 * mt + (e & 1);   // operand registers: rows g, g + 8, then the same rows eight k slots on
                a[e] = dequant<BF16>(h ? w[r].y : w[r].x, 2 * st + (e >> 1), bs[r]);
              }
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) mma_16x8x16<BF16>(acc[mt][nt], a, st ? x[nt].z : x[nt].x, st ? x[nt].w : x[nt].y);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[s]);
      if (++s == STAGES) { s = 0; parity ^= 1u; }
    }
    if (!ok && p.status) atomicExch(p.status, kStatusTimeoutEpilogue);
    // every warp has read its last stage: the partial tile may go over them
    asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) part[(nt * 8 + 2 * t + (e & 1)) * kRows + row0 + 16 * mt + 8 * (e >> 1)] = acc[mt][nt][e];
  }

  if (C > 1) cluster_sync_all();
  else __syncthreads();

  if (warp < kComputeWarps) {
    // token columns that this CTA finishes: warp w takes columns w, w + 4, ..., lane l weight rows 4 l .. 4 l + 3
    const int cols_per = BN / C, j_begin = rank * cols_per;
    const uint32_t part_addr = smem_u32(part);
    const int n = n0 + 4 * lane;
    float bias_v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (p.bias != nullptr && n + e < p.N) bias_v[e] = load16(p.bias, n + e, p.dtype);
    const bool vec = (((reinterpret_cast<uintptr_t>(p.out) | reinterpret_cast<uintptr_t>(p.residual)) & 7) == 0) &&
                     ((p.ldo | (p.residual ? p.ldr : 0)) & 3) == 0 && n + 4 <= p.N;
#pragma unroll 1
    for (int j = j_begin + warp; j < j_begin + cols_per; j += kComputeWarps) {
      const int m = m0 + j;
      if (m >= p.M) break;
      const uint32_t off = static_cast<uint32_t>((j * kRows + 4 * lane) * 4);
      float y[4];
      switch (C) {
        case 1: sum_partials<1>(part_addr + off, y); break;
        case 2: sum_partials<2>(part_addr + off, y); break;
        case 4: sum_partials<4>(part_addr + off, y); break;
        default: sum_partials<8>(part_addr + off, y); break;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = act_apply(p.act, y[e] * p.alpha + bias_v[e]);
      const long long o = m * p.ldo + n, ro = m * p.ldr + n;
      if (vec) {
        if (p.residual) {
          const uint2 rr = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p.residual) + ro);
          const float2 a = unpack16(rr.x, p.dtype), b = unpack16(rr.y, p.dtype);
          y[0] += a.x; y[1] += a.y; y[2] += b.x; y[3] += b.y;
        }
        *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p.out) + o) = make_uint2(pack16(y[0], y[1], p.dtype), pack16(y[2], y[3], p.dtype));
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (n + e >= p.N) break;
          if (p.residual) y[e] += load16(p.residual, ro + e, p.dtype);
          static_cast<uint16_t*>(p.out)[o + e] = static_cast<uint16_t>(pack16(y[e], 0.f, p.dtype));
        }
      }
    }
  }
  // nobody leaves while a peer may still read its partial tile
  if (C > 1) cluster_sync_all();
}

template <int BN, bool BF16>
int launch_q4(const CUtensorMap& tx, const SmallGemmParams& p, dim3 grid, bool use_pdl, cudaStream_t stream) {
  using S = Q4Smem<BN>;
  auto kern = gemm_q4_kernel<BN, BF16>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal) != cudaSuccess) return -10;
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = S::kTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int nattr = 0;
  if (p.cluster > 1) {
    attrs[nattr].id = cudaLaunchAttributeClusterDimension;
    attrs[nattr].val.clusterDim.x = p.cluster;
    attrs[nattr].val.clusterDim.y = 1;
    attrs[nattr].val.clusterDim.z = 1;
    ++nattr;
  }
  if (use_pdl) {
    attrs[nattr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[nattr].val.programmaticStreamSerializationAllowed = 1;
    ++nattr;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = nattr;
  return cudaLaunchKernelEx(&cfg, kern, tx, p) == cudaSuccess ? 0 : -11;
}

// Split of K over a cluster.  The SMs should be loaded evenly, and a CTA's start and end (about what two units take: first
// loads, cluster barriers, the reduction) should be a small part of it.  57344 x 8192, one token, C = 1 / 2 / 4 / 8: 102, 90, 85
// and 88 us; 8192 x 28672: 139, 76, 57 and 51 (launch included).
int split_q4(int tiles, int num_kb, int bn, int sms) {
  const int units = (num_kb + kUnit - 1) / kUnit;
  int best = 1;
  double best_cost = 0.0;
  for (int c = 1; c <= 8 && bn % c == 0 && (c == 1 || units / c >= 4); c *= 2) {
    const long long ctas = static_cast<long long>(tiles) * c, per_sm = (ctas + sms - 1) / sms;
    // an SM with few CTAs cannot keep its pipes busy: count at least four
    const double cost = static_cast<double>(per_sm < 4 ? 4 : per_sm) * (static_cast<double>(units) / c + 2.0);
    if (c == 1 || cost <= best_cost) {
      best_cost = cost;
      best = c;
    }
  }
  return best;
}

}  // namespace

int launch_gemm_q4(const ortb200_gemm_args* a, cudaStream_t stream, int* cluster_out, int* stages_out) {
  const int bn = a->M <= 8 ? 8 : 16;
  CUtensorMap tx;
  const CUtensorMapDataType dt = a->dtype == ORTB200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  if (make_tensor_map_2d(&tx, a->x, dt, 2, a->K, a->M, static_cast<int64_t>(a->K) * 2, kBK, bn) != 0) return -6;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles_n = (a->N + kRows - 1) / kRows, tiles_m = (a->M + bn - 1) / bn;
  SmallGemmParams p{};
  p.M = a->M; p.N = a->N; p.K = a->K; p.num_kb = a->K / kBK;
  p.cluster = a->force_splits > 0 ? pick_cluster(tiles_n * tiles_m, (p.num_kb + kUnit - 1) / kUnit, bn, a->force_splits)
                                  : split_q4(tiles_n * tiles_m, p.num_kb, bn, sms);
  p.dtype = a->dtype; p.act = a->act; p.alpha = a->alpha;
  p.out = a->out; p.ldo = a->ldo; p.bias = a->bias; p.residual = a->residual; p.ldr = a->ldr; p.status = a->status;
  p.nbits_blob = a->w;
  const dim3 grid(tiles_n * p.cluster, tiles_m, 1);
  const bool bf16 = a->dtype == ORTB200_BF16, pdl = a->use_pdl != 0;
  *cluster_out = p.cluster;
  *stages_out = Q4Smem<8>::kStages;
  if (bn == 8) return bf16 ? launch_q4<8, true>(tx, p, grid, pdl, stream) : launch_q4<8, false>(tx, p, grid, pdl, stream);
  return bf16 ? launch_q4<16, true>(tx, p, grid, pdl, stream) : launch_q4<16, false>(tx, p, grid, pdl, stream);
}

}  // namespace ortb200
