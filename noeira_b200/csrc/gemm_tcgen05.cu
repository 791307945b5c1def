// bf16 GEMM on the 5th generation tensor cores: D = epilogue(A · B), fp32 accumulation in TMEM.
//
//   * operands are fetched by TMA (128-byte swizzle, no multicast) into a multi-stage shared
//     memory ring; one elected thread issues tcgen05.mma (M=128, N=BN, K=16) four times per
//     64-wide k-block; tcgen05.commit releases the stage / publishes the accumulator;
//   * persistent CTAs (one per SM) walk the tile list; two TMEM accumulators let the epilogue
//     of tile i overlap the main loop of tile i+1;
//   * warp roles (352 threads): warp 0 = TMA producer of A, warp 1 = MMA issuer + TMEM owner, warp 2 = TMA producer of B,
//     warps 3..10 = epilogue (TMEM quarter = warp_id % 4, two warps per quarter);
//   * both operands may be K-major ([rows, K] row-major) or MN-major ([K, rows] row-major), so
//     forward (x·W, W stored [IN, OUT]), dgrad (dy·Wᵀ) and wgrad (xᵀ·dy) all run from the
//     natural layouts without a transpose pass;
//   * epilogue: +bias[n], activation, or multiplication by the activation derivative taken from
//     a saved tensor (dgrad of tanh / relu / gelu / silu), optional accumulate into fp32 output
//     (dW += …), bf16 or fp32 store;
//   * every mbarrier wait is bounded; on a timeout the CTA records it in `status`, all roles
//     drain, TMEM is released and the kernel returns.
//
// Counterpart in the reference: library GEMMs only (cuBLAS / cuBLASLt epilogues / MAX matmul;
// noeira/nn/primitives/linear.mojo:1295-1387, noeira/nn/core/cublaslt_gemm.mojo:66-73).
#include <cuda.h>

#include "common.cuh"
#include "gemm_api.h"

namespace {

using namespace nb;

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
// Eight epilogue warps: two share a 32-row quarter of the accumulator and take its column groups in turn.  With four the
// epilogue of a 256 x 256 tile (bias, GELU, residual, bf16 store) took longer than the twelve k-blocks of K = 768, and the
// tensor core waited for a free accumulator: 24576 x 3072 x 768 with GELU took 240 us, 176 us with eight.
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 96 + 32 * EPI_WARPS;     // A loads, MMA, B loads, epilogue
constexpr int NUM_THREADS2 = 64 + 32 * EPI_WARPS;    // CTA pairs: loads, MMA, epilogue

struct GemmParams {
  int M, N, K;
  int a_mn, b_mn;  // operand majors
  int tf32;        // 1: operands are fp32 read as TF32 (kind::tf32, 8 k per instruction, 32 elements per 128-byte row)
  int ldd;         // output row pitch (elements)
  int ld_aux;      // aux row pitch (elements, bf16)
  int out_f32, accumulate, act, dact;
  int tiles_m, tiles_n, num_kb;
  int splits, kb_per_split;  // split-K: work item = (tile, split); partial tiles meet in `ws`
  int tile_rows;             // rows of a tile: BM, 2 BM for CTA pairs
  float alpha;
  float* ws;                 // splits>1: fp32 partial tiles, [tile][split][BM*BN]
  unsigned int* tile_ctr;    // splits>1: one arrival counter per tile (zero between launches)
  void* D;
  const float* bias;
  const __nv_bfloat16* aux;
  unsigned int* status;
  // implicit-GEMM convolution (conv != 0): A is never materialised; the producer reads activation patches of the NHWC
  // input through a 4-D tensor map (c, w, h, b), one box of conv_bw output pixels x 64 channels per TMA
  // conv == 2: weight gradient.  A = patches^T is MN-major: the SAME shared-memory image as the forward's A tile (rows =
  // pixels, 128 bytes of channels), now read with the pixels as the reduction dimension; B = dy, MN-major
  int conv, conv_c, conv_ow, conv_oh, conv_kw, conv_pad, conv_bw, conv_taps, conv_b;
};

__device__ __forceinline__ void tma_load_4d_g(void* smem_dst, const void* tmap, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}

// MUFU tanh: one instruction, max relative error 2^-11 — below bf16 resolution of the stored result.
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The activation code is selected ONCE per 16-column chunk and the taken case is a short straight run: the
// epilogue executes few instructions per tile, so its speed is set by instruction fetch, i.e. by code size.
__device__ __forceinline__ void act_apply16(int act, float (&v)[16]) {
  switch (act) {
    case NB_ACT_RELU:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j], 0.f);
      break;
    case NB_ACT_TANH:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = tanh_fast(v[j]);
      break;
    case NB_ACT_GELU:
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        // 0.5 x (1 + tanh(c (x + 0.044715 x^3))) in five multiply-adds around the tanh
        const float x = v[j], h = 0.5f * x;
        v[j] = fmaf(h, tanh_fast(x * fmaf(0.7978845608028654f * 0.044715f, x * x, 0.7978845608028654f)), h);
      }
      break;
    case NB_ACT_SILU:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = v[j] / (1.f + __expf(-v[j]));
      break;
    case NB_ACT_SIGMOID:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = 1.f / (1.f + __expf(-v[j]));
      break;
    default: break;
  }
}
// derivative factor from the SAVED tensor: tanh/relu/sigmoid save the output y, gelu/silu save the input x
__device__ __forceinline__ float dact_apply(int dact, float s) {
  switch (dact) {
    case NB_ACT_RELU: return s > 0.f ? 1.f : 0.f;
    case NB_ACT_TANH: return 1.f - s * s;
    case NB_ACT_SIGMOID: return s * (1.f - s);
    case NB_ACT_GELU: {
      const float c = 0.7978845608028654f;
      const float u = c * (s + 0.044715f * s * s * s);
      const float t = tanh_fast(u);
      return 0.5f * (1.f + t) + 0.5f * s * (1.f - t * t) * c * (1.f + 3.f * 0.044715f * s * s);
    }
    case NB_ACT_SILU: {
      const float sg = 1.f / (1.f + __expf(-s));
      return sg * (1.f + s * (1.f - sg));
    }
    default: return 1.f;
  }
}
__device__ __forceinline__ void dact_apply16(int dact, float (&v)[16], const float (&sv)[16]) {
  switch (dact) {
    case NB_ACT_RELU:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = sv[j] > 0.f ? v[j] : 0.f;
      break;
    case NB_ACT_TANH:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] *= 1.f - sv[j] * sv[j];
      break;
    case NB_ACT_SIGMOID:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] *= sv[j] * (1.f - sv[j]);
      break;
    case NB_ACT_GELU:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] *= dact_apply(NB_ACT_GELU, sv[j]);
      break;
    case NB_ACT_SILU:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] *= dact_apply(NB_ACT_SILU, sv[j]);
      break;
    case NB_AUX_ADD:
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] += sv[j];
      break;
    default: break;
  }
}

// Epilogue for 16 consecutive columns of one output row, in two phases so that the global loads it needs (the saved
// activation for a fused derivative, the old output when accumulating) can be issued one chunk ahead of their use:
// a chunk costs a DRAM / L2 round trip otherwise, which made narrow-K GEMMs epilogue-bound.
struct EpiPrefetch {
  uint4 aux[2];   // 16 bf16 of the saved tensor
  float4 old[4];  // 16 fp32 of the previous output (accumulate)
};

__device__ __forceinline__ void epilogue_prefetch16(const GemmParams& p, int row, int col0, bool active, EpiPrefetch& pf) {
  if (!active || col0 + 16 > p.N) return;
  if (p.dact && (p.ld_aux % 8 == 0)) {
    const __nv_bfloat16* ax = p.aux + (size_t)row * p.ld_aux + col0;
    pf.aux[0] = __ldg(reinterpret_cast<const uint4*>(ax));
    pf.aux[1] = __ldg(reinterpret_cast<const uint4*>(ax + 8));
  }
  if (p.out_f32 && p.accumulate && (p.ldd % 4 == 0)) {
    const float* o = reinterpret_cast<const float*>(p.D) + (size_t)row * p.ldd + col0;
#pragma unroll
    for (int j = 0; j < 4; ++j) pf.old[j] = *reinterpret_cast<const float4*>(o + 4 * j);
  }
}

// What a tile's epilogue does is part of the kernel: the frequent forms have instances of their own.  With the tests for
// bias, activation and saved tensor inside the loop over 16-column chunks every chunk jumped across the whole switch, and a
// chunk without any of them took 530 clocks, most of them instruction fetch; it takes 165 now.  (All forms side by side in
// one kernel spilled 4 KB of registers.)  The bias is a run-time test everywhere: one jump over 16 shuffles.
enum EpiMode { EPI_PLAIN, EPI_RELU, EPI_GELU, EPI_ADD, EPI_BF16, EPI_F32, EPI_F32_ANY, EPI_MODES };   // EPI_BF16, EPI_F32_ANY: the rest
__host__ inline EpiMode epi_mode(const GemmParams& p, bool split) {
  if (split) return EPI_F32;                                                   // raw partial tiles
  if (p.out_f32) return (!p.bias && !p.act && !p.dact) ? EPI_F32 : EPI_F32_ANY;
  if (!p.dact) return !p.act ? EPI_PLAIN : (p.act == NB_ACT_RELU ? EPI_RELU : (p.act == NB_ACT_GELU ? EPI_GELU : EPI_BF16));
  return (!p.act && p.dact == NB_AUX_ADD) ? EPI_ADD : EPI_BF16;
}

// alpha, bias and activation of 16 consecutive columns; `sv`: the 16 values of the saved / residual tensor when dact is set.
// The bias comes from the lanes that hold it (see load_bias): lane b0 + j has columns 4j .. 4j + 3 of the chunk.
template <int MODE>
__device__ __forceinline__ void epilogue_math16(const GemmParams& p, const float4& bias, int b0, float (&v)[16], const float (&sv)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] *= p.alpha;
  if (p.bias) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[4 * j] += __shfl_sync(0xffffffffu, bias.x, b0 + j);
      v[4 * j + 1] += __shfl_sync(0xffffffffu, bias.y, b0 + j);
      v[4 * j + 2] += __shfl_sync(0xffffffffu, bias.z, b0 + j);
      v[4 * j + 3] += __shfl_sync(0xffffffffu, bias.w, b0 + j);
    }
  }
  if (MODE == EPI_RELU) act_apply16(NB_ACT_RELU, v);
  if (MODE == EPI_GELU) act_apply16(NB_ACT_GELU, v);
  if (MODE == EPI_ADD) dact_apply16(NB_AUX_ADD, v, sv);
  if (MODE == EPI_BF16 || MODE == EPI_F32_ANY) {
    if (p.act) act_apply16(p.act, v);
    if (p.dact) dact_apply16(p.dact, v, sv);
  }
}
// The bias of a warp's column groups (`half`, `half` + 2, ... of G columns each; at most 128 columns), four per lane, fetched
// while the accumulator is still being computed.  Loaded inside the chunk loop it cost an L2 round trip per 16 columns (most
// of the L1 is shared memory here): 24576 x 2304 x 768 took 101 us with it and 77 us without a bias.
template <int BN, int G>
__device__ __forceinline__ float4 load_bias(const GemmParams& p, int n0, int half, int lane) {
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  const int idx = 4 * lane, c = half * G + idx / G * 2 * G + idx % G, col = n0 + c;
  if (p.bias && c < BN) {
    if (col < p.N) b.x = p.bias[col];
    if (col + 1 < p.N) b.y = p.bias[col + 1];
    if (col + 2 < p.N) b.z = p.bias[col + 2];
    if (col + 3 < p.N) b.w = p.bias[col + 3];
  }
  return b;
}
__device__ __forceinline__ void unpack16(const uint4 (&w)[2], float (&f)[16]) {
  const __nv_bfloat162* h0 = reinterpret_cast<const __nv_bfloat162*>(&w[0]);
  const __nv_bfloat162* h1 = reinterpret_cast<const __nv_bfloat162*>(&w[1]);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f[2 * j] = __low2float(h0[j]);
    f[2 * j + 1] = __high2float(h0[j]);
    f[8 + 2 * j] = __low2float(h1[j]);
    f[8 + 2 * j + 1] = __high2float(h1[j]);
  }
}
__device__ __forceinline__ uint4 pack8f(const float* v) {
  uint4 pk;
  __nv_bfloat162 h0 = __floats2bfloat162_rn(v[0], v[1]), h1 = __floats2bfloat162_rn(v[2], v[3]),
                 h2 = __floats2bfloat162_rn(v[4], v[5]), h3 = __floats2bfloat162_rn(v[6], v[7]);
  pk.x = *reinterpret_cast<uint32_t*>(&h0);
  pk.y = *reinterpret_cast<uint32_t*>(&h1);
  pk.z = *reinterpret_cast<uint32_t*>(&h2);
  pk.w = *reinterpret_cast<uint32_t*>(&h3);
  return pk;
}

// direct store of 16 columns by the thread that owns them (second phase of a split-K GEMM)
__device__ __forceinline__ void epilogue_store16(const GemmParams& p, int row, int col0, float (&v)[16],
                                                 const EpiPrefetch& pf) {
  const bool full = (col0 + 16 <= p.N);
  float sv[16];
  if (p.dact) {
    if (full && (p.ld_aux % 8 == 0)) {
      unpack16(pf.aux, sv);
    } else {
      const __nv_bfloat16* ax = p.aux + (size_t)row * p.ld_aux + col0;
#pragma unroll
      for (int j = 0; j < 16; ++j) sv[j] = (col0 + j < p.N) ? __bfloat162float(ax[j]) : 0.f;
    }
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] *= p.alpha;
  if (p.bias) {
    if (full) {
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 bv = __ldg(reinterpret_cast<const float4*>(p.bias + col0 + j));
        v[j] += bv.x; v[j + 1] += bv.y; v[j + 2] += bv.z; v[j + 3] += bv.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (col0 + j < p.N) v[j] += p.bias[col0 + j];
    }
  }
  if (p.act) act_apply16(p.act, v);
  if (p.dact) dact_apply16(p.dact, v, sv);
  if (p.out_f32) {
    float* o = reinterpret_cast<float*>(p.D) + (size_t)row * p.ldd + col0;
    if (full && (p.ldd % 4 == 0)) {
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        float4 x = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        if (p.accumulate) {
          const float4 y = pf.old[j >> 2];
          x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
        }
        *reinterpret_cast<float4*>(o + j) = x;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (col0 + j < p.N) o[j] = p.accumulate ? o[j] + v[j] : v[j];
    }
  } else {
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.D) + (size_t)row * p.ldd + col0;
    if (full && (p.ldd % 8 == 0)) {
#pragma unroll
      for (int j = 0; j < 16; j += 8) *reinterpret_cast<uint4*>(o + j) = pack8f(v + j);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (col0 + j < p.N) o[j] = __float2bfloat16(v[j]);
    }
  }
}

// Epilogue of one warp: rows [row0, row0 + 32) of the tile (lane = row), column groups `half`, `half` + 2, ... of the tile's
// BN columns that start at column n0 of the output.
//
// Tensor memory hands every lane a whole row, and a store straight from there touches 32 rows with 16 bytes each: 32 L2
// requests per instruction, which made GEMMs with K <= 1024 epilogue-bound (24576 x 2304 x 768 with bias: 142 us with direct
// stores from four warps, 105 us from eight, 101 us staged, 82 us with the bias fetched ahead, see load_bias,
// and 71 with a kernel per epilogue form, see EpiMode).  So a group goes through 4 KB of shared memory per warp: the lane that
// owns the row does the arithmetic and writes its packed row (16-byte chunks XOR-swizzled, no bank conflicts), then the warp
// copies the group out with whole 64- or 128-byte row segments per request.  The saved / residual tensor comes in the same
// way in front of the arithmetic, the old fp32 output is added during the copy.
constexpr int EPI_STAGE_BYTES = 4096;   // per warp

// byte offset of 16-byte chunk `ch` of row `r`; CPR = chunks per row (8: 128-byte rows, 4: 64-byte rows)
template <int CPR>
__device__ __forceinline__ int epi_off(int r, int ch) {
  return CPR == 8 ? r * 128 + ((ch ^ (r & 7)) << 4) : r * 64 + ((ch ^ ((r >> 1) & 3)) << 4);
}

template <int BN>
__host__ __device__ constexpr int epi_group() { return BN >= 128 ? 64 : 32; }   // columns per group, bf16 output
template <int BN, int MODE>
__device__ __forceinline__ void epilogue_groups_bf16(const GemmParams& p, const float4& bias, uint32_t taddr, uint8_t* st, int row0,
                                                   int n0, int half, int lane) {
  constexpr int G = epi_group<BN>(), CPR = G / 8, NV = CPR;   // columns per group; 16-byte vectors per lane and group
  constexpr int NC = (BN < G ? BN : G) / 16;                      // 16-column chunks per group
  constexpr int RS = 32 / CPR;                                    // rows per copy instruction
  const int rr0 = lane / CPR, ch = lane % CPR;                    // copies: this lane's first row and its chunk of every row
  const bool vec_d = p.ldd % 8 == 0, vec_a = p.ld_aux % 8 == 0;
  uint4 ax[NV];
  auto load_aux = [&](int c) {
    const int col = n0 + c + ch * 8;
    const __nv_bfloat16* a = p.aux + (size_t)(row0 + rr0) * p.ld_aux + col;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      ax[i] = make_uint4(0, 0, 0, 0);
      if (row0 + rr0 + i * RS < p.M && col < p.N) {
        if (vec_a && col + 8 <= p.N) {
          ax[i] = __ldg(reinterpret_cast<const uint4*>(a));
        } else {
          auto at = [&](int j) { return col + j < p.N ? (uint32_t)__bfloat16_as_ushort(a[j]) : 0u; };
          ax[i] = make_uint4(at(0) | at(1) << 16, at(2) | at(3) << 16, at(4) | at(5) << 16, at(6) | at(7) << 16);
        }
      }
      a += (size_t)RS * p.ld_aux;
    }
  };
  const bool with_aux = MODE == EPI_ADD || (MODE == EPI_BF16 && p.dact != 0);
  if (with_aux && half * G < BN && n0 + half * G < p.N) load_aux(half * G);
#pragma unroll 1
  for (int c = half * G; c < BN && n0 + c < p.N; c += 2 * G) {
    if (with_aux) {
#pragma unroll
      for (int i = 0; i < NV; ++i) *reinterpret_cast<uint4*>(st + epi_off<CPR>(rr0 + i * RS, ch)) = ax[i];
      __syncwarp();
      if (c + 2 * G < BN && n0 + c + 2 * G < p.N) load_aux(c + 2 * G);
    }
    auto chunk = [&](int k, const uint32_t* r) {
      float v[16], sv[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
      uint8_t* s0 = st + epi_off<CPR>(lane, 2 * k);
      uint8_t* s1 = st + epi_off<CPR>(lane, 2 * k + 1);
      if (with_aux) {
        const uint4 w[2] = {*reinterpret_cast<const uint4*>(s0), *reinterpret_cast<const uint4*>(s1)};
        unpack16(w, sv);
      }
      epilogue_math16<MODE>(p, bias, ((c / (2 * G)) * G + 16 * k) >> 2, v, sv);
      *reinterpret_cast<uint4*>(s0) = pack8f(v);
      *reinterpret_cast<uint4*>(s1) = pack8f(v + 8);
    };
    if (NC == 1) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(taddr + (uint32_t)c, r);
      tmem_ld_wait();
      chunk(0, r);
    } else {
#pragma unroll 1
      for (int k = 0; k < NC; k += 2) {       // two chunks per tensor-memory load
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + (uint32_t)(c + 16 * k), r);
        tmem_ld_wait();
        chunk(k, r);
        chunk(k + 1, r + 16);
      }
    }
    __syncwarp();
    const int col = n0 + c + ch * 8;
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.D) + (size_t)(row0 + rr0) * p.ldd + col;
    const int rows = (col < p.N && ch * 8 < BN) ? p.M - row0 : 0;
    if (vec_d && col + 8 <= p.N) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (rr0 + i * RS < rows) *reinterpret_cast<uint4*>(o) = *reinterpret_cast<const uint4*>(st + epi_off<CPR>(rr0 + i * RS, ch));
        o += (size_t)RS * p.ldd;
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < NV; ++i) {
        const uint4 w = *reinterpret_cast<const uint4*>(st + epi_off<CPR>(rr0 + i * RS, ch));
        const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&w);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (rr0 + i * RS < rows && col + j < p.N) o[j] = e[j];
        o += (size_t)RS * p.ldd;
      }
    }
    __syncwarp();
  }
}

// fp32 output, or (split) the raw fp32 partial tile of a split-K item at `part` (row pitch BN)
template <int BN, int MODE>
__device__ __forceinline__ void epilogue_groups_f32(const GemmParams& p, const float4& bias, uint32_t taddr, uint8_t* st, int row0,
                                                  int n0, int half, int lane, float* part) {
  constexpr int G = 32;
  constexpr int NC = (BN < G ? BN : G) / 16;
  const bool vec_d = p.ldd % 4 == 0;
#pragma unroll 1
  for (int c = half * G; c < BN && n0 + c < p.N; c += 2 * G) {
    auto chunk = [&](int k, const uint32_t* r) {
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
      const int col0 = n0 + c + 16 * k;
      if (MODE == EPI_F32_ANY) {
        float sv[16];
        if (p.dact) {
          const __nv_bfloat16* ax = p.aux + (size_t)(row0 + lane) * p.ld_aux + col0;
#pragma unroll
          for (int j = 0; j < 16; ++j) sv[j] = (row0 + lane < p.M && col0 + j < p.N) ? __bfloat162float(ax[j]) : 0.f;
        }
        epilogue_math16<MODE>(p, bias, ((c / (2 * G)) * G + 16 * k) >> 2, v, sv);
      } else if (!part) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] *= p.alpha;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4*>(st + epi_off<8>(lane, 4 * k + j)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    };
    if (NC == 1) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(taddr + (uint32_t)c, r);
      tmem_ld_wait();
      chunk(0, r);
    } else {
      uint32_t r[32];
      tmem_ld_32x32b_x32(taddr + (uint32_t)c, r);
      tmem_ld_wait();
      chunk(0, r);
      chunk(1, r + 16);
    }
    __syncwarp();
    const int rr0 = lane >> 3, ch = lane & 7, col = n0 + c + ch * 4;
    if (part) {
      float* o = part + (size_t)rr0 * BN + c + ch * 4;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (ch * 4 < BN) *reinterpret_cast<float4*>(o + (size_t)i * 4 * BN) = *reinterpret_cast<const float4*>(st + epi_off<8>(rr0 + 4 * i, ch));
    } else {
      float* o = reinterpret_cast<float*>(p.D) + (size_t)(row0 + rr0) * p.ldd + col;
      const int rows = (col < p.N && ch * 4 < BN) ? p.M - row0 : 0;
      if (vec_d && col + 4 <= p.N) {
#pragma unroll 1
        for (int h = 0; h < 8; h += 4) {      // four rows of this lane at a time: their old values are in flight together
          float4 old[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (p.accumulate && rr0 + 4 * (h + i) < rows) old[i] = *reinterpret_cast<const float4*>(o + (size_t)i * 4 * p.ldd);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float4 w = *reinterpret_cast<const float4*>(st + epi_off<8>(rr0 + 4 * (h + i), ch));
            if (p.accumulate) { w.x += old[i].x; w.y += old[i].y; w.z += old[i].z; w.w += old[i].w; }
            if (rr0 + 4 * (h + i) < rows) *reinterpret_cast<float4*>(o + (size_t)i * 4 * p.ldd) = w;
          }
          o += (size_t)16 * p.ldd;
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
          const float4 w = *reinterpret_cast<const float4*>(st + epi_off<8>(rr0 + 4 * i, ch));
          const float e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (rr0 + 4 * i < rows && col + j < p.N) o[j] = p.accumulate ? o[j] + e[j] : e[j];
          o += (size_t)4 * p.ldd;
        }
      }
    }
    __syncwarp();
  }
}

// Bounded wait of a pipeline role.  The common case is one test of the barrier; the abort flag of the CTA is looked at only
// while the barrier is not there yet.
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status,
                                              unsigned int where) {
  if (mbar_try_wait(bar, parity)) return true;
  for (uint32_t it = 0; it < NB_SPIN_LIMIT; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 0u && *abort_flag) return false;
  }
  report(status, NB_ST_MBAR_TIMEOUT, where, parity);
  return false;
}

// The four instructions of one k-block.  `ad` / `bd` are complete descriptors of the stage's operands, `astep` / `bstep` the
// advance per instruction in descriptor units (16 bytes).  Nothing but additions stands between two instructions: with the
// descriptors built from the operand majors in front of each one, the issuing thread needed 880 clocks per k-block, three to
// six times what the tensor core needs for it (M = 128: 512 clocks at 256 columns, 128 at 64), and every one-CTA tile ran at
// 416 ns per k-block whatever its width; 190 to 280 ns now.
template <bool TF32>
__device__ __forceinline__ void mma_kblock(uint32_t d_tmem, uint64_t ad, uint64_t bd, uint32_t astep, uint32_t bstep, uint32_t idesc,
                                           uint32_t accumulate) {
#pragma unroll
  for (int k = 0; k < BK / UMMA_K; ++k) {
    if (TF32) umma_tf32(d_tmem, ad, bd, idesc, k == 0 ? accumulate : 1u);
    else umma_f16(d_tmem, ad, bd, idesc, k == 0 ? accumulate : 1u);
    ad += astep;
    bd += bstep;
  }
}

__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int tiles_n, int& mb, int& nb_) {
  constexpr int GM = 8;
  const int per_group = GM * tiles_n;
  const int group = tile / per_group;
  const int first_m = group * GM;
  const int gsz = min(tiles_m - first_m, GM);
  const int in_group = tile - group * per_group;
  mb = first_m + in_group % gsz;
  nb_ = in_group / gsz;
}

template <int BN, int STAGES, int MODE>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const GemmParams p) {
  constexpr uint32_t A_BYTES = BM * BK * 2;
  constexpr uint32_t B_BYTES = BN * BK * 2;
  constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = (2 * BN <= 32) ? 32 : (2 * BN <= 64 ? 64 : (2 * BN <= 128 ? 128 : (2 * BN <= 256 ? 256 : 512)));

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi_stage = smem + STAGES * STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi_stage + EPI_WARPS * EPI_STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_items = p.tiles_m * p.tiles_n * p.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 2);   // both producers announce their bytes
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], EPI_WARPS);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0 || warp == 2) {
    // ------------------------------------------------------------------ TMA producers
    // One thread for A, one for B: a thread needs about 100 ns per k-block and 50 ns per copy, which for one thread with the
    // two to six copies of a stage is more than the tensor core needs for it (M = N = 128: 209 to 317 ns per k-block with
    // one producer thread, 191 to 238 with two).
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      // a k-block is one 128-byte swizzle row of K: 64 bf16 or 32 fp32 elements; an MN-major operand arrives in chunks of
      // that many MN elements, each chunk bk rows of 128 bytes
      const int bk = p.tf32 ? BK / 2 : BK, chunk = bk;
      for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
        int mb, nb_;
        const int tile = item / p.splits, split = item - tile * p.splits;
        tile_coords(tile, p.tiles_m, p.tiles_n, mb, nb_);
        const int kb0 = split * p.kb_per_split, kb1 = min(p.num_kb, kb0 + p.kb_per_split);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&empty_bar[stage], phase ^ 1u, abort_flag, p.status, 1)) { ok = false; *abort_flag = 1; break; }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          mbar_expect_tx(&full_bar[stage], warp == 0 ? A_BYTES : B_BYTES);
          if (warp == 2) {
            if (!p.b_mn) {
              tma_load_2d(sb, &tmB, &full_bar[stage], kb * bk, nb_ * BN);
            } else {
              for (int h = 0; h < (BN + chunk - 1) / chunk; ++h)
                tma_load_2d(sb + h * (bk * 128), &tmB, &full_bar[stage], nb_ * BN + h * chunk, kb * bk);
            }
          } else if (p.conv == 2) {
            // rows of the tile = 2 chunks of 64 channels of one filter tap each; k-block kb = 64 output pixels as runs of
            // bw consecutive pixels of one output row.  A chunk past the last tap and pixels past the last image read the
            // zero fill (image index out of range), so the byte count of the stage stays the same.
            const int bw = p.conv_bw, per_img = p.conv_oh * p.conv_ow;
            for (int h = 0; h < BM / 64; ++h) {
              const int kpos = mb * BM + h * 64, tap = kpos / p.conv_c, c0 = kpos - tap * p.conv_c;
              const int kh = tap / p.conv_kw, kw = tap - kh * p.conv_kw;
              for (int i = 0; i < BK / bw; ++i) {
                const int m0 = kb * BK + i * bw;
                int bimg = m0 / per_img;
                const int rem = m0 - bimg * per_img;
                const int oh = rem / p.conv_ow, ow0 = rem - oh * p.conv_ow;
                if (tap >= p.conv_taps) bimg = p.conv_b;
                tma_load_4d_g(sa + h * (64 * BK * 2) + i * bw * 128, &tmA, &full_bar[stage], c0, ow0 - p.conv_pad + kw,
                              oh - p.conv_pad + kh, bimg);
              }
            }
          } else if (p.conv) {
            // k-block kb = 64 channels [c0, c0+64) of filter tap (kh, kw); the 128 output pixels of the tile are
            // 128 / bw runs of bw consecutive pixels of one output row (bw divides OW and 128), stride 1:
            // input pixel = output pixel + tap − pad; coordinates outside the image read the zero fill
            const int kpos = kb * BK, tap = kpos / p.conv_c, c0 = kpos - tap * p.conv_c;
            const int kh = tap / p.conv_kw, kw = tap - kh * p.conv_kw;
            const int bw = p.conv_bw, per_img = p.conv_oh * p.conv_ow;
            for (int i = 0; i < BM / bw; ++i) {
              const int m0 = mb * BM + i * bw;
              const int bimg = m0 / per_img, rem = m0 - bimg * per_img;
              const int oh = rem / p.conv_ow, ow0 = rem - oh * p.conv_ow;
              tma_load_4d_g(sa + i * bw * 128, &tmA, &full_bar[stage], c0, ow0 - p.conv_pad + kw, oh - p.conv_pad + kh, bimg);
            }
          } else if (!p.a_mn) {
            tma_load_2d(sa, &tmA, &full_bar[stage], kb * bk, mb * BM);
          } else {
            for (int h = 0; h < BM / chunk; ++h)
              tma_load_2d(sa + h * (bk * 128), &tmA, &full_bar[stage], mb * BM + h * chunk, kb * bk);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc(p.tf32 ? 2u : 1u, BM, BN, (uint32_t)p.a_mn, (uint32_t)p.b_mn);
      // one instruction consumes 32 bytes of K: 16 bf16 or 8 tf32.  K-major: 32 bytes further inside the swizzle row;
      // MN-major: that many k-rows of 128 bytes further, chunks of MN one k-block of rows apart.
      // An MN-major TF32 operand is in the 32-byte-atom form of the 128-byte swizzle (descriptor layout 1): its pattern
      // repeats every 4 k-rows, so the stride between row groups is 512 bytes instead of 1024.
      const bool tf32 = p.tf32 != 0;
      const uint32_t kadv_mn = tf32 ? 8u * 128u : 16u * 128u, lbo_mn = tf32 ? 32u * 128u : 64u * 128u;
      const uint32_t sbo_mn = tf32 ? 512u : 1024u, lay_mn = tf32 ? 1u : 2u;
      const uint32_t s0 = smem_u32(smem);
      const uint64_t ad0 = p.a_mn ? make_smem_desc(s0, lbo_mn, sbo_mn, lay_mn) : make_smem_desc(s0, 16, 1024, 2);
      const uint64_t bd0 = p.b_mn ? make_smem_desc(s0 + A_BYTES, lbo_mn, sbo_mn, lay_mn) : make_smem_desc(s0 + A_BYTES, 16, 1024, 2);
      const uint32_t astep = (p.a_mn ? kadv_mn : UMMA_K * 2) >> 4, bstep = (p.b_mn ? kadv_mn : UMMA_K * 2) >> 4;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
        if (!wait_or_abort(&tempty_bar[acc], acc_phase ^ 1u, abort_flag, p.status, 2)) { ok = false; *abort_flag = 1; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
        const int split = item % p.splits;
        const int kb0 = split * p.kb_per_split, kb1 = min(p.num_kb, kb0 + p.kb_per_split);
        uint32_t accumulate = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&full_bar[stage], phase, abort_flag, p.status, 3)) { ok = false; *abort_flag = 1; break; }
          tc_fence_after();
          const uint32_t off = (uint32_t)stage * (STAGE_BYTES >> 4);
          if (tf32) mma_kblock<true>(d_tmem, ad0 + off, bd0 + off, astep, bstep, idesc, accumulate);
          else mma_kblock<false>(d_tmem, ad0 + off, bd0 + off, astep, bstep, idesc, accumulate);
          accumulate = 1;
          umma_commit(&empty_bar[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit(&tfull_bar[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 3..10)
    const int quarter = warp & 3, half = (warp - 3) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      int mb, nb_;
      const int tile = item / p.splits;
      tile_coords(tile, p.tiles_m, p.tiles_n, mb, nb_);
      const float4 bias = load_bias<BN, (MODE == EPI_F32 || MODE == EPI_F32_ANY) ? 32 : epi_group<BN>()>(p, nb_ * BN, half, lane);
      if (!wait_or_abort(&tfull_bar[acc], acc_phase, abort_flag, p.status, 4)) { ok = false; *abort_flag = 1; break; }
      tc_fence_after();
      const int row_in_tile = quarter * 32;
      const uint32_t taddr0 = tmem_base + ((uint32_t)row_in_tile << 16) + (uint32_t)(acc * BN);
      uint8_t* st = epi_stage + (warp - 3) * EPI_STAGE_BYTES;
      if (MODE == EPI_F32 || MODE == EPI_F32_ANY)   // split: park the partial tile; a second kernel sums the splits in order
        epilogue_groups_f32<BN, MODE>(p, bias, taddr0, st, mb * BM + row_in_tile, nb_ * BN, half, lane,
                                      p.splits > 1 ? p.ws + (size_t)item * (BM * BN) + (size_t)row_in_tile * BN : nullptr);
      else
        epilogue_groups_bf16<BN, MODE>(p, bias, taddr0, st, mb * BM + row_in_tile, nb_ * BN, half, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------ two-CTA tiles
// The same GEMM with cta_group::2: a cluster of two CTAs (two SMs) owns one 256 x 256 output tile.  Each CTA stages 128
// rows of A and 128 of the 256 B columns; ONE thread of the leader CTA issues tcgen05.mma.cta_group::2 (M = 256,
// N = 256), which reads both CTAs' shared memory and writes rows [0,128) of the tile into the leader's tensor memory
// and rows [128,256) into the peer's.  Per SM that is half the B bytes of a 128 x 256 one-CTA tile for the same
// FLOPs, i.e. 64 instead of 96 shared-memory bytes per tensor-core clock.
//   * both CTAs' TMA loads complete on the LEADER's full barrier (cp.async.bulk.tensor with cta_group::2 may signal a
//     barrier of the peer; no multicast is used); the leader arms it with the bytes of both;
//   * tcgen05.commit with a two-CTA mask frees the stage / publishes the accumulator in both CTAs;
//   * the peer's epilogue warps release the accumulator on the leader's barrier (remote arrive).
constexpr int BN2 = 256;       // tile columns (both CTAs together)
constexpr int STAGES2 = 6;     // 6 x (16 KB A + 16 KB B) per CTA

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load whose completion bytes go to a barrier given as a shared::cluster address (possibly the peer CTA's)
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this shared-memory offset in BOTH CTAs of the pair once the MMAs issued so far have retired
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"((unsigned short)3)
               : "memory");
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS2, 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  constexpr uint32_t A_BYTES = BM * BK * 2;            // this CTA's 128 rows of A
  constexpr uint32_t B_BYTES = (BN2 / 2) * BK * 2;     // this CTA's 128 of the 256 B columns
  constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = 512;                  // two accumulators of 256 columns

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi_stage = smem + STAGES2 * STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi_stage + EPI_WARPS * EPI_STAGE_BYTES);   // used in the leader only
  uint64_t* empty_bar = full_bar + STAGES2;
  uint64_t* tfull_bar = empty_bar + STAGES2;
  uint64_t* tempty_bar = tfull_bar + 2;                                             // used in the leader only
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();           // 0 = leader
  const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;
  const int num_items = p.tiles_m * p.tiles_n * p.splits;   // tiles of 256 x 256, each in `splits` ranges of k-blocks

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES2; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * EPI_WARPS);   // the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmB);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = cluster_id; item < num_items && ok; item += num_clusters) {
        int mb, nb_;
        const int tile = item / p.splits, split = item - tile * p.splits;
        tile_coords(tile, p.tiles_m, p.tiles_n, mb, nb_);
        const int kb0 = split * p.kb_per_split, kb1 = min(p.num_kb, kb0 + p.kb_per_split);
        const int m0 = mb * (2 * BM) + (int)rank * BM;          // this CTA's rows of A
        const int n0 = nb_ * BN2 + (int)rank * (BN2 / 2);       // this CTA's columns of B
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&empty_bar[stage], phase ^ 1u, abort_flag, p.status, 21)) { ok = false; *abort_flag = 1; break; }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          const uint32_t fb = mapa_rank(smem_u32(&full_bar[stage]), 0);
          if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * STAGE_BYTES);
          if (!p.a_mn) {
            tma_load_2d_pair(sa, &tmA, fb, kb * BK, m0);
          } else {
#pragma unroll
            for (int h = 0; h < BM / 64; ++h) tma_load_2d_pair(sa + h * (64 * BK * 2), &tmA, fb, m0 + h * 64, kb * BK);
          }
          if (!p.b_mn) {
            tma_load_2d_pair(sb, &tmB, fb, kb * BK, n0);
          } else {
#pragma unroll
            for (int h = 0; h < BN2 / 128; ++h) tma_load_2d_pair(sb + h * (64 * BK * 2), &tmB, fb, n0 + h * 64, kb * BK);
          }
          if (++stage == STAGES2) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc(1u, 2 * BM, BN2, (uint32_t)p.a_mn, (uint32_t)p.b_mn);
      const uint32_t s0 = smem_u32(smem);
      const uint64_t ad0 = p.a_mn ? make_smem_desc(s0, 64 * BK * 2, 1024, 2) : make_smem_desc(s0, 16, 1024, 2);
      const uint64_t bd0 = p.b_mn ? make_smem_desc(s0 + A_BYTES, 64 * BK * 2, 1024, 2) : make_smem_desc(s0 + A_BYTES, 16, 1024, 2);
      const uint32_t astep = (p.a_mn ? UMMA_K * 128 : UMMA_K * 2) >> 4, bstep = (p.b_mn ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int item = cluster_id; item < num_items && ok; item += num_clusters) {
        if (!wait_or_abort(&tempty_bar[acc], acc_phase ^ 1u, abort_flag, p.status, 22)) { ok = false; *abort_flag = 1; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN2);
        const int split = item % p.splits, kb0 = split * p.kb_per_split, kb1 = min(p.num_kb, kb0 + p.kb_per_split);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&full_bar[stage], phase, abort_flag, p.status, 23)) { ok = false; *abort_flag = 1; break; }
          tc_fence_after();
          uint64_t ad = ad0 + (uint32_t)stage * (STAGE_BYTES >> 4), bd = bd0 + (uint32_t)stage * (STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            umma_f16_pair(d_tmem, ad, bd, idesc, ((kb - kb0) | k) != 0 ? 1u : 0u);
            ad += astep;
            bd += bstep;
          }
          umma_commit_pair(&empty_bar[stage]);
          if (++stage == STAGES2) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit_pair(&tfull_bar[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9 of both CTAs)
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int item = cluster_id; item < num_items && ok; item += num_clusters) {
      int mb, nb_;
      tile_coords(item / p.splits, p.tiles_m, p.tiles_n, mb, nb_);
      const float4 bias = load_bias<BN2, (MODE == EPI_F32 || MODE == EPI_F32_ANY) ? 32 : epi_group<BN2>()>(p, nb_ * BN2, half, lane);
      if (!wait_or_abort(&tfull_bar[acc], acc_phase, abort_flag, p.status, 24)) { ok = false; *abort_flag = 1; break; }
      tc_fence_after();
      const int row0 = mb * (2 * BM) + (int)rank * BM + quarter * 32;
      const uint32_t taddr0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN2);
      uint8_t* st = epi_stage + (warp - 2) * EPI_STAGE_BYTES;
      if (MODE == EPI_F32 || MODE == EPI_F32_ANY) epilogue_groups_f32<BN2, MODE>(
          p, bias, taddr0, st, row0, nb_ * BN2, half, lane,
          p.splits > 1 ? p.ws + (size_t)item * (2 * BM * BN2) + (size_t)((int)rank * BM + quarter * 32) * BN2 : nullptr);
      else epilogue_groups_bf16<BN2, MODE>(p, bias, taddr0, st, row0, nb_ * BN2, half, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_rank(smem_u32(&tempty_bar[acc]), 0));
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // neither CTA leaves (or frees tensor memory) while the other may still read or signal it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// Second phase of a split-K GEMM: one thread per (row, 16-column chunk) of the output sums that chunk over the
// splits in index order (deterministic) and runs the epilogue.  A separate launch, not a "last CTA reduces" tail:
// the serial tail cost 20 us for 18 splits, and a tail that waits for sibling CTAs could deadlock against a
// second split-K kernel running on another stream.
__global__ void __launch_bounds__(128)
splitk_reduce_kernel(const GemmParams p, int BN) {
  const int chunks = BN / 16;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)p.tiles_m * p.tiles_n * p.tile_rows * chunks;
  if (idx >= total) return;
  const int c = (int)(idx % chunks);
  const int row_in_tile = (int)((idx / chunks) % p.tile_rows);
  const int tile = (int)(idx / ((long long)chunks * p.tile_rows));
  int mb, nb_;
  tile_coords(tile, p.tiles_m, p.tiles_n, mb, nb_);
  const int row = mb * p.tile_rows + row_in_tile, col0 = nb_ * BN + c * 16;
  if (row >= p.M || col0 >= p.N) return;
  EpiPrefetch pf;
  epilogue_prefetch16(p, row, col0, true, pf);
  const size_t tile_elems = (size_t)p.tile_rows * BN;
  const float* src = p.ws + (size_t)tile * p.splits * tile_elems + (size_t)row_in_tile * BN + c * 16;
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = 0.f;
  int sp = 0;
  for (; sp + 8 <= p.splits; sp += 8) {
    float4 x[8][4];
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j) x[u][j] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)(sp + u) * tile_elems) + j);
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[4 * j] += x[u][j].x; v[4 * j + 1] += x[u][j].y; v[4 * j + 2] += x[u][j].z; v[4 * j + 3] += x[u][j].w;
      }
  }
  for (; sp < p.splits; ++sp) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 x = __ldcg(reinterpret_cast<const float4*>(src + (size_t)sp * tile_elems) + j);
      v[4 * j] += x.x; v[4 * j + 1] += x.y; v[4 * j + 2] += x.z; v[4 * j + 3] += x.w;
    }
  }
  epilogue_store16(p, row, col0, v, pf);
}

// The weight-gradient case (fp32 output, plain or accumulating, no bias / activation): one thread per FOUR output
// columns, so a 256 x 256 gradient has 16 k threads in flight instead of 4 k and every split's load of a warp is one
// contiguous 512-byte run.  Splits are still added in index order.
__global__ void __launch_bounds__(256)
splitk_reduce_f32_kernel(const GemmParams p, int BN) {
  const int quads = BN / 4;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)p.tiles_m * p.tiles_n * p.tile_rows * quads;
  if (idx >= total) return;
  const int c = (int)(idx % quads);
  const int row_in_tile = (int)((idx / quads) % p.tile_rows);
  const int tile = (int)(idx / ((long long)quads * p.tile_rows));
  int mb, nb_;
  tile_coords(tile, p.tiles_m, p.tiles_n, mb, nb_);
  const int row = mb * p.tile_rows + row_in_tile, col0 = nb_ * BN + c * 4;
  if (row >= p.M || col0 >= p.N) return;
  const size_t tile_elems = (size_t)p.tile_rows * BN;
  const float* src = p.ws + (size_t)tile * p.splits * tile_elems + (size_t)row_in_tile * BN + c * 4;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  int sp = 0;
  for (; sp + 8 <= p.splits; sp += 8) {
    float4 x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)(sp + u) * tile_elems));
#pragma unroll
    for (int u = 0; u < 8; ++u) { v.x += x[u].x; v.y += x[u].y; v.z += x[u].z; v.w += x[u].w; }
  }
  for (; sp < p.splits; ++sp) {
    const float4 x = __ldcg(reinterpret_cast<const float4*>(src + (size_t)sp * tile_elems));
    v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
  }
  v.x *= p.alpha; v.y *= p.alpha; v.z *= p.alpha; v.w *= p.alpha;
  float* o = reinterpret_cast<float*>(p.D) + (size_t)row * p.ldd + col0;
  if (col0 + 4 <= p.N && (p.ldd % 4 == 0)) {
    if (p.accumulate) {
      const float4 y = *reinterpret_cast<const float4*>(o);
      v.x += y.x; v.y += y.y; v.z += y.z; v.w += y.w;
    }
    *reinterpret_cast<float4*>(o) = v;
  } else {
    const float e[4] = {v.x, v.y, v.z, v.w};
    for (int j = 0; j < 4; ++j)
      if (col0 + j < p.N) o[j] = p.accumulate ? o[j] + e[j] : e[j];
  }
}

// ------------------------------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// 2-D bf16 tensor map: inner extent `inner` (contiguous), outer extent `outer`, row pitch `ld` elements.
// `mn_major` matters for 32-bit elements only: an MN-major TF32 operand has to use the 128-byte swizzle with 32-byte
// atoms (two-bit XOR of the 32-byte chunk index with the row index modulo 4); every other operand uses the 16-byte-atom form
int make_tmap_elt(CUtensorMap* tm, const void* base, long long inner, long long outer, long long ld, int box_inner,
                  int box_outer, int elt_bytes, int mn_major = 0) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return NB_ERR_NO_DRIVER_SYMBOL;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || ((ld * elt_bytes) & 15)) return NB_ERR_UNALIGNED;
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  cuuint64_t strides[1] = {(cuuint64_t)ld * elt_bytes};
  cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
  cuuint32_t estr[2] = {1, 1};
  // fp32 operands are loaded as TFLOAT32: the copy rounds them to the 10-bit mantissa the tensor core reads
  CUresult r = enc(tm, elt_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_TFLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                   const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   (elt_bytes == 4 && mn_major) ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? NB_OK : NB_ERR_TENSORMAP;
}
int make_tmap_bf16(CUtensorMap* tm, const void* base, long long inner, long long outer, long long ld, int box_inner,
                   int box_outer) {
  return make_tmap_elt(tm, base, inner, outer, ld, box_inner, box_outer, 2);
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

int g_two_cta_mode = 0;  // 0 = by expected time, 1 = never, 2 = whenever the shape allows it

// ---- choice of tile form and split
// Time in nanoseconds that a form is expected to take, from measurements on one B200 (graph of ten launches, operands in L2):
//   * a k-block (64 bf16 of K) costs the issuing threads or the tensor core kb_ns, or the L2 its bytes at about 17 KB/ns over
//     all SMs, whichever is longer;
//   * launch, first loads and the last epilogue cost fixed_ns; in further rounds of tiles the epilogue hides behind the next
//     main loop unless that is shorter (epi_ns);
//   * a split-K adds a launch and its partial tiles twice through the L2.
// 4816 x 512 x 3200 (us): 128-column tiles, the earlier choice, 28.6; 256 columns 21.0; pairs 21.5.  512 x 3200 x 4816: 64
// columns 41.7, 256 in two splits 24.7.  200 x 512 x 512: two splits 7.8, none 5.9.  4096 x 384 x 49152: 64 columns 296,
// pairs 222, pairs in two splits 145.
struct TileForm { int bn, rows, kb_bytes, slots, kb_ns, fixed_ns, epi_ns; };   // slots: tiles in flight on 148 SMs
constexpr TileForm TILE_64 = {64, BM, 24576, 1, 200, 3900, 600}, TILE_128 = {128, BM, 32768, 1, 210, 4600, 900},
                   TILE_256 = {256, BM, 49152, 1, 280, 4900, 1700}, TILE_PAIR = {256, 2 * BM, 65536, 2, 280, 5300, 1700};

long long form_ns(const TileForm& f, long long tiles, int num_kb, int splits, int sms) {
  const long long items = tiles * splits, slots = sms / f.slots, waves = ceil_div_ll(items, slots);
  const long long active = items < slots ? items : slots, l2_ns = active * f.kb_bytes / 17000;
  const long long loop = (long long)ceil_div(num_kb, splits) * (f.kb_ns > l2_ns ? f.kb_ns : l2_ns);
  long long t = f.fixed_ns + loop + (waves - 1) * (loop > f.epi_ns ? loop : f.epi_ns);
  if (splits > 1) t += 2500 + items * f.rows * f.bn * 8 / 5000;
  return t;
}
// Best number of splits of one form; 1 unless the workspace holds the partial tiles.
long long best_split(const TileForm& f, int M, int N, int num_kb, long long ws_bytes, int sms, int* splits) {
  const long long tiles = (long long)ceil_div(M, f.rows) * ceil_div(N, f.bn), slots = sms / f.slots;
  long long best = form_ns(f, tiles, num_kb, 1, sms);
  *splits = 1;
  if (tiles * 2 > slots || tiles > NB_GEMM_WS_COUNTERS || num_kb < 8) return best;
  for (int sp = 2; sp <= num_kb / 4 && tiles * sp <= slots; ++sp) {
    if (tiles * sp * f.rows * f.bn * 4 > ws_bytes) break;
    const long long t = form_ns(f, tiles, num_kb, sp, sms);
    if (t < best) { best = t; *splits = sp; }
  }
  return best;
}

int finish_split(const GemmParams& p, int BN, cudaStream_t stream) {
  if (p.splits <= 1) return NB_OK;
  const long long rows = (long long)p.tiles_m * p.tiles_n * p.tile_rows;
  if (p.out_f32 && !p.bias && !p.act && !p.dact)
    splitk_reduce_f32_kernel<<<(unsigned)((rows * (BN / 4) + 255) / 256), 256, 0, stream>>>(p, BN);
  else
    splitk_reduce_kernel<<<(unsigned)((rows * (BN / 16) + 127) / 128), 128, 0, stream>>>(p, BN);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

// `splits`: wanted number of ranges of k-blocks (the workspace holds their partial tiles)
template <int BN, int STAGES>
int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmParams& p, int splits, cudaStream_t stream) {
  constexpr size_t smem = (size_t)STAGES * (BM * BK * 2 + BN * BK * 2) + EPI_WARPS * EPI_STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static_assert(smem <= 232448, "shared memory budget of one CTA");
  p.tiles_m = ceil_div(p.M, BM);
  p.tiles_n = ceil_div(p.N, BN);
  p.tile_rows = BM;
  p.num_kb = ceil_div(p.K, p.tf32 ? BK / 2 : BK);
  p.kb_per_split = ceil_div(p.num_kb, splits);
  p.splits = ceil_div(p.num_kb, p.kb_per_split);
  const int items = p.tiles_m * p.tiles_n * p.splits;
  const int grid = items < sm_count() ? items : sm_count();
  typedef void (*Kernel)(CUtensorMap, CUtensorMap, GemmParams);
  // narrow tiles (heads of a few columns) run the general epilogues only
  static const Kernel kernels[EPI_MODES] = {
      gemm_bf16_kernel<BN, STAGES, BN < 64 ? EPI_BF16 : EPI_PLAIN>, gemm_bf16_kernel<BN, STAGES, BN < 64 ? EPI_BF16 : EPI_RELU>,
      gemm_bf16_kernel<BN, STAGES, BN < 64 ? EPI_BF16 : EPI_GELU>,  gemm_bf16_kernel<BN, STAGES, BN < 64 ? EPI_BF16 : EPI_ADD>,
      gemm_bf16_kernel<BN, STAGES, EPI_BF16>,                       gemm_bf16_kernel<BN, STAGES, EPI_F32>,
      gemm_bf16_kernel<BN, STAGES, EPI_F32_ANY>};
  static bool configured[EPI_MODES] = {};
  const EpiMode mode = epi_mode(p, p.splits > 1);
  if (!configured[mode]) {
    NB_CUDA(cudaFuncSetAttribute(kernels[mode], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[mode] = true;
  }
  kernels[mode]<<<grid, NUM_THREADS, smem, stream>>>(tmA, tmB, p);
  NB_LAUNCH_CHECK();
  return finish_split(p, BN, stream);
}

int launch_two_cta(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmParams& p, int splits, cudaStream_t stream) {
  constexpr size_t smem = (size_t)STAGES2 * (BM * BK * 2 + (BN2 / 2) * BK * 2) + EPI_WARPS * EPI_STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static_assert(smem <= 232448, "shared memory budget of one CTA");
  p.tiles_m = ceil_div(p.M, 2 * BM);
  p.tiles_n = ceil_div(p.N, BN2);
  p.tile_rows = 2 * BM;
  p.num_kb = ceil_div(p.K, BK);
  p.kb_per_split = ceil_div(p.num_kb, splits);
  p.splits = ceil_div(p.num_kb, p.kb_per_split);
  const int items = p.tiles_m * p.tiles_n * p.splits;
  const int clusters = items < sm_count() / 2 ? items : sm_count() / 2;
  typedef void (*Kernel)(CUtensorMap, CUtensorMap, GemmParams);
  static const Kernel kernels[EPI_MODES] = {gemm2_bf16_kernel<EPI_PLAIN>, gemm2_bf16_kernel<EPI_RELU>, gemm2_bf16_kernel<EPI_GELU>,
                                            gemm2_bf16_kernel<EPI_ADD>,   gemm2_bf16_kernel<EPI_BF16>, gemm2_bf16_kernel<EPI_F32>,
                                            gemm2_bf16_kernel<EPI_F32_ANY>};
  static bool configured[EPI_MODES] = {};
  const EpiMode mode = epi_mode(p, p.splits > 1);
  if (!configured[mode]) {
    NB_CUDA(cudaFuncSetAttribute(kernels[mode], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[mode] = true;
  }
  kernels[mode]<<<2 * clusters, NUM_THREADS2, smem, stream>>>(tmA, tmB, p);
  NB_LAUNCH_CHECK();
  return finish_split(p, BN2, stream);
}


}  // namespace

extern "C" {

// Selects between one-CTA tiles and two-CTA (cta_group::2) 256 x 256 tiles; returns the previous setting.
int nb_gemm_two_cta_mode(int mode) {
  const int old = g_two_cta_mode;
  if (mode >= 0 && mode <= 2) g_two_cta_mode = mode;
  return old;
}

// D[M,N] = epi(alpha * A·B).  A: a_mn=0 → [M,K] row-major (lda = pitch of a row of K), a_mn=1 → [K,M]
// row-major (lda = pitch of a row of M).  B: b_mn=0 → [N,K] row-major, b_mn=1 → [K,N] row-major.
// Pitches in elements; every pitch*2 bytes and every base must be 16-byte aligned (TMA).
static int gemm_any(int tf32, const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb, int ldd, int a_mn,
                    int b_mn, int out_f32, int accumulate, float alpha, const float* bias, int act, const void* aux,
                    int ld_aux, int dact, unsigned int* status, int bn_hint, void* workspace, long long workspace_bytes,
                    void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return NB_ERR_BAD_ARG;
  const int elt = tf32 ? 4 : 2, bk = 128 / elt;   // elements per 128-byte row = k-block depth = MN-major chunk width
  if (accumulate && !out_f32) return NB_ERR_BAD_ARG;
  if (dact && !aux) return NB_ERR_BAD_ARG;
  // workspace layout: [NB_GEMM_WS_COUNTERS u32 tile counters (zero at rest)] [fp32 partial tiles]
  const bool have_ws = workspace && workspace_bytes > NB_GEMM_WS_COUNTERS * 4 + (1 << 20);
  const long long ws_bytes = have_ws ? workspace_bytes - NB_GEMM_WS_COUNTERS * 4 : 0;
  const int num_kb = ceil_div(K, bk), sms = sm_count();
  int BN = bn_hint, splits = 1;
  bool two_cta = false;
  if (b_mn && BN && BN < bk) BN = bk;
  if (BN == 0 && N <= 32 && !b_mn) {
    BN = N <= 16 ? 16 : 32;                        // heads of a few columns
    best_split(TILE_64, M, N, num_kb, ws_bytes, sms, &splits);
  } else if (BN == 0) {
    // the form with the smallest expected time; MN-major B needs whole 64-column boxes
    long long best = best_split(TILE_64, M, N, num_kb, ws_bytes, sms, &splits);
    BN = 64;
    int sp;
    for (const TileForm* f : {&TILE_128, &TILE_256}) {
      if (N <= f->bn / 2) break;
      const long long t = best_split(*f, M, N, num_kb, ws_bytes, sms, &sp);
      if (t < best) { best = t; BN = f->bn; splits = sp; }
    }
    if (!tf32 && g_two_cta_mode != 1 && M >= 256 && N >= 256 && K >= 128) {
      const long long t = best_split(TILE_PAIR, M, N, num_kb, ws_bytes, sms, &sp);
      if (t < best || g_two_cta_mode == 2) { two_cta = true; splits = sp; }
    }
  } else {
    const TileForm f = BN == 256 ? TILE_256 : (BN == 128 ? TILE_128 : TILE_64);
    best_split(TileForm{BN, BM, f.kb_bytes, 1, f.kb_ns, f.fixed_ns, f.epi_ns}, M, N, num_kb, ws_bytes, sms, &splits);
  }
  if (two_cta) BN = BN2 / 2;   // the B box of one CTA
  CUtensorMap tmA, tmB;
  int rc;
  if (!a_mn) rc = make_tmap_elt(&tmA, A, K, M, lda, bk, BM, elt);
  else rc = make_tmap_elt(&tmA, A, M, K, lda, bk, bk, elt, 1);
  if (rc) return rc;
  if (!b_mn) rc = make_tmap_elt(&tmB, B, K, N, ldb, bk, BN, elt);
  else rc = make_tmap_elt(&tmB, B, N, K, ldb, bk, bk, elt, 1);
  if (rc) return rc;
  GemmParams p;
  p.M = M; p.N = N; p.K = K;
  p.a_mn = a_mn; p.b_mn = b_mn; p.tf32 = tf32;
  p.ldd = ldd; p.ld_aux = ld_aux;
  p.out_f32 = out_f32; p.accumulate = accumulate; p.act = act; p.dact = dact;
  p.alpha = alpha;
  p.D = D; p.bias = bias; p.aux = (const __nv_bfloat16*)aux; p.status = status;
  p.conv = 0;
  p.ws = have_ws ? (float*)((char*)workspace + NB_GEMM_WS_COUNTERS * 4) : nullptr;
  p.tile_ctr = have_ws ? (unsigned int*)workspace : nullptr;
  cudaStream_t s = (cudaStream_t)stream;
  if (two_cta) return launch_two_cta(tmA, tmB, p, splits, s);
  switch (BN) {
    case 256: return launch<256, 4>(tmA, tmB, p, splits, s);
    case 128: return launch<128, 6>(tmA, tmB, p, splits, s);
    case 64: return launch<64, 8>(tmA, tmB, p, splits, s);
    case 32: return launch<32, 8>(tmA, tmB, p, splits, s);
    case 16: return launch<16, 8>(tmA, tmB, p, splits, s);
    default: return NB_ERR_BAD_ARG;
  }
}

int nb_gemm_bf16(const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb, int ldd, int a_mn,
                 int b_mn, int out_f32, int accumulate, float alpha, const float* bias, int act, const void* aux,
                 int ld_aux, int dact, unsigned int* status, int bn_hint, void* workspace, long long workspace_bytes,
                 void* stream) {
  return gemm_any(0, A, B, D, M, N, K, lda, ldb, ldd, a_mn, b_mn, out_f32, accumulate, alpha, bias, act, aux, ld_aux, dact,
                  status, bn_hint, workspace, workspace_bytes, stream);
}
// The same contraction on fp32 operands read as TF32 (10-bit mantissa, fp32 accumulation): `kind::tf32`, one-CTA tiles.
// Pitches in fp32 elements (multiples of 4); `aux` stays a bf16 tensor.
int nb_gemm_tf32(const void* A, const void* B, void* D, int M, int N, int K, int lda, int ldb, int ldd, int a_mn,
                 int b_mn, int out_f32, int accumulate, float alpha, const float* bias, int act, const void* aux,
                 int ld_aux, int dact, unsigned int* status, int bn_hint, void* workspace, long long workspace_bytes,
                 void* stream) {
  return gemm_any(1, A, B, D, M, N, K, lda, ldb, ldd, a_mn, b_mn, out_f32, accumulate, alpha, bias, act, aux, ld_aux, dact,
                  status, bn_hint, workspace, workspace_bytes, stream);
}

// Implicit-GEMM convolution forward, stride 1: y[B·OH·OW, OC] = epi(patches(x) · W), x NHWC bf16 [B, H, W, C] with
// C % 64 == 0, W in GEMM layout [KH·KW·C, OC] (row pitch ldw).  OW must have a power-of-two factor bw >= 8 (the run
// length of one TMA box).  Output spatial size: OH = H + 2·pad − KH + 1, OW likewise.
int nb_conv_implicit_fwd(const void* x, const void* Wt, void* y, int B, int H, int Wd, int C, int OC, int KH, int KW, int pad,
                         int ldw, int ldy, const float* bias, int act, const void* residual, int ld_res,
                         unsigned int* status, void* stream) {
  const int OH = H + 2 * pad - KH + 1, OW = Wd + 2 * pad - KW + 1;
  if (B <= 0 || OH <= 0 || OW <= 0 || C % 64 || OC <= 0) return NB_ERR_BAD_ARG;
  int bw = 1;
  while (bw < 128 && OW % (bw * 2) == 0) bw *= 2;
  if (bw < 8) return NB_ERR_BAD_ARG;   // every box then starts on a 1024-byte swizzle atom of the A tile
  EncodeTiledFn enc = get_encode();
  if (!enc) return NB_ERR_NO_DRIVER_SYMBOL;
  if (reinterpret_cast<uintptr_t>(x) & 15) return NB_ERR_UNALIGNED;
  CUtensorMap tmA, tmB;
  {
    cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)Wd, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)Wd * C * 2, (cuuint64_t)H * Wd * C * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)bw, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    if (enc(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(x), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return NB_ERR_TENSORMAP;
  }
  const int M = B * OH * OW, K = KH * KW * C;
  int BN = 128;
  if (OC <= 64 || (long long)ceil_div(M, BM) * ceil_div(OC, 128) < sm_count()) BN = 64;
  int rc = make_tmap_bf16(&tmB, Wt, OC, K, ldw, 64, BK);
  if (rc) return rc;
  GemmParams p;
  p.M = M; p.N = OC; p.K = K;
  p.a_mn = 0; p.b_mn = 1; p.tf32 = 0;
  p.ldd = ldy; p.ld_aux = ld_res;
  p.out_f32 = 0; p.accumulate = 0; p.act = act; p.dact = residual ? NB_AUX_ADD : 0;
  p.alpha = 1.f;
  p.D = y; p.bias = bias; p.aux = (const __nv_bfloat16*)residual; p.status = status;
  p.ws = nullptr; p.tile_ctr = nullptr;
  p.conv = 1; p.conv_c = C; p.conv_ow = OW; p.conv_oh = OH; p.conv_kw = KW; p.conv_pad = pad; p.conv_bw = bw;
  p.conv_taps = KH * KW; p.conv_b = B;
  cudaStream_t s = (cudaStream_t)stream;
  if (BN == 128) return launch<128, 6>(tmA, tmB, p, 1, s);
  return launch<64, 8>(tmA, tmB, p, 1, s);
}


// Implicit-GEMM weight gradient of a stride-1 convolution: dW[KH·KW·C, OC] (+)= patches(x)^T · dy without the patch
// matrix.  x NHWC bf16 [B, H, W, C], C % 64 == 0; dy bf16 [B·OH·OW, OC] (row pitch ld_dy); dW fp32 (row pitch ld_dw), the
// result is ADDED to it.  OW needs a power-of-two factor bw in [8, 64].  Split-K over the pixels through `workspace`.
int nb_conv_implicit_wgrad(const void* x, const void* dy, float* dW, int B, int H, int Wd, int C, int OC, int KH, int KW, int pad,
                           int ld_dy, int ld_dw, unsigned int* status, void* workspace, long long workspace_bytes, void* stream) {
  const int OH = H + 2 * pad - KH + 1, OW = Wd + 2 * pad - KW + 1;
  if (B <= 0 || OH <= 0 || OW <= 0 || C % 64 || OC <= 0) return NB_ERR_BAD_ARG;
  int bw = 1;
  while (bw < 64 && OW % (bw * 2) == 0) bw *= 2;
  if (bw < 8) return NB_ERR_BAD_ARG;
  EncodeTiledFn enc = get_encode();
  if (!enc) return NB_ERR_NO_DRIVER_SYMBOL;
  if (reinterpret_cast<uintptr_t>(x) & 15) return NB_ERR_UNALIGNED;
  CUtensorMap tmA, tmB;
  {
    cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)Wd, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)Wd * C * 2, (cuuint64_t)H * Wd * C * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)bw, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    if (enc(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(x), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return NB_ERR_TENSORMAP;
  }
  const int Mpix = B * OH * OW, Kc = KH * KW * C;
  int BN = 128;
  if (OC <= 64 || (long long)ceil_div(Kc, BM) * ceil_div(OC, 128) * 2 < sm_count()) BN = 64;
  int rc = make_tmap_bf16(&tmB, dy, OC, Mpix, ld_dy, 64, BK);
  if (rc) return rc;
  GemmParams p;
  p.M = Kc; p.N = OC; p.K = Mpix;
  p.a_mn = 1; p.b_mn = 1; p.tf32 = 0;
  p.ldd = ld_dw; p.ld_aux = 0;
  p.out_f32 = 1; p.accumulate = 1; p.act = 0; p.dact = 0;
  p.alpha = 1.f;
  p.D = dW; p.bias = nullptr; p.aux = nullptr; p.status = status;
  p.ws = nullptr; p.tile_ctr = nullptr;
  long long ws_bytes = 0;
  if (workspace && workspace_bytes > NB_GEMM_WS_COUNTERS * 4 + (1 << 20)) {
    p.tile_ctr = (unsigned int*)workspace;
    p.ws = (float*)((char*)workspace + NB_GEMM_WS_COUNTERS * 4);
    ws_bytes = workspace_bytes - NB_GEMM_WS_COUNTERS * 4;
  }
  p.conv = 2; p.conv_c = C; p.conv_ow = OW; p.conv_oh = OH; p.conv_kw = KW; p.conv_pad = pad; p.conv_bw = bw;
  p.conv_taps = KH * KW; p.conv_b = B;
  cudaStream_t s = (cudaStream_t)stream;
  int splits;
  best_split(BN == 128 ? TILE_128 : TILE_64, Kc, OC, ceil_div(Mpix, BK), ws_bytes, sm_count(), &splits);
  if (BN == 128) return launch<128, 6>(tmA, tmB, p, splits, s);
  return launch<64, 8>(tmA, tmB, p, splits, s);
}

}  // extern "C"
