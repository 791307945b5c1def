// What the tcgen05 GEMM kernels share (plain GEMM, CTA pairs, convolution with a gathering producer): parameters, the staged
// epilogue, the bounded pipeline wait, the instructions of one k-block, tensor maps and the expected-time model of the tile
// forms.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "gemm_api.h"

namespace nbgemm {

using namespace nb;

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
// Eight epilogue warps: two share a 32-row quarter of the accumulator and take its column groups in turn.  With four the
// epilogue of a 256 x 256 tile (bias, GELU, residual, bf16 store) took longer than the twelve k-blocks of K = 768, and the
// tensor core waited for a free accumulator: 24576 x 3072 x 768 with GELU took 240 us, 176 us with eight.
constexpr int EPI_WARPS = 8;

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
  bool vec_d, vec_aux, vec_bias;   // rows of the output / saved tensor and the bias start on 16-byte boundaries (set_vec)
  float alpha;
  float* ws;                 // splits>1: fp32 partial tiles, [tile][split][BM*BN]
  void* D;
  const float* bias;
  const __nv_bfloat16* aux;
  unsigned int* status;
};

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

// What a tile's epilogue does is part of the kernel: the frequent forms have instances of their own.  With the tests for
// bias, activation and saved tensor inside the loop over 16-column chunks every chunk jumped across the whole switch, and a
// chunk without any of them took 530 clocks, most of them instruction fetch; it takes 165 now.  (All forms side by side in
// one kernel spilled 4 KB of registers.)  The bias is a run-time test everywhere: one jump over 16 shuffles.
enum EpiMode { EPI_PLAIN, EPI_RELU, EPI_GELU, EPI_ADD, EPI_BF16, EPI_F32, EPI_F32_ANY, EPI_MODES };   // EPI_BF16, EPI_F32_ANY: the rest
inline EpiMode epi_mode(const GemmParams& p, bool split) {
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
  const bool vec_d = p.vec_d, vec_a = p.vec_aux;
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
  const bool vec_d = p.vec_d;
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
// The same for a whole warp, whose lanes then exchange values (bias shuffles, staged rows): they go on or give up together.  A
// lane that gave up alone, because the abort flag was set between two lanes' looks at it, would leave the others waiting.
__device__ __forceinline__ bool warp_wait_or_abort(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status,
                                                   unsigned int where) {
  return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag, status, where));
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

// ------------------------------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode() {
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
inline int make_tmap_elt(CUtensorMap* tm, const void* base, long long inner, long long outer, long long ld, int box_inner,
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
inline int make_tmap_bf16(CUtensorMap* tm, const void* base, long long inner, long long outer, long long ld, int box_inner,
                   int box_outer) {
  return make_tmap_elt(tm, base, inner, outer, ld, box_inner, box_outer, 2);
}

inline int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// The base counts as well as the pitch: an output may be a few columns of a wider tensor.
inline void set_vec(GemmParams& p) {
  auto rows16 = [](const void* base, long long pitch) { return ((reinterpret_cast<uintptr_t>(base) | (uintptr_t)pitch) & 15) == 0; };
  p.vec_d = rows16(p.D, (long long)p.ldd * (p.out_f32 ? 4 : 2));
  p.vec_aux = rows16(p.aux, (long long)p.ld_aux * 2);
  p.vec_bias = rows16(p.bias, 0);
}

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

inline long long form_ns(const TileForm& f, long long tiles, int num_kb, int splits, int sms) {
  const long long items = tiles * splits, slots = sms / f.slots, waves = ceil_div_ll(items, slots);
  const long long active = items < slots ? items : slots, l2_ns = active * f.kb_bytes / 17000;
  const long long loop = (long long)ceil_div(num_kb, splits) * (f.kb_ns > l2_ns ? f.kb_ns : l2_ns);
  long long t = f.fixed_ns + loop + (waves - 1) * (loop > f.epi_ns ? loop : f.epi_ns);
  if (splits > 1) t += 2500 + items * f.rows * f.bn * 8 / 5000;
  return t;
}
// Best number of splits of one form; 1 unless the workspace holds the partial tiles.
inline long long best_split(const TileForm& f, int M, int N, int num_kb, long long ws_bytes, int sms, int* splits) {
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

// second phase of a split-K launch: sums the partial tiles in split order and runs the epilogue (gemm_tcgen05.cu)
int finish_split(const GemmParams& p, int BN, cudaStream_t stream);

}  // namespace nbgemm
