// Convolution on the tensor cores without a patch matrix: a GEMM whose A tile is gathered from the NHWC input.
//
//   forward   y[B·OH·OW, OC]       = epi(patches(x) · W)            any stride, padding and width, C % 8 == 0
//   dgrad     the forward on dy with mirrored taps (stride 1); W is read in place, taps from the last to the first
//   wgrad     dW[KH·KW·C, OC]     += patches(x)^T · dy
//
// The patch matrix of a 3x3 layer is nine times its input: 16 x 120 x 160 x 64 became 354 MB, written (186 us) and read twice
// (62 us forward, 68 us weight gradient), where this kernel takes 62 and 54 us.  Gathering with TMA boxes, which
// this replaces, needed widths with a power-of-two factor of 16 and stride 1, issued up to 16 small copies per k-block from
// one thread, and was no faster than the patch matrix.
//
//   * eight producer warps copy 16-byte chunks (8 channels of one filter tap of one output pixel) with cp.async straight into
//     the 128-byte-swizzled A stage; a chunk outside the image or past the last tap is written as zeros.  Eight lanes cover
//     the 128 bytes of a row, so a warp instruction reads four runs of up to 128 bytes; neighbouring taps hit L1 and L2.
//   * the copies of a warp's last k-blocks (CP_LAG) stay in flight; a stage is announced after its copies have landed and every
//     producer thread has made them visible to the tensor core (fence.proxy.async);
//   * B (weights or dy) arrives by TMA from a warp of its own; MMA issue, epilogue, split-K and bounded waits are those of
//     the GEMM (gemm_tile.cuh).
// Bound by the gather: 1024 16-byte copies per 128 x 64 block and SM, 360 to 410 ns, so wider B tiles come almost free.
// Counterpart in the reference: im2col + GEMM (noeira/nn/primitives/conv2d.mojo:437,652,723) or cuDNN.
#include "conv_index.h"
#include "gemm_tile.cuh"

namespace {

using namespace nb;
using namespace nbgemm;
using namespace nbconv;
static_assert(TILE_ROWS == BM && K_BLOCK == BK, "one tiling for the kernel and its index functions");

// Two groups of four gathering warps take the k-blocks in turn: a k-block costs its warps about 900 clocks, most of them
// latency (barrier, proxy fence, address arithmetic of one warp per scheduler), and only half of that is left per k-block.
// 16 x 120 x 160, 64 -> 64: 89 us with one group and divisions, 72 with multiplications, 62 with two groups.
constexpr int CP_GROUPS = 2, CP_GROUP_WARPS = 4, CP_WARPS = CP_GROUPS * CP_GROUP_WARPS;
constexpr int CONV_EPI_WARPS = 4;   // enough behind a main loop this long, and leaves 128 registers per thread
constexpr int CONV_THREADS = 32 * (CP_WARPS + 2 + CONV_EPI_WARPS);   // gather, MMA, B loads, epilogue

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void gather(const ConvGeom& g, uint32_t dst, const Corner& c, const Tap& k) {
  int off;
  bool in = chunk_of(g, c, k, off);
  if (!NB_IN_BOUNDS(!in || (off >= 0 && off <= g.elems - 8), 641, off)) in = false;
  cp_async16(dst, (const __nv_bfloat16*)g.x + (in ? off : 0), in);
}

template <int BN, int STAGES, int MODE>
__global__ void __launch_bounds__(CONV_THREADS, 1)
conv_gemm_kernel(const __grid_constant__ CUtensorMap tmB, const GemmParams p, const ConvGeom g) {
  constexpr uint32_t A_BYTES = BM * BK * 2;
  constexpr uint32_t B_BYTES = BN * BK * 2;
  constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = 2 * BN;
  static_assert(TMEM_COLS == 128 || TMEM_COLS == 256 || TMEM_COLS == 512, "two accumulators, a power of two of columns");
  static_assert(STAGES % CP_GROUPS == 0 && STAGES >= 2 * CP_GROUPS, "a group keeps to its stages");
  constexpr int CP_LAG = 1;   // k-blocks of a group in flight behind the newest (two were 5% slower)

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi_stage = smem + STAGES * STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi_stage + CONV_EPI_WARPS * EPI_STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_items = p.tiles_m * p.tiles_n * p.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], CP_GROUP_WARPS + 1);   // the gathering warps of one group, and B's bytes
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], CONV_EPI_WARPS);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmB);
  }
  if (warp == CP_WARPS) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < CP_WARPS) {
    // ------------------------------------------------------------------ gather of A
    // thread = chunk `ch` of the rows r0, r0 + 16, ... of a stage (rows: 128 pixels; weight gradient: 2 x 64, two groups of
    // 64 patch elements for the same 64 pixels)
    const int group = warp / CP_GROUP_WARPS, tid = threadIdx.x % (32 * CP_GROUP_WARPS);
    const int ch = tid & 7, r0 = tid >> 3;
    const uint32_t dst0 = smem_u32(smem) + (uint32_t)(r0 * 128 + ((ch ^ (r0 & 7)) << 4));   // rows 16 apart swizzle alike
    int stage = 0, turn = 0;
    int done = group, pending = 0;            // `done`: next stage to announce, `pending`: k-blocks not announced yet
    uint32_t phase = 0;
    bool ok = true;
    auto announce = [&]() {                   // this warp's copies of stage `done` have landed
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[done]);
      if ((done += CP_GROUPS) >= STAGES) done = group;
      --pending;
    };
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      int mb, nb_;
      const int tile = item / p.splits, split = item - tile * p.splits;
      tile_coords(tile, p.tiles_m, p.tiles_n, mb, nb_);
      const int kb0 = split * p.kb_per_split, kb1 = min(p.num_kb, kb0 + p.kb_per_split);
      Corner c[8];
      Tap k0, k1;
      if (g.wgrad) {
        k0 = tap_of(g, mb * 16 + ch);
        k1 = tap_of(g, mb * 16 + 8 + ch);
      } else {
        Pixel px = pixel_of(g, mb * BM + r0);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          c[i] = corner_of(g, px, mb * BM + r0 + 16 * i);
          pixel_step(g, px, 16);
        }
      }
      for (int kb = kb0; kb < kb1; ++kb) {
        const bool mine = turn == group;
        if (++turn == CP_GROUPS) turn = 0;
        if (!mine) {
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
          continue;
        }
        if (!wait_or_abort(&empty_bar[stage], phase ^ 1u, abort_flag, p.status, 31)) { ok = false; *abort_flag = 1; }
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        const uint32_t dst = dst0 + (uint32_t)stage * STAGE_BYTES;
        if (g.wgrad) {
          const int m = kb * BK + r0;
          Pixel px = pixel_of(g, m);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const Corner q = corner_of(g, px, m + 16 * i);
            gather(g, dst + (uint32_t)(i * 16 * 128), q, k0);
            gather(g, dst + (uint32_t)((64 + i * 16) * 128), q, k1);
            pixel_step(g, px, 16);
          }
        } else {
          const Tap k = tap_of(g, kb * 8 + ch);
#pragma unroll
          for (int i = 0; i < 8; ++i) gather(g, dst + (uint32_t)(i * 16 * 128), c[i], k);
        }
        cp_commit();
        if (++pending > CP_LAG) {
          cp_wait<CP_LAG>();
          announce();
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
    cp_wait<0>();
    while (pending > 0 && ok) announce();
  } else if (warp == CP_WARPS) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t a_mn = g.wgrad ? 1u : 0u, b_mn = g.mirror ? 0u : 1u;
      const uint32_t idesc = make_idesc(1u, BM, BN, a_mn, b_mn);
      const uint32_t s0 = smem_u32(smem);
      const uint64_t ad0 = a_mn ? make_smem_desc(s0, 64 * 128, 1024, 2) : make_smem_desc(s0, 16, 1024, 2);
      const uint64_t bd0 = b_mn ? make_smem_desc(s0 + A_BYTES, 64 * 128, 1024, 2) : make_smem_desc(s0 + A_BYTES, 16, 1024, 2);
      const uint32_t astep = (a_mn ? UMMA_K * 128 : UMMA_K * 2) >> 4, bstep = (b_mn ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
        if (!wait_or_abort(&tempty_bar[acc], acc_phase ^ 1u, abort_flag, p.status, 32)) { ok = false; *abort_flag = 1; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
        const int split = item % p.splits;
        const int kb0 = split * p.kb_per_split, kb1 = min(p.num_kb, kb0 + p.kb_per_split);
        uint32_t accumulate = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&full_bar[stage], phase, abort_flag, p.status, 33)) { ok = false; *abort_flag = 1; break; }
          tc_fence_after();
          const uint32_t off = (uint32_t)stage * (STAGE_BYTES >> 4);
          mma_kblock<false>(d_tmem, ad0 + off, bd0 + off, astep, bstep, idesc, accumulate);
          accumulate = 1;
          umma_commit(&empty_bar[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit(&tfull_bar[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else if (warp == CP_WARPS + 1) {
    // ------------------------------------------------------------------ TMA loads of B
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
        int mb, nb_;
        const int tile = item / p.splits, split = item - tile * p.splits;
        tile_coords(tile, p.tiles_m, p.tiles_n, mb, nb_);
        const int kb0 = split * p.kb_per_split, kb1 = min(p.num_kb, kb0 + p.kb_per_split);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&empty_bar[stage], phase ^ 1u, abort_flag, p.status, 34)) { ok = false; *abort_flag = 1; break; }
          uint8_t* sb = smem + stage * STAGE_BYTES + A_BYTES;
          mbar_expect_tx(&full_bar[stage], B_BYTES);
          if (g.mirror) {
            // k-block = 64 of the C channels of one tap: C % 64 == 0; rows of W: (tap, output channel of this product)
            const int t = kb * BK / g.C, c0 = kb * BK - t * g.C;
            tma_load_2d(sb, &tmB, &full_bar[stage], c0, (g.taps - 1 - t) * p.N + nb_ * BN);
          } else {
#pragma unroll
            for (int h = 0; h < BN / 64; ++h)
              tma_load_2d(sb + h * (64 * 128), &tmB, &full_bar[stage], nb_ * BN + h * 64, kb * BK);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3;
    uint8_t* st = epi_stage + (warp - CP_WARPS - 2) * EPI_STAGE_BYTES;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
      int mb, nb_;
      tile_coords(item / p.splits, p.tiles_m, p.tiles_n, mb, nb_);
      const int row_in_tile = quarter * 32, row0 = mb * BM + row_in_tile, n0 = nb_ * BN;
      constexpr int G = MODE == EPI_F32 ? 32 : epi_group<BN>();
      const float4 bias0 = load_bias<BN, G>(p, n0, 0, lane), bias1 = load_bias<BN, G>(p, n0, 1, lane);
      if (!warp_wait_or_abort(&tfull_bar[acc], acc_phase, abort_flag, p.status, 35)) { ok = false; *abort_flag = 1; break; }
      tc_fence_after();
      const uint32_t taddr0 = tmem_base + ((uint32_t)row_in_tile << 16) + (uint32_t)(acc * BN);
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
        const float4 bias = half ? bias1 : bias0;
        if (MODE == EPI_F32)
          epilogue_groups_f32<BN, MODE>(p, bias, taddr0, st, row0, n0, half, lane,
                                        p.splits > 1 ? p.ws + (size_t)item * (BM * BN) + (size_t)row_in_tile * BN : nullptr);
        else
          epilogue_groups_bf16<BN, MODE>(p, bias, taddr0, st, row0, n0, half, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }

  // ---------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == CP_WARPS) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Expected time of the forms (see gemm_tile.cuh): the gather sets the time of a k-block.  A 3 x 3 layer with one tile per SM (148 x 128
// pixels, 64 to 512 channels, graph of ten launches, input in L2) takes 261, 296 and 407 ns per k-block and 4.6, 5.2 and 6.9 us
// besides with 64, 128 and 256 columns; with several tiles per SM (16 x 120 x 160) a k-block takes 360 to 410 ns, which the choice
// between forms is about.
constexpr TileForm CONV_64 = {64, BM, 24576, 1, 380, 5000, 1200}, CONV_128 = {128, BM, 32768, 1, 390, 5600, 1800},
                   CONV_256 = {256, BM, 49152, 1, 430, 6500, 3400};

template <int BN, int STAGES>
int launch_conv(const CUtensorMap& tmB, GemmParams& p, const ConvGeom& g, int splits, cudaStream_t stream) {
  constexpr size_t smem = (size_t)STAGES * (BM * BK * 2 + BN * BK * 2) + CONV_EPI_WARPS * EPI_STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static_assert(smem <= 232448, "shared memory budget of one CTA");
  set_vec(p);
  p.tiles_m = ceil_div(p.M, BM);
  p.tiles_n = ceil_div(p.N, BN);
  p.tile_rows = BM;
  p.num_kb = ceil_div(p.K, BK);
  p.kb_per_split = ceil_div(p.num_kb, splits);
  p.splits = ceil_div(p.num_kb, p.kb_per_split);
  const int items = p.tiles_m * p.tiles_n * p.splits;
  const int grid = items < sm_count() ? items : sm_count();
  typedef void (*Kernel)(CUtensorMap, GemmParams, ConvGeom);
  static const Kernel kernels[3] = {conv_gemm_kernel<BN, STAGES, EPI_PLAIN>, conv_gemm_kernel<BN, STAGES, EPI_RELU>,
                                    conv_gemm_kernel<BN, STAGES, EPI_F32>};
  static bool configured[3] = {};
  const EpiMode mode = epi_mode(p, p.splits > 1);
  const int k = mode == EPI_F32 ? 2 : (mode == EPI_PLAIN ? 0 : 1);
  if (!configured[k]) {
    NB_CUDA(cudaFuncSetAttribute(kernels[k], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured[k] = true;
  }
  kernels[k]<<<grid, CONV_THREADS, smem, stream>>>(tmB, p, g);
  NB_LAUNCH_CHECK();
  return finish_split(p, BN, stream);
}

// B operand: `inner` contiguous elements of `outer` rows with pitch ld; K-major tiles take BN rows per box
int conv_any(const ConvGeom& g, GemmParams& p, const void* Bmat, long long inner, long long outer, long long ld, void* workspace,
             long long workspace_bytes, cudaStream_t s) {
  const bool have_ws = workspace && workspace_bytes > NB_GEMM_WS_COUNTERS * 4 + (1 << 20);
  const long long ws_bytes = have_ws ? workspace_bytes - NB_GEMM_WS_COUNTERS * 4 : 0;
  p.ws = have_ws ? (float*)((char*)workspace + NB_GEMM_WS_COUNTERS * 4) : nullptr;
  const int num_kb = ceil_div(p.K, BK), sms = sm_count();
  int splits, sp, BN = 64;
  long long best = best_split(CONV_64, p.M, p.N, num_kb, ws_bytes, sms, &splits);
  for (const TileForm* f : {&CONV_128, &CONV_256}) {
    if (p.N <= f->bn / 2) break;
    const long long t = best_split(*f, p.M, p.N, num_kb, ws_bytes, sms, &sp);
    if (t < best) { best = t; BN = f->bn; splits = sp; }
  }
  CUtensorMap tmB;
  const int rc = make_tmap_bf16(&tmB, Bmat, inner, outer, ld, 64, g.mirror ? BN : 64);
  if (rc) return rc;
  if (BN == 256) return launch_conv<256, 4>(tmB, p, g, splits, s);
  if (BN == 128) return launch_conv<128, 6>(tmB, p, g, splits, s);
  return launch_conv<64, 6>(tmB, p, g, splits, s);
}

int conv_geom(ConvGeom& g, const void* x, int B, int H, int W, int C, int KH, int KW, int stride, int pad) {
  if (B <= 0 || H <= 0 || W <= 0 || C <= 0 || C % 8 || KH <= 0 || KW <= 0 || stride <= 0 || pad < 0) return NB_ERR_BAD_ARG;
  if (H + 2 * pad < KH || W + 2 * pad < KW) return NB_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(x) & 15) return NB_ERR_UNALIGNED;
  if (!conv_fits(B, H, W, C, KH, KW, stride, pad)) return NB_ERR_TOO_LARGE;
  g.x = x;
  conv_geom_set(g, B, H, W, C, KH, KW, stride, pad);
  return NB_OK;
}

}  // namespace

NB_BOUNDS_REGISTER(conv_gemm)

extern "C" {

// y[B·OH·OW, OC] = act(patches(x) · W + bias), act none or ReLU: x NHWC bf16 [B, H, W, C], C % 8 == 0.  mirror = 0: W in GEMM layout
// [KH·KW·C, OC] (row pitch ldw).  mirror = 1 (data gradient of a stride-1 layer): x is dy, C % 64 == 0, and W is that layer's
// weight [KH·KW·OC, C], read with its taps from the last to the first.
int nb_conv_gemm(const void* x, const void* Wt, void* y, int B, int H, int W, int C, int OC, int KH, int KW, int stride, int pad,
                 int mirror, int ldw, int ldy, const float* bias, int act, unsigned int* status, void* workspace,
                 long long workspace_bytes, void* stream) {
  ConvGeom g;
  const int rc = conv_geom(g, x, B, H, W, C, KH, KW, stride, pad);
  if (rc) return rc;
  if (OC <= 0 || (mirror && (C % 64 || stride != 1)) || (act != NB_ACT_NONE && act != NB_ACT_RELU)) return NB_ERR_BAD_ARG;
  g.mirror = mirror;
  GemmParams p = {};
  p.M = g.pixels; p.N = OC; p.K = g.taps * C;
  p.b_mn = !mirror;
  p.ldd = ldy;
  p.act = act;
  p.alpha = 1.f;
  p.D = y; p.bias = bias; p.status = status;
  if (mirror) return conv_any(g, p, Wt, C, (long long)g.taps * OC, ldw, workspace, workspace_bytes, (cudaStream_t)stream);
  return conv_any(g, p, Wt, OC, p.K, ldw, workspace, workspace_bytes, (cudaStream_t)stream);
}

// dW[KH·KW·C, OC] += patches(x)^T · dy: dy bf16 [B·OH·OW, OC] (row pitch ld_dy), dW fp32 (row pitch ld_dw)
int nb_conv_gemm_wgrad(const void* x, const void* dy, float* dW, int B, int H, int W, int C, int OC, int KH, int KW, int stride,
                       int pad, int ld_dy, int ld_dw, unsigned int* status, void* workspace, long long workspace_bytes,
                       void* stream) {
  ConvGeom g;
  const int rc = conv_geom(g, x, B, H, W, C, KH, KW, stride, pad);
  if (rc) return rc;
  if (OC <= 0) return NB_ERR_BAD_ARG;
  g.wgrad = 1;
  GemmParams p = {};
  p.M = g.taps * C; p.N = OC; p.K = g.pixels;
  p.a_mn = p.b_mn = 1;
  p.ldd = ld_dw;
  p.out_f32 = p.accumulate = 1;
  p.alpha = 1.f;
  p.D = dW; p.status = status;
  return conv_any(g, p, dy, OC, g.pixels, ld_dy, workspace, workspace_bytes, (cudaStream_t)stream);
}

}  // extern "C"
