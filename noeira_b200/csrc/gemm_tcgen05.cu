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
#include "gemm_tile.cuh"

namespace {

using namespace nb;
using namespace nbgemm;

constexpr int NUM_THREADS = 96 + 32 * EPI_WARPS;     // A loads, MMA, B loads, epilogue
constexpr int NUM_THREADS2 = 64 + 32 * EPI_WARPS;    // CTA pairs: loads, MMA, epilogue

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
      if (!warp_wait_or_abort(&tfull_bar[acc], acc_phase, abort_flag, p.status, 4)) { ok = false; *abort_flag = 1; break; }
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
      if (!warp_wait_or_abort(&tfull_bar[acc], acc_phase, abort_flag, p.status, 24)) { ok = false; *abort_flag = 1; break; }
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

// Epilogue for 16 consecutive columns of one output row, in two phases so that the global loads it needs (the saved
// activation for a fused derivative, the old output when accumulating) can be issued one chunk ahead of their use:
// a chunk costs a DRAM / L2 round trip otherwise, which made narrow-K GEMMs epilogue-bound.
struct EpiPrefetch {
  uint4 aux[2];   // 16 bf16 of the saved tensor
  float4 old[4];  // 16 fp32 of the previous output (accumulate)
};

__device__ __forceinline__ void epilogue_prefetch16(const GemmParams& p, int row, int col0, bool active, EpiPrefetch& pf) {
  if (!active || col0 + 16 > p.N) return;
  if (p.dact && p.vec_aux) {
    const __nv_bfloat16* ax = p.aux + (size_t)row * p.ld_aux + col0;
    pf.aux[0] = __ldg(reinterpret_cast<const uint4*>(ax));
    pf.aux[1] = __ldg(reinterpret_cast<const uint4*>(ax + 8));
  }
  if (p.out_f32 && p.accumulate && p.vec_d) {
    const float* o = reinterpret_cast<const float*>(p.D) + (size_t)row * p.ldd + col0;
#pragma unroll
    for (int j = 0; j < 4; ++j) pf.old[j] = *reinterpret_cast<const float4*>(o + 4 * j);
  }
}

// direct store of 16 columns by the thread that owns them (second phase of a split-K GEMM)
__device__ __forceinline__ void epilogue_store16(const GemmParams& p, int row, int col0, float (&v)[16],
                                                 const EpiPrefetch& pf) {
  const bool full = (col0 + 16 <= p.N);
  float sv[16];
  if (p.dact) {
    if (full && p.vec_aux) {
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
    if (full && p.vec_bias) {
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
    if (full && p.vec_d) {
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
    if (full && p.vec_d) {
#pragma unroll
      for (int j = 0; j < 16; j += 8) *reinterpret_cast<uint4*>(o + j) = pack8f(v + j);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (col0 + j < p.N) o[j] = __float2bfloat16(v[j]);
    }
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
  if (col0 + 4 <= p.N && p.vec_d) {
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
int g_two_cta_mode = 0;  // 0 = by expected time, 1 = never, 2 = whenever the shape allows it

}  // namespace

int nbgemm::finish_split(const GemmParams& p, int BN, cudaStream_t stream) {
  if (p.splits <= 1) return NB_OK;
  const long long rows = (long long)p.tiles_m * p.tiles_n * p.tile_rows;
  if (p.out_f32 && !p.bias && !p.act && !p.dact)
    splitk_reduce_f32_kernel<<<(unsigned)((rows * (BN / 4) + 255) / 256), 256, 0, stream>>>(p, BN);
  else
    splitk_reduce_kernel<<<(unsigned)((rows * (BN / 16) + 127) / 128), 128, 0, stream>>>(p, BN);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

namespace {

// `splits`: wanted number of ranges of k-blocks (the workspace holds their partial tiles)
template <int BN, int STAGES>
int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, GemmParams& p, int splits, cudaStream_t stream) {
  constexpr size_t smem = (size_t)STAGES * (BM * BK * 2 + BN * BK * 2) + EPI_WARPS * EPI_STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static_assert(smem <= 232448, "shared memory budget of one CTA");
  set_vec(p);
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
  set_vec(p);
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
  // workspace: fp32 partial tiles behind NB_GEMM_WS_COUNTERS words (gemm_api.h)
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
  p.ws = have_ws ? (float*)((char*)workspace + NB_GEMM_WS_COUNTERS * 4) : nullptr;
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

}  // extern "C"
