// Convolution support kernels for the NHWC bf16 path: patch matrix (im2col) for transposed convolutions and for callers that
// ask for it (the convolution itself gathers its patches, conv_gemm_tcgen05.cu), its adjoint as a deterministic gather (no
// atomics) for strided data gradients, BatchNorm2D in training mode (per-channel batch
// statistics, fused scale/shift/ReLU/residual), max pooling, and the uint8 camera-image normaliser.
//
// A convolution is  Y[B·OH·OW, OC] = col[B·OH·OW, KH·KW·C] · W[KH·KW·C, OC]  with the bias / ReLU in the GEMM
// epilogue; dgrad is  dcol = dY · Wᵀ  followed by the gather below; wgrad is  dW += colᵀ · dY  (TN GEMM).
// Reference: im2col + GEMM (noeira/nn/primitives/conv2d.mojo:437,652,723) or cuDNN (nn/core/cudnn_conv.mojo),
// BatchNorm 2-D NHWC kernels (batch_norm_2d.mojo:550-1250), max_pool_2d.mojo, act/data_gpu.mojo:157 (gather +
// /255 + ImageNet mean/std).
#include "common.cuh"

namespace {
using namespace nb;

// col[m, (kh*KW + kw)*C + c] = x[b, oh*s - p + kh, ow*s - p + kw, c]  (zero outside); C % 8 == 0, 16-byte copies
__global__ void __launch_bounds__(256)
im2col_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ col, int B, int H, int W, int C, int KH,
              int KW, int stride, int pad, int OH, int OW, int ldc) {
  const int cv = C / 8;
  const long long total = (long long)B * OH * OW * KH * KW * cv;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    const int c8 = (int)(i % cv);
    long long r = i / cv;
    const int kw = (int)(r % KW); r /= KW;
    const int kh = (int)(r % KH); r /= KH;
    const int ow = (int)(r % OW); r /= OW;
    const int oh = (int)(r % OH);
    const int b = (int)(r / OH);
    const int ih = oh * stride - pad + kh, iw = ow * stride - pad + kw;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (ih >= 0 && ih < H && iw >= 0 && iw < W)
      v = *reinterpret_cast<const uint4*>(x + (((size_t)b * H + ih) * W + iw) * C + c8 * 8);
    const size_t m = ((size_t)b * OH + oh) * OW + ow;
    *reinterpret_cast<uint4*>(col + m * ldc + ((size_t)kh * KW + kw) * C + c8 * 8) = v;
  }
}

// dx[b, h, w, c] = Σ_{kh,kw : (h+p-kh) % s == 0, ...} dcol[b, oh, ow, kh, kw, c]   (gather: one writer per element).  A block owns
// part of one input row, a thread 8 channels of a pixel; only the taps of the pixel's residue modulo the stride are visited.
// 19200 x 1152 -> 16 x 60 x 80 x 128 (44 MB read, 20 MB written): 25.5 us with 64-bit divisions and all taps tested, 14.3 now.
__global__ void __launch_bounds__(256)
col2im_kernel(const __nv_bfloat16* __restrict__ dcol, __nv_bfloat16* __restrict__ dx, int H, int W, int C, int KH, int KW,
              int stride, int pad, int OH, int OW, int ldc) {
  const int cv = C / 8, b = blockIdx.x / H, h = blockIdx.x - b * H;
  for (int i = blockIdx.y * 256 + threadIdx.x; i < W * cv; i += gridDim.y * 256) {
    const int w = i / cv, c8 = i - w * cv;
    float acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
    const int th = h + pad, tw = w + pad;
    // the last output row / column whose window starts at or before this pixel, then backwards through the windows
    for (int oh = min(OH - 1, th / stride); oh >= 0 && th - oh * stride < KH; --oh) {
      const int kh = th - oh * stride;
      for (int ow = min(OW - 1, tw / stride); ow >= 0 && tw - ow * stride < KW; --ow) {
        const int kw = tw - ow * stride;
        const size_t m = ((size_t)b * OH + oh) * OW + ow;
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(dcol + m * ldc + ((size_t)kh * KW + kw) * C + c8 * 8));
        const __nv_bfloat162* hp = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          acc[2 * k] += __low2float(hp[k]);
          acc[2 * k + 1] += __high2float(hp[k]);
        }
      }
    }
    uint4 o;
    __nv_bfloat162 h0 = __floats2bfloat162_rn(acc[0], acc[1]), h1 = __floats2bfloat162_rn(acc[2], acc[3]),
                   h2 = __floats2bfloat162_rn(acc[4], acc[5]), h3 = __floats2bfloat162_rn(acc[6], acc[7]);
    o.x = *reinterpret_cast<uint32_t*>(&h0); o.y = *reinterpret_cast<uint32_t*>(&h1);
    o.z = *reinterpret_cast<uint32_t*>(&h2); o.w = *reinterpret_cast<uint32_t*>(&h3);
    *reinterpret_cast<uint4*>(dx + (((size_t)b * H + h) * W + w) * C + c8 * 8) = o;
  }
}

// ---- BatchNorm2D over an [M, C] view (M = B·H·W).  Every pass is bound by DRAM bytes, so all of them share one mapping: a
// thread owns 8 channels (16 bytes) for good and walks down the rows, which keeps the channel's parameters in registers and
// leaves no division in the loop; BN_UNROLL rows are in flight per thread.  16 x 120 x 160 x 64 (39 MB a tensor), with scalar
// parameter loads and a 64-bit remainder per vector before: apply 25.9 us -> 19.5, statistics forward and backward together 47 -> 31,
// backward dx 35.5 -> 30.3 (16 x 240 x 320 x 64: 109 us = 5.7 TB/s).
constexpr int BN_UNROLL = 4;

struct BnMap {
  int ch, rows;        // first channel, rows per sweep of the grid
  long long row;       // first row
  bool active;
};
// `lanes` threads span a row (or 256 of the vectors of a wide one, blockIdx.y the next 256)
__device__ __forceinline__ BnMap bn_map(int C, int blk, int nblk) {
  const int cv = C / 8, lanes = cv < 256 ? cv : 256, per = 256 / lanes;
  const int l = threadIdx.x % lanes, r = threadIdx.x / lanes;
  BnMap m;
  m.ch = (blockIdx.y * lanes + l) * 8;
  m.row = (long long)blk * per + r;
  m.rows = nblk * per;
  m.active = r < per && m.ch < C;
  return m;
}
__device__ __forceinline__ void bn_unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int k = 0; k < 4; ++k) { f[2 * k] = __low2float(h[k]); f[2 * k + 1] = __high2float(h[k]); }
}
__device__ __forceinline__ uint4 bn_pack8(const float (&o)[8]) {
  uint4 vo;
  __nv_bfloat162 h0 = __floats2bfloat162_rn(o[0], o[1]), h1 = __floats2bfloat162_rn(o[2], o[3]),
                 h2 = __floats2bfloat162_rn(o[4], o[5]), h3 = __floats2bfloat162_rn(o[6], o[7]);
  vo.x = *reinterpret_cast<uint32_t*>(&h0); vo.y = *reinterpret_cast<uint32_t*>(&h1);
  vo.z = *reinterpret_cast<uint32_t*>(&h2); vo.w = *reinterpret_cast<uint32_t*>(&h3);
  return vo;
}
__device__ __forceinline__ void load8f(const float* p, float (&f)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) f[k] = p[k];
}

// Stage 1: per-block Σa, Σa² (BWD = false) or Σg, Σg·x̂ with g = dy masked by the ReLU output (BWD = true).
template <bool BWD>
__global__ void __launch_bounds__(256)
bn_reduce_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ x, const float* __restrict__ mean,
                 const float* __restrict__ rstd, const __nv_bfloat16* __restrict__ relu_out, float* __restrict__ p0,
                 float* __restrict__ p1, long long M, int C) {
  __shared__ float s0[256][9], s1[256][9];
  const BnMap m = bn_map(C, blockIdx.x, gridDim.x);
  float a0[8], a1[8], mu[8], rs[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a0[k] = a1[k] = 0.f;
  if (m.active) {
    if (BWD) { load8f(mean + m.ch, mu); load8f(rstd + m.ch, rs); }
    const bool masked = BWD && relu_out;
    for (long long r0 = m.row; r0 < M; r0 += BN_UNROLL * (long long)m.rows) {
      uint4 va[BN_UNROLL], vx[BN_UNROLL], vo[BN_UNROLL];
#pragma unroll
      for (int u = 0; u < BN_UNROLL; ++u) {
        const long long r = r0 + (long long)u * m.rows;
        if (r < M) {
          const size_t o = (size_t)r * C + m.ch;
          va[u] = __ldg(reinterpret_cast<const uint4*>(a + o));
          if (BWD) vx[u] = __ldg(reinterpret_cast<const uint4*>(x + o));
          if (masked) vo[u] = __ldg(reinterpret_cast<const uint4*>(relu_out + o));
        }
      }
#pragma unroll
      for (int u = 0; u < BN_UNROLL; ++u) {
        if (r0 + (long long)u * m.rows >= M) break;
        float fa[8], fx[8], fo[8];
        bn_unpack8(va[u], fa);
        if (BWD) {
          bn_unpack8(vx[u], fx);
          if (masked) bn_unpack8(vo[u], fo);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float g = (!masked || fo[k] > 0.f) ? fa[k] : 0.f;
            a0[k] += g;
            a1[k] += g * (fx[k] - mu[k]) * rs[k];
          }
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) { a0[k] += fa[k]; a1[k] += fa[k] * fa[k]; }
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) { s0[threadIdx.x][k] = a0[k]; s1[threadIdx.x][k] = a1[k]; }
  __syncthreads();
  const int cv = C / 8, lanes = cv < 256 ? cv : 256, per = 256 / lanes;
  for (int i = threadIdx.x; i < lanes * 8; i += 256) {
    const int l = i >> 3, k = i & 7, c = blockIdx.y * lanes * 8 + i;
    float t0 = 0.f, t1 = 0.f;
    for (int g = 0; g < per; ++g) { t0 += s0[g * lanes + l][k]; t1 += s1[g * lanes + l][k]; }
    if (c < C) { p0[(size_t)blockIdx.x * C + c] = t0; p1[(size_t)blockIdx.x * C + c] = t1; }
  }
}

// Σ over the blocks' partials of 32 channels per block: 32 warps take every 32nd partial each, then the 32 sums are added in
// order.  (One thread per channel walked all of them, a chain of up to 1024 dependent additions: 67 us, 8.4 with 8 warps,
// 4.5 with 32.)
constexpr int BN_FIN_WARPS = 32;
__device__ __forceinline__ bool bn_finish_sums(const float* p0, const float* p1, int split, int C, int& c, float& s, float& ss) {
  __shared__ float q0[BN_FIN_WARPS][33], q1[BN_FIN_WARPS][33];
  const int l = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  c = blockIdx.x * 32 + l;
  float t0 = 0.f, t1 = 0.f;
  if (c < C) {
#pragma unroll 8
    for (int k = w; k < split; k += warps) { t0 += p0[(size_t)k * C + c]; t1 += p1[(size_t)k * C + c]; }
  }
  q0[w][l] = t0;
  q1[w][l] = t1;
  __syncthreads();
  s = ss = 0.f;
  if (w == 0) {
#pragma unroll 8
    for (int k = 0; k < warps; ++k) { s += q0[k][l]; ss += q1[k][l]; }
  }
  return w == 0 && c < C;
}
// forward finish: mean, rstd, running stats
__global__ void __launch_bounds__(32 * BN_FIN_WARPS)
bn_stats_finish_kernel(const float* __restrict__ p0, const float* __restrict__ p1, int split, long long M, int C, float eps,
                       float momentum, float* __restrict__ mean, float* __restrict__ rstd, float* __restrict__ run_mean,
                       float* __restrict__ run_var) {
  int c;
  float s, ss;
  if (!bn_finish_sums(p0, p1, split, C, c, s, ss)) return;
  const float mu = s / M, var = fmaxf(ss / M - mu * mu, 0.f);
  mean[c] = mu;
  rstd[c] = rsqrtf(var + eps);
  if (run_mean) {
    run_mean[c] = (1.f - momentum) * run_mean[c] + momentum * mu;
    run_var[c] = (1.f - momentum) * run_var[c] + momentum * var * ((float)M / fmaxf(M - 1.f, 1.f));
  }
}
// backward finish: dgamma += Σdy·x̂, dbeta += Σdy ; keeps the sums for the dx kernel
__global__ void __launch_bounds__(32 * BN_FIN_WARPS)
bn_bwd_finish_kernel(const float* __restrict__ p0, const float* __restrict__ p1, int split, int C, float* __restrict__ sum_dy,
                     float* __restrict__ sum_dyx, float* __restrict__ dgamma, float* __restrict__ dbeta) {
  int c;
  float s, ss;
  if (!bn_finish_sums(p0, p1, split, C, c, s, ss)) return;
  sum_dy[c] = s;
  sum_dyx[c] = ss;
  if (dgamma) dgamma[c] += ss;
  if (dbeta) dbeta[c] += s;
}

// y = relu?( (x - mean) * rstd * gamma + beta + residual? ).  run_mean given (inference): the statistics are the running ones, and
// `mean` and `rstd` receive what was used, for a backward pass that may come after the running ones have changed.
__global__ void __launch_bounds__(256)
bn_apply_kernel(const __nv_bfloat16* __restrict__ x, float* __restrict__ mean, float* __restrict__ rstd,
                const float* __restrict__ run_mean, const float* __restrict__ run_var, float eps, const float* __restrict__ gamma,
                const float* __restrict__ beta, const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ y, long long M, int C,
                int relu) {
  const BnMap m = bn_map(C, blockIdx.x, gridDim.x);
  if (!m.active) return;
  float mu[8], rs[8], ga[8], be[8];
  if (!run_mean) {
    load8f(mean + m.ch, mu);
    load8f(rstd + m.ch, rs);
  } else {
    load8f(run_mean + m.ch, mu);
    load8f(run_var + m.ch, rs);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      rs[k] = rsqrtf(rs[k] + eps);
      if (m.row == 0) { mean[m.ch + k] = mu[k]; rstd[m.ch + k] = rs[k]; }
    }
  }
  load8f(gamma + m.ch, ga);
  load8f(beta + m.ch, be);
  for (long long r0 = m.row; r0 < M; r0 += BN_UNROLL * (long long)m.rows) {
    uint4 vx[BN_UNROLL], vr[BN_UNROLL];
#pragma unroll
    for (int u = 0; u < BN_UNROLL; ++u) {
      const long long r = r0 + (long long)u * m.rows;
      if (r < M) {
        vx[u] = __ldg(reinterpret_cast<const uint4*>(x + (size_t)r * C + m.ch));
        if (res) vr[u] = __ldg(reinterpret_cast<const uint4*>(res + (size_t)r * C + m.ch));
      }
    }
#pragma unroll
    for (int u = 0; u < BN_UNROLL; ++u) {
      const long long r = r0 + (long long)u * m.rows;
      if (r >= M) break;
      float fx[8], fr[8];
      bn_unpack8(vx[u], fx);
      if (res) bn_unpack8(vr[u], fr);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float o = (fx[k] - mu[k]) * rs[k] * ga[k] + be[k] + (res ? fr[k] : 0.f);
        fx[k] = relu ? fmaxf(o, 0.f) : o;
      }
      *reinterpret_cast<uint4*>(y + (size_t)r * C + m.ch) = bn_pack8(fx);
    }
  }
}

// dx = gamma·rstd·( g − Σg/M − x̂·Σ(g·x̂)/M ),  g = dy masked by the ReLU output; dres = g (residual branch)
__global__ void __launch_bounds__(256)
bn_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                 const __nv_bfloat16* __restrict__ relu_out, const float* __restrict__ mean,
                 const float* __restrict__ rstd, const float* __restrict__ gamma, const float* __restrict__ sum_dy,
                 const float* __restrict__ sum_dyx, __nv_bfloat16* __restrict__ dx, __nv_bfloat16* __restrict__ dres,
                 long long M, int C) {
  const BnMap m = bn_map(C, blockIdx.x, gridDim.x);
  if (!m.active) return;
  const float invM = 1.f / (float)M;
  float mu[8], rs[8], gr[8], k1[8], k2[8];
  load8f(mean + m.ch, mu);
  load8f(rstd + m.ch, rs);
  load8f(gamma + m.ch, gr);
  load8f(sum_dy + m.ch, k1);
  load8f(sum_dyx + m.ch, k2);
#pragma unroll
  for (int k = 0; k < 8; ++k) { gr[k] *= rs[k]; k1[k] *= invM; }
  for (long long r0 = m.row; r0 < M; r0 += BN_UNROLL * (long long)m.rows) {
    uint4 vd[BN_UNROLL], vx[BN_UNROLL], vo[BN_UNROLL];
#pragma unroll
    for (int u = 0; u < BN_UNROLL; ++u) {
      const long long r = r0 + (long long)u * m.rows;
      if (r < M) {
        const size_t o = (size_t)r * C + m.ch;
        vd[u] = __ldg(reinterpret_cast<const uint4*>(dy + o));
        vx[u] = __ldg(reinterpret_cast<const uint4*>(x + o));
        if (relu_out) vo[u] = __ldg(reinterpret_cast<const uint4*>(relu_out + o));
      }
    }
#pragma unroll
    for (int u = 0; u < BN_UNROLL; ++u) {
      const long long r = r0 + (long long)u * m.rows;
      if (r >= M) break;
      float g[8], fx[8], fo[8];
      bn_unpack8(vd[u], g);
      bn_unpack8(vx[u], fx);
      if (relu_out) bn_unpack8(vo[u], fo);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (relu_out && !(fo[k] > 0.f)) g[k] = 0.f;
        const float xh = (fx[k] - mu[k]) * rs[k];
        fx[k] = gr[k] * (g[k] - k1[k] - xh * k2[k] * invM);
      }
      const size_t o = (size_t)r * C + m.ch;
      *reinterpret_cast<uint4*>(dx + o) = bn_pack8(fx);
      if (dres) *reinterpret_cast<uint4*>(dres + o) = bn_pack8(g);
    }
  }
}

// grid of the row-walking kernels: up to `blocks` blocks, each thread with a round of BN_UNROLL rows, or with fewer while that
// leaves less than BN_FIN_WARPS blocks (the finish takes a partial per warp).  Forward + backward, us, four rows / fewer: 1024 x 8
// 18.0 / 16.0, 64 x 256 17.3 / 15.4; more blocks than that cost more in the finish (1024 x 512 with 149 blocks 19.5 / 23.7)
inline dim3 bn_grid(long long M, int C, int blocks) {
  const int cv = C / 8, lanes = cv < 256 ? cv : 256, per = 256 / lanes;
  const long long one = ceil_div_ll(M, per), four = ceil_div_ll(M, (long long)per * BN_UNROLL);
  const long long b = four >= BN_FIN_WARPS ? four : (one < BN_FIN_WARPS ? one : BN_FIN_WARPS);
  return dim3((unsigned)(b < 1 ? 1 : (b > blocks ? blocks : b)), (unsigned)ceil_div(cv, lanes));
}
// a warp per partial
inline int bn_fin_threads(unsigned split) { return 32 * (int)(split < (unsigned)BN_FIN_WARPS ? split : (unsigned)BN_FIN_WARPS); }

// Average pooling with window K, stride = K (non-overlapping) on NHWC: forward averages, backward spreads dy / K².
// `back != 0`: `src` is dy [B, OH, OW, C] and `dst` is dx [B, H, W, C] (pixels outside the pooled area get zero).
__global__ void __launch_bounds__(256)
avgpool_kernel(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst, int B, int H, int W, int C, int K, int OH,
               int OW, int back) {
  const long long total = back ? (long long)B * H * W * C : (long long)B * OH * OW * C, step = (long long)gridDim.x * blockDim.x;
  const float inv = 1.f / (float)(K * K);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    const int c = (int)(i % C);
    long long r = i / C;
    if (back) {
      const int w = (int)(r % W); r /= W;
      const int h = (int)(r % H);
      const int b = (int)(r / H);
      const int oh = h / K, ow = w / K;
      dst[i] = (oh < OH && ow < OW) ? __float2bfloat16(__bfloat162float(src[(((long long)b * OH + oh) * OW + ow) * C + c]) * inv)
                                    : __float2bfloat16(0.f);
    } else {
      const int ow = (int)(r % OW); r /= OW;
      const int oh = (int)(r % OH);
      const int b = (int)(r / OH);
      float acc = 0.f;
      for (int kh = 0; kh < K; ++kh)
        for (int kw = 0; kw < K; ++kw)
          acc += __bfloat162float(src[(((long long)b * H + oh * K + kh) * W + ow * K + kw) * C + c]);
      dst[i] = __float2bfloat16(acc * inv);
    }
  }
}
// Nearest-neighbour upsampling by an integer factor S on NHWC: forward replicates, backward sums the S x S block.
__global__ void __launch_bounds__(256)
upsample_kernel(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst, int B, int H, int W, int C, int S, int back) {
  const int OH = H * S, OW = W * S;
  const long long total = back ? (long long)B * H * W * C : (long long)B * OH * OW * C, step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    const int c = (int)(i % C);
    long long r = i / C;
    if (back) {
      const int w = (int)(r % W); r /= W;
      const int h = (int)(r % H);
      const int b = (int)(r / H);
      float acc = 0.f;
      for (int kh = 0; kh < S; ++kh)
        for (int kw = 0; kw < S; ++kw)
          acc += __bfloat162float(src[(((long long)b * OH + h * S + kh) * OW + w * S + kw) * C + c]);
      dst[i] = __float2bfloat16(acc);
    } else {
      const int ow = (int)(r % OW); r /= OW;
      const int oh = (int)(r % OH);
      const int b = (int)(r / OH);
      dst[i] = src[(((long long)b * H + oh / S) * W + ow / S) * C + c];
    }
  }
}

// 3x3 / stride 2 / pad 1 style max pooling on NHWC; idx stores the tap kh·K + kw of the maximum (the type's largest value:
// none), one byte wherever the taps fit.  A block owns part of one output row, a thread VEC consecutive channels of a pixel.
// Bound by DRAM bytes: 16 x 240 x 320 x 64 -> 120 x 160 reads 157 MB and writes 39 + 20 MB.  One element per thread with
// 64-bit divisions and 4-byte offsets took 270 us, this form 70 us; the backward 194 us -> 144 (54 for the 3x3 / 2 window, below).
// KC != 0: the window size at compile time, so that all loads of a window are in flight together (3: the window of a
// residual network's stem).
template <int VEC, typename I, int KC>
__global__ void __launch_bounds__(256)
maxpool_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, I* __restrict__ idx, int H, int W, int C,
                   int K_, int stride, int pad, int OH, int OW) {
  const int CV = C / VEC, b = blockIdx.x / OH, oh = blockIdx.x - b * OH;
  for (int i = blockIdx.y * 256 + threadIdx.x; i < OW * CV; i += gridDim.y * 256) {
    const int ow = i / CV, c0 = (i - ow * CV) * VEC;
    float best[VEC];
    __align__(8) I tap[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) { best[j] = -INFINITY; tap[j] = (I)-1; }
    const int K = KC ? KC : K_, h0 = oh * stride - pad, w0 = ow * stride - pad;
    const __nv_bfloat16* base = x + (((ptrdiff_t)b * H + h0) * W + w0) * C + c0;     // of the window's corner, maybe outside
    auto take = [&](const uint4& u, int kh, int kw) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const float v = (j & 1) ? __high2float(h[j >> 1]) : __low2float(h[j >> 1]);
        if (v > best[j]) { best[j] = v; tap[j] = (I)(kh * K + kw); }
      }
    };
    auto load = [&](int kh, int kw) {
      const __nv_bfloat16* q = base + ((ptrdiff_t)kh * W + kw) * C;
      uint4 u = make_uint4(0, 0, 0, 0);
      if (VEC == 8) u = __ldg(reinterpret_cast<const uint4*>(q));
      else *reinterpret_cast<__nv_bfloat16*>(&u) = *q;
      return u;
    };
    if (KC) {
      constexpr int KK = KC ? KC : 1;
      const uint4 lowest = make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);    // -inf: never the maximum
      uint4 u[KK][KK];
#pragma unroll
      for (int kh = 0; kh < KK; ++kh)
#pragma unroll
        for (int kw = 0; kw < KK; ++kw)
          u[kh][kw] = (h0 + kh >= 0 && h0 + kh < H && w0 + kw >= 0 && w0 + kw < W) ? load(kh, kw) : lowest;
#pragma unroll
      for (int kh = 0; kh < KK; ++kh)
#pragma unroll
        for (int kw = 0; kw < KK; ++kw) take(u[kh][kw], kh, kw);
    } else {
      for (int kh = max(0, -h0); kh < min(K, H - h0); ++kh)
        for (int kw = max(0, -w0); kw < min(K, W - w0); ++kw) take(load(kh, kw), kh, kw);
    }
    const size_t o = (((size_t)b * OH + oh) * OW + ow) * C + c0;
#pragma unroll
    for (int j = 0; j < VEC; j += 8) {
      if (VEC == 8) {
        const float (&f)[8] = reinterpret_cast<const float (&)[8]>(best);
        *reinterpret_cast<uint4*>(y + o) = bn_pack8(f);
        if (sizeof(I) == 1) *reinterpret_cast<uint2*>(idx + o) = *reinterpret_cast<const uint2*>(tap);
        else
#pragma unroll
          for (int q = 0; q < VEC; q += 4) *reinterpret_cast<int4*>(idx + o + q) = make_int4(tap[q], tap[q + 1], tap[q + 2], tap[q + 3]);
      } else {
        y[o] = __float2bfloat16(best[0]);
        idx[o] = tap[0];
      }
    }
  }
}
// dx = gather over the windows that contain the element (at most ceil(K/stride)^2 = 4 for 3x3 / 2): deterministic.
// One thread owns VEC consecutive channels of one input pixel; the candidate output range is computed directly instead of
// testing all K*K taps, and a window gives its gradient where its stored tap is the one that this pixel is for it.
// S1: the 3x3 / stride 1 window, whose nine windows are all loaded before the first is used (16 x 120 x 160 x 64: 74 us one by
// one, 54 so; 4 x 56 x 56 x 64: 6.4, 4.6).
template <int VEC, typename I, bool S1>
__global__ void __launch_bounds__(256)
maxpool_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const I* __restrict__ idx, __nv_bfloat16* __restrict__ dx, int H, int W,
                   int C, int K, int stride, int pad, int OH, int OW) {
  const int CV = C / VEC, b = blockIdx.x / H, h = blockIdx.x - b * H;
  for (int i = blockIdx.y * 256 + threadIdx.x; i < W * CV; i += gridDim.y * 256) {
    const int w = i / CV, c0 = (i - w * CV) * VEC;
    // output rows oh with oh*stride - pad <= h <= oh*stride - pad + K - 1
    const int oh_lo = max(0, (h + pad - K + stride) / stride), oh_hi = min(OH - 1, (h + pad) / stride);
    const int ow_lo = max(0, (w + pad - K + stride) / stride), ow_hi = min(OW - 1, (w + pad) / stride);
    float acc[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) acc[j] = 0.f;
    auto add = [&](const I (&id)[VEC], const uint4& g, I mine) {
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g);
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const float gv = (j & 1) ? __high2float(gh[j >> 1]) : __low2float(gh[j >> 1]);
        if (id[j] == mine) acc[j] += gv;
      }
    };
    auto load = [&](int oh, int ow, I (&id)[VEC], uint4& g) {
      const size_t o = (((size_t)b * OH + oh) * OW + ow) * C + c0;
      if (VEC == 8) {
        if (sizeof(I) == 1) *reinterpret_cast<uint2*>(id) = __ldg(reinterpret_cast<const uint2*>(idx + o));
        else
#pragma unroll
          for (int q = 0; q < VEC; q += 4) {
            const int4 v = __ldg(reinterpret_cast<const int4*>(idx + o + q));
            id[q] = (I)v.x; id[q + 1] = (I)v.y; id[q + 2] = (I)v.z; id[q + 3] = (I)v.w;
          }
        g = __ldg(reinterpret_cast<const uint4*>(dy + o));
      } else {
        id[0] = idx[o];
        *reinterpret_cast<__nv_bfloat16*>(&g) = dy[o];
      }
    };
    auto tap_of = [&](int oh, int ow) { return (I)((h + pad - oh * stride) * K + (w + pad - ow * stride)); };
    if (S1) {
      __align__(8) I id[9][VEC];
      uint4 g[9];
#pragma unroll
      for (int t = 0; t < 9; ++t) {
        const int oh = h + pad - t / 3, ow = w + pad - t % 3;              // this pixel is tap t of that window
        if (oh >= 0 && oh < OH && ow >= 0 && ow < OW) load(oh, ow, id[t], g[t]);
        else *reinterpret_cast<uint2*>(id[t]) = make_uint2(0xffffffffu, 0xffffffffu);     // no tap
      }
#pragma unroll
      for (int t = 8; t >= 0; --t) add(id[t], g[t], (I)t);                 // windows in row order, as below
    } else
    for (int oh = oh_lo; oh <= oh_hi; ++oh)
      for (int ow = ow_lo; ow <= ow_hi; ++ow) {
        __align__(8) I id[VEC];
        uint4 g = make_uint4(0, 0, 0, 0);
        load(oh, ow, id, g);
        add(id, g, tap_of(oh, ow));
      }
    __nv_bfloat16* d = dx + (((size_t)b * H + h) * W + w) * C + c0;
    if (VEC == 8) {
      const float (&f)[8] = reinterpret_cast<const float (&)[8]>(acc);
      *reinterpret_cast<uint4*>(d) = bn_pack8(f);
    } else {
      d[0] = __float2bfloat16(acc[0]);
    }
  }
}

// The 3x3 / stride 2 window (the layer's default) with 8 channels a thread.  With h' = h + pad, rows h' = 2a and 2a + 1 touch
// the windows oh = a − 1 (tap 2 for the first) and oh = a (taps 0 and 1), columns alike: a thread owns such a 2 x 2 block of
// pixels, loads its four windows once, and tests 9 (pixel, window) pairs where four threads tested 16.  The pass is bound by
// instructions, not bytes: the general kernel takes 144 us for 16 x 240 x 320 x 64, this one 54 us.
__global__ void __launch_bounds__(256)
maxpool_bwd_3s2_kernel(const __nv_bfloat16* __restrict__ dy, const unsigned char* __restrict__ idx, __nv_bfloat16* __restrict__ dx,
                       int H, int W, int C, int pad, int OH, int OW, int a0, int na, int nw) {
  const int CV = C / 8, b = blockIdx.x / na, ah = a0 + blockIdx.x - b * na;
  for (int i = blockIdx.y * 256 + threadIdx.x; i < nw * CV; i += gridDim.y * 256) {
    const int aw0 = i / CV, c0 = (i - aw0 * CV) * 8, aw = a0 + aw0;
    uint2 id[2][2];
    uint4 g[2][2];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int oh = ah - 1 + p, ow = aw - 1 + q;
        id[p][q] = make_uint2(0xffffffffu, 0xffffffffu);     // no tap
        if (oh >= 0 && oh < OH && ow >= 0 && ow < OW) {
          const size_t o = (((size_t)b * OH + oh) * OW + ow) * C + c0;
          id[p][q] = __ldg(reinterpret_cast<const uint2*>(idx + o));
          g[p][q] = __ldg(reinterpret_cast<const uint4*>(dy + o));
        }
      }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int h = 2 * ah + r - pad, w = 2 * aw + c - pad;
        if (h < 0 || h >= H || w < 0 || w >= W) continue;
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll
        for (int p = r; p < 2; ++p)
#pragma unroll
          for (int q = c; q < 2; ++q) {
            const uint32_t mine = (uint32_t)((r + 2 - 2 * p) * 3 + (c + 2 - 2 * q));
            const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g[p][q]);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t t = ((j < 4 ? id[p][q].x : id[p][q].y) >> (8 * (j & 3))) & 0xffu;
              const float gv = (j & 1) ? __high2float(gh[j >> 1]) : __low2float(gh[j >> 1]);
              if (t == mine) acc[j] += gv;
            }
          }
        *reinterpret_cast<uint4*>(dx + (((size_t)b * H + h) * W + w) * C + c0) = bn_pack8(acc);
      }
  }
}

// uint8 [B, 3, H, W] (CHW camera frames) → bf16 NHWC with C padded to 8: (x/255 − mean) / std.  PX pixels per thread (4 when
// an image is a whole number of 4-byte words): 4-byte loads, and the block's image comes from blockIdx.y, so that no
// division per pixel is left.  16 x 480 x 640 (15 MB in, 79 MB out): 35.4 us one pixel at a time, 25.8 now.
template <int PX>
__global__ void __launch_bounds__(256)
image_normalize_kernel(const unsigned char* __restrict__ img, __nv_bfloat16* __restrict__ out, long long HW, float m0,
                       float m1, float m2, float s0, float s1, float s2) {
  const long long px = ((long long)blockIdx.x * 256 + threadIdx.x) * PX;
  if (px >= HW) return;
  const unsigned char* p = img + (size_t)blockIdx.y * 3 * HW + px;
  __align__(4) unsigned char v[3][PX];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (PX == 4) *reinterpret_cast<uint32_t*>(v[c]) = __ldg(reinterpret_cast<const uint32_t*>(p + (size_t)c * HW));
    else v[c][0] = p[(size_t)c * HW];
  }
  __nv_bfloat16* o = out + ((size_t)blockIdx.y * HW + px) * 8;
#pragma unroll
  for (int i = 0; i < PX; ++i) {
    const float f[8] = {(v[0][i] * (1.f / 255.f) - m0) / s0, (v[1][i] * (1.f / 255.f) - m1) / s1, (v[2][i] * (1.f / 255.f) - m2) / s2,
                        0.f, 0.f, 0.f, 0.f, 0.f};
    *reinterpret_cast<uint4*>(o + i * 8) = bn_pack8(f);
  }
}

inline unsigned pool_blocks(int n) { return (unsigned)(n > 65535 * 256 ? 65535 : ceil_div(n, 256)); }
inline int g1(long long n) {
  long long b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 148 * 16 ? 148 * 16 : b));
}
}  // namespace

extern "C" {

int nb_im2col(const void* x, void* col, int B, int H, int W, int C, int KH, int KW, int stride, int pad, int OH, int OW,
              int ldc, void* stream) {
  if (C % 8 || ldc % 8) return NB_ERR_UNALIGNED;
  im2col_kernel<<<g1((long long)B * OH * OW * KH * KW * (C / 8)), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, (__nv_bfloat16*)col, B, H, W, C, KH, KW, stride, pad, OH, OW, ldc);
  NB_LAUNCH_CHECK();
  return NB_OK;
}
int nb_col2im(const void* dcol, void* dx, int B, int H, int W, int C, int KH, int KW, int stride, int pad, int OH, int OW,
              int ldc, void* stream) {
  if (C % 8 || ldc % 8) return NB_ERR_UNALIGNED;
  if (B <= 0 || H <= 0 || W <= 0 || C <= 0) return NB_OK;   // an empty batch: a grid of no blocks is an error
  col2im_kernel<<<dim3((unsigned)(B * H), pool_blocks(W * (C / 8))), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)dcol, (__nv_bfloat16*)dx, H, W, C, KH, KW, stride, pad, OH, OW, ldc);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

// most blocks of the statistics pass = most partials: four blocks per SM
int nb_bn_split(long long M) { return (int)(M < 1 ? 1 : (M > 592 ? 592 : M)); }
// partials: 2 * nb_bn_split(M) * C floats.  mean, rstd: the statistics of this call (inference: the running ones), for nb_bn_bwd
int nb_bn_fwd(const void* x, const float* gamma, const float* beta, const void* residual, void* y, float* mean, float* rstd,
              float* run_mean, float* run_var, float* partials, long long M, int C, float eps, float momentum, int relu,
              int training, void* stream) {
  if (C % 8) return NB_ERR_UNALIGNED;
  cudaStream_t s = (cudaStream_t)stream;
  if (training) {
    const dim3 g = bn_grid(M, C, nb_bn_split(M));
    float* p0 = partials;
    float* p1 = partials + (size_t)g.x * C;
    bn_reduce_kernel<false><<<g, 256, 0, s>>>((const __nv_bfloat16*)x, nullptr, nullptr, nullptr, nullptr, p0, p1, M, C);
    NB_LAUNCH_CHECK();
    bn_stats_finish_kernel<<<ceil_div(C, 32), bn_fin_threads(g.x), 0, s>>>(p0, p1, (int)g.x, M, C, eps, momentum, mean, rstd, run_mean,
                                                          run_var);
    NB_LAUNCH_CHECK();
  }
  bn_apply_kernel<<<bn_grid(M, C, 1 << 20), 256, 0, s>>>((const __nv_bfloat16*)x, mean, rstd, training ? nullptr : run_mean,
                                                        run_var, eps, gamma, beta, (const __nv_bfloat16*)residual,
                                                        (__nv_bfloat16*)y, M, C, relu);
  NB_LAUNCH_CHECK();
  return NB_OK;
}
// relu_out: the forward output when ReLU was fused (masks dy), else null.  sums: 2*C floats of scratch.
int nb_bn_bwd(const void* dy, const void* x, const void* relu_out, const float* mean, const float* rstd,
              const float* gamma, void* dx, void* dres, float* dgamma, float* dbeta, float* partials, float* sums,
              long long M, int C, void* stream) {
  if (C % 8) return NB_ERR_UNALIGNED;
  cudaStream_t s = (cudaStream_t)stream;
  const dim3 g = bn_grid(M, C, nb_bn_split(M));
  float* p0 = partials;
  float* p1 = partials + (size_t)g.x * C;
  bn_reduce_kernel<true><<<g, 256, 0, s>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, mean, rstd,
                                          (const __nv_bfloat16*)relu_out, p0, p1, M, C);
  NB_LAUNCH_CHECK();
  bn_bwd_finish_kernel<<<ceil_div(C, 32), bn_fin_threads(g.x), 0, s>>>(p0, p1, (int)g.x, C, sums, sums + C, dgamma, dbeta);
  NB_LAUNCH_CHECK();
  bn_bwd_dx_kernel<<<bn_grid(M, C, 1 << 20), 256, 0, s>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,
                                                         (const __nv_bfloat16*)relu_out, mean, rstd, gamma, sums, sums + C,
                                                         (__nv_bfloat16*)dx, (__nv_bfloat16*)dres, M, C);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

// idx: one byte per output element when nb_maxpool_idx_bytes(K, stride) == 1, else four.  A pixel in more than nine windows takes
// four: taking bytes out of words is then what the backward spends its time on (16 x 16 / 4 over 16 x 120 x 160 x 64: 139 us with bytes, 86
// with words).
int nb_maxpool_idx_bytes(int K, int stride) { return K * K < 255 && ceil_div(K, stride) <= 3 ? 1 : 4; }
int nb_maxpool_fwd(const void* x, void* y, void* idx, int B, int H, int W, int C, int K, int stride, int pad, int OH, int OW,
                   void* stream) {
  if (B <= 0 || OH <= 0 || OW <= 0 || C <= 0) return NB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  // A large window is walked tap by tap, which needs threads to hide its latency: with few outputs, or few per row of blocks, a thread
  // takes one channel instead of eight (us, eight / one: 8 x 8 / 8 over 16 x 56 x 56 x 64 18.5 / 6.2, 5 x 5 / 3 over 256 x 20 x 20 x 32
  // 13.3 / 11.5; the other side, 5 x 5 / 3 over 16 x 56 x 56 x 64: 9.0 / 11.7).
  const bool few = K >= 4 && ((long long)B * OH * OW * C < 148LL * 288 * 8 || OW * (C / 8) < 64);
  const bool vec = !few && C % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(idx) & 15) == 0;
#define NB_POOL(V, I, KC)                                                                                                   \
  maxpool_fwd_kernel<V, I, KC><<<dim3((unsigned)(B * OH), pool_blocks(OW * (C / V))), 256, 0, s>>>(                         \
      (const __nv_bfloat16*)x, (__nv_bfloat16*)y, (I*)idx, H, W, C, K, stride, pad, OH, OW)
  const bool byte = nb_maxpool_idx_bytes(K, stride) == 1;
  if (vec) {
    if (K == 3) NB_POOL(8, unsigned char, 3);
    else if (byte) NB_POOL(8, unsigned char, 0);
    else NB_POOL(8, int, 0);
  } else {
    if (byte) NB_POOL(1, unsigned char, 0);
    else NB_POOL(1, int, 0);
  }
#undef NB_POOL
  NB_LAUNCH_CHECK();
  return NB_OK;
}
int nb_maxpool_bwd(const void* dy, const void* idx, void* dx, int B, int H, int W, int C, int K, int stride, int pad, int OH,
                   int OW, void* stream) {
  if (B <= 0 || H <= 0 || W <= 0 || C <= 0) return NB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const bool vec = C % 8 == 0 && ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx)) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(idx) & 15) == 0;
#define NB_POOL(V, I, S1)                                                                                                   \
  maxpool_bwd_kernel<V, I, S1><<<dim3((unsigned)(B * H), pool_blocks(W * (C / V))), 256, 0, s>>>(                           \
      (const __nv_bfloat16*)dy, (const I*)idx, (__nv_bfloat16*)dx, H, W, C, K, stride, pad, OH, OW)
  const bool byte = nb_maxpool_idx_bytes(K, stride) == 1;
  if (vec && K == 3 && stride == 2) {
    const int a0 = pad / 2, na = (H - 1 + pad) / 2 - a0 + 1, nw = (W - 1 + pad) / 2 - a0 + 1;   // pixel pairs per direction
    maxpool_bwd_3s2_kernel<<<dim3((unsigned)(B * na), pool_blocks(nw * (C / 8))), 256, 0, s>>>(
        (const __nv_bfloat16*)dy, (const unsigned char*)idx, (__nv_bfloat16*)dx, H, W, C, pad, OH, OW, a0, na, nw);
  } else if (vec) {
    if (K == 3 && stride == 1) NB_POOL(8, unsigned char, true);
    else if (byte) NB_POOL(8, unsigned char, false);
    else NB_POOL(8, int, false);
  } else {
    if (byte) NB_POOL(1, unsigned char, false);
    else NB_POOL(1, int, false);
  }
#undef NB_POOL
  NB_LAUNCH_CHECK();
  return NB_OK;
}
int nb_avgpool(const void* src, void* dst, int B, int H, int W, int C, int K, int OH, int OW, int back, void* stream) {
  if (K <= 0 || OH * K > H || OW * K > W) return NB_ERR_BAD_ARG;
  const long long total = back ? (long long)B * H * W * C : (long long)B * OH * OW * C;
  avgpool_kernel<<<g1(total), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)src, (__nv_bfloat16*)dst, B, H, W, C, K, OH, OW, back);
  NB_LAUNCH_CHECK();
  return NB_OK;
}
// H, W are the LOW-resolution sizes in both directions
int nb_upsample_nearest(const void* src, void* dst, int B, int H, int W, int C, int S, int back, void* stream) {
  if (S <= 0) return NB_ERR_BAD_ARG;
  const long long total = back ? (long long)B * H * W * C : (long long)B * H * S * W * S * C;
  upsample_kernel<<<g1(total), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)src, (__nv_bfloat16*)dst, B, H, W, C, S, back);
  NB_LAUNCH_CHECK();
  return NB_OK;
}
int nb_image_normalize(const unsigned char* img, void* out, int B, int H, int W, float m0, float m1, float m2, float s0,
                       float s1, float s2, void* stream) {
  const long long hw = (long long)H * W;
  if (B <= 0 || hw <= 0) return NB_OK;
  const bool by4 = hw % 4 == 0 && (reinterpret_cast<uintptr_t>(img) & 3) == 0;
  for (int b0 = 0; b0 < B; b0 += 65535) {          // grid.y limit
    const int n = B - b0 < 65535 ? B - b0 : 65535;
    const unsigned char* in = img + (size_t)b0 * 3 * hw;
    __nv_bfloat16* o = (__nv_bfloat16*)out + (size_t)b0 * hw * 8;
    if (by4)
      image_normalize_kernel<4><<<dim3((unsigned)ceil_div_ll(hw, 1024), n), 256, 0, (cudaStream_t)stream>>>(in, o, hw, m0, m1, m2,
                                                                                                           s0, s1, s2);
    else
      image_normalize_kernel<1><<<dim3((unsigned)ceil_div_ll(hw, 256), n), 256, 0, (cudaStream_t)stream>>>(in, o, hw, m0, m1, m2,
                                                                                                          s0, s1, s2);
  }
  NB_LAUNCH_CHECK();
  return NB_OK;
}

}  // extern "C"
