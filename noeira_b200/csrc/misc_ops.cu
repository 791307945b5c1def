// RoPE, embedding gather / scatter-add, and fused loss forward+gradient kernels (MSE, masked L1, KL to a
// standard normal, softmax cross-entropy).  Losses accumulate into device-resident fp32 accumulators so the
// hot loop never copies to the host (noeira/deep_agents/training/device_mean_accum.mojo:157); gradients
// are written in bf16 for the backward GEMMs.
// Reference: noeira/nn/primitives/rope.mojo:84,114; embedding.mojo:54-406; noeira/nn/loss/*.mojo.
#include "common.cuh"

namespace {
using namespace nb;

// x [B, S, H, D] (strides sb, ss, sh, 1), rotate-half pairing (i, i + D/2), angle = (pos0 + s) * theta^(-2i/D).
// dir = +1 forward, -1 backward (the transpose of a rotation is the opposite rotation).  In place.
__global__ void __launch_bounds__(256)
rope_kernel(__nv_bfloat16* __restrict__ x, int B, int S, int H, int D, long long sb, long long ss, long long sh,
            float log2_theta, int pos0, float dir) {
  const int half = D / 2;
  const long long total = (long long)B * S * H * half;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int d = (int)(i % half);
    long long r = i / half;
    const int h = (int)(r % H);
    r /= H;
    const int s = (int)(r % S);
    const int b = (int)(r / S);
    const float inv_freq = exp2f(-(2.f * d / D) * log2_theta);
    float sn, cs;
    sincosf((float)(pos0 + s) * inv_freq, &sn, &cs);
    sn *= dir;
    __nv_bfloat16* p = x + b * sb + s * ss + h * sh;
    const float x1 = __bfloat162float(p[d]), x2 = __bfloat162float(p[d + half]);
    p[d] = __float2bfloat16(x1 * cs - x2 * sn);
    p[d + half] = __float2bfloat16(x2 * cs + x1 * sn);
  }
}

// The same rotation in vectors of 8: a thread owns 8 frequencies of one token and walks over up to ROPE_HEADS heads with the
// same sines.  The scalar kernel takes a sine and a cosine per pair and head and was bound by them: 3200 tokens x 15 heads
// x 64 10.1 us, 4.5 here.
constexpr int ROPE_HEADS = 4;
__global__ void __launch_bounds__(128)
rope_vec_kernel(__nv_bfloat16* __restrict__ x, int B, int S, int H, int D, long long sb, long long ss, long long sh,
                float log2_theta, int pos0, float dir) {
  const int half = D / 2, nc = half / 8, hg = (H + ROPE_HEADS - 1) / ROPE_HEADS;
  const long long total = (long long)B * S * hg * nc;
  for (long long i = (long long)blockIdx.x * 128 + threadIdx.x; i < total; i += (long long)gridDim.x * 128) {
    const int c = (int)(i % nc);
    long long r = i / nc;
    const int h0 = (int)(r % hg) * ROPE_HEADS;
    r /= hg;
    const int s = (int)(r % S), b = (int)(r / S);
    float sn[8], cs[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      sincosf((float)(pos0 + s) * exp2f(-(2.f * (c * 8 + k) / D) * log2_theta), &sn[k], &cs[k]);
      sn[k] *= dir;
    }
    __nv_bfloat16* p = x + b * sb + s * ss + h0 * sh + c * 8;
    uint4 v1[ROPE_HEADS], v2[ROPE_HEADS];
#pragma unroll
    for (int h = 0; h < ROPE_HEADS; ++h)
      if (h0 + h < H) {
        v1[h] = *reinterpret_cast<const uint4*>(p + h * sh);
        v2[h] = *reinterpret_cast<const uint4*>(p + h * sh + half);
      }
#pragma unroll
    for (int h = 0; h < ROPE_HEADS; ++h)
      if (h0 + h < H) {
        __nv_bfloat162* a = reinterpret_cast<__nv_bfloat162*>(&v1[h]);
        __nv_bfloat162* e = reinterpret_cast<__nv_bfloat162*>(&v2[h]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float x0 = __low2float(a[k]), x1 = __high2float(a[k]), y0 = __low2float(e[k]), y1 = __high2float(e[k]);
          a[k] = __floats2bfloat162_rn(x0 * cs[2 * k] - y0 * sn[2 * k], x1 * cs[2 * k + 1] - y1 * sn[2 * k + 1]);
          e[k] = __floats2bfloat162_rn(y0 * cs[2 * k] + x0 * sn[2 * k], y1 * cs[2 * k + 1] + x1 * sn[2 * k + 1]);
        }
        *reinterpret_cast<uint4*>(p + h * sh) = v1[h];
        *reinterpret_cast<uint4*>(p + h * sh + half) = v2[h];
      }
  }
}

// out[t, :] = table[idx[t], :] * scale
__global__ void __launch_bounds__(256)
embedding_fwd_kernel(const __nv_bfloat16* __restrict__ table, int ldt, const long long* __restrict__ idx,
                     __nv_bfloat16* __restrict__ out, int ldo, int T, int D, float scale, int vocab) {
  const int nvec = D / 8;
  const long long total = (long long)T * nvec;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int t = (int)(i / nvec), v = (int)(i % nvec);
    if (!NB_IN_BOUNDS(idx[t] >= 0 && (vocab <= 0 || idx[t] < vocab), 601, idx[t])) continue;
    uint4 w = *reinterpret_cast<const uint4*>(table + (size_t)idx[t] * ldt + v * 8);
    if (scale != 1.f) {
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&w);
#pragma unroll
      for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(__low2float(h[k]) * scale, __high2float(h[k]) * scale);
    }
    *reinterpret_cast<uint4*>(out + (size_t)t * ldo + v * 8) = w;
  }
}
// dtable[idx[t], :] += dy[t, :] * scale   (fp32 atomics: order, hence the last bit, is not reproducible)
__global__ void __launch_bounds__(256)
embedding_bwd_kernel(float* __restrict__ dtable, int ldt, const long long* __restrict__ idx,
                     const __nv_bfloat16* __restrict__ dy, int ldy, int T, int D, float scale, int vocab) {
  const long long total = (long long)T * D;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int t = (int)(i / D), d = (int)(i % D);
    if (!NB_IN_BOUNDS(idx[t] >= 0 && (vocab <= 0 || idx[t] < vocab), 602, idx[t])) continue;
    atomicAdd(dtable + (size_t)idx[t] * ldt + d, __bfloat162float(dy[(size_t)t * ldy + d]) * scale);
  }
}

// Σ w·(pred − target)² over [M, N] (first n_real columns only); dpred = 2·w·(pred − target)·gscale.
// `rowmask` (optional, [M]) zeroes whole rows.  One partial per block, ordered finish by the caller's finish.
template <typename TP>
__global__ void __launch_bounds__(256)
mse_kernel(const TP* __restrict__ pred, int ldp, const float* __restrict__ target, int ldt,
           const float* __restrict__ rowmask, __nv_bfloat16* __restrict__ dpred, int ldd, float* __restrict__ partials,
           int M, int N, int n_real, float gscale, int l1) {
  __shared__ float sh[32];
  const long long total = (long long)M * N;
  const long long stride = (long long)gridDim.x * blockDim.x;
  float acc = 0.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int m = (int)(i / N), n = (int)(i % N);
    float g = 0.f;
    if (n < n_real && (!rowmask || rowmask[m] != 0.f)) {
      const float d = (float)pred[(size_t)m * ldp + n] - target[(size_t)m * ldt + n];
      if (l1) {
        acc += fabsf(d);
        g = (d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f)) * gscale;
      } else {
        acc += d * d;
        g = 2.f * d * gscale;
      }
    }
    if (dpred) dpred[(size_t)m * ldd + n] = __float2bfloat16(g);
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

__global__ void finish_sum_kernel(const float* __restrict__ partials, int n, float scale, float* __restrict__ out) {
  __shared__ float sh[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partials[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) out[0] += s * scale;
}

// KL(N(mu, exp(logvar)) || N(0,1)) summed over latent, mean over batch; info = [mu | logvar] fp32 [B, 2L].
// dinfo (bf16 [B, 2L]) = weight/B * (mu, 0.5 (exp(logvar) − 1)).
__global__ void kl_stdnormal_kernel(const float* __restrict__ info, int ld, __nv_bfloat16* __restrict__ dinfo, int ldd,
                                    float* __restrict__ partials, int B, int L, float weight) {
  __shared__ float sh[32];
  float acc = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B * L; i += gridDim.x * blockDim.x) {
    const int b = i / L, j = i % L;
    const float mu = info[(size_t)b * ld + j], lv = info[(size_t)b * ld + L + j];
    const float ev = __expf(lv);
    acc += -0.5f * (1.f + lv - mu * mu - ev);
    if (dinfo) {
      dinfo[(size_t)b * ldd + j] = __float2bfloat16(weight / B * mu);
      dinfo[(size_t)b * ldd + L + j] = __float2bfloat16(weight / B * 0.5f * (ev - 1.f));
    }
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

// Softmax cross-entropy, one block per row: loss_row = lse − logit[target]; dlogits = (softmax − onehot)·gscale
// written IN PLACE over the bf16 logits.  ignore_index rows contribute nothing.
__global__ void __launch_bounds__(256)
cross_entropy_kernel(__nv_bfloat16* __restrict__ logits, int ld, const long long* __restrict__ target, int V,
                     float* __restrict__ row_loss, float gscale, long long ignore_index, int write_grad) {
  __shared__ float sh[32];
  const int row = blockIdx.x;
  __nv_bfloat16* lr = logits + (size_t)row * ld;
  long long tg = target[row];
  if (!NB_IN_BOUNDS(tg == ignore_index || (tg >= 0 && tg < V), 603, tg)) tg = ignore_index;
  float mx = -INFINITY;
  for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, __bfloat162float(lr[i]));
  mx = block_max(mx, sh);
  float s = 0.f;
  for (int i = threadIdx.x; i < V; i += blockDim.x) s += __expf(__bfloat162float(lr[i]) - mx);
  s = block_sum(s, sh);
  const float lse = mx + logf(s);
  const bool live = tg != ignore_index && tg >= 0 && tg < V;
  if (threadIdx.x == 0) row_loss[row] = live ? lse - __bfloat162float(lr[tg]) : 0.f;
  if (write_grad) {
    __syncthreads();
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
      float g = 0.f;
      if (live) g = (__expf(__bfloat162float(lr[i]) - lse) - (i == tg ? 1.f : 0.f)) * gscale;
      lr[i] = __float2bfloat16(g);
    }
  }
}

// The same loss with the row kept in shared memory: one read and one write of the logits, in 16-byte vectors, where the
// kernel above reads them three times element by element.  Bound by DRAM bytes and, close behind, by the two exponentials
// per logit; two rows of 49152 fit on an SM, so one loads while the other computes.  4096 x 49152 (403 MB): 1044 us above,
// 220 here.  Rows that are not 16-byte aligned or do not fit in shared memory take the kernel above.
template <int T>
__global__ void __launch_bounds__(T)
cross_entropy_smem_kernel(__nv_bfloat16* __restrict__ logits, int ld, const long long* __restrict__ target, int V,
                          float* __restrict__ row_loss, float gscale, long long ignore_index, int write_grad) {
  extern __shared__ uint4 ce_row[];
  __shared__ float sh[32];
  const int row = blockIdx.x, nv = V / 8, tail = V - nv * 8;
  __nv_bfloat16* lr = logits + (size_t)row * ld;
  __nv_bfloat16* tl = reinterpret_cast<__nv_bfloat16*>(ce_row + nv);      // the V % 8 last logits
  long long tg = target[row];
  if (!NB_IN_BOUNDS(tg == ignore_index || (tg >= 0 && tg < V), 603, tg)) tg = ignore_index;
  const bool live = tg != ignore_index && tg >= 0 && tg < V;
  float mx = -INFINITY;
#pragma unroll 4
  for (int i = threadIdx.x; i < nv; i += T) {
    const uint4 v = *reinterpret_cast<const uint4*>(lr + i * 8);
    ce_row[i] = v;
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) mx = fmaxf(mx, fmaxf(__low2float(h[k]), __high2float(h[k])));
  }
  if ((int)threadIdx.x < tail) {
    tl[threadIdx.x] = lr[nv * 8 + threadIdx.x];
    mx = fmaxf(mx, __bfloat162float(tl[threadIdx.x]));
  }
  mx = block_max(mx, sh);
  float s = 0.f;
#pragma unroll 2
  for (int i = threadIdx.x; i < nv; i += T) {
    const uint4 v = ce_row[i];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) s += __expf(__low2float(h[k]) - mx) + __expf(__high2float(h[k]) - mx);
  }
  if ((int)threadIdx.x < tail) s += __expf(__bfloat162float(tl[threadIdx.x]) - mx);
  s = block_sum(s, sh);
  const float lse = mx + logf(s);
  if (threadIdx.x == 0) row_loss[row] = live ? lse - __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ce_row)[tg]) : 0.f;
  if (!write_grad) return;
  const int hot = live ? (int)tg : -1;
  for (int i = threadIdx.x; i < nv; i += T) {
    const uint4 v = ce_row[i];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
    uint4 o = make_uint4(0, 0, 0, 0);
    if (live) {
      __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        oh[k] = __floats2bfloat162_rn((__expf(__low2float(h[k]) - lse) - (8 * i + 2 * k == hot ? 1.f : 0.f)) * gscale,
                                      (__expf(__high2float(h[k]) - lse) - (8 * i + 2 * k + 1 == hot ? 1.f : 0.f)) * gscale);
    }
    *reinterpret_cast<uint4*>(lr + i * 8) = o;
  }
  if ((int)threadIdx.x < tail) {
    const int c = nv * 8 + threadIdx.x;
    lr[c] = __float2bfloat16(live ? (__expf(__bfloat162float(tl[threadIdx.x]) - lse) - (c == hot ? 1.f : 0.f)) * gscale : 0.f);
  }
}

// Sinusoidal embedding of a scalar per row: out[b, :] = [sin(t·w_i) | cos(t·w_i)], periods geometric in
// [min_period, max_period] (flow-matching time embedding).
__global__ void sincos_embed_kernel(const float* __restrict__ t, __nv_bfloat16* __restrict__ out, int ld, int B, int D,
                                    float min_period, float max_period) {
  const int half = D / 2;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B * half; i += gridDim.x * blockDim.x) {
    const int b = i / half, j = i % half;
    const float frac = half > 1 ? (float)j / (half - 1) : 0.f;
    const float period = min_period * powf(max_period / min_period, frac);
    const float a = t[b] * 6.283185307179586f / period;
    float sn, cs;
    sincosf(a, &sn, &cs);
    out[(size_t)b * ld + j] = __float2bfloat16(sn);
    out[(size_t)b * ld + half + j] = __float2bfloat16(cs);
  }
}

inline int g1(long long n) {
  long long b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 1184 ? 1184 : b));
}
}  // namespace

NB_BOUNDS_REGISTER(misc_ops)

extern "C" {

int nb_rope(void* x, int B, int S, int H, int D, long long sb, long long ss, long long sh, float theta, int pos0,
            int backward, void* stream) {
  if (D % 2) return NB_ERR_BAD_ARG;
  // fewer than 1024 pairs per SM: a thread's eight sines in a row take longer than one each in the kernel above (256 tokens x 15 x 64:
  // 3.0 us against 3.5; 512 tokens: 4.0 / 3.5)
  if ((long long)B * S * H * (D / 2) >= 148 * 1024 && D % 16 == 0 && sb % 8 == 0 && ss % 8 == 0 && sh % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    const long long n = (long long)B * S * ceil_div(H, ROPE_HEADS) * (D / 16);
    const long long blocks = (n + 127) / 128;
    rope_vec_kernel<<<(int)(blocks < 1 ? 1 : (blocks > 148 * 16 ? 148 * 16 : blocks)), 128, 0, (cudaStream_t)stream>>>(
        (__nv_bfloat16*)x, B, S, H, D, sb, ss, sh, log2f(theta), pos0, backward ? -1.f : 1.f);
    NB_LAUNCH_CHECK();
    return NB_OK;
  }
  rope_kernel<<<g1((long long)B * S * H * (D / 2)), 256, 0, (cudaStream_t)stream>>>(
      (__nv_bfloat16*)x, B, S, H, D, sb, ss, sh, log2f(theta), pos0, backward ? -1.f : 1.f);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

// vocab: number of table rows (<= 0: unknown; only the bounds-checked build reads it)
int nb_embedding_fwd(const void* table, int ldt, const long long* idx, void* out, int ldo, int T, int D, float scale,
                     int vocab, void* stream) {
  if (D % 8 || ldt % 8 || ldo % 8) return NB_ERR_UNALIGNED;
  embedding_fwd_kernel<<<g1((long long)T * D / 8), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)table, ldt, idx, (__nv_bfloat16*)out, ldo, T, D, scale, vocab);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

int nb_embedding_bwd(float* dtable, int ldt, const long long* idx, const void* dy, int ldy, int T, int D, float scale,
                     int vocab, void* stream) {
  embedding_bwd_kernel<<<g1((long long)T * D), 256, 0, (cudaStream_t)stream>>>(dtable, ldt, idx,
                                                                              (const __nv_bfloat16*)dy, ldy, T, D, scale, vocab);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

// loss_acc[0] += loss_scale · Σ …;  partials: >= 1184 floats.
int nb_mse_loss(const void* pred, int ldp, const float* target, int ldt, const float* rowmask, void* dpred, int ldd,
                float* partials, float* loss_acc, int M, int N, int n_real, float gscale, float loss_scale, int l1,
                int pred_f32, void* stream) {
  const int grid = g1((long long)M * N);
  cudaStream_t s = (cudaStream_t)stream;
  if (pred_f32)
    mse_kernel<float><<<grid, 256, 0, s>>>((const float*)pred, ldp, target, ldt, rowmask, (__nv_bfloat16*)dpred, ldd,
                                           partials, M, N, n_real, gscale, l1);
  else
    mse_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>((const __nv_bfloat16*)pred, ldp, target, ldt, rowmask,
                                                   (__nv_bfloat16*)dpred, ldd, partials, M, N, n_real, gscale, l1);
  NB_LAUNCH_CHECK();
  finish_sum_kernel<<<1, 256, 0, s>>>(partials, grid, loss_scale, loss_acc);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

int nb_kl_stdnormal(const float* info, int ld, void* dinfo, int ldd, float* partials, float* loss_acc, int B, int L,
                    float weight, void* stream) {
  const int grid = g1((long long)B * L);
  cudaStream_t s = (cudaStream_t)stream;
  kl_stdnormal_kernel<<<grid, 256, 0, s>>>(info, ld, (__nv_bfloat16*)dinfo, ldd, partials, B, L, weight);
  NB_LAUNCH_CHECK();
  finish_sum_kernel<<<1, 256, 0, s>>>(partials, grid, weight / B, loss_acc);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

// row_loss: M floats of scratch; loss_acc[0] += loss_scale · Σ row_loss
int nb_cross_entropy(void* logits, int ld, const long long* target, int M, int V, float* row_loss, float* loss_acc,
                     float gscale, float loss_scale, long long ignore_index, int write_grad, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const size_t smem = (size_t)ceil_div(V, 8) * 16;
  // few short rows: reading them three times is quicker than the detour (us, three reads / shared memory: 256 x 256 3.6 / 4.0, 1024 x 256
  // 5.5 / 4.8, 256 x 1000 4.7 / 4.7)
  if ((V >= 512 || M > 512) && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && smem <= 200 * 1024) {
    // threads by row length: 4 to 13 vectors per thread from 32768 logits, 2 to 16 from 4096, up to 8 below
#define NB_CE(T)                                                                                                        \
  do {                                                                                                                  \
    NB_CUDA(cudaFuncSetAttribute(cross_entropy_smem_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)); \
    cross_entropy_smem_kernel<T><<<M, T, smem, s>>>((__nv_bfloat16*)logits, ld, target, V, row_loss, gscale,            \
                                                    ignore_index, write_grad);                                          \
  } while (0)
    if (V >= 32768) NB_CE(1024);
    else if (V >= 4096) NB_CE(256);
    else NB_CE(64);
#undef NB_CE
  } else {
    cross_entropy_kernel<<<M, 256, 0, s>>>((__nv_bfloat16*)logits, ld, target, V, row_loss, gscale, ignore_index,
                                           write_grad);
  }
  NB_LAUNCH_CHECK();
  finish_sum_kernel<<<1, 1024, 0, s>>>(row_loss, M, loss_scale, loss_acc);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

int nb_sincos_embed(const float* t, void* out, int ld, int B, int D, float min_period, float max_period,
                    void* stream) {
  sincos_embed_kernel<<<g1((long long)B * D / 2), 256, 0, (cudaStream_t)stream>>>(t, (__nv_bfloat16*)out, ld, B, D,
                                                                                min_period, max_period);
  NB_LAUNCH_CHECK();
  return NB_OK;
}

}  // extern "C"

// ------------------------------------------------------------------------------------------ Q4_0 weights
// Block of 32 values along a ROW of the [IN, OUT] weight: one fp16 scale d and 16 bytes of 4-bit codes q in [0, 15];
// byte j of a block holds element j (low nibble) and element j + 16 (high nibble); value = (q − 8)·d.
// (Same block format as noeira/nn/quant/q4_0.mojo.)  Output: bf16 [rows, ld] — the tcgen05 GEMM then reads it.
namespace {
__global__ void __launch_bounds__(256)
q4_0_dequant_kernel(const unsigned char* __restrict__ codes, const __half* __restrict__ scales, __nv_bfloat16* __restrict__ out,
                    int rows, int cols, int ld) {
  const int blocks_per_row = cols / 32;
  const long long total = (long long)rows * blocks_per_row;
  for (long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x; b < total; b += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(b / blocks_per_row), cb = (int)(b % blocks_per_row);
    const float d = __half2float(scales[b]);
    const uint4 q = *reinterpret_cast<const uint4*>(codes + b * 16);
    const unsigned char* qb = reinterpret_cast<const unsigned char*>(&q);
    __nv_bfloat16* o = out + (size_t)r * ld + cb * 32;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      o[j] = __float2bfloat16(((int)(qb[j] & 15) - 8) * d);
      o[j + 16] = __float2bfloat16(((int)(qb[j] >> 4) - 8) * d);
    }
  }
}
}  // namespace

extern "C" int nb_q4_0_dequant(const unsigned char* codes, const void* scales, void* out, int rows, int cols, int ld,
                               void* stream) {
  if (cols % 32 || ((uintptr_t)codes & 15)) return NB_ERR_UNALIGNED;
  const long long total = (long long)rows * (cols / 32);
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks < 1) blocks = 1;
  q4_0_dequant_kernel<<<(int)blocks, 256, 0, (cudaStream_t)stream>>>(codes, (const __half*)scales, (__nv_bfloat16*)out, rows,
                                                                    cols, ld);
  NB_LAUNCH_CHECK();
  return NB_OK;
}
