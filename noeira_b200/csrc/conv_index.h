// Index arithmetic of the gathering convolution (conv_gemm_tcgen05.cu): which 16 bytes of the NHWC input a chunk of the patch
// matrix is.  Plain C++ for host and device, so that a CPU test walks the same functions that the kernel runs.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define NBCI_HD __host__ __device__ __forceinline__
#else
#define NBCI_HD inline
#endif

namespace nbconv {

constexpr int TILE_ROWS = 128, K_BLOCK = 64;   // rows of an A tile, reduction elements of a k-block

// n / d for 0 <= n < 2^31 by one multiplication (Granlund and Montgomery, "Division by invariant integers using
// multiplication"): with l = ceil(log2 d), m = floor(2^(31 + l) / d) + 1 fits in 32 bits and n / d = (n m) >> (31 + l).
struct FastDiv {
  uint32_t mul, shift;   // shift = l − 1 after the high word; d = 1: mul = 0
  void set(uint32_t d) {
    uint32_t l = 0;
    while ((1ull << l) < d) ++l;
    mul = d == 1 ? 0u : (uint32_t)((1ull << (31 + l)) / d + 1);
    shift = d == 1 ? 0u : l - 1;
  }
  NBCI_HD int div(int n) const { return mul ? (int)((uint32_t)(((uint64_t)(uint32_t)n * mul) >> 32) >> shift) : n; }
};

struct ConvGeom {
  const void* x;                                        // bf16 [B, H, W, C]
  int H, W, C, KW, taps, stride, pad, OH, OW, pixels;   // pixels = B·OH·OW
  int elems;                                            // B·H·W·C
  FastDiv by_cv, by_kw, by_image, by_row;               // chunks per tap, taps per filter row, OH·OW, OW
  int wgrad;    // A = patches^T (MN-major), reduction over the pixels
  int mirror;   // B rows of tap t are those of tap taps − 1 − t, K-major (data gradient)
};

// Sizes whose offsets fit: they are 32-bit element counts, with the window's corner up to pad rows and columns outside, and
// pixels are counted up to two tiles past the last one.
inline bool conv_fits(long long B, long long H, long long W, long long C, long long KH, long long KW, long long stride, long long pad) {
  const long long OH = (H + 2 * pad - KH) / stride + 1, OW = (W + 2 * pad - KW) / stride + 1;
  return (B * H + 2 * pad) * (W + 2 * pad) * C <= 0x7fffffffLL && B * OH * OW <= 0x7fffffffLL - 256;
}

inline void conv_geom_set(ConvGeom& g, int B, int H, int W, int C, int KH, int KW, int stride, int pad) {
  g.H = H; g.W = W; g.C = C; g.KW = KW; g.taps = KH * KW; g.stride = stride; g.pad = pad;
  g.OH = (H + 2 * pad - KH) / stride + 1;
  g.OW = (W + 2 * pad - KW) / stride + 1;
  g.pixels = B * g.OH * g.OW;
  g.elems = B * H * W * C;
  g.by_cv.set(C / 8);
  g.by_kw.set(KW);
  g.by_image.set(g.OH * g.OW);
  g.by_row.set(g.OW);
  g.wgrad = g.mirror = 0;
}

// A pixel past the last one and a tap past the last one both get this row.  Corner row + tap row is negative as soon as either
// is: a valid corner row is below H and a valid tap row at most H + 2·pad, both below 2^28 (conv_fits, C >= 8).  The two have
// to have the same sign: a tile can hold both at once, and with opposite ones they cancelled to row 0 and were read.
constexpr int OUTSIDE = -(1 << 28);

struct Pixel { int b, oh, ow; };
struct Corner { int h, w, off; };   // of an output pixel's window in the input; off: element offset of (h, w, channel 0), may be negative
struct Tap { int kh, kw, off; };    // of a 16-byte chunk: 8 channels of one tap

NBCI_HD Pixel pixel_of(const ConvGeom& g, int m) {
  const int b = g.by_image.div(m), r = m - b * (g.OH * g.OW), oh = g.by_row.div(r);
  return Pixel{b, oh, r - oh * g.OW};
}
NBCI_HD void pixel_step(const ConvGeom& g, Pixel& p, int n) {
  p.ow += n;
  while (p.ow >= g.OW) {
    p.ow -= g.OW;
    if (++p.oh == g.OH) { p.oh = 0; ++p.b; }
  }
}
NBCI_HD Corner corner_of(const ConvGeom& g, const Pixel& p, int m) {
  Corner c;
  c.h = m < g.pixels ? p.oh * g.stride - g.pad : OUTSIDE;
  c.w = p.ow * g.stride - g.pad;
  c.off = ((p.b * g.H + p.oh * g.stride - g.pad) * g.W + c.w) * g.C;
  return c;
}
NBCI_HD Tap tap_of(const ConvGeom& g, int q) {
  const int t = g.by_cv.div(q), c8 = q - t * (g.C >> 3);
  Tap k;
  k.kh = g.by_kw.div(t);
  k.kw = t - k.kh * g.KW;
  k.off = (k.kh * g.W + k.kw) * g.C + c8 * 8;
  if (t >= g.taps) k.kh = OUTSIDE;
  return k;
}
// the chunk lies in the image (else it is zeros); `off`: its element offset
NBCI_HD bool chunk_of(const ConvGeom& g, const Corner& c, const Tap& k, int& off) {
  off = c.off + k.off;
  return (unsigned)(c.h + k.kh) < (unsigned)g.H && (unsigned)(c.w + k.kw) < (unsigned)g.W;
}

}  // namespace nbconv
