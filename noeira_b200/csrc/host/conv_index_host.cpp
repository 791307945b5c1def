// Walk of the gathering convolution's A tiles on the host, chunk by chunk in the kernel's own order and with its index functions
// (conv_index.h): the oracle for what the kernel reads.
#include "conv_index.h"

using namespace nbconv;

extern "C" {

// 1 when the convolution kernels take these sizes
int nbh_conv_fits(int B, int H, int W, int C, int KH, int KW, int stride, int pad) {
  return conv_fits(B, H, W, C, KH, KW, stride, pad) ? 1 : 0;
}

// off[row · chunks + q]: element offset in x of chunk q (8 channels of one tap) of output pixel `row`, −1 where zeros are
// written; rows and chunks are rounded up to whole tiles (128 pixels x 8 chunks, weight gradient 64 pixels x 16 chunks).
// Returns 0, or 1 when the sizes are refused.
int nbh_conv_gather(int B, int H, int W, int C, int KH, int KW, int stride, int pad, int wgrad, int* off, long long rows,
                        long long chunks) {
  if (!conv_fits(B, H, W, C, KH, KW, stride, pad)) return 1;
  ConvGeom g;
  conv_geom_set(g, B, H, W, C, KH, KW, stride, pad);
  const int step = wgrad ? K_BLOCK : TILE_ROWS, per = wgrad ? TILE_ROWS / 8 : K_BLOCK / 8;
  for (int m0 = 0; m0 < rows; m0 += step)
    for (int q0 = 0; q0 < chunks; q0 += per)
      for (int r0 = 0; r0 < 16; ++r0) {            // a thread's rows: r0, r0 + 16, ...
        Pixel px = pixel_of(g, m0 + r0);
        for (int i = 0; i < step / 16; ++i) {
          const int m = m0 + r0 + 16 * i;
          const Corner c = corner_of(g, px, m);
          for (int q = q0; q < q0 + per; ++q) {
            int o;
            off[m * chunks + q] = chunk_of(g, c, tap_of(g, q), o) ? o : -1;
          }
          pixel_step(g, px, 16);
        }
      }
  return 0;
}

}  // extern "C"
