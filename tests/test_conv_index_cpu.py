"""What the gathering convolution reads: the kernel's index functions, walked on the host, against an independent im2col index."""
import ctypes

import numpy as np
import pytest

from noeira_b200._native import host_lib

# (ic as stored, k, stride, pad, b, h, w): the shapes of the GPU test, odd camera frames, remainders of every kind
SHAPES = [(64, 3, 1, 1, 2, 17, 23), (64, 3, 2, 1, 3, 15, 21), (128, 3, 2, 1, 1, 9, 8), (8, 7, 2, 3, 2, 33, 45), (64, 1, 2, 0, 2, 11, 13),
          (8, 3, 1, 0, 1, 5, 4), (72, 5, 3, 2, 2, 19, 14), (256, 3, 1, 1, 2, 7, 7), (512, 3, 1, 1, 1, 5, 6), (64, 3, 1, 2, 1, 4, 3),
          (128, 3, 1, 1, 1, 1, 1), (16, 2, 2, 1, 2, 6, 9), (8, 7, 2, 3, 1, 481, 639), (8, 7, 2, 3, 1, 97, 131), (64, 3, 1, 1, 3, 25, 33),
          (8, 8, 4, 0, 3, 84, 84), (24, 4, 2, 1, 5, 9, 11), (40, 3, 1, 2, 300, 1, 1), (8, 3, 1, 1, 1, 1, 300), (16, 1, 1, 0, 129, 1, 1)]


def _expected(c, k, stride, pad, b, h, w):
    """Offset of every (pixel, tap, 8-channel chunk) in NHWC, −1 outside the image."""
    oh, ow = (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1
    bi, y, x, kh, kw, c8 = np.ix_(range(b), range(oh), range(ow), range(k), range(k), range(c // 8))
    ih, iw = y * stride - pad + kh, x * stride - pad + kw
    off = ((bi * h + ih) * w + iw) * c + c8 * 8
    inside = (ih >= 0) & (ih < h) & (iw >= 0) & (iw < w) & (bi >= 0) & (c8 >= 0)
    return np.where(inside, off, -1).reshape(b * oh * ow, k * k * (c // 8))


@pytest.mark.parametrize("wgrad", [0, 1])
@pytest.mark.parametrize("c,k,stride,pad,b,h,w", SHAPES)
def test_gather_stays_inside_the_input(c, k, stride, pad, b, h, w, wgrad):
    want = _expected(c, k, stride, pad, b, h, w)
    up = lambda n, m: -(-n // m) * m
    rows, chunks = up(want.shape[0], 64 if wgrad else 128), up(want.shape[1], 16 if wgrad else 8)
    off = np.full((rows, chunks), -2, np.int32)
    rc = host_lib().nbh_conv_gather(*(ctypes.c_int(v) for v in (b, h, w, c, k, k, stride, pad, wgrad)),
                                        off.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(rows), ctypes.c_longlong(chunks))
    assert rc == 0 and off.max() <= b * h * w * c - 8
    full = np.full((rows, chunks), -1, np.int64)             # pixels past the last and taps past the last are zeros
    full[: want.shape[0], : want.shape[1]] = want
    assert np.array_equal(off, full)


def test_host_guards_are_the_kernels():
    """A layer chooses the gathering kernel exactly for the sizes that the kernel takes, in both directions."""
    from noeira_b200 import nn
    from noeira_b200.nn.conv import _gather_fits
    fits = lambda *v: bool(host_lib().nbh_conv_fits(*(ctypes.c_int(i) for i in v)))
    rng = np.random.default_rng(0)
    both = set()
    for _ in range(3000):
        k, stride = int(rng.integers(1, 8)), int(rng.integers(1, 4))
        pad, c, h, w = int(rng.integers(0, k)), 8 * int(rng.integers(1, 33)), int(rng.integers(k, 60)), int(rng.integers(k, 3000))
        b = max(1, int(2 ** 31 / (h * w * c) * rng.uniform(0.4, 1.5)))
        got = fits(b, h, w, c, k, k, stride, pad)
        assert _gather_fits(b, h, w, c, k, stride, pad) == got
        both.add(got)
    assert both == {True, False}
    # dy of a 'full' layer is larger than x: 20000 x 3 x 1002 x 64 elements for 20000 x 1 x 1000 x 64
    conv = nn.Conv2D(64, 64, 3, 1, 2)
    for b in (10000, 11159, 11165, 20000, 40000):
        conv._in = (b, 1, 1000)
        assert conv._implicit_dgrad_ok(1000) == fits(b, 3, 1002, 64, 3, 3, 1, 0)
        assert conv._implicit_ok(64, 1002) == fits(b, 1, 1000, 64, 3, 3, 1, 2)
