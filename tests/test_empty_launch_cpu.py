"""Launchers called with nothing to do return at once, without a launch (a grid of no blocks is an error)."""
import ctypes

from noeira_b200._native import cuda_lib

I, F, N = ctypes.c_int, ctypes.c_float, None


def test_empty_batches():
    lib = cuda_lib()
    for b, h, w, oh, ow in ((0, 8, 8, 4, 4), (2, 0, 8, 0, 4), (2, 8, 0, 4, 0)):
        geo = [I(v) for v in (b, h, w, 16, 3, 2, 1, oh, ow)]
        assert lib.nb_maxpool_fwd(N, N, N, *geo, N) == 0
        assert lib.nb_maxpool_bwd(N, N, N, *geo, N) == 0
        assert lib.nb_col2im(N, N, *(I(v) for v in (b, h, w, 16, 3, 3, 2, 1, oh, ow, 144)), N) == 0
        assert lib.nb_image_normalize(N, N, I(b), I(h), I(w), *(F(v) for v in (0, 0, 0, 1, 1, 1)), N) == 0
    for m, hid in ((0, 64), (4, 0)):
        assert lib.nb_swiglu_fwd(N, I(128), N, I(64), I(m), I(hid), N) == 0
        assert lib.nb_swiglu_bwd(N, I(128), N, I(64), N, I(m), I(hid), N) == 0
