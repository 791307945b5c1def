"""Scratch buffers that grow after a graph has been captured with the smaller one."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_captured_bias_gradient_survives_growth():
    from noeira_b200._native import cuda_lib
    from noeira_b200.nn import layers
    from noeira_b200.ops.streams import Scratch
    pool = Scratch(256 * 8192)
    old, layers._colsum_workspace = layers._colsum_workspace, pool.get       # nothing of earlier tests
    try:
        split = cuda_lib().nb_colsum_split(ctypes.c_int(1 << 20))
        dy = torch.randn(1 << 15, 64, device="cuda").bfloat16()
        out = torch.zeros(64, device="cuda")
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            layers.colsum_into(dy, out, 64)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            layers.colsum_into(dy, out, 64, accumulate=False)
        small = pool.get(dy.device, 1)
        where, n = small.data_ptr(), small.numel()
        del small
        wide = n // split + 8
        big = torch.randn(4096, wide, device="cuda").bfloat16()
        while cuda_lib().nb_colsum_split(ctypes.c_int(big.shape[0])) * wide <= n:
            big = torch.cat([big, big])
        layers.colsum_into(big, torch.zeros(wide, device="cuda"), wide)
        fills = [torch.full((n,), 3.0, device="cuda") for _ in range(4)]
        assert pool.get(dy.device, 1).data_ptr() != where
        g.replay()
        torch.cuda.synchronize()
        assert all(bool((f == 3.0).all()) for f in fills)
        # fp32 sums of 32768 terms of order one
        assert torch.allclose(out.double(), dy.double().sum(0), rtol=1e-5, atol=1e-5 * dy.shape[0] ** 0.5 * 4)
    finally:
        layers._colsum_workspace = old
