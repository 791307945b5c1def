"""Tile form and split choice of the GEMM: every form and layout on shapes around the lines between them, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(200, 512, 512), (200, 520, 3200), (300, 264, 8192), (512, 3200, 1000), (1204, 512, 3200), (256, 256, 16384),
                                   (17, 256, 4096), (256, 6, 4096), (2048, 384, 6144), (4816, 512, 712), (3200, 960, 720)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, True), (False, False), (True, True)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_forms(m, n, k, a_mn, b_mn, mode):
    from noeira_b200 import ops
    from noeira_b200.ops.gemm import set_two_cta_mode
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    pad = lambda v: (v + 7) // 8 * 8
    a = (torch.randn(k, pad(m), device="cuda", generator=g) if a_mn else torch.randn(m, k, device="cuda", generator=g)).bfloat16()
    b = (torch.randn(k, pad(n), device="cuda", generator=g) if b_mn else torch.randn(n, k, device="cuda", generator=g)).bfloat16()
    a, b = (a[:, :m] if a_mn else a), (b[:, :n] if b_mn else b)
    bias = torch.randn(n, device="cuda", generator=g)
    out = torch.randn(m, pad(n), device="cuda", generator=g)[:, :n]
    old, before = set_two_cta_mode(mode), out.double()
    try:
        y = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, act="relu", n=n)
        ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=True, n=n)
    finally:
        set_two_cta_mode(old)
    exact = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    # the tensor core adds 16 products at a time into an fp32 sum and may truncate: k / 16 steps, each off by up to one unit in
    # the last place of a partial sum, which is of order sqrt(k) and here below 4 sqrt(k)
    tol = k / 16 * 2.0 ** -23 * 4 * k ** 0.5
    ref = torch.relu(exact + bias.double())
    assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + tol).all())
    assert bool(((out.double() - before - exact).abs() <= tol + 2.0 ** -22 * exact.abs()).all())
