"""The gathering convolution (forward, input and weight gradient) at odd widths, strides, paddings and channel counts, against
fp64 convolutions of the same bf16 tensors."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ic,oc,k,stride,pad,b,h,w", [
    (64, 64, 3, 1, 1, 2, 17, 23), (64, 128, 3, 2, 1, 3, 15, 21), (128, 256, 3, 2, 1, 1, 9, 8), (3, 64, 7, 2, 3, 2, 33, 45),
    (64, 128, 1, 2, 0, 2, 11, 13), (8, 8, 3, 1, 0, 1, 5, 4), (72, 40, 5, 3, 2, 2, 19, 14), (256, 320, 3, 1, 1, 2, 7, 7),
    (512, 512, 3, 1, 1, 1, 5, 6), (64, 64, 3, 1, 2, 1, 4, 3), (128, 64, 3, 1, 1, 1, 1, 1), (16, 192, 2, 2, 1, 2, 6, 9)])
def test_gathered_convolution(ic, oc, k, stride, pad, b, h, w):
    from noeira_b200 import nn
    from noeira_b200.ops import check_status
    nn.manual_seed(ic + oc)
    c = nn.Conv2D(ic, oc, k, stride, pad, bias=True, relu=False).to("cuda")
    c.bias.set_(torch.randn(oc))
    g = torch.Generator(device="cuda").manual_seed(h * w)
    x = torch.zeros(b, h, w, c.icp, device="cuda", dtype=torch.bfloat16)
    x[..., :ic] = torch.randn(b, h, w, ic, device="cuda", generator=g).bfloat16()
    y = c.forward(x)
    assert c._col is None
    dy = torch.randn(y.shape, device="cuda", generator=g).bfloat16()
    c.weight.grad_storage.fill_(0.5)
    dx = c.vjp(dy)
    torch.cuda.synchronize()
    check_status()
    wt = c.weight.file_view(c.weight.shadow[:, :oc].float()).double()
    xd, dyd = x[..., :ic].double().permute(0, 3, 1, 2), dy.double().permute(0, 3, 1, 2)
    ref = torch.nn.functional.conv2d(xd, wt, c.bias.data.double(), stride, pad).permute(0, 2, 3, 1)
    n = ic * k * k
    # fp32 accumulation of n products of order 1 / sqrt(n) (weights) with truncation per 16, one bf16 rounding
    assert torch.allclose(y.double(), ref, rtol=2 ** -8, atol=n / 16 * 2 ** -23 * 8 + 1e-6)
    gw = torch.nn.grad.conv2d_weight(xd, wt.shape, dyd, stride, pad)
    m = y.numel() // oc
    got = c.weight.file_view((c.weight.grad - 0.5).contiguous())
    assert torch.allclose(got.double(), gw, rtol=1e-5, atol=(m / 16 + 40) * 2 ** -23 * 4 * m ** 0.5 + 1e-5)
    gx = torch.nn.grad.conv2d_input(xd.shape, wt, dyd, stride, pad).permute(0, 2, 3, 1)
    # strided layers and narrow outputs go through a bf16 patch-gradient matrix: k*k rounded terms of order sqrt(oc / n) instead
    # of one rounding
    tol = 2 ** -8 * (oc / n) ** 0.5 * 4 * k if stride > 1 or oc % 64 else oc * k * k / 16 * 2 ** -23 * 8 + 1e-6
    assert torch.allclose(dx[..., :ic].double(), gx, rtol=2 ** -8, atol=tol)


def test_gathered_convolution_repeats_bits():
    from noeira_b200 import nn
    c = nn.Conv2D(64, 64, 3, 1, 1).to("cuda")
    x = torch.randn(4, 50, 62, 64, device="cuda").bfloat16()
    out = []
    for _ in range(2):
        c.weight.grad_storage.zero_()
        y = c.forward(x)
        out.append((y.clone(), c.vjp(y).clone(), c.weight.grad.clone()))
    assert all(torch.equal(p, q) for p, q in zip(*out))


def test_convolution_captured_before_any_eager_product():
    """The forward needs no workspace: a graph may be captured before one exists on the device."""
    from noeira_b200 import nn
    from noeira_b200.ops import check_status, device_status
    from noeira_b200.ops.gemm import _WS
    device_status()
    c = nn.Conv2D(512, 64, 3, 1, 1).to("cuda")               # long reduction, few tiles: splits when it has a workspace
    x = torch.randn(1, 8, 16, 512, device="cuda").bfloat16()
    c.weight.shadow
    torch.cuda.synchronize()
    kept = dict(_WS)
    _WS.clear()
    try:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y = c.forward(x)
    finally:
        _WS.update(kept)
    g.replay()
    torch.cuda.synchronize()
    check_status()
    z = c.forward(x)
    # two orders of 4608 / 16 fp32 additions of partial sums below 4, one bf16 rounding each
    assert torch.allclose(y.float(), z.float(), rtol=2 ** -7, atol=288 * 2 ** -23 * 8)
