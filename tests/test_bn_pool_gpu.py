"""BatchNorm, max-pool and image-normalise passes at the edges of their row / channel mapping, against fp64 or torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,w,c", [(1, 1, 2, 8), (1, 3, 5, 24), (2, 7, 9, 64), (3, 33, 31, 136), (2, 5, 3, 2056), (4, 61, 47, 512), (1, 33, 31, 8), (2, 3, 3, 2048),
                                     (1, 8, 8, 256)])
@pytest.mark.parametrize("res", [False, True])
def test_batchnorm_edges(b, h, w, c, res):
    from noeira_b200 import nn
    g = torch.Generator(device="cuda").manual_seed(c + h)
    bn = nn.BatchNorm2D(c, relu=True).to("cuda")
    bn.gamma.set_(torch.rand(c) + 0.5)
    bn.beta.set_(torch.randn(c))
    x = torch.randn(b, h, w, c, device="cuda", generator=g).bfloat16()
    r = torch.randn(b, h, w, c, device="cuda", generator=g).bfloat16() if res else None
    dy = torch.randn(b, h, w, c, device="cuda", generator=g).bfloat16()
    y = bn.forward(x, residual=r)
    out = bn.vjp(dy)
    dx, dres = out if res else (out, None)
    xd, M = x.double().reshape(-1, c), b * h * w
    ga, be = bn.gamma.data.double(), bn.beta.data.double()
    mean, var = xd.mean(0), xd.var(0, unbiased=False)
    rstd = torch.rsqrt(var + bn.eps)
    xh = (xd - mean) * rstd
    pre = xh * ga + be + (r.double().reshape(-1, c) if res else 0)
    assert torch.allclose(y.double().reshape(-1, c), pre.clamp_min(0), rtol=2 ** -8, atol=1e-4)
    gm = dy.double().reshape(-1, c) * (y.reshape(-1, c) > 0)          # the mask is the stored output's
    # fp32 sums of M terms of order one, one bf16 rounding of dx
    tol = 1e-5 * M ** 0.5 + 1e-5
    assert torch.allclose(bn.beta.grad.double(), gm.sum(0), rtol=1e-5, atol=tol)
    assert torch.allclose(bn.gamma.grad.double(), (gm * xh).sum(0), rtol=1e-4, atol=10 * tol)
    ref = ga * rstd * (gm - gm.mean(0) - xh * (gm * xh).mean(0))
    scale = float((ga * rstd).max())                                    # two pixels per channel: rstd reaches 1 / sqrt(eps)
    assert torch.allclose(dx.double().reshape(-1, c), ref, rtol=2 ** -8, atol=2e-4 * max(scale, 1.0))
    if res:
        assert torch.equal(dres.double().reshape(-1, c), gm)


@pytest.mark.parametrize("b,h,w,c", [(1, 1, 1, 8), (2, 7, 9, 64), (2, 5, 3, 2056), (3, 33, 31, 136)])
@pytest.mark.parametrize("res", [False, True])
def test_batchnorm_inference_backward_uses_the_forward_statistics(b, h, w, c, res):
    """Running statistics that change between forward and vjp (weights loaded, an averaged copy swapped in) change neither."""
    from noeira_b200 import nn
    g = torch.Generator(device="cuda").manual_seed(c)
    bn = nn.BatchNorm2D(c, relu=True).to("cuda").eval()
    bn.gamma.set_(torch.rand(c) + 0.5)
    bn.beta.set_(torch.randn(c))
    bn.running_mean.data.copy_(torch.randn(c, device="cuda", generator=g))
    bn.running_var.data.copy_(torch.rand(c, device="cuda", generator=g) + 0.25)
    mean, rstd = bn.running_mean.data.double(), torch.rsqrt(bn.running_var.data.double() + bn.eps)
    x = torch.randn(b, h, w, c, device="cuda", generator=g).bfloat16()
    r = torch.randn(b, h, w, c, device="cuda", generator=g).bfloat16() if res else None
    dy = torch.randn(b, h, w, c, device="cuda", generator=g).bfloat16()
    y = bn.forward(x, residual=r)
    bn.running_mean.data.fill_(100.0)
    bn.running_var.data.fill_(100.0)
    out = bn.vjp(dy)
    dx = out[0] if res else out
    M, ga = b * h * w, bn.gamma.data.double()
    xh = (x.double().reshape(-1, c) - mean) * rstd
    pre = xh * ga + bn.beta.data.double() + (r.double().reshape(-1, c) if res else 0)
    assert torch.allclose(y.double().reshape(-1, c), pre.clamp_min(0), rtol=2 ** -8, atol=1e-4)
    gm = dy.double().reshape(-1, c) * (y.reshape(-1, c) > 0)
    tol = 1e-5 * M ** 0.5 + 1e-5                                      # fp32 sums of M terms of order one
    assert torch.allclose(bn.gamma.grad.double(), (gm * xh).sum(0), rtol=1e-4, atol=10 * tol)
    ref = ga * rstd * (gm - gm.mean(0) - xh * (gm * xh).mean(0))
    assert torch.allclose(dx.double().reshape(-1, c), ref, rtol=2 ** -8, atol=2e-4 * max(1.0, float((ga * rstd).max())))


@pytest.mark.parametrize("k,stride,pad", [(3, 2, 1), (3, 2, 0), (2, 2, 0), (5, 3, 2), (16, 4, 3), (1, 1, 0), (3, 1, 1), (3, 1, 0), (4, 1, 2), (8, 8, 0)])
@pytest.mark.parametrize("b,h,w,c", [(2, 17, 19, 64), (1, 16, 30, 12), (3, 40, 21, 8), (200, 20, 20, 32), (7, 90, 16, 64)])
def test_maxpool_edges(k, stride, pad, b, h, w, c):
    from noeira_b200 import nn
    g = torch.Generator(device="cuda").manual_seed(k * 100 + c)
    x = torch.randn(b, h, w, c, device="cuda", generator=g).bfloat16()
    pool = nn.MaxPool2D(k, stride, pad)
    y = pool.forward(x)
    xr = x.float().permute(0, 3, 1, 2).requires_grad_(True)
    yr = torch.nn.functional.max_pool2d(xr, k, stride, pad)
    assert torch.equal(y.float().permute(0, 3, 1, 2), yr)
    dy = torch.randn(y.shape, device="cuda", generator=g).bfloat16()
    yr.backward(dy.float().permute(0, 3, 1, 2))
    # torch and the kernel both take the first maximum of a window in row order; one bf16 rounding of the sum
    assert torch.allclose(pool.vjp(dy).float().permute(0, 3, 1, 2), xr.grad, rtol=2 ** -8, atol=1e-6)


@pytest.mark.parametrize("b,h,w", [(1, 1, 1), (2, 5, 7), (3, 6, 10), (2, 97, 131), (1, 64, 64)])
def test_normalize_images_edges(b, h, w):
    from noeira_b200 import nn
    img = torch.randint(0, 256, (b, 3, h, w), dtype=torch.uint8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(h))
    out = nn.normalize_images(img)
    mean, std = (torch.tensor(v, dtype=torch.float64, device="cuda").view(1, 3, 1, 1) for v in ((0.485, 0.456, 0.406), (0.229, 0.224, 0.225)))
    ref = ((img.double() / 255 - mean) / std).permute(0, 2, 3, 1)
    assert torch.allclose(out[..., :3].double(), ref, rtol=2 ** -8, atol=1e-6) and bool((out[..., 3:] == 0).all())
