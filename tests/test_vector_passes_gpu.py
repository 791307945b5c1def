"""Norm backward, SwiGLU, activation, rotary and column-sum passes at odd sizes, pitches and alignments, against fp64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _g(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("m", [1, 9, 150, 2500])
@pytest.mark.parametrize("d", [8, 248, 264, 720, 1032, 2048, 2056])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_backward(m, d, rms):
    from noeira_b200 import nn
    g = _g(m * 7 + d)
    n = (nn.RMSNorm if rms else nn.LayerNorm)(d).to("cuda")
    n.gamma.set_(torch.rand(d) + 0.5)
    x = torch.randn(m, d, device="cuda", generator=g).bfloat16()
    dy = torch.randn(m, d, device="cuda", generator=g).bfloat16()
    n.forward(x)
    dx = n.vjp(dy)
    xd = x.double().requires_grad_(True)
    ga = n.gamma.data.double().requires_grad_(True)
    if rms:
        y = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + n.eps) * ga
    else:
        be = n.beta.data.double().requires_grad_(True)
        y = torch.nn.functional.layer_norm(xd, (d,), ga, be, n.eps)
    y.backward(dy.double())
    assert torch.allclose(dx.double(), xd.grad, rtol=2 ** -8, atol=1e-4)            # one bf16 rounding
    tol = 4e-6 * m ** 0.5 * 4 + 1e-5                                                # fp32 sums of m terms of order one
    assert torch.allclose(n.gamma.grad.double(), ga.grad, rtol=1e-5, atol=tol)
    if not rms:
        assert torch.allclose(n.beta.grad.double(), be.grad, rtol=1e-5, atol=tol)


@pytest.mark.parametrize("m,h,extra", [(1, 8, 0), (3, 10, 0), (67, 2056, 0), (5, 24, 8), (5, 24, 2), (300, 2048, 0),
                                       (70001, 8, 0), (8191, 72, 0), (2700, 200, 8), (1100, 512, 8), (257, 2056, 0), (25, 22536, 0)])
def test_swiglu(m, h, extra):
    from noeira_b200 import nn
    g = _g(m + h)
    buf = torch.randn(m, 2 * h + extra, device="cuda", generator=g).bfloat16()
    gu = buf[:, : 2 * h] if extra == 0 else buf.as_strided((m, 2 * h), (2 * h + extra, 1))
    dh = torch.randn(m, h, device="cuda", generator=g).bfloat16()
    act = nn.SwiGLU(h)
    if extra:                                                                       # pitched rows: the kernel entry itself
        from noeira_b200._native import check, cuda_lib, ptr, stream_ptr
        y = torch.empty(m, h, device="cuda", dtype=torch.bfloat16)
        check(cuda_lib().nb_swiglu_fwd(ptr(gu), ctypes.c_int(gu.stride(0)), ptr(y), ctypes.c_int(h), ctypes.c_int(m), ctypes.c_int(h),
                                       stream_ptr()), "swiglu_fwd")
        dgu = None
    else:
        y, dgu = act.forward(gu), act.vjp(dh)
    gd = gu.double().requires_grad_(True)
    ref = torch.nn.functional.silu(gd[:, :h]) * gd[:, h:]
    ref.backward(dh.double())
    assert torch.allclose(y.double(), ref, rtol=2 ** -8 + 1e-5, atol=1e-6)
    if dgu is not None:
        assert torch.allclose(dgu.double(), gd.grad, rtol=2 ** -8 + 1e-5, atol=1e-6)


@pytest.mark.parametrize("n", [1, 7, 8, 4097, 100000, (1 << 18) - 1, (1 << 18) + 5])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("act", ["relu", "gelu", "silu"])
def test_activation(n, off, act):
    from noeira_b200 import nn
    x = torch.randn(n + off, device="cuda", generator=_g(n)).bfloat16()[off:]
    dy = torch.randn(n, device="cuda", generator=_g(n + 1)).bfloat16()
    m = nn.Elementwise(act)
    y, dx = m.forward(x), m.vjp(dy)
    xd = x.double().requires_grad_(True)
    f = {"relu": torch.relu, "gelu": lambda t: torch.nn.functional.gelu(t, approximate="tanh"), "silu": torch.nn.functional.silu}[act]
    ref = f(xd)
    ref.backward(dy.double())
    assert torch.allclose(y.double(), ref, rtol=2 ** -8 + 1e-5, atol=1e-6)
    assert torch.allclose(dx.double(), xd.grad, rtol=2 ** -8 + 1e-5, atol=2e-6)


@pytest.mark.parametrize("b,s,h,d", [(1, 1, 1, 16), (2, 33, 5, 64), (3, 7, 15, 128), (2, 9, 3, 8), (1, 300, 6, 48), (2, 401, 7, 64), (3, 300, 9, 48),
                                     (17, 300, 1, 64)])
@pytest.mark.parametrize("packed", [False, True])
def test_rope(b, s, h, d, packed):
    from noeira_b200.nn import rope_
    g = _g(b * s + d)
    full = torch.randn(b, s, h + (3 if packed else 0), d, device="cuda", generator=g).bfloat16()
    x = full[:, :, :h]
    ref = x.double().clone()
    inv = 1e4 ** (-torch.arange(d // 2, dtype=torch.float64, device="cuda") * 2 / d)
    a = (5 + torch.arange(s, dtype=torch.float64, device="cuda"))[:, None] * inv
    sn, cs = a.sin()[None, :, None], a.cos()[None, :, None]
    r = torch.cat([ref[..., : d // 2] * cs - ref[..., d // 2:] * sn, ref[..., d // 2:] * cs + ref[..., : d // 2] * sn], -1)
    keep = full[:, :, h:].clone()
    rope_(x, 1e4, pos0=5)
    # angles of up to ~300 in fp32 (2^-24 each), one bf16 rounding
    assert torch.allclose(x.double(), r, rtol=2 ** -8, atol=2e-3)
    assert torch.equal(full[:, :, h:], keep)


@pytest.mark.parametrize("m,n", [(1, 8), (63, 40), (64, 33), (5000, 264), (20000, 16)])
def test_colsum(m, n):
    from noeira_b200.nn.layers import colsum_into
    x = torch.randn(m, n, device="cuda", generator=_g(m + n)).bfloat16()
    out = torch.ones(n, device="cuda")
    colsum_into(x, out, n)
    assert torch.allclose(out.double(), x.double().sum(0) + 1, rtol=1e-5, atol=4e-6 * m ** 0.5 * 4 + 1e-5)
