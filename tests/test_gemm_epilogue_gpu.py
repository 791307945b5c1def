"""The staged GEMM epilogue at the edges of its column groups and row quarters, against fp64 on the same bf16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ACTS = {None: lambda x: x, "relu": torch.relu, "gelu": lambda x: torch.nn.functional.gelu(x, approximate="tanh")}


@pytest.mark.parametrize("m,n", [(1, 8), (33, 24), (127, 40), (129, 64), (130, 72), (255, 136), (300, 200), (513, 264), (700, 328)])
@pytest.mark.parametrize("form", ["bias", "gelu", "residual", "f32", "accumulate", "pitch"])
@pytest.mark.parametrize("tiles", [1, 2])
def test_epilogue_edges(m, n, form, tiles):
    from noeira_b200 import ops
    from noeira_b200.ops.gemm import set_two_cta_mode
    g = torch.Generator(device="cuda").manual_seed(m * 1000 + n)
    k = 192
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    b = torch.randn(k, n, device="cuda", generator=g).bfloat16()
    bias = torch.randn(n, device="cuda", generator=g)
    res = torch.randn(m, n, device="cuda", generator=g).bfloat16()
    exact = a.double() @ b.double()
    kw, out = {}, None
    if form in ("bias", "gelu"):
        act = "gelu" if form == "gelu" else None
        kw, exact = dict(bias=bias, act=act), ACTS[act](exact + bias.double())
    elif form == "residual":
        kw, exact = dict(bias=bias, residual=res), exact + bias.double() + res.double()
    elif form == "f32":
        kw, exact = dict(bias=bias, out_dtype=torch.float32), exact + bias.double()
    elif form == "accumulate":
        out = torch.randn(m, n, device="cuda", generator=g)
        exact = exact + out.double()
        kw = dict(out=out, accumulate=True)
    else:                                                  # a row pitch without 16-byte rows: scalar copies, neighbours untouched
        buf = torch.full((m, n + 3), 7.0, device="cuda", dtype=torch.bfloat16)
        kw = dict(out=buf[:, :n])
    old = set_two_cta_mode(tiles)
    try:
        y = ops.gemm(a, b, b_mn=True, **kw)
    finally:
        set_two_cta_mode(old)
    # one rounding of the result to its type; the 192 fp32 products and additions; GELU through the 2^-11 hardware tanh
    eps = 2.0 ** -8 if y.dtype == torch.bfloat16 else 0.0
    err = (y.double() - exact).abs()
    bound = eps * exact.abs() + 192 * 2.0 ** -23 * k ** 0.5 * 4 + (2.0 ** -9 * exact.abs() + 2e-3 if form == "gelu" else 0.0)
    assert bool((err <= bound).all()), float((err - bound).max())
    if form == "pitch":
        assert bool((buf[:, n:] == 7.0).all())


@pytest.mark.parametrize("n", [4, 8, 12, 15, 16, 40, 72])
@pytest.mark.parametrize("shift", [1, 2, 3, 5])
@pytest.mark.parametrize("k", [64, 4096])                   # one range of K, and split ranges with a second kernel
@pytest.mark.parametrize("form", ["bf16", "f32", "accumulate", "residual"])
def test_outputs_off_the_16_byte_grid(n, shift, k, form):
    """Columns of a wider tensor whose pitch is a whole number of 16-byte words and whose base is not; residual and bias alike."""
    from noeira_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n * 100 + shift)
    m = 37
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    b = torch.randn((n + 7) // 8 * 8, k, device="cuda", generator=g).bfloat16()[:n]
    dt = torch.float32 if form in ("f32", "accumulate") else torch.bfloat16
    buf = torch.full((m, 96), 7.0, device="cuda", dtype=dt)
    out, kw = buf[:, shift:shift + n], {}
    exact = a.double() @ b.double().t()
    if form == "accumulate":
        kw, exact = dict(accumulate=True), exact + 7.0
    else:
        bias = torch.randn(n + shift, device="cuda", generator=g)[shift:]
        kw, exact = dict(bias=bias), exact + bias.double()
        if form == "residual":
            res = torch.randn(m, 96, device="cuda", generator=g).bfloat16()[:, shift:shift + n]
            kw["residual"], exact = res, exact + res.double()
    ops.gemm(a, b, out=out, n=n, **kw)
    # one rounding to the result's type; k / 16 additions into an fp32 sum of order sqrt(k)
    bound = (2.0 ** -8 if dt is torch.bfloat16 else 2.0 ** -22) * exact.abs() + (k / 16 + 4) * 2.0 ** -23 * 4 * k ** 0.5
    err = (out.double() - exact).abs()
    assert bool((err <= bound).all()), float((err - bound).max())
    assert bool((buf[:, :shift] == 7.0).all()) and bool((buf[:, shift + n:] == 7.0).all())


def test_output_of_another_rank():
    """`out` may be [M] for one column or [M, 1, N]: rows are what its first stride says."""
    from noeira_b200 import ops
    a, b = torch.randn(40, 64, device="cuda").bfloat16(), torch.randn(8, 64, device="cuda").bfloat16()
    ref = ops.gemm(a, b, out_dtype=torch.float32)
    one, mid = torch.zeros(40, device="cuda"), torch.zeros(40, 1, 8, device="cuda")
    ops.gemm(a, b[:1], out=one, n=1)
    ops.gemm(a, b, out=mid)
    assert torch.equal(mid[:, 0], ref) and torch.equal(one, ref[:, 0])
