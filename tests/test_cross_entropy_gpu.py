"""Cross-entropy over rows of every form its dispatch knows, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v,pitch", [(5, 8), (8, 8), (65, 72), (513, 520), (4099, 4104), (32768, 32768), (49152, 49152), (102400, 102400),
                                     (130001, 130008), (37, 37), (100, 102)])
@pytest.mark.parametrize("m", [1, 7])
def test_cross_entropy_forms(v, pitch, m):
    from noeira_b200 import nn
    g = torch.Generator(device="cuda").manual_seed(v + m)
    buf = torch.full((m, pitch), 3.0, device="cuda", dtype=torch.bfloat16)
    x = (torch.randn(m, v, device="cuda", generator=g) * 3).bfloat16()
    x[0, v // 2] = float("-inf")                                        # a masked class
    buf[:, :v] = x
    t = torch.randint(0, v, (m,), device="cuda", generator=g)
    t[0] = v - 1 if v // 2 != v - 1 else 0
    if m > 2:
        t[2] = -100                                                     # ignored: no loss, zero gradient
    xd = x.double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(xd, t, ignore_index=-100, reduction="sum") / m
    ref.backward()
    acc = torch.zeros(1, device="cuda")
    d = nn.cross_entropy(buf[:, :v], t, acc)
    assert abs(float(acc) - ref.item()) <= 1e-5 * abs(ref.item()) + 1e-5      # fp32 sums
    # fast exponentials: a few units of 2^-22 per argument unit (at most ~30), one bf16 rounding
    assert torch.allclose(d.double(), xd.grad, rtol=2 ** -8 + 30 * 2 ** -21, atol=1e-9)
    assert bool((buf[:, v:] == 3.0).all())
