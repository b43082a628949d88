"""GELU (erf form) and its gradient against float64 on every bf16 input whose result is a normal number.

Tolerance: one rounding to bf16 (2^-8), plus for the forward the fit's error (2^-14 relative, also in the lower tail) and for
the gradient, whose two terms cancel near its zero, 2^-18 of the larger one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_every_bf16_input():
    from rtp_b200.ops import kernels as K
    x = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda()
    d = x.double()
    cdf = 0.5 * torch.special.erfc(-d / 2.0 ** 0.5)
    ref = d * cdf
    ok = torch.isfinite(d) & ((ref.abs() > 1e-35) | (d == 0)) & (d.abs() < 1e30)
    y = K.gelu_fwd(x).double()
    assert bool(((y - ref).abs() <= (2.0 ** -8 + 2.0 ** -14) * ref.abs())[ok].all()), (y - ref)[ok].abs().max()
    second = d * torch.exp(-0.5 * d * d) / (2 * torch.pi) ** 0.5
    g = K.gelu_bwd(x, torch.ones_like(x)).double()
    ref = cdf + second
    assert bool(((g - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -18 * torch.maximum(cdf, second.abs()) + 1e-35)[ok].all())
    assert torch.isnan(K.gelu_fwd(torch.full((8,), float("nan"), device="cuda", dtype=torch.bfloat16))).all()
    assert torch.isinf(K.gelu_fwd(torch.full((8,), float("inf"), device="cuda", dtype=torch.bfloat16))).all()
