"""Flash attention on scores that are not finite: a NaN or an infinity has to show in the output at whatever key it sits (one
exponential in four is a polynomial, which knows neither), and a key whose score is -inf has no weight.

Tolerance of the finite results: P and the result are each rounded to bf16 once (2^-9 of the value, at random): 2^-7 of the norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
# keys of one row tile and of two a CTA, one launch that fits the SMs and one that does not; heads of 64 and 128
SHAPES = [(1, 2, 256, 64), (2, 90, 300, 64), (2, 80, 256, 128)]


def inputs(B, H, S, hd):
    g = torch.Generator(device="cuda").manual_seed(S + hd)
    q, k, v = (torch.randn(B, S, H, hd, generator=g, device="cuda").to(BF) for _ in range(3))
    q[..., 0] = 1.0                       # the sign of a key's first column is that of an infinite score
    return q, k, v


def forward(q, k, v, **kw):
    from rtp_b200.ops import _lib
    from rtp_b200.ops.flash import flash_attention
    with torch.no_grad():
        o = flash_attention(q, k, v, **kw)
    _lib.check_status()
    return o


@pytest.mark.parametrize("B,H,S,hd", SHAPES)
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_not_finite_shows(B, H, S, hd, value):
    for key in [*range(8), *range(128, 136), S - 1]:
        q, k, v = inputs(B, H, S, hd)
        k[0, key, 0, 0] = value
        o = forward(q, k, v)
        assert not o[0, :, 0].isfinite().any(), key
        o[0, :, 0] = 0
        assert o.isfinite().all()
        o = forward(q, k, v, causal=True)
        assert o[0, :key, 0].isfinite().all() and not o[0, key:, 0].isfinite().any(), key


@pytest.mark.parametrize("B,H,S,hd", SHAPES)
def test_minus_infinity_has_no_weight(B, H, S, hd):
    q, k, v = inputs(B, H, S, hd)
    gone = torch.zeros(S, dtype=torch.bool, device="cuda")
    gone[[1, 6, 7, 130, 134]] = True
    k[:, gone, :, 0] = float("-inf")
    v[:, gone] = 1e4
    x, y, z = (t.double().transpose(1, 2) for t in (q, k, v))
    p = torch.softmax((x @ y.transpose(-1, -2) * hd ** -0.5).masked_fill(gone, float("-inf")), -1)
    ref = (p @ z).transpose(1, 2)
    assert ((forward(q, k, v).double() - ref).norm() <= 2.0 ** -7 * ref.norm()).item()
    k[0, :, 0, 0] = float("-inf")         # no key at all: zeros
    o = forward(q, k, v)
    assert bool((o[0, :, 0] == 0).all())
    assert ((o[:, :, 1:].double() - ref[:, :, 1:]).norm() <= 2.0 ** -7 * ref[:, :, 1:].norm()).item()


@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("B,H,S,hd", SHAPES)
def test_negative_scale(B, H, S, hd, padded):
    """Scores far apart, so that a reference other than their maximum overflows."""
    from rtp_b200.ops.flash import flash_attention
    q, k, v = (t.requires_grad_() for t in inputs(B, H, S, hd))
    do = torch.randn_like(q)
    kpm = None
    if padded:
        kpm = torch.zeros(B, S, dtype=torch.bool, device="cuda")
        kpm[:, 200:] = True
    o = flash_attention(q, k, v, key_padding_mask=kpm, sm_scale=-8.0)
    got = [o.detach(), *torch.autograd.grad(o, (q, k, v), do)]
    x, y, z = (t.detach().double().transpose(1, 2).requires_grad_() for t in (q, k, v))
    s = x @ y.transpose(-1, -2) * -8.0
    if padded:
        s = s.masked_fill(kpm[:, None, None], float("-inf"))
    r = (torch.softmax(s, -1) @ z).transpose(1, 2)
    # Scores are sums of hd products in fp32, a few hundred in size: 2^-23 * 2^9 * sqrt(hd) < 2^-10 of a weight, below P's rounding.
    # Gradients: dS = P (dP - delta), and delta is made of the output as bf16.  Rows with nearly all weight on one key have dP close
    # to delta there, so that its rounding counts as much as those of dS and of the result: twice the bound.
    ref = [r, *(t.transpose(1, 2) for t in torch.autograd.grad(r, (x, y, z), do.double()))]
    for name, a, b in zip(("o", "dq", "dk", "dv"), got, ref):
        assert a.isfinite().all(), name
        bound = 2.0 ** -7 if name == "o" else 2.0 ** -6
        assert ((a.double() - b).norm() <= bound * b.norm()).item(), (name, ((a.double() - b).norm() / b.norm()).item())
