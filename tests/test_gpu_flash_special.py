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
