"""Rotary attention and SwiGLU on packed projections against the separate split, rotation and activation that they replace:
the same arithmetic per element, read and written through other strides.

SwiGLU gives the same bits.  In a rotation the compiler may fuse either product of a * c - b * s into the subtraction, which
flips a rounding to bf16 (2^-7 of the element) in a few of 10^5 elements; attention spreads that out, it does not amplify
it: 2^-11 of the norm covers one flip in 10^4 elements (2^-7 * 10^-2) four times."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("B,S,H,hd", [(2, 100, 4, 64), (1, 257, 8, 128), (3, 97, 8, 64)])
@pytest.mark.parametrize("nshard", [1, 2, 4])
def test_rope_attention(B, S, H, hd, nshard):
    from rtp_b200.models.llama import apply_rope, rope_tables
    from rtp_b200.ops import functional as FO
    torch.manual_seed(S)
    D = H * hd
    qkv = torch.randn(B, S, 3 * D, device="cuda").to(BF).requires_grad_()
    do = torch.randn(B, S, D, device="cuda").to(BF)
    cos, sin = rope_tables(S, hd, 10000.0, "cuda")
    out = FO.rope_attention_packed(qkv, cos, sin, H, nshard)
    q, k, v = (t.view(B, S, H, hd) for t in FO._split_packed(qkv, 3, nshard))
    ref = FO.causal_attention(apply_rope(q, cos, sin), apply_rope(k, cos, sin), v).reshape(B, S, D)
    def close(a, b):
        assert ((a.double() - b.double()).norm() / b.double().norm()).item() <= 2.0 ** -11
    close(out, ref)
    before = qkv.detach().clone()
    (g,) = torch.autograd.grad(out, qkv, do)
    (r,) = torch.autograd.grad(ref, qkv, do)
    for i in range(3):
        close(FO._split_packed(g, 3, nshard)[i], FO._split_packed(r, 3, nshard)[i])
    assert torch.equal(qkv.detach(), before)


@pytest.mark.parametrize("rows,F", [((1,), 8), ((3, 37), 72), ((2, 250), 1536)])
@pytest.mark.parametrize("nshard", [1, 2, 4])
def test_swiglu(rows, F, nshard):
    from rtp_b200.ops import functional as FO
    torch.manual_seed(F)
    y = torch.randn(*rows, 2 * F * nshard, device="cuda").to(BF).requires_grad_()
    dy = torch.randn(*rows, F * nshard, device="cuda").to(BF)
    out, ref = FO.swiglu_packed(y, nshard), FO.swiglu(*FO._split_packed(y, 2, nshard))
    assert torch.equal(out, ref)
    assert torch.equal(FO.recompute(*out._rtp_recompute), out)
    assert torch.equal(torch.autograd.grad(out, y, dy)[0], torch.autograd.grad(ref, y, dy)[0])
