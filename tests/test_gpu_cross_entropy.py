"""Softmax cross-entropy over vocabularies on both sides of what a block's registers hold, with
ignored targets, masked (-inf) logits, padded row pitches and incoming gradients other than one.

Tolerance: the loss is an fp32 sum of at most 60 000 exponentials (2^-18 relative of a value near log V); a gradient is an
fp32 value rounded to bf16 (2^-8 of itself for each rounding), plus the fp32 error of a probability near one (2^-20 of
the factor)."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [8, 1032, 8192, 12296, 16392, 20488, 32000, 36864, 50304, 65536, 65544])
@pytest.mark.parametrize("M", [1, 150, 611])
@pytest.mark.parametrize("factor", [1.0, 3.0])
def test_loss_and_gradient(V, M, factor):
    from rtp_b200.ops import functional as FO
    g = torch.Generator(device="cuda").manual_seed(V + M)
    wide = (4 * torch.randn(M, V + 16, generator=g, device="cuda")).to(torch.bfloat16)
    wide[0, : V // 2] = float("-inf")
    t = torch.randint(V // 2, V, (M,), generator=g, device="cuda")
    if M > 1:
        t[1] = -100
    lg = wide[:, :V].requires_grad_()
    before = wide.clone()
    loss = FO.cross_entropy(lg, t)
    (grad,) = torch.autograd.grad(loss * factor, lg)
    ref_in = before[:, :V].double().requires_grad_()
    ref = F.cross_entropy(ref_in, t, ignore_index=-100)
    (rg,) = torch.autograd.grad(ref * factor, ref_in)
    assert torch.equal(wide.detach(), before)
    assert abs(loss.item() - ref.item()) <= 2.0 ** -16 * (1 + abs(ref.item()))
    n = max(1, int((t != -100).sum()))
    # roundings to bf16 (2^-8 each): the gradient, and again its product with the incoming factor; beyond the registers the
    # probability, the factor and their product
    rel = 2.0 ** -8 * (3 if V > 65536 else 1 if factor == 1.0 else 2)
    assert bool(((grad.double() - rg).abs() <= rel * rg.abs() + 2.0 ** -20 * factor / n).all())
    with torch.no_grad():
        assert FO.cross_entropy(lg, t).item() == loss.item()


@pytest.mark.parametrize("M,V", [(511, 16392), (512, 16392), (512, 20472), (3, 32776), (513, 50304), (64, 65536), (2047, 8200),
                                 (2048, 8192), (2048, 8200), (2048, 16384)])
def test_loss_alone_has_the_same_bits(M, V):
    """Losses without a gradient may come from another kernel: row by row the same bits, whatever was ignored or masked; and
    a gradient that overwrites the logits is the one that goes to a buffer of its own."""
    from rtp_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + V)
    lg = (3 * torch.randn(M, V, generator=g, device="cuda")).to(torch.bfloat16)
    lg[0, 5:] = float("-inf")
    t = torch.randint(0, V, (M,), generator=g, device="cuda")
    t[0], t[1], t[2] = 0, -100, V + 3          # one of the few finite logits, ignored, out of range
    alone = K.cross_entropy_to(lg, t, None)
    grad, over = torch.empty_like(lg), lg.clone()
    assert torch.equal(alone, K.cross_entropy_to(lg, t, grad, grad_scale=0.5))
    assert torch.equal(alone, K.cross_entropy_(over, t, grad_scale=0.5)) and torch.equal(grad, over)
    assert not grad[1].any() and not grad[2].any()
    ref = F.cross_entropy(lg[3:].double(), t[3:], reduction="none") if M > 3 else None
    if ref is not None:
        assert bool(((alone[3:].double() - ref).abs() <= 2.0 ** -16 * (1 + ref.abs())).all())
    assert alone[1].item() == 0 and alone[2].item() == 0


def test_two_backward_passes():
    """The gradient buffer is scaled in place: a second pass over the same graph is refused, as for any tensor that was
    saved for backward and then modified."""
    from rtp_b200.ops import functional as FO
    lg = torch.randn(4, 64, device="cuda").to(torch.bfloat16).requires_grad_()
    loss = FO.cross_entropy(lg, torch.zeros(4, dtype=torch.int64, device="cuda"))
    loss.backward(retain_graph=True)
    with pytest.raises(RuntimeError):
        loss.backward()
