"""Flash attention at the edges of its tiles and of its choices: sequences that end inside, at and one past a 128-row tile, one
and two row tiles a CTA, keys shared out between the two halves of a CTA, launches of one round and of several (persistent
CTAs), groups of heads, fully padded key blocks and rows.

Tolerance: P, dS and the results are each rounded to bf16 once (2^-9 of the value, at random), the inputs are exact: the norm of
the error stays under 2^-7 of the norm of the result; a tile that is stale or misplaced is off by as much as the result."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def exact(q, k, v, do, causal, kpm):
    q, k, v = (t.double().transpose(1, 2).requires_grad_() for t in (q, k, v))
    s = q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    if kpm is not None:
        s = s.masked_fill(kpm[:, None, None, :], float("-inf"))
    p = torch.softmax(s, -1).nan_to_num(0.0)          # a row without keys gives zeros
    o = (p @ v).transpose(1, 2)
    return [o, *(t.transpose(1, 2) for t in torch.autograd.grad(o, (q, k, v), do.double()))]


@pytest.mark.parametrize("B,H,Sq,Sk,hd,causal,pad", [
    (1, 1, 1, 1, 64, True, False), (1, 2, 127, 127, 64, True, False), (1, 2, 128, 129, 128, False, False),
    (2, 3, 129, 128, 64, False, False), (1, 2, 257, 257, 128, True, False), (1, 1, 300, 1100, 64, False, False),
    (1, 1, 1100, 300, 128, False, False), (2, 3, 260, 300, 64, False, True), (1, 2, 640, 640, 128, True, False),
    (9, 17, 129, 129, 64, True, False), (9, 17, 130, 385, 64, False, True), (10, 16, 513, 513, 128, True, False),
    (1, 150, 385, 200, 64, False, False), (5, 16, 700, 700, 128, True, True), (2, 40, 640, 1300, 64, False, True)])
def test_tiles(B, H, Sq, Sk, hd, causal, pad):
    from rtp_b200.ops import _lib
    from rtp_b200.ops.flash import flash_attention
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + Sq)
    q, do = (torch.randn(B, Sq, H, hd, generator=g, device="cuda").to(BF) for _ in range(2))
    k, v = (torch.randn(B, Sk, H, hd, generator=g, device="cuda").to(BF) for _ in range(2))
    kpm = None
    if pad:
        n = torch.randint(1, Sk + 1, (B, 1), generator=g, device="cuda")
        n[0] = Sk // 3                                # whole blocks of padding at the end
        kpm = torch.arange(Sk, device="cuda")[None] >= n
        kpm[-1] = False
        kpm[-1, :min(Sk - 1, 140)] = True             # and at the beginning
    for t in (q, k, v):
        t.requires_grad_()
    o = flash_attention(q, k, v, causal=causal, key_padding_mask=kpm)
    got = [o.detach(), *torch.autograd.grad(o, (q, k, v), do)]
    _lib.check_status()
    for name, x, r in zip(("o", "dq", "dk", "dv"), got, exact(q.detach(), k.detach(), v.detach(), do, causal, kpm)):
        assert x.isfinite().all(), name
        assert ((x.double() - r).norm() <= 2.0 ** -7 * r.norm() + 1e-6).item(), (name, ((x.double() - r).norm() / r.norm()).item())
        for b in range(B):                            # a single wrong tile of one head is seen as well
            for h in range(0, H, max(H // 4, 1)):
                e, n = (x[b, :, h].double() - r[b, :, h]).norm(), r[b, :, h].norm()
                assert (e <= 2.0 ** -6 * n + 1e-6).item(), (name, b, h, (e / n).item())


@pytest.mark.parametrize("B,H,S", [(1, 2, 300), (9, 18, 300)])
def test_repeats_are_equal(B, H, S):
    """Nothing is summed in an order that depends on who is first: two calls give the same bits."""
    from rtp_b200.ops.flash import flash_attention
    q, k, v = (torch.randn(B, S, H, 64, device="cuda").to(BF).requires_grad_() for _ in range(3))
    do = torch.randn(B, S, H, 64, device="cuda").to(BF)
    runs = []
    for _ in range(2):
        o = flash_attention(q, k, v, causal=True)
        runs.append([o.detach(), *torch.autograd.grad(o, (q, k, v), do)])
    assert all(torch.equal(a, b) for a, b in zip(*runs))
