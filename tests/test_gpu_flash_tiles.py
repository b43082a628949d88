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


@pytest.mark.parametrize("B,H,Sq,Sk,hd,causal,pad", [
    (10, 8, 64, 64, 64, True, False), (10, 8, 1, 128, 64, False, False), (37, 4, 128, 128, 128, True, False),
    (25, 3, 127, 65, 64, False, True), (9, 16, 65, 127, 128, False, True), (8, 16, 100, 100, 128, True, False)])
def test_one_head_a_cta(B, H, Sq, Sk, hd, causal, pad):
    """Heads of one block of keys and of queries, more than half as many as SMs and no more than SMs.  Padding leaves every batch entry
    half of its keys: with a single one dS is 0 and what is left of it the rounding of two fp32 sums, which no norm measures."""
    from rtp_b200.ops import _lib
    from rtp_b200.ops.flash import flash_attention
    g = torch.Generator(device="cuda").manual_seed(B * 1000 + Sq)
    q, do = (torch.randn(B, Sq, H, hd, generator=g, device="cuda").to(BF) for _ in range(2))
    k, v = (torch.randn(B, Sk, H, hd, generator=g, device="cuda").to(BF) for _ in range(2))
    kpm = torch.arange(Sk, device="cuda")[None] >= torch.randint(Sk // 2, Sk + 1, (B, 1), generator=g, device="cuda") if pad else None
    for t in (q, k, v):
        t.requires_grad_()
    o = flash_attention(q, k, v, causal=causal, key_padding_mask=kpm)
    got = [o.detach(), *torch.autograd.grad(o, (q, k, v), do)]
    _lib.check_status()
    for name, x, r in zip(("o", "dq", "dk", "dv"), got, exact(q.detach(), k.detach(), v.detach(), do, causal, kpm)):
        assert x.isfinite().all(), name
        assert ((x.double() - r).norm() <= 2.0 ** -7 * r.norm()).item(), (name, ((x.double() - r).norm() / r.norm()).item())
        e, n = (x.double() - r).norm(dim=(1, 3)), r.norm(dim=(1, 3))          # head by head
        assert bool((e <= 2.0 ** -6 * n).all()), (name, (e / n).max().item())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("masked", [False, True])
def test_one_head_a_cta_with_dropout(hd, masked):
    """The same heads in a launch of few, which takes two CTAs a head: the same dropout bits, the same results (P and dS are rounded to
    bf16 from sums in another orientation: 2^-7 of the norm)."""
    from rtp_b200.ops.flash import flash_attention
    g = torch.Generator(device="cuda").manual_seed(hd)
    q, k, v, do = (torch.randn(10, 100, 8, hd, generator=g, device="cuda").to(BF) for _ in range(4))
    mask = torch.randn(100, 100, generator=g, device="cuda") if masked else None

    def run(n):
        x, y, z = (t[:n].clone().requires_grad_() for t in (q, k, v))
        o = flash_attention(x, y, z, attn_mask=mask, causal=not masked, dropout_p=0.2, seed=3, offset=9)
        return [o.detach(), *torch.autograd.grad(o, (x, y, z), do[:n])]
    for a, b in zip(run(10), run(4)):
        a, b = a[:4].double(), b.double()
        assert b.norm() > 0 and ((a - b).norm() <= 2.0 ** -7 * b.norm()).item()
