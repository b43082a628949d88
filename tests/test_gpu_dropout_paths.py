"""Dropout inside flash attention and the norms, with values: the masks are read off the kernels themselves (unit vectors as
values, ones as the residual) and the results compared with float64 under those masks.

Tolerance: attention keeps probabilities and their gradients in bf16 (2^-9 each, at random) and rounds its results once more;
2^-6 of the norm is four times what that gives, and a wrong mask or factor is of the order of one.  Norms: as in
test_gpu_norm_paths.py, a rounding to bf16 (2^-8) of fp32 arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("Sq,Sk,hd,causal,pad", [(300, 300, 64, False, False), (140, 260, 64, False, False),
                                                 (260, 132, 128, False, False), (300, 300, 128, True, False),
                                                 (388, 388, 64, True, True), (130, 300, 64, False, True),
                                                 (300, 516, 128, False, True)])
def test_flash(Sq, Sk, hd, causal, pad):
    from rtp_b200.ops.flash import flash_attention
    B, H, p = 2, 3, 0.25
    g = torch.Generator(device="cuda").manual_seed(Sq + Sk)
    q, do = (torch.randn(B, Sq, H, hd, generator=g, device="cuda").to(BF) for _ in range(2))
    k, v = (torch.randn(B, Sk, H, hd, generator=g, device="cuda").to(BF) for _ in range(2))
    kpm = None
    if pad:          # the second sequence has holes and a padded end
        kpm = torch.zeros(B, Sk, dtype=torch.bool, device="cuda")
        kpm[0, Sk - Sk // 3:] = True
        kpm[1] = torch.rand(Sk, generator=g, device="cuda") < 0.3
        kpm[1, 0] = False
    kw = dict(causal=causal, key_padding_mask=kpm, dropout_p=p, seed=11, offset=5)
    keep = torch.zeros(B, H, Sq, Sk, dtype=torch.float64, device="cuda")
    for c in range(0, Sk, hd):
        n = min(hd, Sk - c)
        unit = torch.zeros(B, Sk, H, hd, device="cuda", dtype=BF)
        unit[:, c:c + n, :, :n] = torch.eye(n, device="cuda", dtype=BF)[None, :, None]
        keep[..., c:c + n] = (flash_attention(q, k, unit, **kw)[..., :n].permute(0, 2, 1, 3) != 0).double() / (1 - p)
    qd, kd, vd = (t.double().permute(0, 2, 1, 3).requires_grad_() for t in (q, k, v))
    s = qd @ kd.transpose(-1, -2) * hd ** -0.5
    dead = torch.zeros(B, 1, Sq, Sk, dtype=torch.bool, device="cuda")
    if causal:
        dead = dead | torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").triu(1)
    if pad:
        dead = dead | kpm[:, None, None]
    alive = (~dead).expand_as(keep)
    assert abs((keep[alive] > 0).double().mean().item() - (1 - p)) < 0.01
    assert not (keep[~alive] > 0).any()
    o = (torch.softmax(s.masked_fill(dead, float("-inf")), -1) * keep) @ vd
    qk, kk, vk = (t.detach().requires_grad_() for t in (q, k, v))
    got = flash_attention(qk, kk, vk, **kw)
    grads = torch.autograd.grad(got, (qk, kk, vk), do)
    ref = torch.autograd.grad(o, (qd, kd, vd), do.double().permute(0, 2, 1, 3))
    for a, r in zip((got.detach(), *grads), (o.detach(), *ref)):
        a = a.double().permute(0, 2, 1, 3)
        assert ((a - r).norm() / r.norm()).item() < 2.0 ** -6
        # block by block of keys or queries, so that a mask that is wrong in one place only does not drown
        for c in range(0, r.shape[2], 64):
            x, y = a[:, :, c:c + 64], r[:, :, c:c + 64]
            assert (x - y).norm().item() <= 2.0 ** -5 * y.norm().item() + 2.0 ** -8 * r.norm().item() * (64 / r.shape[2]) ** 0.5


@pytest.mark.parametrize("D", [8, 256, 264, 512, 520, 1024, 1032, 1536, 2048, 2056, 4104, 5120, 8192])
@pytest.mark.parametrize("M", [1, 140, 297, 1030, 2500, 4099])
@pytest.mark.parametrize("rms", [False, True])
def test_norm(D, M, rms):
    from rtp_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(D + M)
    p = 0.3

    def rnd(*s):
        return torch.randn(*s, generator=g, device="cuda").to(BF)
    x, sub, dy, dres, gamma, beta = rnd(M, D), rnd(M, D), rnd(M, D), rnd(M, D), rnd(D), rnd(D)
    kw = dict(rms=rms, drop_p=p, seed=5, offset=9)
    ones = torch.ones(M, D, device="cuda", dtype=BF)
    keep = K.norm_fwd(torch.zeros_like(x), ones, gamma, None if rms else beta, **kw)[1] != 0
    if M * D > 10000:
        assert abs(keep.double().mean().item() - (1 - p)) < 0.02
    scale = keep.double() / (1 - p)
    y, h, mean, rstd = K.norm_fwd(x, sub, gamma, None if rms else beta, **kw)

    def close(a, r, mag, rel=2.0 ** -8):
        assert bool(((a.double() - r).abs() <= rel * r.abs() + 2.0 ** -16 * mag).all()), (a.double() - r).abs().max().item()
    href = x.double() + sub.double() * scale
    close(h, href, href.abs().max())
    hd, gd = h.double().requires_grad_(), gamma.double()
    mu = hd.mean(-1, keepdim=True) if not rms else 0.0
    ref = (hd - mu) * torch.rsqrt((hd - mu).pow(2).mean(-1, keepdim=True) + 1e-5) * gd + (0.0 if rms else beta.double())
    close(y, ref.detach(), ref.detach().abs().max())
    dx, dsub, dg, db = K.norm_bwd(dy, h, gamma, mean, rstd, has_beta=not rms, dres=dres, **kw)
    (rx,) = torch.autograd.grad(ref, hd, dy.double())
    rx = rx + dres.double()
    mag = (dy.double() * gd).abs().amax() * rstd.double().max() * 4 + dres.double().abs().max()
    close(dx, rx, mag)
    close(dsub, rx * scale, mag)
    if not rms:
        close(db, dy.double().sum(0), dy.double().abs().sum(0), 0.0)
