"""Stacked-heads attention (csrc/attn_tc.cu): numbers of heads that leave its last CTA partly or wholly to one head, both
lengths, against the fp32 kernels on the same dropout stream.

Tolerance: P and dS are rounded to bf16 (2^-9 of the value, at random) where the fp32 kernels keep them, both results once more:
2^-7 of the norm of the result."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("S", [32, 64])
@pytest.mark.parametrize("B,H,N,causal,p", [(1, 1, 1, True, 0.0), (1, 3, 1, False, 0.3), (3, 3, 1, True, 0.3), (5, 6, 2, True, 0.1),
                                            (37, 8, 1, True, 0.0)])
def test_partial_stacks(S, B, H, N, causal, p):
    from rtp_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(S + B)
    qkv = torch.randn(S * B, 3 * H * 64, generator=g, device="cuda").to(BF)
    do = torch.randn(S * B, H * 64, generator=g, device="cuda").to(BF)
    kw = dict(nshard=N, causal=causal, drop_p=p, seed=11, offset=5)
    try:
        K.set_attn_tc(False)
        ref = [K.attn_small_fwd(qkv, S, B, H, **kw), K.attn_small_bwd(qkv, do, S, B, H, **kw)]
    finally:
        K.set_attn_tc(True)
    got = [K.attn_small_fwd(qkv, S, B, H, **kw), K.attn_small_bwd(qkv, do, S, B, H, **kw)]
    assert K.attn_tc_error() == 0
    for x, r in zip(got, ref):
        x, r = x.double().view(S * B, -1, 64), r.double().view(S * B, -1, 64)
        err, n = (x - r).norm(dim=(0, 2)), r.norm(dim=(0, 2))        # head by head
        assert bool((err <= 2.0 ** -7 * n).all()), (err / n).max().item()


@pytest.mark.parametrize("S", [32, 64])
@pytest.mark.parametrize("where", ["q", "k", "v", "do"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_heads_stay_apart(S, where, value):
    """A value that is not finite in one head of one sequence leaves the results of all others as they are, bit for bit."""
    from rtp_b200.ops import kernels as K
    B, H = 5, 3
    g = torch.Generator(device="cuda").manual_seed(S)
    qkv = torch.randn(S, B, 3, H, 64, generator=g, device="cuda").to(BF)
    do = torch.randn(S, B, H, 64, generator=g, device="cuda").to(BF)

    def run():
        a, d = qkv.view(S * B, 3 * H * 64), do.view(S * B, H * 64)
        kw = dict(nshard=1, causal=True, drop_p=0.1, seed=11, offset=5)
        return (K.attn_small_fwd(a, S, B, H, **kw).view(S, B, 1, H, 64), K.attn_small_bwd(a, d, S, B, H, **kw).view(S, B, 3, H, 64))
    clean = run()
    if where == "do":
        do[7, 2, 1, 5] = value
    else:
        qkv[7, 2, "qkv".index(where), 1, 5] = value
    dirty = run()
    assert K.attn_tc_error() == 0
    for c, d in zip(clean, dirty):
        assert c.isfinite().all()
        d[:, 2, :, 1] = c[:, 2, :, 1]
        assert torch.equal(c, d)
    assert where == "do" or not run()[0][7:, 2, 0, 1].isfinite().all()
