"""Short-sequence attention in fp32 (every length that the tensor-core kernels do not take) against float64, at lengths
around its 2 x 2 tiles and up to the longest that fits shared memory.

Tolerance: inputs are exact, everything up to the final rounding to bf16 (2^-8) is fp32; 2^-16 of the largest value covers
the exponentials and sums of up to 117 terms."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _close(got, ref):
    err = (got.double() - ref).abs()
    assert bool((err <= 2.0 ** -8 * ref.abs() + 2.0 ** -16 * ref.abs().max()).all()), err.max().item()


@pytest.mark.parametrize("S,p", [(1, 0.0), (2, 0.3), (17, 0.3), (41, 0.3), (50, 0.3), (63, 0.0), (96, 0.0), (117, 0.0)])
@pytest.mark.parametrize("causal", [True, False])
def test_against_float64(S, p, causal):
    from rtp_b200.ops import kernels as K
    B, H = 3, 2
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v, do = (torch.randn(S, B, H, 64, generator=g, device="cuda").to(BF) for _ in range(4))

    def pack(*t):
        return torch.cat([x.reshape(S * B, H * 64) for x in t], 1).contiguous()
    kw = dict(nshard=1, causal=causal, drop_p=p, seed=11, offset=5)
    keep = torch.ones(B, H, S, S, dtype=torch.float64, device="cuda")
    if p:        # with unit vectors as values the output is the matrix of dropped probabilities
        eye = torch.eye(S, 64, device="cuda", dtype=BF)[:, None, None].expand(S, B, H, 64)
        pd = K.attn_small_fwd(pack(q, k, eye), S, B, H, **kw).view(S, B, H, 64)[..., :S].permute(1, 2, 0, 3)
        keep = (pd != 0).double() / (1 - p)
        if S > 16:
            seen = keep[:, :, -1] if causal else keep
            assert abs((seen > 0).double().mean().item() - (1 - p)) < 0.15
    qd, kd, vd = (t.double().permute(1, 2, 0, 3).requires_grad_() for t in (q, k, v))
    s = qd @ kd.transpose(-1, -2) / 8
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    o = (torch.softmax(s, -1) * keep) @ vd
    out = K.attn_small_fwd(pack(q, k, v), S, B, H, **kw)
    _close(out.view(S, B, H, 64).permute(1, 2, 0, 3), o.detach())
    grads = torch.autograd.grad(o, (qd, kd, vd), do.double().permute(1, 2, 0, 3))
    dqkv = K.attn_small_bwd(pack(q, k, v), pack(do), S, B, H, **kw).view(S, B, 3, H, 64).permute(2, 1, 3, 0, 4)
    for got, ref in zip(dqkv, grads):
        _close(got, ref)


@pytest.mark.parametrize("S", [1, 4, 5, 12, 13])
def test_bits_do_not_depend_on_the_number_of_blocks(S):
    """Many blocks may run with fewer threads each; every sum keeps its order."""
    from rtp_b200.ops import kernels as K
    H, many, few = 2, 300, 3
    g = torch.Generator(device="cuda").manual_seed(S)
    qkv, do = (torch.randn(S, many, w * H * 64, generator=g, device="cuda").to(BF) for w in (3, 1))
    for p in (0.0, 0.3):
        def run(n):
            x, y = qkv[:, :n].reshape(S * n, -1).contiguous(), do[:, :n].reshape(S * n, -1).contiguous()
            kw = dict(causal=True, drop_p=p, seed=7, offset=2)
            return [t.view(S, n, -1)[:, :few] for t in (K.attn_small_fwd(x, S, n, H, **kw), K.attn_small_bwd(x, y, S, n, H, **kw))]
        for a, b in zip(run(many), run(few)):
            assert torch.equal(a, b)
