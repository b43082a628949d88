"""GEMM jobs of a ring of one rank (csrc/gemm_local.cu) against fp32 PyTorch, at the edges of its tiles: rows and columns
that end inside a tile, contractions that end inside a k-block, one and many tiles per unit, every epilogue, the column
sums beside the weight gradient, and several experts in one launch.

Tolerance: a result is one bf16 rounding (2^-8 of the result) of an fp32 sum whose terms are exact products (2^-18 of the
sum of absolute products)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _close(got, ref, mag):
    err = (got.double() - ref).abs()
    assert bool((err <= 2.0 ** -8 * ref.abs() + 2.0 ** -18 * mag + 1e-30).all()), err.max().item()


def near(got, ref, rel):
    assert ((got.double() - ref).norm() / ref.norm()).item() < rel


def _linear(M, I, O, seed=0):
    from rtp_b200.parallel import engine as E
    from rtp_b200.parallel.context import get_context
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rnd(*s):
        return torch.randn(*s, generator=g, device="cuda").to(BF)
    off = (O * I + 63) // 64 * 64
    flat = torch.zeros(off + (O + 63) // 64 * 64, dtype=BF, device="cuda")
    flat[:O * I] = rnd(O * I)
    flat[off:off + O] = rnd(O)
    return E, E.get_engine(get_context()), flat, (True, off, E._round_up(flat.numel() * 2, 16)), off, rnd


@pytest.mark.parametrize("M,I,O", [(1, 64, 8), (8, 8, 8), (127, 72, 136), (129, 200, 264), (257, 520, 120), (650, 768, 3080),
                                   (1000, 1032, 520), (2500, 2048, 1160), (2200, 136, 4104), (4500, 72, 8200)])
def test_linear(M, I, O):
    E, eng, flat, info, off, rnd = _linear(M, I, O)
    x, dy, c, mask = rnd(M, I), rnd(M, O), rnd(M, I), rnd(M, I)
    w, b = flat[:O * I].view(O, I).double(), flat[off:off + O].double()
    xd, dyd = x.double(), dy.double()
    y = E.linear_fwd_raw(eng, flat, info, x, False, I, O)
    _close(y, xd @ w.t() + b, xd.abs() @ w.abs().t() + b.abs())
    y = E.linear_fwd_raw(eng, flat, info, x, False, I, O, act=1)
    _close(y, torch.relu(xd @ w.t() + b), xd.abs() @ w.abs().t() + b.abs())
    dx, mag = dyd @ w, dyd.abs() @ w.abs()
    out, g = E.linear_bwd_raw(eng, flat, info, x, dy, False, I, O, dx_out=c.clone(), dx_accumulate=True)
    _close(out, dx + c.double(), mag + c.double().abs())
    _close(g[:O * I].view(O, I), dyd.t() @ xd, dyd.abs().t() @ xd.abs())
    _close(g[off:off + O], dyd.sum(0), dyd.abs().sum(0))
    out, _ = E.linear_bwd_raw(eng, flat, info, x, dy, False, I, O, mask=mask, mask_scale=2.0)
    _close(out, torch.where(mask > 0, 2.0 * dx, torch.zeros_like(dx)), 2.0 * mag)
    out, _ = E.linear_bwd_raw(eng, flat, info, x, dy, False, I, O, mask=mask, mask_scale=2.0, dx_out=c.clone(), dx_accumulate=True)
    _close(out, torch.where(mask > 0, 2.0 * (dx + c.double()), torch.zeros_like(dx)), 2.0 * (mag + c.double().abs()))
    eng.check()


@pytest.mark.parametrize("M,I,O", [(8191, 288, 64), (8192, 288, 64), (8200, 72, 8), (36864, 288, 64), (9001, 1032, 128)])
def test_long_contraction(M, I, O):
    """Weight gradients of few tiles: one slice of the contraction, eight, and eight with a short last one."""
    E, eng, flat, info, off, rnd = _linear(M, I, O)
    x, dy = rnd(M, I), rnd(M, O)
    xd, dyd, w = x.double(), dy.double(), flat[:O * I].view(O, I).double()
    dx, g = E.linear_bwd_raw(eng, flat, info, x, dy, False, I, O)
    _close(dx, dyd @ w, dyd.abs() @ w.abs())
    _close(g[:O * I].view(O, I), dyd.t() @ xd, dyd.abs().t() @ xd.abs())
    _close(g[off:off + O], dyd.sum(0), dyd.abs().sum(0))
    eng.check()


def test_long_batch_is_captured():
    """The first backward of a biased linear over more rows than any before it may be one that a CUDA graph captures."""
    E, eng, flat, info, off, rnd = _linear(40008, 72, 8)
    x, dy = rnd(40008, 72), rnd(40008, 8)
    E.linear_bwd_raw(eng, flat, info, x[:64], dy[:64], False, 72, 8)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        _, g = E.linear_bwd_raw(eng, flat, info, x, dy, False, 72, 8)
    graph.replay()
    torch.cuda.synchronize()
    _close(g[off:off + 8], dy.double().sum(0), dy.double().abs().sum(0))
    _close(g[:8 * 72].view(8, 72), dy.double().t() @ x.double(), dy.double().abs().t() @ x.double().abs())
    eng.check()


def test_dropout_mask_of_the_general_kernel():
    """The same (seed, offset) drops the same elements as the rotation kernel, which a forced tile width selects."""
    from rtp_b200.ops import gemm as G
    a, b = torch.randn(300, 128, device="cuda").to(BF), torch.randn(200, 128, device="cuda").to(BF)
    kw = dict(drop_p=0.3, seed=11, offset=5)
    got, ref = G.gemm(a, b, **kw), a.double() @ b.double().t()
    assert torch.equal(got == 0, G.gemm(a, b, bn=128, **kw) == 0)
    kept = got != 0
    assert abs(kept.double().mean().item() - 0.7) < 0.01
    # one rounding to bf16 of an fp32 product with 1 / (1 - p), which is rounded itself
    _close(got[kept], (ref / 0.7)[kept], ((a.double().abs() @ b.double().abs().t()) / 0.7)[kept] + 2.0 ** -5 * ref.abs()[kept])


@pytest.mark.parametrize("cap", [8, 40, 136, 320])
def test_experts(cap):
    import torch.nn as nn
    from rtp_b200.module.moe import WeightMOELayer
    from rtp_b200.parallel.engine import fused_experts
    torch.manual_seed(cap)
    E, D, H = 4, 72, 200

    class Expert(nn.Module):
        def __init__(self):
            super().__init__()
            self.linear1, self.linear2, self.activation = nn.Linear(D, H), nn.Linear(H, D), nn.ReLU()
    layer = WeightMOELayer(nn.Identity(), nn.ModuleList([Expert() for _ in range(E)]), device="cuda", dtype=BF)
    x = torch.randn(E, cap, D, device="cuda").to(BF).requires_grad_()
    dy = torch.randn(E, cap, D, device="cuda").to(BF)
    params = [p for e in layer.experts for p in (e.linear1.weight, e.linear1.bias, e.linear2.weight, e.linear2.bias)]
    y = fused_experts(layer, x)
    got = torch.autograd.grad(y, [x, *params], dy)
    for e in range(E):
        w1, b1, w2, b2 = (p.detach().double() for p in params[4 * e:4 * e + 4])
        xd, dyd = x[e].detach().double(), dy[e].double()
        h = torch.relu((xd @ w1.t() + b1).to(BF).double())      # the kernels keep the hidden activation in bf16
        _close(y[e].detach(), h @ w2.t() + b2, 4 * (h.abs() @ w2.abs().t() + b2.abs()) * 2.0 ** 9)
        # a hidden unit whose rounding to bf16 flips is rare: in the norm little more than the rounding of the result is left
        near(y[e].detach(), h @ w2.t() + b2, 2.0 ** -8)
        g = got[1 + 4 * e:5 + 4 * e]
        # sums over exactly this expert's rows: nothing of the next expert's rows may leak into the last k-block
        _close(g[3], dyd.sum(0), dyd.abs().sum(0))
        ref = dyd.t() @ h
        assert ((g[2].double() - ref).norm() / ref.norm()).item() < 2.0 ** -6
        dh = torch.where(h > 0, dyd @ w2, torch.zeros_like(h))
        ref = dh.t() @ xd
        assert ((g[0].double() - ref).norm() / ref.norm()).item() < 2.0 ** -5
        # the hidden gradient is kept in bf16 (2^-9 at random), sums and the input gradient are rounded once more
        near(g[1], dh.sum(0), 2.0 ** -6)
        near(got[0][e], dh @ w1, 2.0 ** -6)
