"""Experts whose capacity is not full: rows that hold no token are left out of the products (csrc/gemm_local.cu), at numbers of
tokens around the edges of its tiles and k-blocks, an expert without any and one that is full.

Tolerance: outputs and gradients are compared with the same layer on a copy of the dispatched tensor, which is not known to have
unused rows: the same sums of the same products, apart from zeros,
which tiles of another shape may round differently once (2^-7 of the value), and once more on the way through the hidden layer."""
import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("E,cap,D,H,counts", [(2, 320, 72, 200, (0, 320)), (4, 320, 72, 200, (1, 63, 64, 65)),
                                              (4, 640, 136, 264, (127, 128, 129, 256)), (8, 1280, 512, 1024, (0, 1, 257, 600, 640, 1000, 1279, 1280))])
def test_unused_rows(E, cap, D, H, counts):
    from rtp_b200.module.moe import WeightMOELayer, combine_by_index, dispatch_by_index
    from rtp_b200.ops.moe import rows_in_use
    from rtp_b200.parallel.engine import fused_experts
    torch.manual_seed(cap)

    class Expert(nn.Module):
        def __init__(self):
            super().__init__()
            self.linear1, self.linear2, self.activation = nn.Linear(D, H), nn.Linear(H, D), nn.GELU()
    layer = WeightMOELayer(nn.Identity(), nn.ModuleList([Expert() for _ in range(E)]), device="cuda", dtype=BF)
    # tokens in random order, each with one choice (the other is dropped), expert e taking counts[e] of them
    idx = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)])
    loc = torch.cat([torch.arange(n) for n in counts])
    perm = torch.randperm(idx.numel())
    idx, loc = idx[perm], loc[perm]
    S = idx.numel()
    pair = torch.stack([idx, torch.zeros_like(idx)], 1).cuda(), torch.stack([loc, torch.zeros_like(loc)], 1).cuda()
    valid = torch.tensor([True, False]).expand(S, 2).cuda()
    gate = torch.rand(S, 2, device="cuda")
    x = torch.randn(S, D, device="cuda").to(BF).requires_grad_()
    dy = torch.randn(S, D, device="cuda").to(BF)
    params = list(layer.experts.parameters())
    results = []
    for known in (True, False):
        d = dispatch_by_index(x, *pair, valid, E, cap)
        fill = rows_in_use(d)
        assert fill.tolist() == list(counts)
        if not known:
            d = d.clone()
            assert rows_in_use(d) is None
        y = combine_by_index(fused_experts(layer, d), *pair, gate, valid)
        results.append([y.detach(), *torch.autograd.grad(y, [x, *params], dy)])
    for a, b in zip(*results):
        assert a.isfinite().all()
        assert bool(((a.double() - b.double()).abs() <= 2.0 ** -7 * b.double().abs() + 1e-3 * b.double().abs().max()).all())


def test_written_rows_count():
    from rtp_b200.ops.moe import dispatch, rows_in_use
    x = torch.randn(8, 64, device="cuda").to(BF)
    idx, loc = torch.zeros(8, 2, dtype=torch.long, device="cuda"), torch.arange(16, device="cuda").view(8, 2)
    d = dispatch(x, idx, loc, torch.ones(8, 2, dtype=torch.bool, device="cuda"), 2, 32)
    assert rows_in_use(d).tolist() == [16, 0]
    d[1, 3] = 1
    assert rows_in_use(d) is None


def layer_of(kind, tokens, D=64, H=128, E=8, capacity=1.0):
    from rtp_b200.models.moe_lm import Expert
    from rtp_b200.module.moe import MOELayer, WeightMOELayer
    from rtp_b200.module.top2gate import Top2Gate, WeightTop2Gate
    torch.manual_seed(1)
    experts = nn.ModuleList([Expert(D, H) for _ in range(E)])
    if kind == "rotating":
        layer = WeightMOELayer(WeightTop2Gate(D, E, device="cuda", dtype=BF, capacity_factor=capacity), experts, device="cuda", dtype=BF)
    else:
        layer = MOELayer(Top2Gate(D, E, capacity), experts).to("cuda", BF)
    x = torch.randn(1, tokens, D, device="cuda").to(BF)

    def run():
        torch.manual_seed(2)                  # the noise of the second choice
        return layer(x), layer.l_aux
    return run


@pytest.mark.parametrize("kind", ["rotating", "all-to-all"])
def test_inference_mode(kind):
    """The same outputs as without gradients (tiles without tokens differ, which reach no output: one rounding, 2^-8, each way)."""
    run = layer_of(kind, 512)
    with torch.no_grad():
        y, aux = run()
    with torch.inference_mode():
        z, aux2 = run()
    assert y.isfinite().all() and y.norm() > 0
    assert torch.equal(aux, aux2)
    assert bool(((y.double() - z.double()).abs() <= 2.0 ** -7 * y.double().abs() + 1e-3 * y.double().abs().max()).all())


def test_no_capacity():
    """Fewer places than one an expert: every token is dropped and the layer gives zeros, and so do its gradients."""
    from rtp_b200.module.moe import dispatch_by_index
    y, _ = layer_of("all-to-all", 8, capacity=0.25)()
    assert y.shape == (1, 8, 64) and bool((y == 0).all())
    x = torch.randn(8, 64, device="cuda").to(BF).requires_grad_()
    idx, none = torch.zeros(8, 2, dtype=torch.long, device="cuda"), torch.zeros(8, 2, dtype=torch.bool, device="cuda")
    d = dispatch_by_index(x, idx, idx, none, 4, 0)
    assert d.shape == (4, 0, 64)
    (g,) = torch.autograd.grad(d, x, torch.empty_like(d))
    assert bool((g == 0).all())


@pytest.mark.parametrize("kind,counted", [("rotating", True), ("all-to-all", False)])
def test_rows_are_counted_for_who_reads_them(kind, counted, monkeypatch):
    from rtp_b200.ops import kernels as K
    seen, scatter = [], K.moe_scatter
    monkeypatch.setattr(K, "moe_scatter", lambda src, slot, scale, rows, fill=None: seen.append(fill) or scatter(src, slot, scale, rows, fill))
    with torch.no_grad():
        layer_of(kind, 64)()
    assert len(seen) == 1 and (seen[0] is not None) == counted


@pytest.mark.parametrize("E,cap,D,H,counts", [(4, 320, 72, 200, (1, 63, 64, 65)), (4, 640, 136, 264, (127, 0, 129, 640))])
def test_against_float64(E, cap, D, H, counts):
    """Four tensors on the way to the output are rounded to bf16 (2^-9 of the value each, at random), eight on the way to a
    gradient: norms of the errors within 2^-7 and 2^-6 of those of the results, expert by expert."""
    from rtp_b200.models.moe_lm import Expert
    from rtp_b200.module.moe import WeightMOELayer, combine_by_index, dispatch_by_index
    from rtp_b200.ops.moe import rows_in_use
    from rtp_b200.parallel.engine import fused_experts
    torch.manual_seed(cap)
    layer = WeightMOELayer(nn.Identity(), nn.ModuleList([Expert(D, H) for _ in range(E)]), device="cuda", dtype=BF)
    idx = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)]).cuda()
    loc = torch.cat([torch.arange(n) for n in counts]).cuda()
    S = idx.numel()
    pair = torch.stack([idx, torch.zeros_like(idx)], 1), torch.stack([loc, torch.zeros_like(loc)], 1)
    valid = torch.tensor([True, False]).expand(S, 2).cuda()
    gate = torch.rand(S, 2, device="cuda")
    x, dy = torch.randn(S, D, device="cuda").to(BF).requires_grad_(), torch.randn(S, D, device="cuda").to(BF)
    params = list(layer.experts.parameters())
    d = dispatch_by_index(x, *pair, valid, E, cap)
    assert rows_in_use(d).tolist() == list(counts)
    y = combine_by_index(fused_experts(layer, d), *pair, gate, valid)
    got = [y.detach(), *torch.autograd.grad(y, [x, *params], dy)]
    xs, ps = x.detach().double().requires_grad_(), [p.detach().double().requires_grad_() for p in params]
    out = torch.zeros(S, D, dtype=torch.float64, device="cuda")
    for e in range(E):
        w1, b1, w2, b2 = ps[4 * e:4 * e + 4]
        rows = (idx == e).nonzero()[:, 0]
        h = torch.nn.functional.gelu(xs[rows] @ w1.t() + b1) @ w2.t() + b2
        out = out.index_add(0, rows, h * gate[rows, :1].double())
    ref = [out.detach(), *torch.autograd.grad(out, [xs, *ps], dy.double())]
    for i, (a, b) in enumerate(zip(got, ref)):
        assert ((a.double() - b).norm() <= (2.0 ** -6 if i else 2.0 ** -7) * b.norm()).item(), (i, ((a.double() - b).norm() / b.norm()).item())
        if i < 2:
            for e in range(E):
                u, v = a[idx == e].double(), b[idx == e]
                assert ((u - v).norm() <= 2.0 ** -6 * v.norm()).item(), (i, e)
