"""Adam: the 16-byte path of full, aligned chunks and the element-wise path (tails, unaligned buffers) are the same
arithmetic, so the same numbers give the same bits whichever of the two takes them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


@pytest.mark.parametrize("moments", [(BF, BF), (F32, F32), (BF, F32)])
@pytest.mark.parametrize("n", [1, 7, 4095, 4096, 4097, 3 * 4096 + 2056])
@pytest.mark.parametrize("adamw", [False, True])
def test_both_paths_agree(moments, n, adamw):
    from rtp_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(n)
    first = [torch.randn(n, generator=g, device="cuda").to(BF), torch.randn(n, generator=g, device="cuda").to(BF),
             (0.1 * torch.randn(n, generator=g, device="cuda")).to(moments[0]),
             (0.01 * torch.rand(n, generator=g, device="cuda")).to(moments[1])]
    out = []
    for shift in (0, 1):           # element offset 1: no buffer is 16-byte aligned
        bufs = []
        for t in first:
            b = torch.zeros(n + 16, dtype=t.dtype, device="cuda")
            b[shift:shift + n] = t
            bufs.append(b)
        plan = K.AdamPlan([tuple(b[shift:shift + n] for b in bufs) + (0.5,)], "cuda")
        step = torch.full((1,), 3, dtype=torch.int64, device="cuda")
        plan.step(step, 1e-2, 0.9, 0.999, 1e-8, 0.1, adamw, 0.5)
        assert all(int((b[:shift] != 0).sum()) == 0 and int((b[shift + n:] != 0).sum()) == 0 for b in bufs)
        out.append([b[shift:shift + n].clone() for b in bufs])
    assert all(torch.equal(a, b) for a, b in zip(*out))
    # and the arithmetic is Adam's (bf16 parameters: one rounding)
    p, gr, m, v = (t.double() for t in first)
    gr = gr.clamp(-0.5, 0.5)
    if not adamw:
        gr = gr + 0.1 * p
    else:
        p = p * (1 - 1e-2 * 0.5 * 0.1)
    m, v = 0.9 * m + 0.1 * gr, 0.999 * v + 0.001 * gr * gr
    p = p - 1e-2 * 0.5 / (1 - 0.9 ** 3) * m / (v.sqrt() / (1 - 0.999 ** 3) ** 0.5 + 1e-8)
    assert bool(((out[0][0].double() - p).abs() <= 2.0 ** -8 * p.abs() + 1e-4).all())


@pytest.mark.parametrize("device", ["cuda", "cpu"])
def test_zero_grad_keeps_the_buffers(device):
    from rtp_b200.optim import ShardedAdam
    ps = [torch.nn.Parameter(torch.randn(n, 3, device=device, dtype=d))
          for n in (1, 7, 70001) for d in (torch.bfloat16, torch.float32)]
    opt = ShardedAdam(ps)
    for i, p in enumerate(ps):
        p.grad = torch.randn_like(p).t().contiguous().t() if i % 2 else torch.randn_like(p)
    ps[1].grad = None
    ps[2].grad = (torch.randn_like(ps[2]).requires_grad_() * 2)        # part of a graph: detached as well
    ptrs = [None if p.grad is None else p.grad.data_ptr() for p in ps]
    opt.zero_grad(set_to_none=False)
    assert [None if p.grad is None else p.grad.data_ptr() for p in ps] == ptrs
    assert all(p.grad is None or (not p.grad.requires_grad and not p.grad.any()) for p in ps)
    opt.zero_grad()
    assert all(p.grad is None for p in ps)
