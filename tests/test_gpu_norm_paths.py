"""LayerNorm / RMSNorm kernels against float64 at the widths where the number of threads per row changes, with row counts
below, at and above what one pass of the grid takes.

Tolerance: h is rounded to bf16 first, as the kernels do; y and dx are one rounding to bf16 (2^-8) of fp32 arithmetic
whose error is 2^-16 of the largest term; dgamma / dbeta are fp32 sums over the rows (2^-16 of the sum of magnitudes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("D", [8, 256, 264, 512, 520, 1024, 1032, 2048, 2056, 4104, 5120, 8192])
@pytest.mark.parametrize("M", [1, 148, 297, 1025, 2500])
@pytest.mark.parametrize("rms,residual", [(False, True), (True, False)])
def test_norm(D, M, rms, residual):
    from rtp_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(D + M)

    def rnd(*s):
        return torch.randn(*s, generator=g, device="cuda").to(BF)
    x, dy, gamma, beta = rnd(M, D), rnd(M, D), rnd(D), rnd(D)
    sub = rnd(M, D) if residual else None
    y, h, mean, rstd = K.norm_fwd(x, sub, gamma, None if rms else beta, rms=rms)
    href = (x.float() + sub.float()).to(BF) if residual else x
    assert torch.equal(h, href)
    hd = href.double().requires_grad_()
    gd = gamma.double().requires_grad_()
    mu = hd.mean(-1, keepdim=True) if not rms else 0.0
    xh = (hd - mu) * torch.rsqrt((hd - mu).pow(2).mean(-1, keepdim=True) + 1e-5)
    ref = xh * gd + (0.0 if rms else beta.double())

    def close(a, r, mag, rel):
        assert bool(((a.double() - r).abs() <= rel * r.abs() + 2.0 ** -16 * mag).all()), (a.double() - r).abs().max().item()
    close(y, ref.detach(), ref.detach().abs().max(), 2.0 ** -8)
    dx, dsub, dg, db = K.norm_bwd(dy, h, gamma, mean, rstd, rms=rms, has_beta=not rms, want_dsub=residual)
    rx, rg = torch.autograd.grad(ref, (hd, gd), dy.double())
    # dx cancels between its three terms: the fp32 error is relative to the largest of them
    close(dx, rx, (dy.double() * gamma.double()).abs().amax() * rstd.double().max() * 4, 2.0 ** -8)
    close(dg, rg, (dy.double() * xh.detach()).abs().sum(0), 0.0)
    if not rms:
        close(db, dy.double().sum(0), dy.double().abs().sum(0), 0.0)
    if residual:
        assert torch.equal(dsub, dx)


@pytest.mark.parametrize("M", [4096, 4098, 8001])
@pytest.mark.parametrize("D", [1032, 1536, 2048])
def test_many_wide_rows(M, D):
    test_norm(D, M, False, True)
    test_norm(D, M, True, False)


@pytest.mark.parametrize("D", [8, 72, 264, 520, 1032, 2048, 5120, 8192])
@pytest.mark.parametrize("M", [1, 5, 297, 4099])
@pytest.mark.parametrize("rms", [False, True])
def test_parameter_gradients_in_place(D, M, rms):
    """Through autograd: gradients of gamma and beta are one rounding to bf16 of the sums, and two calls give the same bits."""
    from rtp_b200.ops import functional as FO
    g = torch.Generator(device="cuda").manual_seed(D + M)
    x, dy = (torch.randn(M, D, generator=g, device="cuda").to(BF) for _ in range(2))
    w, b = (torch.randn(D, generator=g, device="cuda").to(BF).requires_grad_() for _ in range(2))
    x.requires_grad_()

    def run():
        y = FO.rms_norm(x, w) if rms else FO.layer_norm(x, w, b)
        return torch.autograd.grad(y, (x, w) if rms else (x, w, b), dy)
    got = run()
    assert all(torch.equal(p, q) for p, q in zip(got, run()))
    hd = x.detach().double()
    mu = 0.0 if rms else hd.mean(-1, keepdim=True)
    xh = (hd - mu) * torch.rsqrt((hd - mu).pow(2).mean(-1, keepdim=True) + 1e-5)
    for t, terms in zip(got[1:], (dy.double() * xh, dy.double())):
        ref = terms.sum(0)
        assert bool(((t.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -16 * terms.abs().sum(0)).all())


@pytest.mark.parametrize("M,D", [(1, 264), (5, 8192), (300, 520), (1024, 2048), (5000, 1032), (4099, 8192)])
@pytest.mark.parametrize("rms", [False, True])
def test_parameter_gradients_workspace(M, D, rms):
    """The workspace is as large as the launch needs: all of it is written, nothing behind it, and it grows with neither the rows
    beyond two blocks an SM nor a beta that is not there."""
    from rtp_b200.ops import _lib
    from rtp_b200.ops import kernels as K
    L = K._L()
    n = L.rtp_norm_bwd_scratch(M, D, int(not rms))
    assert n % (D * 4 * (1 if rms else 2)) == 0 and n <= min(M, 296) * D * 4 * (1 if rms else 2)
    buf = torch.full((n // 4 + 64,), float("inf"), device="cuda")
    x, dy = (torch.randn(M, D, device="cuda").to(BF) for _ in range(2))
    w, out, dx = torch.ones(D, device="cuda", dtype=BF), torch.empty(2, D, device="cuda", dtype=BF), torch.empty_like(dy)
    mean, rstd = torch.zeros(M, device="cuda"), torch.ones(M, device="cuda")
    K._check(L.rtp_norm_bwd_params(K._p(dy), K._p(x), K._p(w), None if rms else K._p(mean), K._p(rstd), K._p(dx), K._p(out[0]),
                                   None if rms else K._p(out[1]), K._p(buf), M, D, int(rms), None, _lib.stream_ptr()), "norm_bwd_params")
    assert buf[:n // 4].isfinite().all() and bool((buf[n // 4:] == float("inf")).all())


def test_parameter_gradients_are_tensors_of_their_own():
    from rtp_b200.ops import functional as FO
    x = torch.randn(7, 64, device="cuda").to(BF)
    w, b = (torch.ones(64, device="cuda", dtype=BF, requires_grad=True) for _ in range(2))
    FO.layer_norm(x, w, b).sum().backward()
    assert w.grad.untyped_storage().data_ptr() != b.grad.untyped_storage().data_ptr()
    w.grad.detach_()
    b.grad.detach_()
