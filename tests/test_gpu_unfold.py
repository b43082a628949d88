"""Patch matrices of the rotated convolution (csrc/im2col.cu) against torch's unfold and fold: sizes around the rows and channels of
a block, strides, dilations and paddings that skip input or never reach it, and inputs too large for shared memory.

im2col copies: equal.  col2im adds up to KH * KW terms in fp32 and rounds once: 2^-8 of the result and 2^-20 of the largest."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("B,C,H,W,k,s,p,d", [
    (1, 1, 3, 3, (3, 3), 1, 0, 1), (64, 32, 26, 26, (3, 3), 1, 0, 1), (3, 5, 9, 13, (3, 2), (2, 1), (1, 0), 1),
    (2, 64, 32, 32, (5, 5), 1, 2, 1), (2, 17, 23, 12, (3, 3), 3, 1, 2), (300, 3, 12, 12, (5, 5), 2, 1, 1),
    (8, 256, 14, 14, (1, 1), 1, 0, 1), (2, 24, 27, 26, (2, 2), 2, 0, 1), (3, 20, 15, 17, (7, 7), 1, 3, 1), (2, 9, 21, 20, (7, 3), 2, 3, 1),
    (1, 130, 40, 56, (5, 5), 1, 1, 1), (1, 600, 20, 60, (5, 5), 1, 0, 1), (2, 8, 30, 2000, (1, 1), 4, 0, 1), (1, 9, 7, 3000, (7, 3), 1, 3, 1)])
def test_unfold_and_fold(B, C, H, W, k, s, p, d):
    from rtp_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(H + W)
    x = torch.randn(B, C, H, W, generator=g, device="cuda").to(BF)
    K_ = C * k[0] * k[1]
    Kp = (K_ + 7) // 8 * 8
    ref = F.unfold(x.float(), k, d, p, s).transpose(1, 2).reshape(-1, K_)
    cols = K.im2col(x, k, s, p, d, Kp=Kp)
    assert torch.equal(cols[:, :K_].float(), ref) and not cols[:, K_:].any()
    dc = torch.randn(cols.shape, generator=g, device="cuda").to(BF)
    back = dc[:, :K_].double().view(B, -1, K_).transpose(1, 2)
    want = F.fold(back, (H, W), k, d, p, s)
    got = K.col2im(dc, x.shape, k, s, p, d).double()
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * want.abs().max()).all())


@pytest.mark.parametrize("B,C,H,W", [(1, 1, 1, 1), (2, 64, 8, 8), (3, 65, 7, 9), (64, 64, 24, 24), (5, 8, 1, 63)])
def test_rows(B, C, H, W):
    from rtp_b200.ops import kernels as K
    x = torch.randn(B, C, H, W, device="cuda").to(BF)
    for t in (x, x.transpose(2, 3), x.contiguous(memory_format=torch.channels_last)):
        assert torch.equal(K.nchw_rows(t), t.permute(0, 2, 3, 1).reshape(-1, C))
