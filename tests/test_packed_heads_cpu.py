"""Which packed projections the rotary attention reads in place.  Heads must not be cut by the column groups of the shards;
where they are (12 heads of 64 on a ring of 8: groups of 96 columns), the caller splits and joins the projection instead."""
import pytest
import torch

from rtp_b200.ops import functional as FO


@pytest.mark.parametrize("heads,nshard", [(12, 8), (6, 4), (4, 8)])
def test_heads_that_shards_cut_are_left_to_the_caller(heads, nshard, monkeypatch):
    monkeypatch.setattr(FO, "use_kernels", lambda x: True)
    B, S, D = 1, 100, heads * 64
    qkv = torch.randn(B, S, 3 * D).to(torch.bfloat16)
    cos, sin = torch.ones(S, 32), torch.zeros(S, 32)
    assert FO.rope_attention_packed(qkv, cos, sin, heads, nshard) is None
    q, k, v = FO._split_packed(qkv, 3, nshard)
    want = qkv.view(B, S, nshard, 3, D // nshard)
    for i, t in enumerate((q, k, v)):
        assert torch.equal(t, want[:, :, :, i].reshape(B, S, D))
