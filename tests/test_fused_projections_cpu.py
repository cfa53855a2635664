"""The one matrix behind several projections is read only while the parameters are its rows."""

import torch
from torch import nn

from mllm_b200.layers.gdn import views_of


def test_replaced_parameters_are_read_on_their_own():
    fused = torch.randn(24, 8)
    parts = [nn.Parameter(fused[a:b], requires_grad=False) for a, b in ((0, 8), (8, 20), (20, 24))]
    assert views_of(fused, parts)
    parts[1].data.copy_(torch.zeros(12, 8))        # written in place: still its rows
    assert views_of(fused, parts) and not fused[8:20].any()
    parts[1].data = torch.zeros(12, 8)
    assert not views_of(fused, parts) and not views_of(None, parts)
