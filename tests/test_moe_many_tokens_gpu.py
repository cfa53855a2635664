"""Experts with many rows each: chunks of 256 by pairs of thread blocks, the counting sort by a cluster."""

import pytest
import torch

from mllm_b200 import ops
from mllm_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skew", [0.0, 3.0])
@pytest.mark.parametrize("tokens,experts,top", [(1283, 8, 2), (5000, 16, 4)])
def test_many_rows_per_expert(tokens, experts, top, skew):
    hidden, inter = 256, 256
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn((tokens, hidden), generator=g, device="cuda").bfloat16()
    w13 = (torch.randn((experts, 2 * inter, hidden), generator=g, device="cuda") * 0.05).bfloat16()
    w2 = (torch.randn((experts, hidden, inter), generator=g, device="cuda") * 0.05).bfloat16()
    # with a skew some experts get most tokens and some none
    score = torch.rand((tokens, experts), generator=g, device="cuda") + skew * torch.linspace(0, 1, experts, device="cuda")
    ids = score.topk(top, -1).indices.to(torch.int32)
    weight = torch.rand((tokens, top), generator=g, device="cuda")
    mixed = torch.stack([ref.interleave_gate_up(w.clone(), ops.SWIGLU_BLOCK) for w in w13])
    got = ops.moe_experts(x, mixed, w2, weight, ids, swiglu_block=ops.SWIGLU_BLOCK)
    ops.check_status()
    want = torch.zeros((tokens, hidden), dtype=torch.float64, device="cuda")
    for e in range(experts):
        t, c = (ids == e).nonzero(as_tuple=True)
        a, b = (x[t].double() @ w13[e].double().t()).chunk(2, -1)
        want.index_add_(0, t, ((torch.nn.functional.silu(a) * b) @ w2[e].double().t()) * weight[t, c].double().unsqueeze(-1))
    # hidden values, expert rows and the sum are each rounded to 8 bits
    assert (got.double() - want).norm() / want.norm() < 2 ** -7
