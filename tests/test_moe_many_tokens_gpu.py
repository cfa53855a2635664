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


def test_many_rows_of_local_experts():
    """The experts of one rank, half of all: pairs of the others have no row."""
    tokens, experts, top, hidden, inter = 3000, 12, 4, 256, 256
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn((tokens, hidden), generator=g, device="cuda").half()
    w13 = (torch.randn((experts // 2, 2 * inter, hidden), generator=g, device="cuda") * 0.05).half()
    w2 = (torch.randn((experts // 2, hidden, inter), generator=g, device="cuda") * 0.05).half()
    ids = torch.rand((tokens, experts), generator=g, device="cuda").topk(top, -1).indices.to(torch.int32)
    weight = torch.rand((tokens, top), generator=g, device="cuda")
    mixed = torch.stack([ref.interleave_gate_up(w.clone(), ops.SWIGLU_BLOCK) for w in w13])
    got = ops.moe_experts(x, mixed, w2, weight, ids, expert_offset=6, swiglu_block=ops.SWIGLU_BLOCK, num_experts_global=experts)
    ops.check_status()
    want = torch.zeros((tokens, hidden), dtype=torch.float64, device="cuda")
    for e in range(experts // 2):
        t, c = (ids == e + 6).nonzero(as_tuple=True)
        a, b = (x[t].double() @ w13[e].double().t()).chunk(2, -1)
        want.index_add_(0, t, ((torch.nn.functional.silu(a) * b) @ w2[e].double().t()) * weight[t, c].double().unsqueeze(-1))
    # hidden values, expert rows and the sum are each rounded to 11 bits
    assert (got.double() - want).norm() / want.norm() < 2 ** -10


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hidden,inter", [(256, 512), (1280, 256)])
def test_many_rows_without_a_gate(hidden, inter, dtype):
    tokens, experts, top = 1283, 8, 2
    g = torch.Generator(device="cuda").manual_seed(hidden)
    x = torch.randn((tokens, hidden), generator=g, device="cuda").to(dtype)
    w1 = (torch.randn((experts, inter, hidden), generator=g, device="cuda") * 0.05).to(dtype)
    w2 = (torch.randn((experts, hidden, inter), generator=g, device="cuda") * 0.05).to(dtype)
    ids = torch.rand((tokens, experts), generator=g, device="cuda").topk(top, -1).indices.to(torch.int32)
    rows = ops.moe_expert_rows(x, w1, w2, torch.ones((tokens, top), device="cuda"), ids, gated=False)
    ops.check_status()
    got = rows.rows[rows.sorted_pos.view(tokens, top).long()].double()
    want = torch.zeros_like(got)
    for e in range(experts):
        t, c = (ids == e).nonzero(as_tuple=True)
        want[t, c] = torch.nn.functional.gelu(x[t].double() @ w1[e].double().t()) @ w2[e].double().t()
    # hidden values and expert rows are each rounded to 8 (11) bits
    assert (got - want).norm() / want.norm() < 2.0 ** (-7 if dtype == torch.bfloat16 else -10)
