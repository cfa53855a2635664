"""Kernels around attention with gated query heads against the operators that they stand for."""

import pytest
import torch

from mllm_b200 import ops
from mllm_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,half", [(64, 8), (64, 32), (128, 16), (256, 32), (256, 128)])
@pytest.mark.parametrize("tokens", [1, 9, 5000])
@pytest.mark.parametrize("axes", [False, True])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_prologue_and_epilogue(dim, half, tokens, axes, dt):
    hq, hkv, eps = 6, 2, 1e-6
    g = torch.Generator(device="cuda").manual_seed(dim + tokens)
    row = torch.randn((tokens, (2 * hq + 2 * hkv) * dim), generator=g, device="cuda").to(dt)
    qw, kw = (1 + 0.1 * torch.randn((dim,), generator=g, device="cuda").to(dt) for _ in range(2))
    positions = torch.randint(0, 30000, (3, tokens) if axes else (tokens,), generator=g, device="cuda")
    axis_map = (torch.arange(half, device="cuda") % 3).to(torch.int8) if axes else None
    inv = 1e6 ** (-torch.arange(half, device="cuda", dtype=torch.float32) / half)
    loc = torch.randperm(tokens + 3, generator=g, device="cuda")[:tokens]
    store = torch.zeros((2, hkv, tokens + 3, dim), dtype=dt, device="cuda")
    kc, vc = store[0].transpose(0, 1), store[1].transpose(0, 1)
    assert ops.gated_heads_ok(row, kc, dim, half)
    q = ops.gated_head_prologue(row, qw, kw, positions, axis_map, inv, loc, kc, vc, hq, dim, eps)

    heads = row[:, :2 * hq * dim].view(tokens, hq, 2, dim)
    angles = (positions.float()[axis_map.long()].t() if axes else positions.float().unsqueeze(1)) * inv

    def turned(t, w):
        t = ref.rmsnorm(t.reshape(-1, dim), w, eps).view(t.shape).float()
        return ref.apply_rope_neox(t, angles.cos(), angles.sin()).to(dt)

    # one rounding of a result may fall the other way
    torch.testing.assert_close(q, turned(heads[:, :, 0], qw), rtol=2 ** -7, atol=2 ** -8)
    k, v = row[:, 2 * hq * dim:].view(tokens, 2, hkv, dim).unbind(1)
    torch.testing.assert_close(kc[loc], turned(k, kw), rtol=2 ** -7, atol=2 ** -8)
    assert torch.equal(vc[loc], v)
    o = torch.randn((tokens, hq, dim), generator=g, device="cuda").to(dt)
    want = o.float() * torch.sigmoid(heads[:, :, 1].float())
    torch.testing.assert_close(ops.gated_head_epilogue(o, row).float(), want, rtol=2 ** -8, atol=1e-6)
