"""Head norm, rotation and cache write in one kernel, at the edges of its two widths."""

import pytest
import torch

from mllm_b200 import ops
from mllm_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,pad", [(1, 1, 0), (4, 2, 0), (5, 1, 8), (4, 2, 4), (3, 2, 4), (32, 8, 0)])
@pytest.mark.parametrize("tokens", [1, 7, 700, 20000])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_norm_rope_write(hq, hkv, pad, tokens, dtype):
    torch.manual_seed(1)
    if tokens == 20000 and hq == 32:
        tokens = 16385
    wide = torch.randn(tokens, (hq + 2 * hkv) * 128 + pad, device="cuda").to(dtype)
    qw, kw = (1 + 0.2 * torch.randn(128, device="cuda")).to(dtype), (1 + 0.2 * torch.randn(128, device="cuda")).to(dtype)
    pos, loc = torch.randint(0, 40000, (tokens,), device="cuda"), torch.randperm(tokens + 3, device="cuda")[:tokens]

    def run(f):
        qkv = wide.clone()[:, :(hq + 2 * hkv) * 128]
        caches = [torch.zeros(tokens + 3, hkv, 128, dtype=dtype, device="cuda") for _ in range(2)]
        f(qkv, qw, kw, pos, loc, *caches, hq, hkv, 128, 1e6, 1e-6, inv_freq=ops.rope_inv_freq(128, 1e6, qkv.device))
        return qkv[:, :(hq + hkv) * 128].float(), caches[0].float(), caches[1].float()

    got, want = run(ops.qk_norm_rope_kv_write), run(ref.qk_norm_rope_kv_write)
    # A rotated feature is a cos + b sin of the normed pair (a, b): the norm's rounding of each of the two may fall the other way (a unit
    # in its last place, at most 2 u of it), and that of the sum (at most 2 u, u = 2^-8 or 2^-11).  sqrt(a^2 + b^2) is the same before
    # and after, so that 2 u (|a| + |b|) + 2 u |a cos + b sin| <= 2 (1 + sqrt(2)) u sqrt(a^2 + b^2).  Angles up to 40000 are rounded
    # to 2^-9 in both, the same way.  Values are copied.
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    for g, w in zip(got[:2], want[:2]):
        w = w.reshape(-1, 2, 64)
        assert ((g.reshape(-1, 2, 64) - w).abs() <= 5 * unit * w.norm(dim=1, keepdim=True)).all()
    assert torch.equal(got[2], want[2])
