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
    # one rounding after the norm and one after the rotation, of values that the rotation adds up: 2 (1 + sqrt(2)) half units in the
    # last place of a bf16 / fp16 number, and of the largest of the two
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    for g, w in zip(got, want):
        assert (g - w).abs().max() <= 5 * unit * w.abs().max()
