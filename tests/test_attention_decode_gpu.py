"""Streaming decode attention: lengths around the edges of a warp's 16 tokens and a tile's 64, groups around the widths of the
column operand, contexts dealt to one and to many thread blocks."""

import pytest
import torch

from mllm_b200 import ops
from mllm_b200.ops import reference as ref

pytestmark = pytest.mark.gpu

# probabilities and results are rounded to 8 bits (bf16), each by at most 2^-9 of itself, in independent directions
TOLERANCE = 2 ** -8

LENGTHS = {
    "edges": [1, 15, 16, 17, 63, 64, 65, 127, 128, 129],
    "one long": [1, 3, 5000, 2],
    "short": [7],
    "many": [(i * 37) % 300 + 1 for i in range(150)],
    "with an empty one": [40, 0, 200, 0, 0, 64],
}


def _run(lens, hq, hkv, hd, dtype=torch.bfloat16, head_major=True, **options):
    g = torch.Generator(device="cuda").manual_seed(len(lens) + hq + hd)
    total = sum(lens) + 8
    shape = (hkv, total, hd) if head_major else (total, hkv, hd)
    k, v = (torch.randn(shape, generator=g, device="cuda").to(dtype) for _ in range(2))
    if head_major:
        k, v = k.transpose(0, 1), v.transpose(0, 1)
    q = torch.randn((len(lens), hq, hd), generator=g, device="cuda").to(dtype)
    slots = torch.randperm(total, generator=g, device="cuda").to(torch.int32)
    table = torch.zeros((len(lens) + 1, max(lens) + 1), dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(lens):
        table[b, :n] = slots[at:at + n]
        at += n
    req = torch.arange(len(lens), dtype=torch.int32, device="cuda")
    seq = torch.tensor(lens, dtype=torch.int32, device="cuda")
    got = ops.attention_decode(q, k, v, table, req, seq, hd ** -0.5, max_seq_len=max(lens), **options)
    rows = [b for b, n in enumerate(lens) if n]
    empty = [b for b, n in enumerate(lens) if not n]
    assert not empty or not got[empty].any()
    want = ref.attention_decode(q[rows].float(), k.float(), v.float(), table, req[rows], seq[rows], hd ** -0.5, **options)
    error = (got[rows].float() - want.float()).norm() / want.float().norm()
    assert error < TOLERANCE, float(error)


@pytest.mark.parametrize("lens", LENGTHS, ids=str)
@pytest.mark.parametrize("hq,hkv,hd", [(8, 8, 128), (32, 4, 128), (18, 2, 128), (34, 2, 128), (32, 1, 128), (16, 4, 64), (32, 1, 64), (8, 2, 256), (16, 1, 256)])
def test_lengths_and_groups(lens, hq, hkv, hd):
    _run(LENGTHS[lens], hq, hkv, hd)


@pytest.mark.parametrize("options", [dict(window=1), dict(window=50), dict(chunk=48), dict(logit_cap=5.0)], ids=str)
@pytest.mark.parametrize("lens", ["edges", "one long"])
def test_masks_and_cap(lens, options):
    _run(LENGTHS[lens], 16, 4, 128, **options)


def test_sink_joins_whole_and_divided_contexts():
    sink = torch.linspace(-4, 4, 16, device="cuda")
    for lens in ("edges", "one long"):
        _run(LENGTHS[lens], 16, 4, 128, sink=sink)


def test_fp16_and_slot_major():
    _run(LENGTHS["edges"], 16, 4, 128, dtype=torch.float16)
    _run(LENGTHS["edges"], 16, 4, 128, head_major=False)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("hq,hkv,hd", [(8, 2, 64), (16, 4, 128), (8, 2, 256)])
def test_scores_that_are_no_numbers(hq, hkv, hd, value):
    """A key of NaN or infinity makes the softmax of its head NaN, whether the context lies in one thread block or in many; it leaves the
    other heads and requests alone."""
    lens = [3, 70, 5000, 40]
    g = torch.Generator(device="cuda").manual_seed(hd)
    table = torch.arange(sum(lens), dtype=torch.int32, device="cuda")
    table = torch.nn.utils.rnn.pad_sequence(table.split(lens), batch_first=True).contiguous()
    k, v = (torch.randn((sum(lens), hkv, hd), generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn((len(lens), hq, hd), generator=g, device="cuda").abs().bfloat16()
    for b in (0, 2):
        k[table[b, 2].item(), 1] = value
    req, seq = torch.arange(len(lens), dtype=torch.int32, device="cuda"), torch.tensor(lens, dtype=torch.int32, device="cuda")
    got = ops.attention_decode(q, k, v, table, req, seq, hd ** -0.5, max_seq_len=max(lens)).view(len(lens), hkv, -1, hd)
    hit = torch.zeros_like(got, dtype=torch.bool)
    hit[0, 1] = hit[2, 1] = True
    assert torch.equal(got.isnan(), hit)
