"""Prefill of the gated delta rule in two kernels: chunks of 64 tokens at their edges, head sizes that are padded, several value
blocks, decays from almost none to almost all, spans of a bounded workspace."""

import pytest
import torch

from mllm_b200 import ops

pytestmark = pytest.mark.gpu


def _rule(q, k, v, g, beta, state, lens, has):
    q, k, v = q.double(), k.double(), v.double()
    rep = v.shape[1] // q.shape[1]
    q, k = (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = q.repeat_interleave(rep, 1) * q.shape[-1] ** -0.5, k.repeat_interleave(rep, 1)
    out, states, at = [], [], 0
    for b, n in enumerate(lens):
        s = state[b].double() * (1 if has[b] else 0)
        for t in range(at, at + n):
            s = s * g[t].double().exp()[:, None, None]
            u = (v[t] - torch.einsum("hkv,hk->hv", s, k[t])) * beta[t].double()[:, None]
            s = s + k[t].unsqueeze(-1) * u.unsqueeze(-2)
            out.append(torch.einsum("hkv,hk->hv", s, q[t]))
        at += n
        states.append(s)
    return torch.stack(out), torch.stack(states)


def _check(lens, heads, key_heads, dk, dv, decay=0.1, max_len=None):
    gen = torch.Generator(device="cuda").manual_seed(sum(lens) + heads)
    T = sum(lens)
    q, k = (torch.randn((T, key_heads, dk), generator=gen, device="cuda").bfloat16() for _ in range(2))
    v = torch.randn((T, heads, dv), generator=gen, device="cuda").bfloat16()
    g = -torch.rand((T, heads), generator=gen, device="cuda") * decay
    beta = torch.rand((T, heads), generator=gen, device="cuda")
    state = torch.randn((len(lens) + 1, heads, dk, dv), generator=gen, device="cuda") * 0.1
    has = [i % 2 for i in range(len(lens))]
    want, after = _rule(q, k, v, g, beta, state, lens, has)
    spare = state[len(lens)].clone()
    i32 = dict(dtype=torch.int32, device="cuda")
    ops.set_gdn_extend_backend("cuda_chunkwise")
    try:
        got = ops.gated_delta_rule(q, k, v, g, beta, state, torch.arange(len(lens), **i32), torch.tensor(lens, **i32), torch.tensor(has, **i32),
                                   max_len=max(lens) if max_len is None else max_len)
    finally:
        ops.set_gdn_extend_backend("auto")
    ops.check_status()
    # outputs are rounded to 8 bits; the state is fp32, and the operands of its products hold 16 bits
    assert (got.double() - want).norm() / want.norm() < 2 ** -8
    assert (state[:len(lens)].double() - after).norm() / after.norm() < 2 ** -14
    assert torch.equal(state[len(lens)], spare)


@pytest.mark.parametrize("lens", [[1], [63], [64], [65], [128, 1, 129], [300, 7, 64, 2]], ids=str)
def test_chunks(lens):
    _check(lens, 4, 4, 128, 128)


@pytest.mark.parametrize("heads,key_heads,dk,dv", [(4, 2, 128, 128), (2, 2, 64, 96), (2, 1, 40, 24), (2, 2, 128, 256), (80, 80, 128, 128), (6, 2, 8, 8)])
def test_heads(heads, key_heads, dk, dv):
    _check([100, 33], heads, key_heads, dk, dv)


@pytest.mark.parametrize("decay", [0.0, 1e-3, 5.0, 60.0])
def test_decays(decay):
    _check([200], 2, 2, 128, 128, decay=decay)


@pytest.mark.parametrize("chunks", [2, 3, 5])
@pytest.mark.parametrize("lens", [[330, 129], [64 * 7 + 1], [1, 0, 640, 65, 200]], ids=str)
def test_spans_of_the_workspace(lens, chunks, monkeypatch):
    """Room for one to five chunks at a time: spans of several chunks, the last one in part, that take the state up where the span before
    left it; fewer chunks than requests, which then come in groups."""
    heads, slot = 6, (2 * 64 * 128 + 2 * 64 * 128 + 2 * 64 * 64) * 2 + 160 * 4 + 64 * 128 * 4      # of a (chunk, head): W in two terms, Q, K, P in two terms, scalars, U0
    monkeypatch.setattr(ops, "GDN_WORKSPACE_BYTES", chunks * heads * slot)
    _check(lens, heads, 3, 128, 128)


def test_workspace_of_many_requests(monkeypatch):
    """One chunk of all requests is more than the workspace may have."""
    monkeypatch.setattr(ops, "GDN_WORKSPACE_BYTES", 1 << 20)
    lens = [40 + 7 * (i % 5) for i in range(24)]
    _check(lens, 2, 2, 128, 128)
    T = sum(lens)
    q, k, v = (torch.randn(T, 2, 128, device="cuda").bfloat16() for _ in range(3))
    g, beta, state = -torch.rand(T, 2, device="cuda"), torch.rand(T, 2, device="cuda"), torch.zeros(24, 2, 128, 128, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    index = (torch.arange(24, **i32), torch.tensor(lens, **i32), torch.zeros(24, **i32))
    torch.cuda.reset_peak_memory_stats()
    inputs = torch.cuda.memory_allocated()
    ops.gated_delta_rule(q, k, v, g, beta, state, *index, max_len=max(lens))
    assert torch.cuda.max_memory_allocated() - inputs < (1 << 20) + v.numel() * 2 + (64 << 10)


def test_spans_of_many_heads():
    """Heads that leave room for one chunk at a time in 512 MB, the longest run not known."""
    _check([330, 129], 1700, 100, 8, 128, max_len=0)


def test_state_between_other_values():
    """A state that does not start on a 16-byte boundary is moved value by value, and nothing beside it is touched."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    lens, heads, dk, dv = [70, 5], 2, 128, 96
    q, k, v = (torch.randn((75, heads, d), generator=gen, device="cuda").bfloat16() for d in (dk, dk, dv))
    g, beta = -torch.rand((75, heads), generator=gen, device="cuda") * 0.1, torch.rand((75, heads), generator=gen, device="cuda")
    room = torch.randn(2 * heads * dk * dv + 6, generator=gen, device="cuda") * 0.1
    plain = room[1:-5].clone().view(2, heads, dk, dv)
    odd = room[1:-5].view(2, heads, dk, dv)
    before = room.clone()
    i32 = dict(dtype=torch.int32, device="cuda")
    got = [ops.gated_delta_rule(q, k, v, g, beta, s, torch.arange(2, **i32), torch.tensor(lens, **i32), torch.ones(2, **i32), max_len=70) for s in (plain, odd)]
    ops.check_status()
    assert torch.equal(got[0], got[1]) and torch.equal(plain, odd)
    assert torch.equal(room[:1], before[:1]) and torch.equal(room[-5:], before[-5:])


@pytest.mark.parametrize("tokens,heads,width", [(256, 16, 128), (819, 5, 128), (1025, 4, 64), (4097, 1, 8), (700, 6, 120), (4100, 3, 256)])
@pytest.mark.parametrize("sigmoid", [False, True])
def test_gated_norm_of_many_rows(tokens, heads, width, sigmoid):
    """Rows at the edges of a warp's and a block's share, widths that leave lanes idle, a gate inside wider rows: the output's rounding
    to 8 bits (at most 2^-8 of it) is the largest error of a row, beside 2^-18 for the fast exponential and division."""
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    x = torch.randn((tokens, heads, width), generator=gen, device="cuda").bfloat16()
    rows = torch.randn((tokens, 16 + heads * width), generator=gen, device="cuda").bfloat16()
    gate, w = rows[:, 8:8 + heads * width], torch.randn(width, generator=gen, device="cuda").bfloat16()
    got = ops.rmsnorm_gated(x.flatten(1), gate, w, 1e-6, round_norm=False, sigmoid=sigmoid).double().reshape(tokens, heads, width)
    g = gate.double().reshape(tokens, heads, width)
    want = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6) * w.double() * (torch.sigmoid(g) if sigmoid else g * torch.sigmoid(g))
    assert ((got - want).abs() <= (2 ** -8 + 2 ** -18) * want.abs() + 1e-30).all()


@pytest.mark.parametrize("where", ["q", "k", "v", "g", "beta"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("token", [16, 31, 60, 64 + 50])
def test_tokens_before_one_that_is_no_number(token, value, where):
    """Tokens of the 16-token tiles in front of it, and other requests, are what they are without it, bit for bit."""
    gen = torch.Generator(device="cuda").manual_seed(token)
    lens, heads, d = [150, 70], 2, 128
    x = {n: torch.randn((220, heads, d), generator=gen, device="cuda").bfloat16() for n in "qkv"}
    x["g"], x["beta"] = -torch.rand((220, heads), generator=gen, device="cuda") * 0.1, torch.rand((220, heads), generator=gen, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")

    def run():
        state = torch.zeros(2, heads, d, d, device="cuda")
        out = ops.gated_delta_rule(x["q"], x["k"], x["v"], x["g"], x["beta"], state, torch.arange(2, **i32), torch.tensor(lens, **i32),
                                   torch.zeros(2, **i32), max_len=150)
        ops.check_status()
        return out, state

    want, state = run()
    x[where][token, 1] = value
    got, after = run()
    clean = token // 16 * 16
    assert not got[token, 1].isfinite().all()
    assert torch.equal(got[:clean], want[:clean]) and torch.equal(got[:, 0], want[:, 0]) and torch.equal(got[150:], want[150:])
    assert torch.equal(after[1], state[1]) and torch.equal(after[0, 0], state[0, 0])
