"""A decoder layer over new tokens as one native call against the calls one by one."""

from types import SimpleNamespace

import pytest
import torch

from mllm_b200 import ops
from mllm_b200.engine.forward_batch import ForwardMode
from mllm_b200.models.qwen3 import Qwen3DecoderLayer

pytestmark = pytest.mark.gpu


def _layer(bias, norm, dtype=torch.bfloat16):
    torch.manual_seed(3)
    config = SimpleNamespace(hidden_size=512, num_attention_heads=4, num_key_value_heads=2, head_dim=128, intermediate_size=768, rms_norm_eps=1e-6,
                             attention_bias=bias, use_qk_norm=norm, rope_theta=1e4)
    layer = Qwen3DecoderLayer(config, 0, params_dtype=dtype).cuda()
    for name, p in layer.named_parameters():
        p.data.copy_(torch.randn_like(p, dtype=torch.float32) * (0.05 if p.dim() > 1 else 0.3) + (1.0 if "norm" in name else 0.0))
    layer.mlp.gate_up_proj.quant_method.process_weights_after_loading(layer.mlp.gate_up_proj)
    return layer


def _batch(lens, prefix, cache=torch.bfloat16):
    new = [n - p for n, p in zip(lens, prefix)]
    width = max(lens)
    table = torch.arange(len(lens) * width, dtype=torch.int32, device="cuda").view(len(lens), width)
    i32 = dict(dtype=torch.int32, device="cuda")
    torch.manual_seed(5)
    pools = [torch.randn(len(lens) * width, 2, 128, device="cuda").to(cache) for _ in range(2)]
    fb = SimpleNamespace(
        forward_mode=ForwardMode.EXTEND, mrope_positions=None, req_to_token_pool=SimpleNamespace(req_to_token=table), extra={},
        token_to_kv_pool=SimpleNamespace(get_kv_buffer=lambda i: pools), req_pool_indices=torch.arange(len(lens), **i32),
        seq_lens=torch.tensor(lens, **i32), extend_prefix_lens=torch.tensor(prefix, **i32), max_extend_len=max(new),
        extend_start_loc=torch.tensor([sum(new[:i]) for i in range(len(new))], **i32),
        positions=torch.cat([torch.arange(p, n, device="cuda") for n, p in zip(lens, prefix)]),
        out_cache_loc=torch.cat([table[i, p:n].long() for i, (n, p) in enumerate(zip(lens, prefix))]))
    return fb, sum(new)


def _compare(layer, make_batch, first, monkeypatch, dtype=torch.bfloat16):
    """The native call serves the layer, and gives what the calls one by one give: the same kernels on the same numbers."""
    def run():
        fb, rows = make_batch()
        torch.manual_seed(7)
        hidden, residual = torch.randn(rows, 512, device="cuda").to(dtype), torch.randn(rows, 512, device="cuda").to(dtype)
        out = layer(hidden, None if first else residual, fb)
        return (*out, *fb.token_to_kv_pool.get_kv_buffer(0))

    results, native = [], ops.prefill_layer
    monkeypatch.setattr(ops, "prefill_layer", lambda *a: results.append(native(*a)) or results[-1])
    got = run()
    assert len(results) == 1 and results[0] is not None
    results.clear()
    hooked = []
    handle = layer.self_attn.attn.register_forward_hook(lambda *a: hooked.append(1))      # a hooked part is called as such
    want = run()
    handle.remove()
    assert hooked and not results
    for g, w in zip(got, want):
        assert torch.equal(g.view(torch.uint8) if g.dtype.itemsize == 1 else g, w.view(torch.uint8) if w.dtype.itemsize == 1 else w)
    return got


@pytest.mark.parametrize("bias,norm", [(False, True), (True, False)])
@pytest.mark.parametrize("lens,prefix", [([9], [0]), ([70, 200], [6, 0]), ([300, 41, 9], [0, 40, 1])], ids=str)
@pytest.mark.parametrize("first", [False, True])
def test_native_layer(bias, norm, lens, prefix, first, monkeypatch):
    _compare(_layer(bias, norm), lambda: _batch(lens, prefix), first, monkeypatch)


@pytest.mark.parametrize("option", ["fp16", "8-bit cache", "window", "soft cap", "three axes", "gelu"])
def test_native_layer_options(option, monkeypatch):
    dtype = torch.float16 if option == "fp16" else torch.bfloat16
    lens, prefix = [70, 200], [6, 0]

    def changed(on):
        layer = _layer(False, True, dtype)
        core = layer.self_attn.attn
        if on and option == "window":
            core.sliding_window = 20
        if on and option == "soft cap":
            core.logit_cap = 0.5
        if on and option == "three axes":
            core.mrope_sections = [24, 20, 20]
        if on and option == "gelu":
            layer.mlp.gate_up_proj.gate_activation = "gelu_tanh"

        def make():
            fb, rows = _batch(lens, prefix, torch.float8_e4m3fn if on and option == "8-bit cache" else dtype)
            if option == "three axes":
                fb.mrope_positions = torch.stack([fb.positions, fb.positions // 3, fb.positions % 5])
            return fb, rows

        return layer, make

    got = _compare(*changed(True), False, monkeypatch, dtype)
    if option != "fp16":        # and the option reached the kernels
        monkeypatch.undo()
        assert not torch.equal(got[0], _compare(*changed(False), False, monkeypatch, dtype)[0])


def _misaligned(w):
    """The same rows two bytes behind a 16-byte boundary."""
    store = torch.empty(w.numel() + 8, dtype=w.dtype, device=w.device)[1:w.numel() + 1].view(w.shape)
    return store.copy_(w.data)


@pytest.mark.parametrize("part", ["weight", "gains", "head sizes"])
def test_declined_before_anything_is_launched(part, monkeypatch):
    """What the native call cannot serve leaves the residual stream as it was."""
    layer = _layer(False, True)
    fb, rows = _batch([70], [6])
    hidden, residual = torch.randn(rows, 512, device="cuda").bfloat16(), torch.randn(rows, 512, device="cuda").bfloat16()
    before = [t.clone() for t in (hidden, residual, *fb.token_to_kv_pool.get_kv_buffer(0))]
    if part == "weight":            # no kernel reads it: the calls one by one say so
        layer.mlp.down_proj.weight.data = _misaligned(layer.mlp.down_proj.weight)
        assert layer._forward_native(hidden, residual, fb) is None
    elif part == "gains":
        layer.post_attention_layernorm.weight.data = torch.ones(511, device="cuda", dtype=torch.bfloat16)
        with pytest.raises(RuntimeError):
            layer._forward_native(hidden, residual, fb)
    else:                           # the switch that takes a head size off the kernels
        monkeypatch.setattr(ops, "_ATTN_HEAD_SIZES", (64, 256))
        assert layer._forward_native(hidden, residual, fb) is None
    for t, b in zip((hidden, residual, *fb.token_to_kv_pool.get_kv_buffer(0)), before):
        assert torch.equal(t, b)
