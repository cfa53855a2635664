"""Prefill and decode steps of the served models, as a serving loop runs them.

A case is one step of one model: ``phase`` "prompt" runs the new tokens of a batch of requests (behind cached prefixes or
not), "reply" runs one new token per request on top of a filled cache.  Weights are random with the shapes of the named
preset and go through the model's own checkpoint loader; the caches of earlier tokens are filled with values of the size
that the models write (keys are normed per head).  ``run`` builds the step's batch and runs it, and returns the logits of
each request's last token with what the step wrote: the rows of the K/V cache and the recurrent states.
"""

from __future__ import annotations

import math
import zlib

import torch

from mllm_b200.configs import ServerConfig
from mllm_b200.executor.model_runner import ModelRunner
from mllm_b200.models.presets import get_preset

# name: preset, layers kept (None: all), weight scheme
MODELS = {
    "dense-0.6b": ("qwen3-0.6b", None, None),
    "dense-8b": ("qwen3-8b", None, None),
    "dense-8b-w4a16": ("qwen3-8b", None, "w4a16"),
    "vl-2b-w8a8": ("qwen3-vl-2b", None, "w8a8"),
    "moe-30b-part": ("qwen3-30b-a3b", 6, None),       # 6 of the 48 layers: the share of one of 8 GPUs
    "hybrid-2b": ("qwen3.5-2b", None, None),
}
CONTEXT = 8192
BATCHES = (1, 8, 32, 64)      # max_running_requests of the runner: a reply batch between two sizes is padded as a server does


def listed():
    return [
        # the smallest calls: one short prompt, and its reply token by token
        dict(name="prompt-0.6b-128", model="dense-0.6b", phase="prompt", requests=1, new=128, spread=0.0, prefix=0, page=16),
        dict(name="reply-0.6b-1x160", model="dense-0.6b", phase="reply", requests=1, new=160, spread=0.0, prefix=0, page=16),
        # the one-batch benchmark: 8 requests of 2048 tokens, prompt and reply
        dict(name="prompt-8b-8x2048", model="dense-8b", phase="prompt", requests=8, new=2048, spread=0.0, prefix=0, page=16),
        dict(name="reply-8b-8x2048", model="dense-8b", phase="reply", requests=8, new=2048, spread=0.0, prefix=0, page=16),
        # serving: a few new requests of odd lengths, some of them behind a shared prefix that is cached already
        dict(name="prompt-8b-ragged", model="dense-8b", phase="prompt", requests=3, new=517, spread=0.8, prefix=1024, page=1),
        # serving: a running batch of unlike lengths, slots given one at a time
        dict(name="reply-8b-29-ragged", model="dense-8b", phase="reply", requests=29, new=1900, spread=0.8, prefix=0, page=1),
        # 4-bit weights, few users
        dict(name="reply-8b-w4a16-2x1500", model="dense-8b-w4a16", phase="reply", requests=2, new=1500, spread=0.3, prefix=0, page=1),
        # an image and a question, 8-bit weights and activations
        dict(name="prompt-vl-2b-w8a8", model="vl-2b-w8a8", phase="prompt", requests=1, new=2048, spread=0.0, prefix=0, page=16),
        # mixture of experts: prompts of a batch, and its replies
        dict(name="prompt-moe-4x2048", model="moe-30b-part", phase="prompt", requests=4, new=2048, spread=0.3, prefix=0, page=16),
        dict(name="reply-moe-64x2048", model="moe-30b-part", phase="reply", requests=64, new=2048, spread=0.5, prefix=0, page=1),
        # delta-net layers beside attention: prompts of a batch, and its replies
        dict(name="prompt-hybrid-4x2000", model="hybrid-2b", phase="prompt", requests=4, new=2000, spread=0.4, prefix=0, page=16),
        dict(name="reply-hybrid-8x2048", model="hybrid-2b", phase="reply", requests=8, new=2048, spread=0.0, prefix=0, page=16),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    model = rng.choice(list(MODELS))
    if model == "vl-2b-w8a8":
        return dict(model=model, phase="prompt", requests=1, new=_log_int(rng, 260, 3000), spread=0.0, prefix=0, page=16)
    page = rng.choice([1, 16])
    if rng.random() < 0.5:
        requests = _log_int(rng, 1, 64)
        return dict(model=model, phase="reply", requests=requests, new=_log_int(rng, 100, min(4096, 65536 // requests)),
                    spread=round(rng.uniform(0.1, 0.8), 2) if page == 1 else 0.0, prefix=0, page=page)
    requests = _log_int(rng, 1, 8)
    top = 1024 if model == "dense-8b-w4a16" else 2048
    return dict(model=model, phase="prompt", requests=requests, new=_log_int(rng, 30, top), spread=round(rng.uniform(0.0, 0.8), 2),
                prefix=rng.choice([0, 0, 1024]) if model != "hybrid-2b" else 0, page=page)


# ---------------------------------------------------------------------------------------------------------------------
# what a case stands for: lengths, slots, weights
# ---------------------------------------------------------------------------------------------------------------------
def _config(case):
    preset, layers, _ = MODELS[case["model"]]
    cfg = get_preset(preset)
    if layers is not None:
        cfg = get_preset(preset, num_hidden_layers=layers)
    return cfg


def _text(cfg):
    return getattr(cfg, "text_config", cfg)


def _lengths(case):
    """(cached tokens, new tokens) of each request.  Lengths are spread evenly around the mean, in an order that mixes them;
    every second prompt has the cached prefix."""
    n, mean, spread = case["requests"], case["new"], case["spread"]
    out = []
    for i in range(n):
        at = (((i * 7) % n) + 0.5) / n * 2 - 1 if n % 7 else (i + 0.5) / n * 2 - 1
        length = max(2, int(round(mean * (1 + spread * at))))
        if case["phase"] == "reply":
            out.append((length - 1, 1))
        else:
            out.append((case["prefix"] if i % 2 == 0 else 0, length))
    return out


def _slots(case):
    """Slots of each request's tokens, in position order, as a fresh allocator gives them.  With pages a request owns whole
    pages; without, a reply batch gets the slots of its new tokens together."""
    page, lens, at, out = case["page"], _lengths(case), case["page"], []
    if page == 1 and case["phase"] == "reply":
        for cached, _ in lens:
            out.append(list(range(at, at + cached)))
            at += cached
        return [s + [at + i] for i, s in enumerate(out)], at + len(lens)
    for cached, new in lens:
        out.append(list(range(at, at + cached + new)))
        at += -(-(cached + new) // page) * page
    return out, at


def _written(case, pool):
    """The view of K/V storage [layer, k|v, head, slot, feature] that holds what the step wrote."""
    slots, end = _slots(case)
    if case["phase"] == "prompt":
        return pool[:, :, :, case["page"]:end]
    if case["page"] == 1:
        return pool[:, :, :, end - len(slots):end]
    step = -(-len(slots[0]) // case["page"]) * case["page"]
    return pool[:, :, :, slots[0][-1]:end:step]


def _generator(name, seed):
    return torch.Generator(device="cuda").manual_seed((zlib.crc32(name.encode()) * 1_000_003 + int(seed)) % 2 ** 63)


def _randn(name, seed, shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(shape, generator=_generator(name, seed), device="cuda", dtype=dtype).mul_(std)


def _tensor_specs(case):
    """Checkpoint name -> (kind, shape) in loading order.  Matrices that write to the residual stream are smaller the deeper
    the model is, so that the stream keeps the size it has in trained models, where no single layer makes up most of it."""
    cfg = _config(case)
    t, scheme = _text(cfg), MODELS[case["model"]][2]
    H, D, V, specs = t.hidden_size, t.head_dim, t.vocab_size, {}
    added = "added-8bit" if scheme == "w8a8" else "added-tied" if t.tie_word_embeddings else "added"

    def linear(name, out, inp, kind="matrix"):
        if scheme == "w4a16":
            specs[name + ".weight_packed"] = ("packed4", (out, inp // 8))
            specs[name + ".weight_scale"] = ("scale4/" + kind, (out, inp // 128))
        elif scheme == "w8a8":
            specs[name + ".weight"] = ("int8", (out, inp))
            specs[name + ".weight_scale"] = ("scale8/" + kind, (out, 1))
        else:
            specs[name + ".weight"] = (kind, (out, inp))

    specs["model.embed_tokens.weight"] = ("matrix" if t.tie_word_embeddings else "table", (V, H))
    hybrid = case["model"] == "hybrid-2b"
    gain = "offset" if hybrid else "gain"
    for i in range(t.num_hidden_layers):
        p = f"model.layers.{i}."
        specs[p + "input_layernorm.weight"] = specs[p + "post_attention_layernorm.weight"] = (gain, (H,))
        if hybrid and t.layer_types[i] == "linear_attention":
            a, kd, vd = p + "linear_attn.", t.linear_num_key_heads * 128, t.linear_num_value_heads * 128
            specs[a + "in_proj_qkv.weight"] = ("matrix", (2 * kd + vd, H))
            specs[a + "in_proj_z.weight"] = ("matrix", (vd, H))
            specs[a + "in_proj_b.weight"] = specs[a + "in_proj_a.weight"] = ("matrix", (t.linear_num_value_heads, H))
            specs[a + "conv1d.weight"] = ("taps", (2 * kd + vd, 1, t.linear_conv_kernel_dim))
            specs[a + "dt_bias"], specs[a + "A_log"] = ("dt_bias", (t.linear_num_value_heads,)), ("a_log", (t.linear_num_value_heads,))
            specs[a + "norm.weight"] = ("gain", (128,))
            linear(a + "out_proj", H, vd, added)
        else:
            a = p + "self_attn."
            linear(a + "q_proj", t.num_attention_heads * D * (2 if hybrid else 1), H)
            linear(a + "k_proj", t.num_key_value_heads * D, H)
            linear(a + "v_proj", t.num_key_value_heads * D, H)
            linear(a + "o_proj", H, t.num_attention_heads * D, added)
            specs[a + "q_norm.weight"] = specs[a + "k_norm.weight"] = (gain, (D,))
        if hasattr(t, "num_experts"):
            E, F = t.num_experts, t.moe_intermediate_size
            specs[p + "mlp.gate.weight"] = ("matrix", (E, H))
            specs[p + "mlp.experts.gate_up_proj"] = ("matrix", (E, 2 * F, H))
            specs[p + "mlp.experts.down_proj"] = (added, (E, H, F))
        else:
            linear(p + "mlp.gate_proj", t.intermediate_size, H)
            linear(p + "mlp.up_proj", t.intermediate_size, H)
            linear(p + "mlp.down_proj", H, t.intermediate_size, added)
    specs["model.norm.weight"] = (gain, (H,))
    if not t.tie_word_embeddings:
        specs["lm_head.weight"] = ("matrix", (V, H))
    vc = getattr(cfg, "vision_config", None)
    if vc is not None:
        W, M = vc.hidden_size, vc.spatial_merge_size ** 2 * vc.hidden_size

        def biased(name, out, inp, kind="matrix"):
            specs[name + ".weight"], specs[name + ".bias"] = (kind, (out, inp)), ("bias", (out,))

        def norm(name, width):
            specs[name + ".weight"], specs[name + ".bias"] = ("gain", (width,)), ("bias", (width,))

        biased("visual.patch_embed.proj", W, vc.in_channels * vc.temporal_patch_size * vc.patch_size ** 2)
        specs["visual.pos_embed.weight"] = ("matrix", (vc.num_position_embeddings, W))
        for i in range(vc.depth):
            b = f"visual.blocks.{i}."
            norm(b + "norm1", W)
            norm(b + "norm2", W)
            biased(b + "attn.qkv", 3 * W, W)
            biased(b + "attn.proj", W, W, "added")
            biased(b + "mlp.linear_fc1", vc.intermediate_size, W)
            biased(b + "mlp.linear_fc2", W, vc.intermediate_size, "added")
        for m in ["visual.merger."] + [f"visual.deepstack_merger_list.{j}." for j in range(len(vc.deepstack_visual_indexes))]:
            norm(m + "norm", W if m == "visual.merger." else M)
            biased(m + "linear_fc1", M, M)
            biased(m + "linear_fc2", vc.out_hidden_size, M)
    return specs


# standard deviations of 16-bit matrices; those of the scaled ones go into the scales.  A tied table has the size of an output
# matrix, and what the layers add to its rows is small to match: in each case all layers together come to about a third of the
# stream, so that a layer's rounding shows and does not drown the result.  (With 8-bit activations a value that rounds to the
# neighbouring code moves a whole step, which takes a smaller share: at a third two correct results differ by a tenth.)
MATRICES = {"matrix": 0.02, "added": 0.02 / 32, "added-tied": 0.02 / 64, "added-8bit": 0.02 / 1024, "table": 1.0}


def _tensor(name, kind, shape, seed):
    g = _generator(name, seed)

    def uniform(low, high):
        return torch.rand(shape, generator=g, device="cuda") * (high - low) + low

    if kind in MATRICES:
        return _randn(name, seed, shape, MATRICES[kind])
    if kind == "taps":
        return _randn(name, seed, shape, 0.5)
    if kind == "bias":
        return _randn(name, seed, shape, 0.02)
    if kind == "gain":
        return _randn(name, seed, shape, 0.1) + 1.0
    if kind == "offset":
        return _randn(name, seed, shape, 0.1)
    if kind == "packed4":      # eight codes from 0 to 15 around 8 in a word
        codes = _randn(name, seed, (8, *shape), 3.0).round_().clamp_(-8, 7).to(torch.int32) + 8
        for i in range(1, 8):
            codes[0] |= codes[i] << (4 * i)
        return codes[0].clone()
    if kind.startswith("scale4/"):
        return (uniform(0.75, 1.25) * (MATRICES[kind[7:]] / 3)).to(torch.bfloat16)
    if kind == "int8":
        return _randn(name, seed, shape, 32.0).round_().clamp_(-127, 127).to(torch.int8)
    if kind.startswith("scale8/"):
        return uniform(0.75, 1.25) * (MATRICES[kind[7:]] / 32)
    if kind == "a_log":
        return uniform(1.0, 16.0).log()
    if kind == "dt_bias":      # steps from 0.001 to 0.1
        return torch.expm1(torch.exp(uniform(math.log(1e-3), math.log(0.1)))).log()
    raise KeyError(kind)


class _Runner(ModelRunner):
    """A runner whose checkpoint is made up while it is read."""

    case, seed = None, 0

    def _iter_weights(self, model_path):
        for name, (kind, shape) in _tensor_specs(self.case).items():
            yield name, _tensor(name, kind, shape, self.seed)


def _inputs(case, seed):
    """Token ids of the new tokens (of all requests in one row), and for an image its pixels and grid."""
    cfg = _config(case)
    n = sum(new for _, new in _lengths(case))
    ids = torch.randint(0, 10000, (n,), generator=_generator("ids", seed), device="cuda")
    if not hasattr(cfg, "vision_config"):
        return ids, None, None
    side = 448 // cfg.vision_config.patch_size
    merged = (side // cfg.vision_config.spatial_merge_size) ** 2
    ids[4], ids[5:5 + merged] = cfg.vision_start_token_id, cfg.image_token_id
    pixels = torch.randint(0, 256, (side * side, 3 * 2 * cfg.vision_config.patch_size ** 2), generator=_generator("pixels", seed), device="cuda")
    return ids, pixels.float() / 127.5 - 1.0, torch.tensor([[1, side, side]], device="cuda")


def _cached_rows(case, seed, layer):
    """K and V of the tokens before the step, [tokens of all requests, 2, kv heads, head size]."""
    t = _text(_config(case))
    return _randn(f"cache.{layer}", seed, (sum(c for c, _ in _lengths(case)), 2, t.num_key_value_heads, t.head_dim))


def _states(case, seed, layer):
    """Recurrent matrices and convolution inputs of the tokens before the step."""
    t, n = _text(_config(case)), case["requests"]
    channels = (2 * t.linear_num_key_heads + t.linear_num_value_heads) * 128
    return (_randn(f"state.{layer}", seed, (n, t.linear_num_value_heads, 128, 128), 0.1, torch.float32),
            _randn(f"history.{layer}", seed, (n, channels, t.linear_conv_kernel_dim - 1)))


def _kinds(case):
    """Attention layers and delta-net layers."""
    t = _text(_config(case))
    types = getattr(t, "layer_types", None) or ["full_attention"] * t.num_hidden_layers
    return [i for i, k in enumerate(types) if k == "full_attention"], [i for i, k in enumerate(types) if k != "full_attention"]


# ---------------------------------------------------------------------------------------------------------------------
# measured
# ---------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    slots, end = _slots(case)
    lens = _lengths(case)
    reply = case["phase"] == "reply"
    sc = ServerConfig(model_path="generated", dtype="bfloat16", context_length=CONTEXT, max_total_tokens=end + 4096,
                      radix_cache_page_size=case["page"], page_size=case["page"],
                      max_running_requests=min(b for b in BATCHES if b >= case["requests"]),
                      disable_cuda_graph=not reply)
    runner = _Runner(sc, hf_config=_config(case), quantization_method=MODELS[case["model"]][2], device="cuda:0")
    runner.case, runner.seed = case, seed
    runner.initialize()
    dev, table = runner.device, runner.req_to_token_pool.req_to_token
    rows = runner.req_to_token_pool.alloc(len(lens))
    for row, s in zip(rows, slots):
        table[row, :len(s)] = torch.tensor(s, dtype=torch.int32, device=dev)
    before = torch.tensor([x for (c, _), s in zip(lens, slots) for x in s[:c]], dtype=torch.int64, device=dev)
    attention, delta = _kinds(case)
    for j in range(len(attention)):
        if before.numel():
            values = _cached_rows(case, seed, j)
            for buffer, value in zip(runner.token_to_kv_pool.get_kv_buffer(j), values.unbind(1)):
                buffer[before] = value
    if delta and reply:
        for j in range(len(delta)):
            for buffer, value in zip(runner.gdn_pool.layer(j), _states(case, seed, j)):
                buffer[rows[0]:rows[0] + len(rows)] = value
    ids, pixels, grid = _inputs(case, seed)

    def ints(values, dtype=torch.int32):
        return torch.tensor(values, dtype=dtype, device=dev)

    return dict(
        case=case, runner=runner, ids=ids, rows=ints(rows), first=rows[0], lens=ints([c + n for c, n in lens]), new=ints([n for _, n in lens]),
        cached=ints([c for c, _ in lens]), loc=ints([x for (c, _), s in zip(lens, slots) for x in s[c:]], torch.int64),
        new_host=[n for _, n in lens], cached_host=[c for c, _ in lens],
        extra={} if pixels is None else dict(pixel_values=pixels, image_grid_thw=grid))


def run(state):
    r, case = state["runner"], state["case"]
    if case["phase"] == "reply":
        batch = r.prepare_forward_batch_decode(state["ids"], state["rows"], state["lens"], state["loc"],
                                               max_seq_len=max(state["cached_host"]) + 1)
    else:
        batch = r.prepare_forward_batch_extend(state["ids"], state["rows"], state["lens"], state["new"], state["cached"], state["loc"],
                                               extend_seq_lens_cpu=state["new_host"], extend_prefix_lens_cpu=state["cached_host"],
                                               **state["extra"])
    out = dict(logits=r.forward(batch).next_token_logits, cache=_written(case, r.token_to_kv_pool.store))
    if r.gdn_pool is not None:
        at = slice(state["first"], state["first"] + case["requests"])
        out.update(state=r.gdn_pool.recurrent[:, at], history=r.gdn_pool.conv[:, at])
    return out


def work(case):
    cfg, lens = _config(case), _lengths(case)
    t = _text(cfg)
    H, D, V = t.hidden_size, t.head_dim, t.vocab_size
    T, B = sum(n for _, n in lens), len(lens)
    attention, delta = _kinds(case)
    size = {"packed4": 4, "int8": 1, "scale8/matrix": 4, "a_log": 4, "dt_bias": 4}
    weights = flops = 0.0
    for name, (kind, shape) in _tensor_specs(case).items():
        n = math.prod(shape)
        if name == "model.embed_tokens.weight":
            weights += T * H * 2 + (n * 2 if t.tie_word_embeddings else 0)
            flops += 2.0 * B * n if t.tie_word_embeddings else 0
            continue
        if "experts" in name:      # experts that T tokens with 8 choices each reach on average
            E, k = t.num_experts, t.num_experts_per_tok
            weights += n * 2 * (1 - (1 - k / E) ** T)
            flops += 2.0 * T * n * k / E
            continue
        weights += n * size.get(kind, 2)
        rows = B if name == "lm_head.weight" else 784 if name.startswith("visual.blocks") or "patch_embed" in name else \
            196 if name.startswith("visual.") else T
        if len(shape) == 2 and (kind in MATRICES or kind in ("int8", "packed4")) and "pos_embed" not in name:
            flops += 2.0 * rows * n * (8 if kind == "packed4" else 1)
    pairs = sum(n * c + n * (n + 1) / 2 for c, n in lens)
    kv = 2 * t.num_key_value_heads * D * 2.0 * len(attention)
    data = kv * sum(c + n for c, n in lens) + B * V * 2.0
    flops += 4.0 * pairs * t.num_attention_heads * D * len(attention)
    if delta:
        state = t.linear_num_value_heads * 128 * 128
        data += len(delta) * B * state * 4.0 * (2 if case["phase"] == "reply" else 1)
        flops += len(delta) * T * state * 6.0
    if hasattr(cfg, "vision_config"):
        flops += 4.0 * 784 * 784 * cfg.vision_config.hidden_size * cfg.vision_config.depth
    return {"bytes": weights + data, "flops": flops}


def tolerance(case):
    # 16-bit activations through all layers: against 64 bits the outputs are 0.004 to 0.007 off where there are six layers, and
    # 0.009 to 0.017 where there are 24 to 36 (8-bit activations among them), and two correct results differ by up to twice that
    return {"rel": 0.02 if case["model"] == "moe-30b-part" else 0.03}


# ---------------------------------------------------------------------------------------------------------------------
# the same step in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _rms(x, gain, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * gain


def _turn(x, angles):
    """x [T, heads, D]: features i and i + n of the first 2n turn by angles [T, n]."""
    n = angles.shape[-1]
    c, s = angles.cos().unsqueeze(1), angles.sin().unsqueeze(1)
    a, b = x[..., :n], x[..., n:2 * n]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * n:]], -1)


def _attend(q, k, v, first):
    """Causal attention of q [n, heads, D] at positions first.. over k, v [m, kv heads, D]."""
    n, heads, D = q.shape
    group = heads // k.shape[1]
    out = torch.empty_like(q)
    at = torch.arange(first, first + n, device=q.device).unsqueeze(1)
    hidden = torch.arange(k.shape[0], device=q.device).unsqueeze(0) > at
    for h in range(k.shape[1]):
        s = torch.einsum("ngd,md->gnm", q[:, h * group:(h + 1) * group], k[:, h]) * D ** -0.5
        out[:, h * group:(h + 1) * group] = torch.einsum("gnm,md->ngd", s.masked_fill_(hidden, -math.inf).softmax(-1), v[:, h])
    return out


def _delta_net(get, p, t, x, lens, states, history):
    """The delta-net mixer, token by token; returns its output, the states and the convolution inputs that follow."""
    hk, hv, taps, B, n_max = t.linear_num_key_heads, t.linear_num_value_heads, t.linear_conv_kernel_dim, len(lens), max(n for _, n in lens)
    kd = hk * 128
    rows = x @ get(p + "in_proj_qkv.weight").t()
    z = (x @ get(p + "in_proj_z.weight").t()).unflatten(-1, (hv, 128))
    beta = torch.sigmoid(x @ get(p + "in_proj_b.weight").t())
    g = -get(p + "A_log").exp() * torch.nn.functional.softplus(x @ get(p + "in_proj_a.weight").t() + get(p + "dt_bias"))
    w, mixed, at = get(p + "conv1d.weight")[:, 0], [], 0
    for i, (_, n) in enumerate(lens):
        seq = torch.cat([history[i].t(), rows[at:at + n]])
        mixed.append(torch.nn.functional.silu(sum(seq[j:j + n] * w[:, j] for j in range(taps))))
        history[i] = seq[-(taps - 1):].t()
        at += n

    def padded(parts):
        return torch.stack([torch.nn.functional.pad(m, (0, 0) * (m.dim() - 1) + (0, n_max - m.shape[0])) for m in parts], 1)

    m = padded(mixed)
    q, k, v = m[..., :kd].unflatten(-1, (hk, 128)), m[..., kd:2 * kd].unflatten(-1, (hk, 128)), m[..., 2 * kd:].unflatten(-1, (hv, 128))
    q, k = (u * torch.rsqrt(u.square().sum(-1, keepdim=True) + 1e-6) for u in (q, k))
    q, k = q.repeat_interleave(hv // hk, 2) * 128 ** -0.5, k.repeat_interleave(hv // hk, 2)
    news = [n for _, n in lens]
    beta, decay = padded(beta.split(news)), padded(g.split(news)).exp()      # behind a request's end: decay 1 and step 0
    S, out = states, torch.empty(n_max, B, hv, 128, dtype=torch.float64, device=x.device)
    for step in range(n_max):
        S = S * decay[step, :, :, None, None]
        u = (v[step] - torch.einsum("bhkv,bhk->bhv", S, k[step])) * beta[step].unsqueeze(-1)
        S = S + k[step].unsqueeze(-1) * u.unsqueeze(-2)
        out[step] = torch.einsum("bhkv,bhk->bhv", S, q[step])
    o = torch.cat([out[:n, i] for i, n in enumerate(news)])
    o = _rms(o, get(p + "norm.weight"), t.rms_norm_eps) * torch.nn.functional.silu(z)
    return o.flatten(1) @ get(p + "out_proj.weight").t(), S, history


def _image(get, cfg, pixels):
    """Vision tower of one square image: image features and one set per deepstack level."""
    vc = cfg.vision_config
    side, heads, W = int(math.isqrt(pixels.shape[0])), vc.num_heads, vc.hidden_size
    m = vc.spatial_merge_size
    dev = pixels.device

    def linear(x, name):
        return x @ get(name + ".weight").t() + get(name + ".bias")

    def norm(x, name):
        return torch.nn.functional.layer_norm(x, x.shape[-1:], get(name + ".weight"), get(name + ".bias"), 1e-6)

    def merge_order(grid):      # [side, side, ...] -> neighbours of a merged patch in a row
        return grid.unflatten(1, (side // m, m)).unflatten(0, (side // m, m)).transpose(1, 2).flatten(0, 3)

    table = int(math.isqrt(vc.num_position_embeddings))
    pos = torch.linspace(0, table - 1, side, dtype=torch.float32).double().to(dev)
    low = pos.floor()
    part, low = pos - low, low.long()
    high = (low + 1).clamp(max=table - 1)
    e = get("visual.pos_embed.weight").view(table, table, W)
    rows = e[low] * (1 - part)[:, None, None] + e[high] * part[:, None, None]
    grid = rows[:, low] * (1 - part)[None, :, None] + rows[:, high] * part[None, :, None]
    x = linear(pixels.to(torch.bfloat16).double(), "visual.patch_embed.proj") + merge_order(grid)
    D = W // heads
    inv = 10000.0 ** (-torch.arange(0, D // 2, 2, dtype=torch.float64, device=dev) / (D // 2))
    at = torch.arange(side, dtype=torch.float64, device=dev)
    rc = merge_order(torch.stack(torch.meshgrid(at, at, indexing="ij"), -1))
    angles = (rc.unsqueeze(-1) * inv).flatten(1)
    levels = []

    def merger(x, p, shuffled):
        y = norm(x.reshape(-1, m * m * W), p + "norm") if shuffled else norm(x, p + "norm").reshape(-1, m * m * W)
        return linear(torch.nn.functional.gelu(linear(y, p + "linear_fc1")), p + "linear_fc2")

    for i in range(vc.depth):
        b = f"visual.blocks.{i}."
        q, k, v = linear(norm(x, b + "norm1"), b + "attn.qkv").view(-1, 3, heads, D).unbind(1)
        q, k = _turn(q, angles), _turn(k, angles)
        s = torch.einsum("nhd,mhd->hnm", q, k) * D ** -0.5
        x = x + linear(torch.einsum("hnm,mhd->nhd", s.softmax(-1), v).flatten(1), b + "attn.proj")
        y = torch.nn.functional.gelu(linear(norm(x, b + "norm2"), b + "mlp.linear_fc1"), approximate="tanh")
        x = x + linear(y, b + "mlp.linear_fc2")
        if i in vc.deepstack_visual_indexes:
            levels.append(merger(x, f"visual.deepstack_merger_list.{len(levels)}.", True))
    return merger(x, "visual.merger.", False), levels


def exact(case, seed):
    cfg, lens = _config(case), _lengths(case)
    t = _text(cfg)
    specs, scheme = _tensor_specs(case), MODELS[case["model"]][2]
    D, heads, kv_heads, eps = t.head_dim, t.num_attention_heads, t.num_key_value_heads, t.rms_norm_eps
    hybrid = case["model"] == "hybrid-2b"
    slots, end = _slots(case)
    news = [n for _, n in lens]

    def get(name):
        kind, shape = specs[name]
        w = _tensor(name, kind, shape, seed).double()
        return w + 1 if kind == "offset" else w

    def linear(x, name):
        if scheme == "w4a16":
            words, scale = _tensor(name + ".weight_packed", *specs[name + ".weight_packed"], seed), get(name + ".weight_scale")
            codes = ((words.unsqueeze(-1) >> torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)) & 15).flatten(1).double() - 8
            return x @ (codes.unflatten(1, (-1, 128)) * scale.unsqueeze(-1)).flatten(1).t()
        if scheme == "w8a8":
            step = x.abs().amax(-1, keepdim=True) / 127
            return ((x / step).round() @ get(name + ".weight").t()) * step * get(name + ".weight_scale")[:, 0]
        return x @ get(name + ".weight").t()

    ids, pixels, _ = _inputs(case, seed)
    x = _tensor("model.embed_tokens.weight", *specs["model.embed_tokens.weight"], seed)[ids].double()
    positions = torch.cat([torch.arange(c, c + n, dtype=torch.float64, device="cuda") for c, n in lens])
    levels = []
    theta = t.rope_parameters["rope_theta"] if hybrid else t.rope_theta
    turned = int(D * t.rope_parameters["partial_rotary_factor"]) if hybrid else D
    angles = positions.unsqueeze(1) * theta ** (-torch.arange(0, turned, 2, dtype=torch.float64, device="cuda") / turned)
    if pixels is not None:
        features, levels = _image(get, cfg, pixels)
        x[5:5 + features.shape[0]] = features
        side = int(math.isqrt(features.shape[0]))
        p3 = positions.repeat(3, 1)
        i = torch.arange(side * side, device="cuda")
        p3[:, 5:5 + side * side] = torch.stack([torch.zeros_like(i), i // side, i % side]) + 5.0
        p3[:, 5 + side * side:] = torch.arange(p3.shape[1] - 5 - side * side, device="cuda") + 5.0 + side
        j = torch.arange(D // 2, device="cuda")
        sections = t.rope_scaling["mrope_section"]
        axis = torch.where((j % 3 == 1) & (j < 3 * sections[1]), 1, torch.where((j % 3 == 2) & (j < 3 * sections[2]), 2, 0))
        angles = p3[axis].t() * theta ** (-2.0 * j / D)
    attention, delta = _kinds(case)
    store = torch.zeros(len(attention), 2, kv_heads, end, D, dtype=torch.float64, device="cuda")
    states, histories = [], []
    for i in range(t.num_hidden_layers):
        p = f"model.layers.{i}."
        h = _rms(x, get(p + "input_layernorm.weight"), eps)
        if i in attention:
            a, layer = p + "self_attn.", attention.index(i)
            q = linear(h, a + "q_proj").unflatten(-1, (heads, -1))
            gate = q[..., D:]
            k, v = linear(h, a + "k_proj").unflatten(-1, (kv_heads, D)), linear(h, a + "v_proj").unflatten(-1, (kv_heads, D))
            q = _turn(_rms(q[..., :D], get(a + "q_norm.weight"), eps), angles)
            k = _turn(_rms(k, get(a + "k_norm.weight"), eps), angles)
            past, at, past_at, parts = _cached_rows(case, seed, layer).double(), 0, 0, []
            for (c, n), s in zip(lens, slots):
                kk = torch.cat([past[past_at:past_at + c, 0], k[at:at + n]])
                vv = torch.cat([past[past_at:past_at + c, 1], v[at:at + n]])
                store[layer, 0, :, s], store[layer, 1, :, s] = kk.transpose(0, 1), vv.transpose(0, 1)
                parts.append(_attend(q[at:at + n], kk, vv, c))
                at, past_at = at + n, past_at + c
            o = torch.cat(parts).flatten(1)
            if hybrid:
                o = o * torch.sigmoid(gate.flatten(1))
            x = x + linear(o, a + "o_proj")
        else:
            S, history = (u.double() for u in _states(case, seed, delta.index(i)))
            if case["phase"] == "prompt":
                S, history = torch.zeros_like(S), torch.zeros_like(history)
            y, S, history = _delta_net(get, p + "linear_attn.", t, h, lens, S, history)
            x = x + y
            states.append(S)
            histories.append(history)
        h = _rms(x, get(p + "post_attention_layernorm.weight"), eps)
        if hasattr(t, "num_experts"):
            prob, choice = (h @ get(p + "mlp.gate.weight").t()).softmax(-1).topk(t.num_experts_per_tok)
            prob = prob / prob.sum(-1, keepdim=True)
            up = _tensor(p + "mlp.experts.gate_up_proj", *specs[p + "mlp.experts.gate_up_proj"], seed)
            down = _tensor(p + "mlp.experts.down_proj", *specs[p + "mlp.experts.down_proj"], seed)
            y = torch.zeros_like(x)
            for e in range(t.num_experts):
                row, col = (choice == e).nonzero(as_tuple=True)
                a, b = (h[row] @ up[e].double().t()).chunk(2, -1)
                y.index_add_(0, row, ((torch.nn.functional.silu(a) * b) @ down[e].double().t()) * prob[row, col].unsqueeze(-1))
            x = x + y
        else:
            y = torch.nn.functional.silu(linear(h, p + "mlp.gate_proj")) * linear(h, p + "mlp.up_proj")
            x = x + linear(y, p + "mlp.down_proj")
        if i < len(levels):
            x[5:5 + levels[i].shape[0]] += levels[i]
    last = torch.tensor(news, device="cuda").cumsum(0) - 1
    head = get("model.embed_tokens.weight" if t.tie_word_embeddings else "lm_head.weight")
    out = dict(logits=_rms(x[last], get("model.norm.weight"), eps) @ head.t(), cache=_written(case, store))
    if delta:
        out.update(state=torch.stack(states), history=torch.stack(histories))
    return out
