"""What the framework's speed is measured on: the calls a program makes, at the sizes it makes them.

Speech (the 0.6B and 1.7B architectures of config.preset, random weights):
  prompt     Engine.prefill: the talker over a prompt's rows -> last-row logits, hidden state, the key / value cache it leaves
  codec      CodecDecoder.decode: codes of an utterance, or of a streaming window whose context is only there for its state -> waveform
  frames     Engine.decode_frames: a chunk of the frame loop for one or several lock-step utterances -> codes, last hidden state
Sequence models (op lists of seq_ops.StepBuilder, sizes of the `--seq-model` benchmark):
  attention  one softmax-attention layer on a prompt, a portion of one, or decoded rows behind a filled cache, bf16 or true f32
  delta      one gated-delta-rule layer on a prompt
  moe        one routed-experts feed-forward with a shared expert
  request    SequenceEngine.step: a whole small model over a prompt and then token by token -> logits of every step

Every case makes its weights and inputs on the GPU from the seed.  `exact` restates each path in float64 torch, without the framework.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # x-vector voice clone: the prompt in front of every streamed utterance (time to first audio)
        dict(name="prompt of a clone", what="prompt", size="0.6B", layers=28, rows=39),
        # voice clone with a reference clip in the context
        dict(name="prompt with a clip", what="prompt", size="0.6B", layers=8, rows=262),
        # the longest prompts that the default cache of 2048 positions takes
        dict(name="longest prompt", what="prompt", size="0.6B", layers=4, rows=1900),
        # streaming: 8 new frames behind 25 frames of context, once per chunk
        dict(name="codec window", what="codec", frames=33, context=25),
        # non-streaming: 20 seconds of audio at once
        dict(name="codec utterance", what="codec", frames=256, context=0),
        # one streamed utterance: a chunk of 8 frames
        dict(name="chunk of frames", what="frames", streams=1, frames=8, before=120),
        # serving: sixteen utterances share the weight sweeps of a chunk
        dict(name="sixteen utterances", what="frames", streams=16, frames=8, before=120),
        # attention layer of a 1024-wide sequence model on a whole prompt: capped scores, sink, output gates, part of a head rotated
        dict(name="attention prompt", what="attention", rows=2048, before=0, heads=16, kv=4, cap=50.0, window=0, gate=True, f32=False),
        # the same mechanism, windowed, in true 32-bit, on a portion of a prompt
        dict(name="attention portion f32", what="attention", rows=384, before=300, heads=8, kv=2, cap=0.0, window=512, gate=False, f32=True),
        # delta-rule layer on a ragged prompt
        dict(name="delta rule prompt", what="delta", rows=1501, width=1024, heads=8, kv=4),
        # routed experts on a batch of prompt rows
        dict(name="experts", what="moe", rows=701, width=1024, experts=16, top=2, ff=768, shared=1536),
        # a short request to a whole model: its prompt, then its tokens one by one
        dict(name="request", what="request", prompt=203, new=24, width=1024),
    ]


def draw(rng):
    def spread(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))

    what = rng.choice(["prompt", "prompt", "codec", "codec", "frames", "attention", "attention", "delta", "moe", "request"])
    if what == "prompt":
        size = rng.choice(["0.6B", "0.6B", "1.7B"])
        rows = spread(17, 1900)
        return dict(what=what, size=size, layers=max(1, min(12, 4000 // rows // (1 if size == "0.6B" else 3))), rows=rows)
    if what == "codec":
        context = rng.choice([0, 25])
        return dict(what=what, frames=context + spread(1, 24 if context else 256), context=context)
    if what == "frames":
        return dict(what=what, streams=spread(1, 16), frames=rng.randint(1, 8), before=spread(20, 300))
    if what == "attention":
        f32 = rng.random() < 0.3
        rows = 1 if rng.random() < 0.15 else spread(2, 500 if f32 else 2048)
        kv = rng.choice([1, 2, 4])
        return dict(what=what, rows=rows, before=rng.choice([0, spread(1, 2048 - min(rows, 2000))]), heads=kv * rng.choice([1, 2, 3, 4]), kv=kv,
                    cap=rng.choice([0.0, 0.0, 50.0]), window=rng.choice([0, 0, spread(16, 1024)]), gate=rng.random() < 0.5, f32=f32)
    if what == "delta":
        kv = rng.choice([2, 4])
        return dict(what=what, rows=spread(2, 2048), width=rng.choice([512, 1024]), heads=kv * rng.choice([1, 2]), kv=kv)
    if what == "moe":
        experts = rng.choice([8, 14, 16, 32])
        return dict(what=what, rows=spread(1, 2048), width=rng.choice([1024, 2048]), experts=experts, top=rng.randint(1, 4), ff=rng.choice([512, 768, 1024]),
                    shared=rng.choice([0, 1536, 2048]))
    return dict(what=what, prompt=spread(5, 500), new=rng.randint(1, 24), width=rng.choice([512, 1024]))


class _Draws:
    """Random tensors on the GPU, in order, from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)

    def n(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        t = torch.randn(*shape, generator=self.g, device=DEV, dtype=torch.float32)
        return (t * std + mean if mean else t * std).to(dtype)

    def u(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, generator=self.g, device=DEV, dtype=torch.float32) * (hi - lo) + lo

    def i(self, *shape, below):
        return torch.randint(0, below, shape, generator=self.g, device=DEV)


def _rms(x, eps, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


# ------------------------------------------------------------------------------------------------------------------------
# speech: talker prompt and frame loop
# ------------------------------------------------------------------------------------------------------------------------
def _tts_config(case):
    from qwen3_tts_cuda_graphs_b200.config import preset, with_layers

    if case["what"] == "frames":
        return preset("0.6B-Base")
    return with_layers(preset(case["size"] + "-Base"), case["layers"], 1)


def _tts_weights(cfg, d):
    from qwen3_tts_cuda_graphs_b200.weights import tensor_specs

    w = {}
    for name, shape, kind in tensor_specs(cfg):
        if "text_embedding" in name or "text_projection" in name:
            continue      # prompts arrive as embeddings here
        if kind == "norm":
            w[name] = d.n(*shape, std=0.1, mean=1.0)
        else:
            w[name] = d.n(*shape, std=0.08 if kind == "head" else 0.64 * cfg.talker.hidden_size ** -0.5)      # 0.02 at the 0.6B width
    return w


def _engine(cfg, w, max_seq, streams):
    from qwen3_tts_cuda_graphs_b200.engine import Engine
    from qwen3_tts_cuda_graphs_b200.weights import pack_arena

    return Engine(cfg, pack_arena(cfg, w, max_seq, torch.device(DEV)), max_seq, max_streams=streams, max_frames=512)


class _DeviceArray:
    """A framework buffer by its device address, for torch.as_tensor; the tensor keeps this object, and with it the buffer's owner."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<i2", data=(int(ptr), False), version=2)


def _prompt_inputs(case, seed):
    d, cfg = _Draws(seed), _tts_config(case)
    w = _tts_weights(cfg, d)
    # rows are sums of text and codec embeddings, larger than what one layer adds to them
    return cfg, w, d.n(case["rows"], cfg.talker.hidden_size, std=0.5)


def _prompt_prepare(case, seed):
    from qwen3_tts_cuda_graphs_b200.engine import SamplingPolicy

    cfg, w, x = _prompt_inputs(case, seed)
    eng = _engine(cfg, w, 2048, 1)
    t = cfg.talker
    kv = [torch.as_tensor(_DeviceArray(eng, eng.lib.fq3_kv_cache_ptr(eng.h, 0, 0, which), (t.num_hidden_layers, t.num_key_value_heads, 2048, t.head_dim)),
                          device=DEV).view(torch.bfloat16) for which in (0, 1)]
    return dict(eng=eng, x=x, policy=SamplingPolicy(do_sample=False), kv=kv)


def _prompt_run(s, case):
    logits = s["eng"].prefill(0, s["x"], 0, s["policy"], want_logits=True)
    return {"logits": logits, "hidden": s["eng"].last_hidden(0), "k": s["kv"][0][:, :, :case["rows"]], "v": s["kv"][1][:, :, :case["rows"]]}


def _half_turn(x, cos, sin):
    h = x.shape[-1] // 2
    return x * cos + torch.cat([-x[..., h:], x[..., :h]], -1) * sin


def _prompt_exact(case, seed):
    cfg, w, x = _prompt_inputs(case, seed)
    t, T = cfg.talker, case["rows"]
    W = {k: v.to(F64) for k, v in w.items() if k.startswith(("talker.model", "talker.codec_head")) and "embedding" not in k}
    x = x.to(F64)
    f = t.rope_theta ** (-torch.arange(0, t.head_dim, 2, device=DEV, dtype=F64) / t.head_dim)
    a = torch.arange(T, device=DEV, dtype=F64)[:, None] * f
    cos, sin = torch.cat([a, a], -1).cos()[:, None], torch.cat([a, a], -1).sin()[:, None]
    H, G, D = t.num_attention_heads, t.num_key_value_heads, t.head_dim
    mask = torch.ones(T, T, device=DEV, dtype=torch.bool).triu(1)
    ks, vs = [], []
    for i in range(t.num_hidden_layers):
        p = f"talker.model.layers.{i}."
        h = _rms(x, t.rms_norm_eps, W[p + "input_layernorm.weight"])
        q = _rms((h @ W[p + "self_attn.q_proj.weight"].T).view(T, H, D), t.rms_norm_eps, W[p + "self_attn.q_norm.weight"])
        k = _rms((h @ W[p + "self_attn.k_proj.weight"].T).view(T, G, D), t.rms_norm_eps, W[p + "self_attn.k_norm.weight"])
        v = (h @ W[p + "self_attn.v_proj.weight"].T).view(T, G, D)
        q, k = _half_turn(q, cos, sin), _half_turn(k, cos, sin)
        ks.append(k.transpose(0, 1))
        vs.append(v.transpose(0, 1))
        o = torch.empty(T, H, D, device=DEV, dtype=F64)
        for g in range(G):
            for hd in range(g * (H // G), (g + 1) * (H // G)):
                s = (q[:, hd] @ k[:, g].T) * D ** -0.5
                o[:, hd] = s.masked_fill_(mask, -math.inf).softmax(-1) @ v[:, g]
        x = x + o.reshape(T, H * D) @ W[p + "self_attn.o_proj.weight"].T
        h = _rms(x, t.rms_norm_eps, W[p + "post_attention_layernorm.weight"])
        x = x + (F.silu(h @ W[p + "mlp.gate_proj.weight"].T) * (h @ W[p + "mlp.up_proj.weight"].T)) @ W[p + "mlp.down_proj.weight"].T
    hid = _rms(x[-1], t.rms_norm_eps, W["talker.model.norm.weight"])
    return {"logits": hid @ W["talker.codec_head.weight"].T, "hidden": hid, "k": torch.stack(ks), "v": torch.stack(vs)}


def _frames_prepare(case, seed):
    from qwen3_tts_cuda_graphs_b200.engine import SamplingPolicy, SubPolicy

    d, cfg = _Draws(seed), _tts_config(case)
    w = _tts_weights(cfg, d)
    S, H = case["streams"], cfg.talker.hidden_size
    eng = _engine(cfg, w, 1024, S)
    policy = SamplingPolicy(min_new_tokens=512, seed=int(seed) & 0xFFFFFF)
    for i in range(S):
        eng.set_text_conditioning(i, d.n(40, H, std=0.3), d.n(H, std=0.3))
        eng.prefill(i, d.n(case["before"], H, std=0.3), 0, policy, dense=False)
    first = [int(v) for v in d.i(S, below=2048).tolist()]
    return dict(eng=eng, policy=policy, sub=SubPolicy(), first=first, hidden=[d.n(H) for _ in range(S)])


def _frames_run(s, case):
    eng = s["eng"]
    for i, (tok, hid) in enumerate(zip(s["first"], s["hidden"])):      # the utterances as they stood when the chunk began
        eng.reset_stream(i)
        eng.set_loop_state(i, tok, hid, case["before"], 0)
    eng.decode_frames(case["streams"], case["frames"], s["policy"], s["sub"])
    return {"hidden": [eng.last_hidden(i) for i in range(case["streams"])], "codes": [eng.read_codes(i, 0, case["frames"]) for i in range(case["streams"])]}


# ------------------------------------------------------------------------------------------------------------------------
# speech: codec decoder
# ------------------------------------------------------------------------------------------------------------------------
def _codec_inputs(case, seed):
    from qwen3_tts_cuda_graphs_b200.codec import codec_tensor_specs
    from qwen3_tts_cuda_graphs_b200.config import CodecDecoderConfig

    d, c = _Draws(seed), CodecDecoderConfig()
    w = {}
    for name, shape, kind in codec_tensor_specs(c):
        if kind in ("lscale", "gamma"):      # residual branches of the transformer and the upsampler: scaled down, as they are from the first training step on
            t = d.n(*shape, std=0.02, mean=0.1, dtype=torch.float32)
        elif kind == "norm":
            t = d.n(*shape, std=0.1, mean=1.0, dtype=torch.float32)
        elif kind == "bias":
            t = d.n(*shape, std=0.02, dtype=torch.float32)
        elif kind == "snake":      # logarithms of the sine's frequency and of what divides it
            t = d.n(*shape, std=0.2, mean=0.7 if name.endswith("beta") else 0.0, dtype=torch.float32)
        else:      # fan-in scaling; residual branches and the last convolution smaller, so that the waveform is a signal inside [-1, 1]
            fan = {"emb": c.num_quantizers, "dw": shape[-1], "tconv": shape[0] * (1 if len(shape) > 2 and shape[2] <= 2 else 2)}.get(kind) or math.prod(shape[1:])
            gain = 0.25 if kind == "conv" and shape[0] == 1 else 0.3 if name.endswith("conv2.conv.weight") else 1.0
            t = d.n(*shape, std=gain / math.sqrt(fan)).to(torch.float32)
        w[name] = t
    return c, w, d.i(case["frames"], c.num_quantizers, below=c.codebook_size)


def _codec_prepare(case, seed):
    from qwen3_tts_cuda_graphs_b200.codec import CodecDecoder

    c, w, codes = _codec_inputs(case, seed)
    return dict(dec=CodecDecoder(c, w, DEV), codes=codes, skip=case["context"] * c.total_upsample)


def _conv(x, w, b, dil=1):
    """x [T, cin], w [cout, cin, k]: causal convolution."""
    k = w.shape[2]
    y = b.expand(x.shape[0], -1).clone()
    for j in range(k):
        back = (k - 1 - j) * dil
        if back < x.shape[0]:
            y[back:] += x[:x.shape[0] - back] @ w[:, :, j].T
    return y


def _tconv(x, w, b, r):
    """Transposed convolution of stride r (kernel r or 2r), trimmed at the end."""
    T, cout = x.shape[0], w.shape[1]
    y = torch.zeros(T + 1, r, cout, device=x.device, dtype=x.dtype)
    for part in range(w.shape[2] // r):
        y[part:part + T] += torch.einsum("tc,cok->tko", x, w[:, :, part * r:(part + 1) * r])
    return (y[:T] + b).reshape(T * r, cout)


def _codec_exact(case, seed):
    c, w, codes = _codec_inputs(case, seed)
    W = {k: v.to(F64) for k, v in w.items()}
    T, D, H = codes.shape[0], c.head_dim, c.num_attention_heads
    books = [W[f"quantizer.codebook.{q}"][codes[:, q]] for q in range(c.num_quantizers)]
    ns = c.num_semantic_quantizers
    x = sum(books[:ns]) @ W["quantizer.rvq_first.output_proj.weight"].squeeze().T + sum(books[ns:]) @ W["quantizer.rvq_rest.output_proj.weight"].squeeze().T
    x = _conv(x, W["pre_conv.conv.weight"], W["pre_conv.conv.bias"])
    a = torch.arange(T, device=DEV, dtype=F64)[:, None] * c.rope_theta ** (-torch.arange(0, D, 2, device=DEV, dtype=F64) / D)
    cos, sin = torch.cat([a, a], -1).cos()[:, None], torch.cat([a, a], -1).sin()[:, None]
    i = torch.arange(T, device=DEV)
    hide = (i[None] > i[:, None]) | (i[None] <= i[:, None] - c.sliding_window)
    for layer in range(c.num_hidden_layers):
        p = f"pre_transformer.layers.{layer}."
        h = _rms(x, c.rms_norm_eps, W[p + "input_layernorm.weight"])
        q, k, v = ((h @ W[p + f"self_attn.{n}_proj.weight"].T).view(T, H, D) for n in "qkv")
        q, k = _half_turn(q, cos, sin), _half_turn(k, cos, sin)
        s = torch.einsum("ihd,jhd->hij", q, k) * D ** -0.5
        o = torch.einsum("hij,jhd->ihd", s.masked_fill(hide, -math.inf).softmax(-1), v).reshape(T, H * D)
        x = x + W[p + "self_attn_layer_scale.scale"] * (o @ W[p + "self_attn.o_proj.weight"].T)
        h = _rms(x, c.rms_norm_eps, W[p + "post_attention_layernorm.weight"])
        x = x + W[p + "mlp_layer_scale.scale"] * ((F.silu(h @ W[p + "mlp.gate_proj.weight"].T) * (h @ W[p + "mlp.up_proj.weight"].T)) @ W[p + "mlp.down_proj.weight"].T)
    x = _rms(x, c.rms_norm_eps, W["pre_transformer.norm.weight"])
    for n, r in enumerate(c.upsampling_ratios):
        p = f"upsample.{n}."
        x = _tconv(x, W[p + "0.conv.weight"], W[p + "0.conv.bias"], r)
        dw = W[p + "1.dwconv.conv.weight"]
        h = W[p + "1.dwconv.conv.bias"] + sum(dw[:, 0, j] * F.pad(x, (0, 0, 6 - j, 0))[:x.shape[0]] for j in range(7))
        h = F.layer_norm(h, (h.shape[-1],), W[p + "1.norm.weight"], W[p + "1.norm.bias"], 1e-6)
        h = F.gelu(h @ W[p + "1.pwconv1.weight"].T + W[p + "1.pwconv1.bias"])
        x = x + W[p + "1.gamma"] * (h @ W[p + "1.pwconv2.weight"].T + W[p + "1.pwconv2.bias"])

    def snake(z, n):
        return z + torch.sin(z * W[n + ".alpha"].exp()) ** 2 / (W[n + ".beta"].exp() + 1e-9)

    x = _conv(x, W["decoder.0.conv.weight"], W["decoder.0.conv.bias"])
    for n, r in enumerate(c.upsample_rates):
        p = f"decoder.{n + 1}.block."
        x = _tconv(snake(x, p + "0"), W[p + "1.conv.weight"], W[p + "1.conv.bias"], r)
        for j, dil in enumerate((1, 3, 9)):
            u = f"{p}{j + 2}."
            h = _conv(snake(x, u + "act1"), W[u + "conv1.conv.weight"], W[u + "conv1.conv.bias"], dil)
            x = x + _conv(snake(h, u + "act2"), W[u + "conv2.conv.weight"], W[u + "conv2.conv.bias"])
    n = len(c.upsample_rates) + 1
    x = _conv(snake(x, f"decoder.{n}"), W[f"decoder.{n + 1}.conv.weight"], W[f"decoder.{n + 1}.conv.bias"]).clamp(-1, 1).reshape(-1)
    return x[case["context"] * c.total_upsample:]


def _codec_macs(c, frames, context):
    """Multiply-adds: everything up to the upsampling for all frames, the vocoder for the wanted ones."""
    H = c.hidden_size
    per = 2 * c.codebook_dim * c.latent_dim + 3 * c.latent_dim * H
    per += c.num_hidden_layers * (4 * H * c.num_attention_heads * c.head_dim + 3 * H * c.intermediate_size)
    rows, voc = 1, 0
    for r in c.upsampling_ratios:
        per += rows * r * H * H
        rows *= r
        per += rows * 8 * H * H
    voc += rows * 7 * H * c.decoder_dim
    ch = c.decoder_dim
    for r in c.upsample_rates:
        voc += rows * 2 * r * ch * (ch // 2)
        rows, ch = rows * r, ch // 2
        voc += rows * 3 * 8 * ch * ch
    return per * frames + voc * (frames - context)


# ------------------------------------------------------------------------------------------------------------------------
# sequence models: layers
# ------------------------------------------------------------------------------------------------------------------------
def _builder(specs, rows, max_pos, f32):
    from qwen3_tts_cuda_graphs_b200.seq_ops import StepBuilder
    from qwen3_tts_cuda_graphs_b200.seq_state import SequenceStateManager

    slot = SequenceStateManager(specs, max_pos, torch.device(DEV), 1).acquire("request")
    return StepBuilder(torch.device(DEV), rows, slot, f32), slot


def _play(s):
    from qwen3_tts_cuda_graphs_b200 import codec

    codec.run_op_plan(codec.load_lib(), s["plan"], True)


def _turn_pairs(x, pos, freq):
    """x [T, heads, d]: the first 2 * len(freq) entries turn in pairs (2i, 2i + 1)."""
    a = pos[:, None].to(F64) * freq
    cos, sin, n = a.cos()[:, None], a.sin()[:, None], 2 * freq.shape[0]
    e, o = x[..., 0:n:2], x[..., 1:n:2]
    return torch.cat([torch.stack([e * cos - o * sin, o * cos + e * sin], -1).flatten(-2), x[..., n:]], -1)


def _attend(q, k, v, first, scale, cap, window, sink):
    """q [M, H, d] at positions first .., k / v [L, G, ..]; causal, windowed, with a sink in the denominator."""
    M, H, _ = q.shape
    L, G, _ = k.shape
    i, j = torch.arange(first, first + M, device=q.device)[:, None], torch.arange(L, device=q.device)[None]
    hide = (j > i) | ((j <= i - window) if window else torch.zeros_like(j > i))
    out = torch.empty(M, H, v.shape[2], device=q.device, dtype=q.dtype)
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        s = torch.cat([s.masked_fill(hide, -math.inf), sink[h].expand(M, 1)], 1) if sink is not None else s.masked_fill(hide, -math.inf)
        out[:, h] = s.softmax(-1)[:, :L] @ v[:, h // (H // G)]
    return out


def _attention_inputs(case, seed):
    from qwen3_tts_cuda_graphs_b200.config import SoftmaxAttentionConfig

    d, H, G, M, W = _Draws(seed), case["heads"], case["kv"], case["rows"], 1024
    dt = torch.float32 if case["f32"] else torch.bfloat16
    c = SoftmaxAttentionConfig(H, G, 128, 128, 128 ** -0.5, case["cap"], 32, 10000.0, window=case["window"], sink=True, gate=case["gate"])
    w = {"wqkv": d.n((H + 2 * G) * 128 + (H if case["gate"] else 0), W, std=W ** -0.5, dtype=dt), "o": d.n(W, H * 128, std=(H * 128) ** -0.5, dtype=dt),
         "freq": (10000.0 ** (-torch.arange(16, device=DEV, dtype=F64) / 16)).to(torch.float32), "sink": d.n(H, std=0.5, dtype=torch.float32)}
    return c, w, d.n(M, W, dtype=dt), d.n(case["before"], G * 128, dtype=dt), d.n(case["before"], G * 128, dtype=dt)


def _attention_prepare(case, seed):
    from qwen3_tts_cuda_graphs_b200.seq_state import StateSpec

    c, w, h, k, v = _attention_inputs(case, seed)
    M, n = case["rows"], case["before"]
    b, slot = _builder([StateSpec("k", "append", k.shape[1], dtype=k.dtype), StateSpec("v", "append", v.shape[1], dtype=v.dtype)], M, n + M, case["f32"])
    slot.cur["k"][:n], slot.cur["v"][:n] = k, v
    slot.pos.fill_(n)
    out = torch.zeros(M, h.shape[1], device=DEV)
    b.softmax_attention(h, c, w, "k", "v", out)
    return dict(plan=b.finish(), out=out, k=slot.cur["k"][n:n + M], v=slot.cur["v"][n:n + M], keep=(b, slot, w, h))


def _attention_exact(case, seed):
    c, w, h, k, v = _attention_inputs(case, seed)
    H, G, M, n = c.heads, c.kv_heads, case["rows"], case["before"]
    p = h.to(F64) @ w["wqkv"].to(F64).T
    pos = torch.arange(n, n + M, device=DEV)
    f = 10000.0 ** (-torch.arange(16, device=DEV, dtype=F64) / 16)
    q, kn = _turn_pairs(p[:, :H * 128].view(M, H, 128), pos, f), _turn_pairs(p[:, H * 128:(H + G) * 128].view(M, G, 128), pos, f)
    vn = p[:, (H + G) * 128:(H + 2 * G) * 128]
    o = _attend(q, torch.cat([k.to(F64).view(n, G, 128), kn]), torch.cat([v.to(F64), vn]).view(n + M, G, 128), n, c.scale, c.softcap, c.window, w["sink"].to(F64))
    if c.gate:
        o = o * torch.sigmoid(p[:, (H + 2 * G) * 128:])[..., None]
    return {"out": o.reshape(M, -1) @ w["o"].to(F64).T, "k": kn.reshape(M, -1), "v": vn}


def _delta_weights(d, W, H, G, dt=torch.bfloat16):
    """A gated-delta-rule layer, heads of 128 x 128, four taps."""
    n = 2 * G * 128 + H * 128
    return {"win": d.n(n + H * 128 + 2 * H, W, std=W ** -0.5, dtype=dt), "conv": d.n(n, 4, std=0.4, dtype=torch.float32), "A_log": torch.log(d.u(H, lo=0.5, hi=4.5)),
            "dt_bias": d.n(H, mean=-1.5, dtype=torch.float32), "norm": d.n(128, std=0.1, mean=1.0, dtype=torch.float32), "o": d.n(W, H * 128, std=(H * 128) ** -0.5, dtype=dt)}


def _delta_layer(h, w, H, G, eps):
    """float64: h [M, W] -> output [M, W], state [H, 128, 128]."""
    M, n = h.shape[0], 2 * G * 128 + H * 128
    raw = h @ w["win"].to(F64).T
    taps = w["conv"].to(F64)
    cv = F.silu(sum(taps[:, j] * F.pad(raw[:, :n], (0, 0, 3 - j, 0))[:M] for j in range(4)))
    unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    rep = lambda z: z.repeat_interleave(H // G, 1)  # noqa: E731
    q, k = rep(unit(cv[:, :G * 128].view(M, G, 128)) * 128 ** -0.5), rep(unit(cv[:, G * 128:2 * G * 128].view(M, G, 128)))
    v = cv[:, 2 * G * 128:].view(M, H, 128)
    decay = torch.exp(-w["A_log"].to(F64).exp() * F.softplus(raw[:, n + H * 128:n + H * 128 + H] + w["dt_bias"].to(F64)))
    beta = torch.sigmoid(raw[:, n + H * 128 + H:])
    S, y = torch.zeros(H, 128, 128, device=h.device, dtype=F64), torch.empty(M, H, 128, device=h.device, dtype=F64)
    for t in range(M):
        S = decay[t, :, None, None] * S
        u = beta[t, :, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        y[t] = torch.einsum("hkv,hk->hv", S, q[t])
    y = (_rms(y, eps, w["norm"].to(F64)) * F.silu(raw[:, n:n + H * 128]).view(M, H, 128)).reshape(M, -1)
    return y @ w["o"].to(F64).T, S


def _delta_inputs(case, seed):
    d = _Draws(seed)
    return _delta_weights(d, case["width"], case["heads"], case["kv"]), d.n(case["rows"], case["width"])


def _delta_prepare(case, seed):
    from qwen3_tts_cuda_graphs_b200.config import DeltaRuleConfig
    from qwen3_tts_cuda_graphs_b200.seq_state import StateSpec

    w, h = _delta_inputs(case, seed)
    H, G = case["heads"], case["kv"]
    b, slot = _builder([StateSpec("dr.conv", "carry", 2 * G * 128 + H * 128, 3), StateSpec("dr.s", "carry", 128, H * 128, in_place=True)], case["rows"], 4096, False)
    out = torch.zeros(case["rows"], case["width"], device=DEV)
    b.delta_rule(h, DeltaRuleConfig(H, G, 128, 128, 4), w, "dr", 1e-5, out)
    b.commit()
    return dict(plan=b.finish(), out=out, slot=slot, keep=(b, w, h))


def _delta_run(s, case):
    s["slot"].reset()      # a new request's state
    _play(s)
    return {"out": s["out"], "state": s["slot"].cur["dr.s"]}


def _moe_inputs(case, seed):
    d, W, E, ff = _Draws(seed), case["width"], case["experts"], case["ff"]
    # an expert's and the shared expert's (gate, up) rows alternate
    w = {"router": d.n(E, W, std=W ** -0.5), "up": d.n(E, 2 * ff, W, std=W ** -0.5), "down": d.n(E, W, ff, std=ff ** -0.5)}
    if case["shared"]:
        w["shared_up"], w["shared_down"] = d.n(2 * case["shared"], W, std=W ** -0.5), d.n(W, case["shared"], std=case["shared"] ** -0.5)
    return w, d.n(case["rows"], W)


def _moe_prepare(case, seed):
    from qwen3_tts_cuda_graphs_b200.config import MoEFFConfig

    w, x = _moe_inputs(case, seed)
    c = MoEFFConfig(case["experts"], 0, case["top"], 1, 1, 1.0, case["ff"], case["shared"], score="sigmoid", renorm=False, weight_input=True, gated=True)
    b, slot = _builder([], case["rows"], 4096, False)
    out, x32 = torch.zeros(case["rows"], case["width"], device=DEV), x.to(torch.float32)
    b.moe_ff(x32, x, c, w, out)
    return dict(plan=b.finish(), out=out, keep=(b, slot, w, x, x32))


def _moe_exact(case, seed):
    w, x = _moe_inputs(case, seed)
    x, W = x.to(F64), {k: v.to(F64) for k, v in w.items()}

    def gated(rows, up, down):
        z = rows @ up.T
        return (F.silu(z[:, 0::2]) * z[:, 1::2]) @ down.T

    score = torch.sigmoid(x @ W["router"].T)
    wt, ids = score.topk(case["top"], -1)
    out = gated(x, W["shared_up"], W["shared_down"]) if case["shared"] else torch.zeros_like(x)
    for e in range(case["experts"]):
        t, j = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            out.index_add_(0, t, gated(x[t] * wt[t, j][:, None], W["up"][e], W["down"][e]))
    return out


# ------------------------------------------------------------------------------------------------------------------------
# sequence models: a whole one
# ------------------------------------------------------------------------------------------------------------------------
_VOCAB, _EPS = 3072, 1e-5


def _request_layers(W):
    """Delta rule, attention, attention on the first one's cache, delta rule; heads of 128."""
    H = W // 64
    att = dict(heads=H, kv_heads=max(1, H // 4), dim=128, vdim=128, scale=128 ** -0.5, softcap=50.0, rot=dict(dims=32, base=10000.0))
    delta = dict(heads=H // 2, kv_heads=H // 4, dim=128, vdim=128, conv=4)
    return [("delta", delta), ("attention", att), ("attention", dict(att, kv_from=1)), ("delta", delta)]


def _request_inputs(case, seed):
    d, W = _Draws(seed), case["width"]
    w = {"embed": d.n(_VOCAB, W), "head": d.n(_VOCAB, W, std=W ** -0.5)}

    def norm(name):
        w[name], w[name + ".b"], w[name + ".alpha"] = d.n(W, std=0.1, mean=1.0), d.n(W, std=0.3), torch.tensor(0.75)

    norm("final.norm")
    for i, (kind, m) in enumerate(_request_layers(W)):
        p, H, G = f"l{i}.", m["heads"], m["kv_heads"]
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            norm(p + n)
        q = p + "mix."
        if kind == "delta":
            L = _delta_weights(d, W, H, G)
            cut = [G * 128, 2 * G * 128, 2 * G * 128 + H * 128, 2 * G * 128 + 2 * H * 128, 2 * G * 128 + 2 * H * 128 + H]
            for n, t in zip(("q", "k", "v", "g", "a", "b"), torch.tensor_split(L["win"], cut)):
                w[q + n] = t
            for n, t in zip(("q.conv", "k.conv", "v.conv"), torch.tensor_split(L["conv"], cut[:2])):
                w[q + n] = t
            w.update({q + n: L[n] for n in ("A_log", "dt_bias", "norm", "o")})
        else:
            for n, rows in [("q", H * 128)] + ([] if "kv_from" in m else [("k", G * 128), ("v", G * 128)]) + [("g", H)]:
                w[q + n] = d.n(rows, W, std=W ** -0.5)
            w[q + "o"], w[q + "sink"] = d.n(W, H * 128, std=(H * 128) ** -0.5), d.n(H, std=0.5)
        w[p + "mlp.up"], w[p + "mlp.down"], w[p + "mlp.act"] = d.n(3 * W, W, std=W ** -0.5), d.n(W, 3 * W, std=(3 * W) ** -0.5), torch.tensor([0.3, -0.2])
        dwa = d.n(i + 2, std=0.1)
        dwa[-1] += 0.8
        w[p + "dwa"] = dwa
    return w, [int(t) for t in d.i(case["prompt"] + case["new"], below=_VOCAB).tolist()]


def _request_prepare(case, seed):
    from qwen3_tts_cuda_graphs_b200.config import sequence_config_from_dict
    from qwen3_tts_cuda_graphs_b200.seq_engine import SequenceEngine, model_class

    w, toks = _request_inputs(case, seed)
    w = {k: v.cpu() for k, v in w.items()}      # a checkpoint's tensors
    cfg = dict(architecture="Redodra", vocab=_VOCAB, width=case["width"], norm=dict(eps=_EPS),
               layers=[dict(type=kind, mixer=m, mlp=dict(kind="dense", ff=3 * case["width"])) for kind, m in _request_layers(case["width"])])
    model = model_class("Redodra")(sequence_config_from_dict(cfg), w.get, torch.device(DEV))
    return dict(eng=SequenceEngine(model, 1024, 1), toks=toks)


def _request_run(s, case):
    eng, toks, n = s["eng"], s["toks"], case["prompt"]
    eng.open("request")
    rows = [eng.step("request", toks[:n], [n - 1]).clone()]
    for t in toks[n:]:
        rows.append(eng.step("request", [t], [0]).clone())
    eng.close("request")
    return torch.cat(rows)


def _request_exact(case, seed):
    w, toks = _request_inputs(case, seed)
    w = {k: v.to(DEV, F64) for k, v in w.items()}
    T, W = len(toks), case["width"]
    pos = torch.arange(T, device=DEV)
    f = 10000.0 ** (-torch.arange(16, device=DEV, dtype=F64) / 16)

    def norm(v, n):
        return torch.tanh(w[n + ".alpha"] * v) * w[n] + w[n + ".b"]

    x = w["embed"][torch.tensor(toks, device=DEV)]
    hist, kv = [x], None
    for i, (kind, m) in enumerate(_request_layers(W)):
        p, H, G = f"l{i}.", m["heads"], m["kv_heads"]
        h, q = norm(x, p + "norm1"), p + "mix."
        if kind == "delta":
            L = {n: w[q + n] for n in ("A_log", "dt_bias", "norm", "o")}
            L["win"] = torch.cat([w[q + n] for n in ("q", "k", "v", "g", "a", "b")])
            L["conv"] = torch.cat([w[q + n] for n in ("q.conv", "k.conv", "v.conv")])
            y, _ = _delta_layer(h, L, H, G, _EPS)
        else:
            qh = _turn_pairs((h @ w[q + "q"].T).view(T, H, 128), pos, f)
            if "kv_from" not in m:
                kv = _turn_pairs((h @ w[q + "k"].T).view(T, G, 128), pos, f), (h @ w[q + "v"].T).view(T, G, 128)
            o = _attend(qh, *kv, 0, m["scale"], m["softcap"], 0, w[q + "sink"]) * torch.sigmoid(h @ w[q + "g"].T)[..., None]
            y = o.reshape(T, -1) @ w[q + "o"].T
        x = x + norm(y, p + "norm1b")
        z = norm(x, p + "norm2") @ w[p + "mlp.up"].T
        ap, aq = F.softplus(w[p + "mlp.act"])
        z = torch.where(z > 0, ap * z * z, (0.5 + aq) * (torch.expm1(z.clamp(max=0)) - z)) + 0.5 * z
        x = x + norm(z @ w[p + "mlp.down"].T, p + "norm2b")
        hist.append(x)
        x = sum(a * b for a, b in zip(w[p + "dwa"], hist))
    return norm(x[case["prompt"] - 1:], "final.norm") @ w["head"].T


# ------------------------------------------------------------------------------------------------------------------------
# the measured interface
# ------------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    s = {"prompt": _prompt_prepare, "codec": _codec_prepare, "frames": _frames_prepare, "attention": _attention_prepare, "delta": _delta_prepare,
         "moe": _moe_prepare, "request": _request_prepare}[case["what"]](case, seed)
    s["case"] = dict(case)
    return s


def run(s):
    case = s["case"]
    what = case["what"]
    if what == "prompt":
        return _prompt_run(s, case)
    if what == "codec":      # a streaming user drops the context's part of the waveform
        return s["dec"].decode(s["codes"], skip_samples=s["skip"])[s["skip"]:]
    if what == "frames":
        return _frames_run(s, case)
    if what == "delta":
        return _delta_run(s, case)
    if what == "request":
        return _request_run(s, case)
    _play(s)
    return {"out": s["out"], "k": s["k"], "v": s["v"]} if what == "attention" else s["out"]


def exact(case, seed):
    if case["what"] == "frames":
        return None      # every code is sampled from what the codes before it led to
    out = {"prompt": _prompt_exact, "codec": _codec_exact, "attention": _attention_exact, "moe": _moe_exact, "request": _request_exact}
    if case["what"] == "delta":
        w, h = _delta_inputs(case, seed)
        y, S = _delta_layer(h.to(F64), w, case["heads"], case["kv"], 1e-5)
        return {"out": y, "state": S.reshape(-1, 128)}
    return out[case["what"]](case, seed)


def work(case):
    """Weights and inputs once, outputs once; products and attention scores, no element-wise arithmetic."""
    what = case["what"]
    if what == "prompt":
        c = _tts_config(case)
        t, T = c.talker, case["rows"]
        par = t.num_hidden_layers * t.layer_params()
        head = t.vocab_size * t.hidden_size
        cache = t.num_hidden_layers * T * 2 * t.kv_dim
        return {"bytes": 2.0 * (par + head + T * t.hidden_size + cache), "flops": 2.0 * par * T + 2.0 * head + t.num_hidden_layers * 2.0 * T * (T + 1) * t.q_dim}
    if what == "codec":
        from qwen3_tts_cuda_graphs_b200.codec import codec_tensor_specs
        from qwen3_tts_cuda_graphs_b200.config import CodecDecoderConfig

        c = CodecDecoderConfig()
        par = sum(math.prod(s) for _, s, kind in codec_tensor_specs(c) if kind != "emb")
        new = case["frames"] - case["context"]
        att = c.num_hidden_layers * c.num_attention_heads * c.head_dim * 4.0 * case["frames"] * min(case["frames"], c.sliding_window)
        return {"bytes": 2.0 * par + 2.0 * case["frames"] * c.num_quantizers * c.codebook_dim + 4.0 * new * c.total_upsample,
                "flops": 2.0 * _codec_macs(c, case["frames"], case["context"]) + att}
    if what == "frames":
        c = _tts_config(case)
        t, p, S, n = c.talker, c.predictor, case["streams"], case["frames"]
        talker = t.num_hidden_layers * t.layer_params() + t.vocab_size * t.hidden_size
        pred, heads = p.num_hidden_layers * p.layer_params(), 15 * p.vocab_size * p.hidden_size
        kv = t.num_hidden_layers * 2 * t.kv_dim * (case["before"] + n / 2.0)
        # per frame: every weight once (all streams share it), the valid part of every stream's cache
        return {"bytes": n * 2.0 * (talker + pred + heads + S * kv), "flops": n * S * 2.0 * (talker + 16 * pred + heads + kv)}
    if what == "attention":
        M, n, H, G, W, e = case["rows"], case["before"], case["heads"], case["kv"], 1024, 4.0 if case["f32"] else 2.0
        N = (H + 2 * G) * 128 + (H if case["gate"] else 0)
        span = sum(min(i + 1, case["window"] or i + 1) for i in range(n, n + M))
        keys = min(n, case["window"]) if case["window"] else n
        return {"bytes": e * (W * (N + H * 128) + M * W + 2 * (keys + M) * G * 128) + 4.0 * M * W, "flops": 2.0 * M * W * (N + H * 128) + 4.0 * 128 * H * span}
    if what == "delta":
        M, W, H, G = case["rows"], case["width"], case["heads"], case["kv"]
        N = 2 * G * 128 + 2 * H * 128 + 2 * H
        return {"bytes": 2.0 * (W * (N + H * 128) + M * W) + 4.0 * M * W + 8.0 * H * 128 * 128, "flops": 2.0 * M * W * (N + H * 128) + 7.0 * M * H * 128 * 128}
    if what == "moe":
        M, W, E, top, ff, sh = (case[k] for k in ("rows", "width", "experts", "top", "ff", "shared"))
        return {"bytes": 2.0 * (min(E, M * top) * 3 * ff * W + 3 * sh * W + E * W + M * W) + 4.0 * M * W, "flops": 2.0 * M * W * (E + top * 3 * ff + 3 * sh)}
    W, P, n = case["width"], case["prompt"], case["new"]
    H = W // 64
    par = 2 * W * (2 * (H // 4) * 128 + 3 * (H // 2) * 128) + W * (4 * H * 128 + 2 * (H // 4) * 128) + 4 * 6 * W * W
    return {"bytes": (n + 1) * 2.0 * (par + _VOCAB * W), "flops": 2.0 * par * (P + n) + 2.0 * _VOCAB * W * (n + 1)}


def tolerance(case):
    """What another order of the sums does: bf16 roundings that fall the other way travel through the layers behind them.  Measured: the prompt
    without split sums and with the other attention kernel 0.017 (28 layers), 0.010 (8), 0.007 (4); the codec without split sums 0.017; the single
    layers round their operands once, and are within 0.003 (true 32-bit: 1.1e-6) of the exact result."""
    return {"prompt": {"rel": 0.03, "max": 0.5}, "codec": {"rel": 0.03, "max": 0.5}, "frames": {"rel": 0.01, "differ": 0.01},
            "attention": {"rel": 1e-5 if case.get("f32") else 6e-3, "max": 1e-4 if case.get("f32") else 5e-2}, "delta": {"rel": 4e-3, "max": 4e-2},
            "moe": {"rel": 4e-3, "max": 4e-2}, "request": {"rel": 0.01, "max": 0.1}}[case["what"]]
