"""Performance cases of the framework: what a user's program has it do, through the public entry points.

Three families, each over the range it is used in:

* ``frames`` / ``prompt`` -- the DualAR decode engine (``RQTransformer``): ``decode_frames`` for a batch of utterances
  against their cached positions, and ``forward_generate`` of a prompt.
* ``codec`` -- the Mimi decoder (``MimiModel``): ``decode`` of whole utterances, or ``decode_step`` frame by frame as the
  streaming loop calls it.
* ``lm`` -- the hybrid language models (``PamasunLM``, ``MaferaxLM``, ``VirusunLM``): ``forward`` of prompts (``steps`` 0)
  or of single decoded tokens against a filled cache (``steps`` > 0).  Prompt cases hold a few layers, one of each kind.

Weights are random (the repository ships none), of the sizes of the repository's own configurations and benchmarks.
Decoded tokens are given, never chosen, so that the logits of two builds can be compared.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from smoltts_b200.config import named_config
from smoltts_b200.lm import MaferaxLM, PamasunLM, VirusunLM
from smoltts_b200.lm_config import MaferaxConfig, PamasunConfig, VirusunConfig
from smoltts_b200.mimi import MimiModel
from smoltts_b200.model import RQTransformer, make_prompt_cache, precompute_freqs_cis
from smoltts_b200.synth import byte_prompt, mimi_state_dict_shapes, prompt_grid, state_dict_shapes

SEMANTIC0 = 320                  # first semantic id of the byte-level tokenizer

# width, heads, key/value heads, head size, feed-forward, vocabulary of the language models
LM_SIZES = {
    "w768": dict(width=768, heads=12, kv_heads=4, dim=64, ff=3072, vocab=2368),
    "w1536": dict(width=1536, heads=12, kv_heads=4, dim=128, ff=4096, vocab=8192),
}


def listed():
    return [
        # one utterance, greedy, in the middle of 1024 frames behind a 200-byte prompt: the latency case of speech synthesis
        dict(name="frames_1", kind="frames", model="smoltts_byte_150m", batch=1, context=724, frames=8),
        # a serving batch whose utterances are at different lengths
        dict(name="frames_64", kind="frames", model="smoltts_byte_150m", batch=64, context=471, frames=3),
        # time to first frame: the 200-byte prompt of one utterance
        dict(name="prompt_212", kind="prompt", model="smoltts_byte_150m", tokens=212),
        # one stream, frame by frame: the streaming loop
        dict(name="codec_stream_1", kind="codec", entry="decode_step", streams=1, frames=8),
        # finished utterances of a batch job through the codec
        dict(name="codec_batch_48", kind="codec", entry="decode", streams=48, frames=4),
        # a long prompt of one request: delta rule, attention, feed-forwards
        dict(name="pamasun_prompt", kind="lm", design="pamasun", size="w768", pattern="da", layers=2, dtype="bfloat16", seqs=1, tokens=2048, steps=0, want="last"),
        # the wide model, every position's logits (scoring a text), odd length
        dict(name="pamasun_score_wide", kind="lm", design="pamasun", size="w1536", pattern="ad", layers=2, dtype="bfloat16", seqs=1, tokens=1801, steps=0, want="all"),
        # prompts of several requests in one step, of unequal lengths; own and lent keys, delta rule, rotary attention beside an mLSTM
        dict(name="virusun_prompts", kind="lm", design="virusun", size="w768", pattern="adbp", layers=4, dtype="bfloat16", seqs=3, tokens=1000, steps=0, want="last"),
        # latent attention, gated linear recurrence, routed experts
        dict(name="maferax_prompt", kind="lm", design="maferax", size="w768", pattern="gl", layers=2, dtype="bfloat16", seqs=1, tokens=1024, steps=0, want="all"),
        # the float32 engine, as the trace replayer runs it
        dict(name="pamasun_f32", kind="lm", design="pamasun", size="w768", pattern="da", layers=2, dtype="float32", seqs=1, tokens=300, steps=0, want="last"),
        # a single chat: one token at a time behind a long context, the whole depth of the model
        dict(name="pamasun_decode_1", kind="lm", design="pamasun", size="w768", pattern="daa", layers=10, dtype="bfloat16", seqs=1, tokens=2048, steps=4, want="last"),
        # a few users of the wide model at different lengths
        dict(name="virusun_decode_5", kind="lm", design="virusun", size="w1536", pattern="adbp", layers=4, dtype="bfloat16", seqs=5, tokens=700, steps=4, want="last"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frames", "prompt", "codec", "lm", "lm", "lm"])
    if kind == "frames":
        return dict(kind=kind, model=rng.choice(["smoltts_byte_150m", "smoltts_byte_70m"]), batch=_log_int(rng, 1, 64),
                    context=_log_int(rng, 30, 900), frames=rng.randint(1, 3))
    if kind == "prompt":
        return dict(kind=kind, model=rng.choice(["smoltts_byte_150m", "smoltts_byte_70m"]), tokens=_log_int(rng, 16, 800))
    if kind == "codec":
        return dict(kind=kind, entry=rng.choice(["decode", "decode_step"]), streams=_log_int(rng, 1, 48), frames=rng.randint(1, 4))
    design, decode = rng.choice(["pamasun", "virusun", "maferax"]), rng.random() < 0.4
    pattern = {"pamasun": ["d", "a", "da"], "virusun": ["a", "d", "p", "adbp"], "maferax": ["g", "l", "gl"]}[design]
    pattern = rng.choice(pattern)
    seqs = rng.choice([1, 1, 2, 4, 7])
    return dict(kind=kind, design=design, size=rng.choice(["w768", "w768", "w1536"]), pattern=pattern, layers=len(pattern),
                dtype="float32" if not decode and rng.random() < 0.15 else "bfloat16", seqs=seqs,
                tokens=_log_int(rng, 9, 1200 // seqs), steps=rng.randint(1, 4) if decode else 0, want=rng.choice(["last", "all"]) if not decode else "last")


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(shape, g, scale):
    return torch.randn(*shape, generator=g, device="cuda") * scale


# ---------------------------------------------------------------------------------------------- DualAR decode engine

def _dualar_weights(cfg, seed):
    g = _gen(seed)
    return {k: (1.0 + _randn(s, g, 0.05) if k.endswith("norm.weight") else _randn(s, g, cfg.initializer_range)).to(torch.bfloat16) for k, s in state_dict_shapes(cfg).items()}


def _contexts(case):
    """Cached positions of every sequence: unequal lengths, the first one the longest."""
    return [max(1, case["context"] - (37 * b) % max(1, case["context"] // 2)) for b in range(case["batch"])]


def _frame_inputs(case, cfg, seed):
    """Pending column, the columns that follow, and the keys and values cached so far [batch, longest, layer, 2, heads, 64]."""
    g = _gen(seed + 1)
    codes = torch.randint(0, cfg.codebook_size, (2, case["batch"], cfg.n_rows), generator=g, device="cuda", dtype=torch.int32)
    codes[:, :, 0] = SEMANTIC0 + codes[:, :, 1]
    kv = torch.randn(case["batch"], max(_contexts(case)), cfg.n_layer, 2, cfg.n_local_heads, 64, generator=g, device="cuda", dtype=torch.bfloat16)
    return codes[0].contiguous(), codes[1].contiguous(), kv


def _prepare_frames(case, seed):
    cfg, lens = named_config(case["model"]), _contexts(case)
    B, L, n = case["batch"], max(lens), case["frames"]
    model = RQTransformer(cfg, max_batch=B, max_seq_len=L + n + 1)
    model.load_state_dict(_dualar_weights(cfg, seed))
    batch = model.new_batch(B, max_positions=L + n + 1, max_frames=n)
    first, force, kv = _frame_inputs(case, cfg, seed)
    pages, ps = batch.block_table.long(), model.page_size
    kv = F.pad(kv, (0, 0, 0, 0, 0, 0, 0, 0, 0, pages.shape[1] * ps - L)).view(B, -1, ps, cfg.n_layer, 2, cfg.n_local_heads, 64)
    model.kv_view()[pages] = kv.permute(0, 1, 3, 4, 5, 2, 6)
    model.set_force(force)
    return dict(kind="frames", model=model, batch=batch, first=first, lens=torch.tensor(lens, dtype=torch.int32, device="cuda"), host=lens, frames=n,
                settings=model.sampling(ignore_stop=True))


def _run_frames(s):
    model, batch = s["model"], s["batch"]
    batch.tokens.copy_(s["first"])
    batch.seq_len.copy_(s["lens"])
    batch.step.zero_()
    batch.host_len = list(s["host"])
    model.decode_frames(batch, s["settings"], s["frames"])
    return {"token_logits": model.debug_buffer("token_logits", batch.batch), "depth_logits": model.debug_buffer("depth_logits", batch.batch)}


def _prepare_prompt(case, seed):
    cfg = named_config(case["model"])
    model = RQTransformer(cfg, max_batch=1, max_seq_len=case["tokens"] + 1)
    model.load_state_dict(_dualar_weights(cfg, seed))
    return dict(kind="prompt", model=model, prompt=_prompt_ids(case, cfg, seed))


def _prompt_ids(case, cfg, seed):
    row = byte_prompt(max(1, case["tokens"] - 12), seed=seed)[-case["tokens"]:]
    return prompt_grid(row, cfg)[None].to(device="cuda", dtype=torch.int32)


def _run_prompt(s):
    cache = make_prompt_cache(s["model"])
    logits, hidden = s["model"].forward_generate(s["prompt"], cache)
    cache.batch.release()
    return {"logits": logits, "hidden": hidden}


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn_pairs(x, table):
    """x [..., n, heads, 64]; table [n, 32, 2] (or with the batch in front)."""
    c, s = table[..., None, :, 0], table[..., None, :, 1]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)


def _dualar_block(x, w, p, cfg, heads, kv_heads, table, past=None, mask=None):
    """x [B, n, D]; past: (keys, values) [B, m, kv_heads, 64] in front; mask [.., n, m + n] of the visible positions."""
    B, n, D = x.shape
    q, k, v = (_rms(x, w[p + "attention_norm.weight"], cfg.norm_eps) @ w[p + "attention.wqkv.weight"].T).split([heads * 64, kv_heads * 64, kv_heads * 64], -1)
    q, k, v = _turn_pairs(q.view(B, n, heads, 64), table), _turn_pairs(k.view(B, n, kv_heads, 64), table), v.view(B, n, kv_heads, 64)
    if past is not None:
        k, v = torch.cat([past[0], k], 1), torch.cat([past[1], v], 1)
    q = q.view(B, n, kv_heads, heads // kv_heads, 64)
    s = torch.einsum("bngrd,bmgd->bgrnm", q, k) / 8.0
    if mask is not None:
        s = s.masked_fill(~mask, float("-inf"))
    y = torch.einsum("bgrnm,bmgd->bngrd", torch.softmax(s, -1), v).reshape(B, n, heads * 64)
    x = x + y @ w[p + "attention.wo.weight"].T
    h = _rms(x, w[p + "ffn_norm.weight"], cfg.norm_eps)
    return x + (F.silu(h @ w[p + "feed_forward.w1.weight"].T) * (h @ w[p + "feed_forward.w3.weight"].T)) @ w[p + "feed_forward.w2.weight"].T, (k, v)


def _dualar_embed(cols, w, cfg):
    """cols [B, rows] -> [B, D]."""
    at = torch.arange(cfg.num_codebooks, device="cuda") * cfg.codebook_size
    vq = w["codebook_embeddings.weight"][cols[:, 1:].long() + at].sum(1)
    return w["embeddings.weight"][cols[:, 0].long()] + vq * (cols[:, 1:2] != 0)


def _exact_frames(case, seed):
    cfg, lens = named_config(case["model"]), _contexts(case)
    w = {k: v.double() for k, v in _dualar_weights(cfg, seed).items()}
    col, force, kv = _frame_inputs(case, cfg, seed)
    B, L, n = case["batch"], max(lens), case["frames"]
    rope = precompute_freqs_cis(L + n + 1, 64, cfg.rope_base).cuda().double()
    lens = torch.tensor(lens, device="cuda")
    kv = F.pad(kv.double(), (0, 0, 0, 0, 0, 0, 0, 0, 0, n))            # the frames' own positions follow a sequence's last one
    m = torch.arange(L + n, device="cuda")
    for f in range(n):
        x, here = _dualar_embed(col, w, cfg)[:, None], lens + f
        table = rope[here][:, None]
        seen = torch.cat([m[None] < here[:, None], torch.ones(B, 1, dtype=torch.bool, device="cuda")], 1)[:, None, None, None]
        for i in range(cfg.n_layer):
            x, (k, v) = _dualar_block(x, w, f"layers.{i}.", cfg, cfg.n_head, cfg.n_local_heads, table, (kv[:, :, i, 0], kv[:, :, i, 1]), seen)
            kv[torch.arange(B), here, i, 0], kv[torch.arange(B), here, i, 1] = k[:, -1], v[:, -1]
        col = force
    logits = _rms(x[:, 0], w["norm.weight"], cfg.norm_eps) @ w["embeddings.weight"].T
    x, fast, depth, C = x, precompute_freqs_cis(cfg.max_fast_seqlen, 64, cfg.rope_base).cuda().double(), [], cfg.codebook_size
    past = [None] * cfg.n_fast_layer
    for i in range(cfg.max_fast_seqlen):
        for j in range(cfg.n_fast_layer):
            x, past[j] = _dualar_block(x, w, f"fast_layers.{j}.", cfg, cfg.fast_n_head, cfg.fast_n_local_heads, fast[i:i + 1], past[j])
        depth.append(_rms(x[:, 0], w["fast_norm.weight"], cfg.norm_eps) @ w["fast_output.weight"][i * C:(i + 1) * C].T)
        if i + 1 < cfg.max_fast_seqlen:
            x = w["fast_embeddings.weight"][force[:, 1 + i].long() + i * C][:, None]
    return {"token_logits": logits, "depth_logits": torch.stack(depth, 1)}


def _exact_prompt(case, seed):
    cfg = named_config(case["model"])
    w = {k: v.double() for k, v in _dualar_weights(cfg, seed).items()}
    ids = _prompt_ids(case, cfg, seed)[0].T
    n = ids.shape[0]
    table = precompute_freqs_cis(n, 64, cfg.rope_base).cuda().double()
    x, mask = _dualar_embed(ids, w, cfg)[None], torch.ones(n, n, dtype=torch.bool, device="cuda").tril()
    for i in range(cfg.n_layer):
        x, _ = _dualar_block(x, w, f"layers.{i}.", cfg, cfg.n_head, cfg.n_local_heads, table, None, mask)
    x = x[:, -1]
    return {"logits": _rms(x, w["norm.weight"], cfg.norm_eps) @ w["embeddings.weight"].T, "hidden": x}


# ---------------------------------------------------------------------------------------------- Mimi decoder

def _codec_weights(seed):
    g, out = _gen(seed), {}
    for name, s in mimi_state_dict_shapes().items():
        if name.endswith("cluster_usage"):
            out[name] = 0.5 + 1.5 * torch.rand(*s, generator=g, device="cuda")
        elif name.endswith("layer_scale.scale"):
            out[name] = 0.1 + 0.2 * torch.rand(*s, generator=g, device="cuda")
        elif name.endswith("layernorm.weight"):
            out[name] = 1.0 + _randn(s, g, 0.1)
        elif name.endswith(".bias"):
            out[name] = _randn(s, g, 0.05)
        elif name.endswith("embed_sum"):
            out[name] = _randn(s, g, 1.0)
        elif name == "upsample.conv.weight":
            out[name] = _randn(s, g, 0.7)
        else:
            turned = name.startswith("decoder.") and len(s) == 3 and s[2] >= 8       # transposed convolution: [in, out, 2 stride]
            out[name] = _randn(s, g, 1.4 / (s[0] * 2 if turned else math.prod(s[1:])) ** 0.5)
    return out


def _codec_codes(case, seed):
    return torch.randint(0, 2048, (case["streams"], 8, case["frames"]), generator=_gen(seed + 1), device="cuda", dtype=torch.int32)


def _prepare_codec(case, seed):
    model = MimiModel(max_streams=case["streams"], max_frames=256)
    model.load_state_dict(_codec_weights(seed))
    return dict(kind="codec", entry=case["entry"], model=model, codes=_codec_codes(case, seed))


def _run_codec(s):
    model, codes = s["model"], s["codes"]
    if s["entry"] == "decode":
        return model.decode(codes)
    caches = [model.make_cache() for _ in range(codes.shape[0])]
    out = [model.decode_step(codes[:, :, t:t + 1], caches).clone() for t in range(codes.shape[2])]
    for c in caches:
        model.release_cache(c)
    return out


def _exact_codec(case, seed):
    w, codes = {k: v.double() for k, v in _codec_weights(seed).items()}, _codec_codes(case, seed).long()
    B, T = codes.shape[0], codes.shape[2]
    x = 0
    for half, cs in (("semantic", codes[:, :1]), ("acoustic", codes[:, 1:])):
        p = f"quantizer.{half}_residual_vector_quantizer."
        e = sum((w[f"{p}layers.{i}.codebook.embed_sum"] / w[f"{p}layers.{i}.codebook.cluster_usage"].clamp(min=1e-5)[:, None])[cs[:, i]] for i in range(cs.shape[1]))
        x = x + e @ w[p + "output_proj.weight"][:, :, 0].T
    x = (x[:, :, None] * w["upsample.conv.weight"][:, 0, :2].T).reshape(B, 2 * T, -1)          # every frame upsampled alone
    n = 2 * T
    half = torch.arange(32, device="cuda", dtype=torch.float64)
    ang = torch.arange(n, device="cuda", dtype=torch.float64)[:, None] * 10000.0 ** (-half / 32)
    cos, sin = ang.cos(), ang.sin()
    turn = lambda z: torch.cat([z[..., :32] * cos - z[..., 32:] * sin, z[..., 32:] * cos + z[..., :32] * sin], -1)  # noqa: E731
    mask = torch.ones(n, n, dtype=torch.bool, device="cuda").tril()
    for i in range(8):
        p = f"decoder_transformer.layers.{i}."
        h = F.layer_norm(x, (512,), w[p + "input_layernorm.weight"], w[p + "input_layernorm.bias"], 1e-5)
        q, k, v = ((h @ w[f"{p}self_attn.{m}_proj.weight"].T).view(B, n, 8, 64).transpose(1, 2) for m in "qkv")
        a = torch.softmax((turn(q) @ turn(k).transpose(-1, -2) / 8.0).masked_fill(~mask, float("-inf")), -1) @ v
        x = x + a.transpose(1, 2).reshape(B, n, 512) @ w[p + "self_attn.o_proj.weight"].T * w[p + "self_attn_layer_scale.scale"]
        h = F.layer_norm(x, (512,), w[p + "post_attention_layernorm.weight"], w[p + "post_attention_layernorm.bias"], 1e-5)
        x = x + F.gelu(h @ w[p + "mlp.fc1.weight"].T) @ w[p + "mlp.fc2.weight"].T * w[p + "mlp_layer_scale.scale"]
    x = x.transpose(1, 2)

    def conv(key, z):
        k = w[key + ".conv.weight"]
        return F.conv1d(F.pad(z, (k.shape[2] - 1, 0)), k, w[key + ".conv.bias"])

    x, at = conv("decoder.layers.0", x), 1
    for r in (8, 6, 5, 4):
        key = f"decoder.layers.{at + 1}.conv."
        x = F.conv_transpose1d(F.elu(x), w[key + "weight"], w[key + "bias"], stride=r)[..., :-r]
        x = x + conv(f"decoder.layers.{at + 2}.block.3", F.elu(conv(f"decoder.layers.{at + 2}.block.1", F.elu(x))))
        at += 3
    x = conv(f"decoder.layers.{at + 1}", F.elu(x))
    return x if case["entry"] == "decode" else [x[..., t * 1920:(t + 1) * 1920] for t in range(T)]


# ---------------------------------------------------------------------------------------------- hybrid language models

def _lm_config(case):
    z = LM_SIZES[case["size"]]
    D, H, G, d, ff = z["width"], z["heads"], z["kv_heads"], z["dim"], z["ff"]
    kinds, layers, last = [case["pattern"][i % len(case["pattern"])] for i in range(case["layers"])], [], 0
    for i, kind in enumerate(kinds):
        mlp = {"kind": "dense", "ff": ff}
        if case["design"] == "pamasun":
            mlp = {"kind": "dense", "ff": ff * 3 // 2}                 # two matrices instead of three
            layers.append({"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5}, "mlp": mlp} if kind == "a"
                          else {"type": "general_delta", "mixer": {"heads": H, "dim": d}, "mlp": mlp})
        elif case["design"] == "maferax":
            if kind == "l":
                mlp = {"kind": "moe", "expert": {"ff": 1024}, "router": {"experts": 16, "identity": 2, "top": 3, "groups": {"count": 3, "keep": 2}, "scale": 2.0}}
                layers.append({"type": "latent_attention", "mlp": mlp,
                               "mixer": {"heads": H, "dim": d, "rot_dim": d // 2, "vdim": d, "q_rank": D // 2, "kv_rank": 128, "scale": (1.5 * d) ** -0.5,
                                         "rot": {"base": 10000.0, "dims": d // 2}}})
            else:
                layers.append({"type": "gla", "mixer": {"heads": H, "dim": d, "vdim": d, "tau": 16.0}, "mlp": mlp})
        elif kind in "ab":
            c, h = (d, H // 2) if d <= 64 else (d // 2, H)
            m = {"heads": h, "kv_heads": G * h // H, "dim": c, "vdim": 2 * c, "scale": c ** -0.5, "diff": 0.5}
            if kind == "b":
                m["kv_from"] = last
            else:
                last = i
            layers.append({"type": "attention", "mixer": m, "mlp": mlp})
        elif kind == "d":
            layers.append({"type": "delta", "mixer": {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "conv": 4}, "mlp": mlp})
        else:
            layers.append({"type": "parallel", "mlp": mlp,
                           "mixer": {"left": {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5,
                                              "rot": {"base": 10000.0, "dims": d, "scaling": {"factor": 4.0, "original": 1024, "fast": 32.0, "slow": 1.0}}},
                                     "right": {"heads": H, "dim": d, "vdim": d, "gate_cap": 15.0}, "left_scale": 1.0, "right_scale": 1.0}})
    out = {"architecture": case["design"].capitalize(), "vocab": z["vocab"], "width": D, "norm": {"eps": 1e-6}, "layers": layers}
    if case["design"] == "pamasun":
        out.update(embedding={"scale": D ** 0.5}, loop={"start": 0, "stop": 0, "times": 1})
    if case["design"] == "maferax":
        out.update(postln_alpha=2.0, logit_scale=1.0)
    return out


CONFIGS = {"pamasun": PamasunConfig, "maferax": MaferaxConfig, "virusun": VirusunConfig}
ENGINES = {"pamasun": PamasunLM, "maferax": MaferaxLM, "virusun": VirusunLM}
RANKS = {"pamasun": 64, "maferax": 16}          # inner size of the low-rank decay projection


def _lm_shapes(case, raw):
    cfg = CONFIGS[case["design"]].from_dict(raw)
    return cfg.tensor_shapes({i: RANKS[case["design"]] for i in range(case["layers"])}) if case["design"] in RANKS else cfg.tensor_shapes()


def _lm_weights(case, seed):
    raw, g, out = _lm_config(case), _gen(seed), {}
    for k, s in _lm_shapes(case, raw).items():
        last = k.rsplit(".", 1)[-1]
        if k == "embed":
            t = _randn(s, g, s[1] ** -0.5 if case["design"] == "pamasun" else 1.0)
        elif last == "conv":
            t = _randn(s, g, 0.5)
        elif len(s) == 2:
            t = _randn(s, g, s[1] ** -0.5 * (4.0 if last == "router" else 1.0))
        elif len(s) == 0:
            t = 1.0 + 0.2 * torch.rand((), generator=g, device="cuda")
        elif last == "dwa":
            t = torch.cat([torch.rand(s[0] - 1, generator=g, device="cuda") * 0.3, torch.ones(1, device="cuda")])
        elif last in ("ls1", "ls2"):
            t = 0.6 + _randn(s, g, 0.1)
        elif last in ("r1", "r2"):
            t = 0.1 + 0.8 * torch.rand(*s, generator=g, device="cuda")
        elif last == "act":
            t = torch.tensor([0.6, 0.3, 0.1, 0.05], device="cuda") + _randn(s, g, 0.02)
        elif k.endswith((".q.norm", ".k.norm", "mix.norm", "right.norm", "dq.norm", "dkv.norm")) or (case["design"] == "virusun" and k == "final.norm"):
            t = 1.0 + _randn(s, g, 0.1)
        elif case["design"] == "virusun" and last in ("norm1", "norm2"):
            t = 0.6 + _randn(s, g, 0.1)
        elif last in ("A_log", "dt_bias"):
            t = -1.0 + _randn(s, g, 0.5)
        elif k.endswith(("f.b", "a2.b")):
            t = 3.0 + _randn(s, g, 0.5)
        else:
            t = _randn(s, g, 0.1)
        out[k] = t.to(torch.bfloat16)
    return raw, out


def _lengths(case):
    """Tokens of every sequence: unequal, the first the longest."""
    return [max(1, case["tokens"] - (case["tokens"] * b) // (2 * case["seqs"]) - b) for b in range(case["seqs"])]


def _lm_tokens(case, seed):
    g = torch.Generator().manual_seed(int(seed) + 1)
    return [torch.randint(0, LM_SIZES[case["size"]]["vocab"], (n + case["steps"],), generator=g).tolist() for n in _lengths(case)]


def _prepare_lm(case, seed):
    raw, w = _lm_weights(case, seed)
    lens, room = _lengths(case), max(256, sum(_lengths(case)))
    model = ENGINES[case["design"]](CONFIGS[case["design"]].from_dict(raw), dtype=getattr(torch, case["dtype"]),
                                    max_tokens=sum(-(-(n + case["steps"]) // 64) * 64 for n in lens), max_seqs=case["seqs"], page_size=64, max_step_tokens=room,
                                    max_want=sum(lens) if case["want"] == "all" else case["seqs"])
    model.load_state_dict({k: v.cpu() for k, v in w.items()})           # as a checkpoint file is read
    toks, s = _lm_tokens(case, seed), dict(kind="lm", model=model, lens=lens, steps=case["steps"])
    if case["steps"]:
        s["seqs"] = [model.open_sequence() for _ in lens]
        model.forward([(q, t[:n], []) for q, t, n in zip(s["seqs"], toks, lens)])
        s["next"] = [[t[n + i:n + i + 1] for t, n in zip(toks, lens)] for i in range(case["steps"])]
    else:
        s["toks"], s["want"] = toks, [list(range(n)) if case["want"] == "all" else [n - 1] for n in lens]
    return s


def _run_lm(s):
    model = s["model"]
    if s["steps"]:
        out = []
        for q, n in zip(s["seqs"], s["lens"]):
            q.length = n                                              # a pass decodes behind the same cached positions
        for step in s["next"]:
            out.append(model.forward([(q, t, [0]) for q, t in zip(s["seqs"], step)]).clone())
        return torch.stack(out)
    seqs = [model.open_sequence() for _ in s["toks"]]
    logits = model.forward(list(zip(seqs, s["toks"], s["want"])))
    for q in seqs:
        model.close_sequence(q)
    return logits


def _divide(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, bias=None, sink=None):
    """q [n, H, d] (scaled), k [n, G, d], v [n, G, dv], causal; bias(distance [n, n], head); sink [H]."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    at = torch.arange(n, device="cuda", dtype=torch.float64)
    dist, out = at[:, None] - at[None], []
    for h in range(H):
        s = q[:, h] @ k[:, h // (H // G)].T
        if bias is not None:
            s = s - bias(dist.clamp(min=0), h)
        s = s.masked_fill(dist < 0, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :n] @ v[:, h // (H // G)])
    return torch.stack(out, 1)


def _turn(x, freqs, mult, halves):
    """x [n, heads, dims]: pairs (2i, 2i + 1), or (i, i + dims / 2) with ``halves``."""
    ang = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None, None] * torch.tensor(freqs, device="cuda", dtype=torch.float64)
    c, s = ang.cos() * mult, ang.sin() * mult
    a, b = x.chunk(2, -1) if halves else (x[..., 0::2], x[..., 1::2])
    u, v = a * c - b * s, b * c + a * s
    return torch.cat([u, v], -1) if halves else torch.stack([u, v], -1).flatten(-2)


def _pamasun_mixer(x, w, m, kind, eps):
    n, H, d = x.shape[0], m["heads"], m["dim"]
    if kind == "attention":
        q, k = (_divide((x @ w[c].T).view(n, -1, d), eps) * w[c + ".norm"] for c in "qk")
        y = _attend(q * m["scale"], k, (x @ w["v"].T).view(n, -1, m["vdim"]), lambda dist, h: w["r1"][h] * torch.log1p(w["r2"][h] * dist), w["sink"])
        return (y.reshape(n, -1) * torch.sigmoid(x @ w["g"].T)) @ w["o"].T
    r, k, v = ((x @ w[c].T).view(n, H, d) for c in "rkv")
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(x @ w["w1"].T) @ w["w2"].T + w["w0"])).view(n, H, d)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au = torch.sigmoid(x @ w["a"].T + w["a.b"]).view(n, H, d) * u
    S, out = torch.zeros(H, d, d, device="cuda", dtype=torch.float64), []
    left, right = torch.stack([-au, k], -1), torch.stack([torch.zeros_like(v), v], 2)            # S <- decay S - au (u S) + k v
    for t in range(n):
        right[t, :, 0] = (u[t][:, None] @ S)[:, 0]
        S = torch.baddbmm(decay[t][:, :, None] * S, left[t], right[t])
        out.append((r[t][:, None] @ S)[:, 0])
    y = _divide(torch.stack(out), eps).reshape(n, -1) * w["norm"]
    return (y * torch.sigmoid(x @ w["g"].T)) @ w["o"].T


def _maferax_mixer(x, w, m, kind, eps):
    n, H, d, dv = x.shape[0], m["heads"], m["dim"], m["vdim"]
    if kind == "latent_attention":
        r, rank = m["rot_dim"], m["kv_rank"]
        freqs = [m["rot"]["base"] ** (-2.0 * i / m["rot"]["dims"]) for i in range(m["rot"]["dims"] // 2)]
        q = (_divide(x @ w["dq"].T, eps) * w["dq.norm"] @ w["uq"].T).view(n, H, d + r)
        kv = x @ w["dkv"].T
        c, kr = _divide(kv[:, :rank], eps) * w["dkv.norm"], _turn(kv[:, None, rank:], freqs, 1.0, False)
        q = torch.cat([q[..., :d], _turn(q[..., d:], freqs, 1.0, False)], -1) * m["scale"]
        k = torch.cat([(c @ w["uk"].T).view(n, H, d), kr.expand(n, H, r)], -1)
        y = _attend(q, k, (c @ w["uv"].T).view(n, H, dv)) * torch.sigmoid(x @ w["g"].T)[:, :, None]
        return y.reshape(n, -1) @ w["o"].T
    q, k, v = ((x @ w[c].T).view(n, H, -1) for c in "qkv")
    decay = torch.exp(F.logsigmoid((x @ w["a1"].T) @ w["a2"].T + w["a2.b"]) / m["tau"]).view(n, H, d)
    S, out = torch.zeros(H, d, dv, device="cuda", dtype=torch.float64), []
    for t in range(n):
        S = torch.baddbmm(decay[t][:, :, None] * S, k[t][:, :, None], v[t][:, None])
        out.append((q[t][:, None] @ S)[:, 0])
    y = _divide(torch.stack(out) * d ** -0.5, eps) * w["norm"]
    return (y.reshape(n, -1) * F.silu(x @ w["g"].T)) @ w["o"].T


def _maferax_feed(x, w, mlp):
    if mlp["kind"] == "dense":
        return (F.gelu(x @ w["gate"].T, approximate="tanh") * (x @ w["up"].T)) @ w["down"].T
    r = mlp["router"]
    E, size = r["experts"] + r["identity"], (r["experts"] + r["identity"]) // r["groups"]["count"]
    s = torch.softmax(x @ w["router"].T, -1)
    pick = s + w["correction"]
    kept = pick.view(-1, r["groups"]["count"], size).amax(-1).topk(r["groups"]["keep"], -1).indices
    allowed = torch.zeros(x.shape[0], r["groups"]["count"], dtype=torch.bool, device="cuda").scatter_(1, kept, True).repeat_interleave(size, 1)
    ids = pick.masked_fill(~allowed, float("-inf")).topk(r["top"], -1).indices
    chosen = s.gather(1, ids)
    weight = torch.zeros_like(s).scatter_(1, ids, chosen / chosen.sum(-1, keepdim=True) * r["scale"])
    out = weight[:, r["experts"]:].sum(-1, keepdim=True) * x
    for e in range(r["experts"]):
        out = out + weight[:, e:e + 1] * ((F.silu(x @ w[f"e{e}.gate"].T) * (x @ w[f"e{e}.up"].T)) @ w[f"e{e}.down"].T)
    return out


def _virusun_mixer(x, w, m, kind, eps, lent):
    """(result, keys and values of an attention layer)."""
    n = x.shape[0]
    if kind == "attention":
        d = m["dim"]
        q = _divide((x @ w["q"].T + w["q.b"]).view(n, -1, 2, d), eps) * w["q.norm"] * m["scale"]
        k, v = lent if lent is not None else (_divide((x @ w["k"].T + w["k.b"]).view(n, -1, 2, d), eps) * w["k.norm"], (x @ w["v"].T + w["v.b"]).view(n, -1, m["vdim"]))
        lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + m["diff"]
        y = _attend(q[:, :, 0], k[:, :, 0], v) - lam * _attend(q[:, :, 1], k[:, :, 1], v)
        y = (_divide(y, eps) * (1.0 - m["diff"])).reshape(n, -1) * torch.sigmoid(x @ w["g"].T)
        return y @ w["o"].T + w["o.b"], (k, v)
    if kind == "delta":
        H, G, d, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
        q, k, v = (F.silu(F.conv1d(F.pad((x @ w[c].T).T[None], (taps - 1, 0)), w[c + ".conv"][:, None], groups=w[c].shape[0])[0].T) for c in "qkv")
        unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k = (unit(z.view(n, G, d)).repeat_interleave(H // G, 1) for z in (q, k))
        v, beta = v.view(n, H, dv), torch.sigmoid(x @ w["b"].T)
        keep = torch.exp(-torch.exp(w["A_log"]) * F.softplus(x @ w["a"].T + w["dt_bias"]))
        S, out = torch.zeros(H, d, dv, device="cuda", dtype=torch.float64), []
        for t in range(n):
            S = keep[t][:, None, None] * S
            S = torch.baddbmm(S, k[t][:, :, None], beta[t][:, None, None] * (v[t][:, None] - k[t][:, None] @ S))
            out.append((q[t][:, None] @ S)[:, 0])
        y = _divide(torch.stack(out) * d ** -0.5, eps) * w["norm"]
        return (y.reshape(n, -1) * F.silu(x @ w["g"].T)) @ w["o"].T, None
    a, r = m["left"], m["right"]
    rot, sc = a["rot"], a["rot"]["scaling"]
    at = lambda t: rot["dims"] * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(rot["base"]))  # noqa: E731
    lo, hi, freqs = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), rot["dims"] - 1), []
    for i in range(rot["dims"] // 2):
        f, ramp = rot["base"] ** (-2.0 * i / rot["dims"]), min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        freqs.append(f / sc["factor"] * ramp + f * (1.0 - ramp))
    q, k = ((_divide(x @ w[f"left.{c}"].T + w[f"left.{c}.b"], eps) * w[f"left.{c}.norm"]).view(n, -1, a["dim"]) for c in "qk")
    mult = 0.1 * math.log(sc["factor"]) + 1.0
    y = _attend(_turn(q, freqs, mult, True) * a["scale"], _turn(k, freqs, mult, True), (x @ w["left.v"].T + w["left.v.b"]).view(n, -1, a["vdim"]))
    left = y.reshape(n, -1) @ w["left.o"].T + w["left.o.b"]
    H, d, cap = r["heads"], r["dim"], r["gate_cap"]
    q, k, v = ((x @ w["right." + c].T).view(n, H, -1) for c in "qkv")
    i_log, f_log = (cap * torch.tanh((x @ w[f"right.{c}"].T + w[f"right.{c}.b"]) / cap) for c in "if")
    f_log, top = F.logsigmoid(f_log), torch.zeros(H, device="cuda", dtype=torch.float64)
    S, out = torch.zeros(H, d, r["vdim"] + 1, device="cuda", dtype=torch.float64), []
    v = torch.cat([v, torch.ones_like(v[..., :1])], -1)                   # a last column of ones: the key sum
    for t in range(n):
        new = torch.maximum(f_log[t] + top, i_log[t])
        S = torch.baddbmm(torch.exp(f_log[t] + top - new)[:, None, None] * S, (torch.exp(i_log[t] - new)[:, None] * k[t])[:, :, None], v[t][:, None])
        top, o = new, (q[t][:, None] @ S)[:, 0] * d ** -0.5
        out.append(o[:, :-1] / (torch.maximum(o[:, -1:].abs(), torch.exp(-top)[:, None]) + 1e-6))
    y = _divide(torch.stack(out), eps).reshape(n, -1) * w["right.norm"] * torch.sigmoid(x @ w["right.g"].T)
    return m["left_scale"] * left + m["right_scale"] * (y @ w["right.o"].T), None


def _exact_lm_sequence(case, raw, w, toks):
    eps, design, lent, results = raw["norm"]["eps"], case["design"], [], []
    x = w["embed"][torch.tensor(toks, device="cuda")]
    if design == "pamasun":
        x = x * raw["embedding"]["scale"]
    if design == "maferax":
        x = _divide(x, eps) * w["embed.norm"]
        results.append(x)
    for i, L in enumerate(raw["layers"]):
        p = f"l{i}."
        mix, feed = ({k[len(p + part):]: v for k, v in w.items() if k.startswith(p + part)} for part in ("mix.", "mlp."))
        if design == "pamasun":
            y = _pamasun_mixer(_divide(x, eps) * (1 + w[p + "norm1"]), mix, L["mixer"], L["type"], eps)
            x = x + _divide(y, eps) * (1 + w[p + "norm1b"]) * w[p + "ls1"]
            z = (_divide(x, eps) * (1 + w[p + "norm2"])) @ feed["up"].T
            a, b, c, e = feed["act"]
            y = (a * _divide(z, eps) + b * _divide(z ** 2, eps) + c * _divide(z ** 3, eps) + e) @ feed["down"].T
            x = x + _divide(y, eps) * (1 + w[p + "norm2b"]) * w[p + "ls2"]
        elif design == "maferax":
            x = _divide(raw["postln_alpha"] * x + _maferax_mixer(x, mix, L["mixer"], L["type"], eps), eps) * w[p + "norm1"]
            x = _divide(raw["postln_alpha"] * x + _maferax_feed(x, feed, L["mlp"]), eps) * w[p + "norm2"]
            results.append(x)
            x = sum(w[p + "dwa"][j] * r for j, r in enumerate(results))
        else:
            src = L["mixer"].get("kv_from")
            y, kv = _virusun_mixer(x, mix, L["mixer"], L["type"], eps, lent[src] if src is not None else None)
            lent.append(kv)
            x = x + _divide(y, eps) * w[p + "norm1"]
            x = x + _divide((F.silu(x @ feed["gate"].T) * (x @ feed["up"].T)) @ feed["down"].T, eps) * w[p + "norm2"]
    want = len(toks) if case["want"] == "all" else case["steps"] or 1
    x = _divide(x[len(toks) - want:], eps) * (1 + w["final.norm"] if design == "pamasun" else w["final.norm"])
    return x @ w["head"].T


def _exact_lm(case, seed):
    raw, w = _lm_weights(case, seed)
    w = {k: v.double() for k, v in w.items()}
    out = [_exact_lm_sequence(case, raw, w, t) for t in _lm_tokens(case, seed)]
    return torch.stack(out, 1) if case["steps"] else torch.cat(out)


def _lm_work(case):
    """Weights (of the experts: as many as the tokens can choose), cached keys, values and states; 2 flops per weight and token,
    scores and sums of the visible keys, the recurrences' updates and reads."""
    raw, z = _lm_config(case), LM_SIZES[case["size"]]
    H, d, wide = z["heads"], z["dim"], 4 if case["dtype"] == "float32" else 2
    rows = [(n + i, 1) for n in _lengths(case) for i in range(case["steps"])] if case["steps"] else [(0, n) for n in _lengths(case)]
    tokens, passes = sum(n for _, n in rows), max(1, case["steps"])
    pairs = sum(p * n + n * (n + 1) // 2 for p, n in rows)                  # (query, visible key)
    wanted = tokens if case["want"] == "all" or case["steps"] else len(rows)
    flops, per_pass, expert = 0, 0, 3 * 1024 * z["width"]
    for k, s in _lm_shapes(case, raw).items():
        if len(s) == 2 and k != "embed" and not k.endswith(".conv") and ".mlp.e" not in k:
            per_pass += s[0] * s[1] * wide
            flops += 2 * s[0] * s[1] * (wanted if k == "head" else tokens)
    moved = tokens * z["width"] * wide + wanted * z["vocab"] * 4
    for L in raw["layers"]:
        if L["mlp"]["kind"] == "moe":
            flops += 2 * 3 * tokens * expert
            per_pass += min(16, 3 * -(-tokens // passes)) * expert * wide
        mixers = [L["mixer"]] if L["type"] != "parallel" else [L["mixer"]["left"], L["mixer"]["right"]]
        for kind, m in zip([L["type"]] if len(mixers) == 1 else ["attention", "mlstm"], mixers):
            if kind in ("attention", "latent_attention"):
                maps, cached = (2 if "diff" in m else 1), (m["kv_rank"] + m["rot_dim"] if kind != "attention" else m["kv_heads"] * (m["dim"] * (2 if "diff" in m else 1) + m["vdim"]))
                flops += 2 * m["heads"] * maps * (m["dim"] + m.get("rot_dim", 0) + m["vdim"]) * pairs
                moved += sum(p + n for p, n in rows) * cached * wide
            else:
                flops += (8 if "delta" in kind else 6) * H * d * d * tokens
                moved += (2 if case["steps"] else 1) * len(rows) * H * d * d * 4
    return {"bytes": per_pass * passes + moved, "flops": flops}


# ---------------------------------------------------------------------------------------------- what is measured

def prepare(case, seed):
    return {"frames": _prepare_frames, "prompt": _prepare_prompt, "codec": _prepare_codec, "lm": _prepare_lm}[case["kind"]](case, seed)


def run(state):
    return {"frames": _run_frames, "prompt": _run_prompt, "codec": _run_codec, "lm": _run_lm}[state["kind"]](state)


def exact(case, seed):
    return {"frames": _exact_frames, "prompt": _exact_prompt, "codec": _exact_codec, "lm": _exact_lm}[case["kind"]](case, seed)


def work(case):
    if case["kind"] == "frames":
        cfg, n = named_config(case["model"]), case["frames"]
        at = [c + f for c in _contexts(case) for f in range(n)]
        return {"bytes": n * cfg.unique_weight_bytes() + sum(a + 1 for a in at) * cfg.kv_bytes_per_position(), "flops": sum(cfg.flops_per_frame(a) for a in at)}
    if case["kind"] == "prompt":
        cfg, n = named_config(case["model"]), case["tokens"]
        weights = cfg.n_layer * cfg.layer_params()
        head = cfg.vocab_size * cfg.dim
        return {"bytes": 2 * (weights + head) + n * cfg.kv_bytes_per_position(), "flops": 2 * (n * weights + head) + 4 * cfg.dim * cfg.n_layer * n * (n + 1) // 2}
    if case["kind"] == "codec":
        macs, elems, rows, ch = 0, 0, 2, 1024
        layers = [(1, 2 * 256 * 512), (2, 8 * (4 * 512 * 512 + 2 * 512 * 2048)), (2, 7 * 512 * 1024)]
        for r in (8, 6, 5, 4):
            layers.append((rows, 2 * ch * r * ch // 2))
            rows, ch = rows * r, ch // 2
            layers.append((rows, 3 * ch * ch // 2 + ch // 2 * ch))
        layers.append((rows, 3 * ch))
        macs, elems = sum(n * m for n, m in layers), sum(m for _, m in layers)
        B, T = case["streams"], case["frames"]
        steps = T if case["entry"] == "decode_step" else 1            # a whole utterance can read every weight once
        return {"bytes": 4 * (steps * elems + B * T * 1920) + B * 8 * 2 * 2048 * sum(2 * t + 2 for t in range(T)), "flops": 2 * B * T * macs}
    return _lm_work(case)


def tolerance(case):
    """bf16 models: one rounding of an activation or a cached value is 2^-9 relative and travels on; float32: sums in another order."""
    if case["kind"] == "codec":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "lm" and case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "lm":
        return {"rel": 0.03 if case["design"] == "maferax" else 0.02, "max": 0.9 if case["design"] == "maferax" else 0.5}   # a close call of the router may fall the other way
    return {"rel": 0.03, "max": 0.5}
