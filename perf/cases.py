"""Workloads of the framework through its public entry points, with their least work and what plain arithmetic gives.

Five kinds of pass, at the widths of the configurations that the package names:

``serve``    ``LLMEngine.replay``: prompts in one ragged batch, then decode steps from CUDA graphs
``step``     ``DecoderModel.forward_hidden`` + ``full_logits`` over a paged cache: a prompt chunk or one decoded token per sequence
``experts``  ``MoeFeedForward``: router, dispatch, grouped products and combination of routed and shared experts
``image``    ``FluxTransformer.forward``: one denoising step
``video``    ``WanTransformer.forward``: one denoising step, one guidance branch
``sample``   ``ops.sample_tokens``: the filter chain and the draw over a batch of logits

Models keep their configuration's widths and vocabulary and take fewer layers, so that a state fits the card
several times. 8-bit weights are drawn on the e4m3 grid with one power of two, which block quantisation keeps as it is.
"""
from __future__ import annotations

import math
import zlib
from dataclasses import replace

import torch

import hartsyinference_b200  # noqa: F401
from hartsyinference_b200 import ops
from hartsyinference_b200.engine import LLMEngine
from hartsyinference_b200.models.dit import flux, wan
from hartsyinference_b200.models.llm import config as llm
from hartsyinference_b200.models.llm.moe import MoeFeedForward, MoeWeights
from hartsyinference_b200.models.llm.transformer import DecoderModel, ForwardBatch

PAGE = 16
GRID = 2.0 ** -12          # 8-bit weights: e4m3 values times this
SUBLAYER = 0.25            # output projections: a sublayer adds a part of the stream's size, as in a trained model


def listed():
    return [
        # one user chats with a small model: latency, launches and host work of the engine count
        dict(name="chat-0.5b", kind="serve", model="qwen2.5-0.5b", layers=24, fp8=False, requests=1, least=29, most=29, steps=12),
        # a few users on a mid-size model: prompts of odd lengths in one batch, then their tokens
        dict(name="serve-8b-ragged", kind="serve", model="llama-3-8b", layers=8, fp8=False, requests=6, least=40, most=400, steps=8),
        # the benchmark's own step: 64 requests of 2048 tokens, 8-bit weights
        dict(name="decode-70b-fp8", kind="step", model="llama-3-70b", layers=4, fp8=True, decode=True, sequences=64, queries=1, least=2048, most=2176),
        # latent attention at decode, 8-bit weights (the leading dense layers of the model)
        dict(name="decode-dsv3-fp8", kind="step", model="deepseek-v3", layers=2, fp8=True, decode=True, sequences=32, queries=1, least=900, most=1152),
        # short prompts of odd lengths, bf16 weights
        dict(name="prefill-8b-ragged", kind="step", model="llama-3-8b", layers=6, fp8=False, decode=False, sequences=3, queries=645, least=0, most=0),
        # the benchmark's prompt chunk: 8192 tokens of four prompts, 8-bit weights
        dict(name="prefill-70b-fp8", kind="step", model="llama-3-70b", layers=2, fp8=True, decode=False, sequences=4, queries=2048, least=0, most=0),
        # a chunk of a long prompt on top of what the cache holds already
        dict(name="prefill-8b-long", kind="step", model="llama-3-8b", layers=4, fp8=False, decode=False, sequences=1, queries=2048, least=6144, most=6144),
        # an expert layer at decode batch size (a quarter of the model's experts, all widths)
        dict(name="experts-dsv3-fp8", kind="experts", model="deepseek-v3", experts=64, fp8=True, tokens=64),
        # one step of a 1024 x 1024 picture, 8-bit weights
        dict(name="image-1024-fp8", kind="image", double=2, single=4, fp8=True, height=64, width=64, text=512),
        # one step of a smaller picture of odd shape, bf16 weights
        dict(name="image-odd-bf16", kind="image", double=2, single=4, fp8=False, height=31, width=45, text=256),
        # one step of 33 frames of 480 x 832, one guidance branch
        dict(name="video-480p-fp8", kind="video", layers=2, fp8=True, frames=9, height=60, width=104),
        # sampling for a decode batch: temperature, top-k, top-p and min-p per request
        dict(name="sample-64", kind="sample", rows=64, vocab=128256),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["serve", "decode", "decode", "prefill", "prefill", "experts", "image", "video", "sample"])
    if kind == "serve":
        model, layers = rng.choice([("qwen2.5-0.5b", 24), ("llama-3-8b", 8)])
        n = _log(rng, 1, 16)
        least = _log(rng, 8, 300)
        return dict(kind="serve", model=model, layers=layers, fp8=False, requests=n, least=least, most=least + rng.randrange(1, 300), steps=rng.randrange(2, 14))
    if kind == "decode":
        model, layers, fp8, most = rng.choice([("llama-3-70b", 3, True, 64), ("llama-3-70b", 2, False, 64), ("llama-3-8b", 4, True, 96), ("deepseek-v3", 2, True, 128)])
        n = _log(rng, 1, most)
        least = _log(rng, 30, 6000 if n <= 16 else 2000)
        return dict(kind="step", model=model, layers=layers, fp8=fp8, decode=True, sequences=n, queries=1, least=least, most=least + rng.randrange(1, 400))
    if kind == "prefill":
        model, layers, fp8 = rng.choice([("llama-3-70b", 2, True), ("llama-3-8b", 4, False), ("llama-3-8b", 4, True), ("qwen2.5-0.5b", 12, False)])
        total = _log(rng, 70, 6000)
        n = min(_log(rng, 1, 12), max(1, total // 40))
        least = rng.choice([0, 0, _log(rng, 20, 4000)])
        return dict(kind="step", model=model, layers=layers, fp8=fp8, decode=False, sequences=n, queries=total // n, least=least, most=least + (rng.randrange(1, 300) if least else 0))
    if kind == "experts":
        return dict(kind="experts", model="deepseek-v3", experts=64, fp8=rng.random() < 0.7, tokens=_log(rng, 1, 700))
    if kind == "image":
        return dict(kind="image", double=2, single=4, fp8=rng.random() < 0.6, height=_log(rng, 16, 64), width=_log(rng, 16, 64), text=rng.choice([128, 256, 512]))
    if kind == "video":
        return dict(kind="video", layers=2, fp8=rng.random() < 0.7, frames=rng.randrange(1, 8), height=2 * _log(rng, 12, 30), width=2 * _log(rng, 12, 52))
    return dict(kind="sample", rows=_log(rng, 1, 128), vocab=rng.choice([32000, 50257, 128256, 151936]))


# ------------------------------------------------------------------------------------------ inputs
def _gen(name, seed):
    return torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()) * 1000003 + seed)


def _weight(name, seed, *shape, std=None, fp8=False):
    """A weight by name: normal values in bf16 that keep the size of a normed row, on the e4m3 grid where it will be held in 8 bits."""
    std = shape[-1] ** -0.5 if std is None else std
    w = torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=_gen(name, seed))
    return (w * (1 / GRID)).clamp_(-448, 448).to(torch.float8_e4m3fn).to(torch.bfloat16) * GRID if fp8 else w


def _near_one(name, seed, n):
    return 1.0 + _weight(name, seed, n, std=0.1)


def _llm_tensor(cfg, fp8, seed, name):
    """The checkpoint's tensor of that name, or None."""
    h, d, m = cfg.hidden_size, cfg.head_dim, cfg.mla
    last = name.split(".")[-2]
    if name == "model.embed_tokens.weight":
        return _weight(name, seed, cfg.vocab_size, h, std=1.0)
    if name == "lm_head.weight":
        return None if cfg.tie_embeddings else _weight(name, seed, cfg.vocab_size, h)
    shapes = {"gate_proj": (cfg.ffn_size, h), "up_proj": (cfg.ffn_size, h), "down_proj": (h, cfg.ffn_size)}
    if m is None:
        shapes.update(q_proj=(cfg.num_heads * d, h), k_proj=(cfg.num_kv_heads * d, h), v_proj=(cfg.num_kv_heads * d, h), o_proj=(h, cfg.num_heads * d))
    else:
        shapes.update(q_a_proj=(m.q_lora_rank, h), q_b_proj=(cfg.num_heads * (m.qk_nope_head_dim + m.qk_rope_head_dim), m.q_lora_rank),
                      kv_a_proj_with_mqa=(m.kv_lora_rank + m.qk_rope_head_dim, h), kv_b_proj=(cfg.num_heads * (m.qk_nope_head_dim + m.v_head_dim), m.kv_lora_rank),
                      o_proj=(h, cfg.num_heads * m.v_head_dim))
    if name.endswith("norm.weight"):
        return _near_one(name, seed, {"q_a_layernorm": m and m.q_lora_rank, "kv_a_layernorm": m and m.kv_lora_rank}.get(last, h))
    if last in ("o_proj", "down_proj"):
        return _weight(name, seed, *shapes[last], std=SUBLAYER * shapes[last][1] ** -0.5, fp8=fp8)
    if last in shapes:
        if name.endswith(".bias"):
            return _weight(name, seed, shapes[last][0], std=0.2) if cfg.qkv_bias else None
        return _weight(name, seed, *shapes[last], fp8=fp8 and last not in ("kv_a_proj_with_mqa", "kv_b_proj"))
    return None


def _llm_config(case):
    return replace(llm.PRESETS[case["model"]], num_layers=case["layers"])


def _lengths(case):
    """Tokens that every sequence holds before the pass (``step``), or prompt lengths (``serve``): spread over the case's range."""
    n = case["sequences"] if case["kind"] == "step" else case["requests"]
    return torch.randint(case["least"], case["most"] + 1, (n,), generator=torch.Generator().manual_seed(case["least"] + 1000003 * n)).tolist()


def _queries(case):
    """Prompt tokens of every sequence of a chunk: the same total, uneven (a whole number more or less per sequence)."""
    n, q = case["sequences"], case["queries"]
    return [q] if n == 1 else [q] * n if q >= 1024 else [q + (i * 2 - (n - 1)) * (q // (2 * n)) for i in range(n)]


def _tokens(cfg, seed, *shape):
    return torch.randint(0, cfg.vocab_size, shape, generator=torch.Generator().manual_seed(seed + 5), dtype=torch.int32)


def _pool_layout(counts, seed):
    """Page ids of every sequence, shuffled over the pool as a running engine leaves them."""
    pages = [(c + PAGE - 1) // PAGE for c in counts]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(seed + 3)).to(torch.int32)
    table, at = torch.zeros(len(counts), max(pages), dtype=torch.int32), 0
    for i, p in enumerate(pages):
        table[i, :p] = order[at:at + p]
        at += p
    return table, at


def _fill_cache(cache, seed):
    """Values of the size that the projections of a normed stream give."""
    g = _gen("cache", seed)
    for layer in cache:
        layer.normal_(0.0, 1.0, generator=g)


def prepare(case, seed):
    return {"serve": _prepare_serve, "step": _prepare_step, "experts": _prepare_experts, "image": _prepare_image, "video": _prepare_video,
            "sample": _prepare_sample}[case["kind"]](case, seed)


def _decoder(case, seed):
    cfg = _llm_config(case)
    model = DecoderModel(cfg, "cuda", fp8=case["fp8"])
    model.load_state_dict(lambda name: _llm_tensor(cfg, case["fp8"], seed, name))
    return cfg, model


def _prepare_serve(case, seed):
    cfg, model = _decoder(case, seed)
    lens, steps = _lengths(case), case["steps"]
    longest = max(lens) + steps
    engine = LLMEngine(model, num_pages=sum((n + steps) // PAGE + 1 for n in lens), page_size=PAGE, max_batch=len(lens), prefill_chunk=sum(lens), max_model_len=longest)
    ids = _tokens(cfg, seed, len(lens), longest).tolist()
    first = [(i, ids[i][:n], [n - 1]) for i, n in enumerate(lens)]
    later = [[(i, [ids[i][n + s]], [0]) for i, n in enumerate(lens)] for s in range(steps)]
    return dict(kind="serve", engine=engine, first=first, later=later, keys=list(range(len(lens))))


def _prepare_step(case, seed):
    cfg, model = _decoder(case, seed)
    held = _lengths(case)
    new = [1] * len(held) if case["decode"] else _queries(case)
    total = [a + b for a, b in zip(held, new)]
    table, pages = _pool_layout(total, seed)
    model.alloc_kv(pages, PAGE)
    _fill_cache(model.kv_cache, seed)
    pos = torch.cat([torch.arange(a, a + b) for a, b in zip(held, new)])
    seq = torch.repeat_interleave(torch.arange(len(new)), torch.tensor(new))
    slots = table[seq, pos // PAGE].long() * PAGE + pos % PAGE
    cu = torch.tensor([0] + new).cumsum(0).to(torch.int32)
    dev = lambda t: t.to("cuda")
    batch = ForwardBatch(tokens=dev(_tokens(cfg, seed, sum(new))), positions=dev(pos.to(torch.int32)), slot_mapping=dev(slots), block_table=dev(table),
                         kv_lens=dev(torch.tensor(total, dtype=torch.int32)), is_decode=case["decode"], cu_q=None if case["decode"] else dev(cu),
                         max_q_len=max(new), max_kv_len=max(total))
    return dict(kind="step", model=model, batch=batch, rows=None if case["decode"] else dev((cu[1:] - 1).long()))


def _prepare_experts(case, seed):
    cfg = llm.PRESETS[case["model"]]
    cfg = replace(cfg, moe=replace(cfg.moe, num_experts=case["experts"]))
    w = _expert_weights(case, cfg, seed)
    lin = lambda name: ops.LinearWeight.from_dense(w[name], fp8=case["fp8"])
    weights = MoeWeights(router=ops.LinearWeight(w["router"]), router_bias=w["bias"], gate_up=lin("gate_up"), down=lin("down"),
                         shared_gate_up=lin("shared_gate_up"), shared_down=lin("shared_down"))
    return dict(kind="experts", layer=MoeFeedForward(cfg, weights), x=w["x"])


def _expert_weights(case, cfg, seed):
    m, h, f8 = cfg.moe, cfg.hidden_size, case["fp8"]
    e, f, fs = m.num_experts, m.expert_ffn, m.shared_ffn * m.num_shared_experts
    return dict(router=_weight("router", seed, e, h), bias=_weight("bias", seed, e, std=0.01).float(), gate_up=_weight("gate_up", seed, e * 2 * f, h, fp8=f8),
                down=_weight("down", seed, e * h, f, fp8=f8), shared_gate_up=_weight("shared_gate_up", seed, 2 * fs, h, fp8=f8),
                shared_down=_weight("shared_down", seed, h, fs, fp8=f8), x=_weight("x", seed, case["tokens"], h, std=1.0))


def _flux_config(case):
    return replace(flux.FLUX_DEV, num_double_blocks=case["double"], num_single_blocks=case["single"])


def _dit_tensor(shape_of, fp8, seed, name):
    if name.endswith(".bias"):
        return _weight(name, seed, shape_of(name[:-5])[0], std=0.02)
    if "norm_" in name.split(".")[-2] or name.split(".")[-2] == "norm3":
        return _near_one(name, seed, shape_of(name)[0])
    base = name[:-7] if name.endswith(".weight") else name
    shape = shape_of(base)
    out = base.endswith((".to_out.0", ".to_add_out", ".net.2", ".proj_out", "_attn.o", ".ffn.2"))
    return _weight(name, seed, *shape, std=(SUBLAYER if out else 1.0) * shape[-1] ** -0.5, fp8=fp8)


def _flux_tensor(cfg, fp8, seed, name):
    h, a, f = cfg.hidden_size, cfg.num_heads * cfg.head_dim, cfg.mlp_dim

    def shape_of(base):
        part = base.split(".")
        if base.endswith(".weight"):
            return (cfg.head_dim,)
        for end, shape in (("x_embedder", (h, cfg.in_channels)), ("context_embedder", (h, cfg.context_dim)), ("proj_out", (h, a + f)), ("proj_mlp", (f, h)),
                           ("net.0.proj", (f, h)), ("net.2", (h, f)), ("to_out.0", (h, a)), ("to_add_out", (h, a)), ("norm1.linear", (6 * h, h)),
                           ("norm1_context.linear", (6 * h, h)), ("norm_out.linear", (2 * h, h)), ("norm.linear", (3 * h, h)), ("linear_2", (h, h))):
            if base.endswith(end):
                return (cfg.latent_channels, h) if base == "proj_out" else shape
        if part[-1] == "linear_1":
            return (h, cfg.pooled_dim if "text_embedder" in base else 256)
        return (a, h)

    # embedders of few inputs are held in bf16
    small = name.startswith("x_embedder") or ".linear_1." in name
    return _dit_tensor(shape_of, fp8 and not small, seed, name)


def _prepare_image(case, seed):
    cfg = _flux_config(case)
    model = flux.FluxTransformer(cfg, "cuda", fp8=case["fp8"], get=lambda name: _flux_tensor(cfg, case["fp8"], seed, name))
    return dict(kind="image", model=model, **_image_inputs(case, cfg, seed))


def _image_inputs(case, cfg, seed):
    img_ids, txt_ids = flux.flux_ids(case["height"], case["width"], case["text"], "cuda")
    return dict(img=_weight("latents", seed, 1, case["height"] * case["width"], cfg.in_channels, std=1.0), txt=_weight("text", seed, 1, case["text"], cfg.context_dim, std=0.3),
                pooled=_weight("pooled", seed, 1, cfg.pooled_dim, std=1.0), sigma=torch.tensor([0.7], device="cuda"), guidance=torch.tensor([3.5], device="cuda"),
                img_ids=img_ids, txt_ids=txt_ids)


def _wan_config(case):
    return replace(wan.WAN_14B, num_layers=case["layers"])


def _wan_tensor(cfg, fp8, seed, name):
    h = cfg.hidden_size

    def shape_of(base):
        if base.endswith(".weight"):
            return (h,)
        if base.endswith("norm3"):
            return (h,)
        if base.endswith("modulation"):
            return (2 if base.startswith("head") else 6, h)
        for end, shape in (("patch_embedding", (h, cfg.patch_dim)), ("text_embedding.0", (h, cfg.text_dim)), ("time_embedding.0", (h, cfg.freq_dim)),
                           ("time_projection.1", (6 * h, h)), ("ffn.0", (cfg.ffn_size, h)), ("ffn.2", (h, cfg.ffn_size)),
                           ("head.head", (cfg.out_channels * math.prod(cfg.patch), h))):
            if base.endswith(end):
                return shape
        return (h, h)

    small = name.startswith(("patch_embedding", "time_embedding.0")) or name.endswith("modulation")
    return _dit_tensor(shape_of, fp8 and not small, seed, name)


def _video_inputs(case, cfg, seed):
    return dict(latents=_weight("latents", seed, cfg.in_channels, case["frames"], case["height"], case["width"], std=1.0),
                text=_weight("text", seed, cfg.text_len, cfg.text_dim, std=0.3), timestep=torch.tensor(700.0, device="cuda"))


def _prepare_video(case, seed):
    cfg = _wan_config(case)
    model = wan.WanTransformer(cfg, "cuda", fp8=case["fp8"], get=lambda name: _wan_tensor(cfg, case["fp8"], seed, name))
    x = _video_inputs(case, cfg, seed)
    return dict(kind="video", model=model, latents=x["latents"], timestep=x["timestep"], context=model.encode_text(x["text"]))


def _prepare_sample(case, seed):
    n = case["rows"]
    g = torch.Generator().manual_seed(seed)
    pick = lambda values: torch.tensor(values)[torch.randint(0, len(values), (n,), generator=g)].to("cuda")
    # peaked logits as a trained head gives them: a few candidates well above a broad floor
    logits = torch.empty(n, case["vocab"], dtype=torch.float32, device="cuda").normal_(0.0, 2.0, generator=_gen("logits", seed))
    logits += 6.0 * (torch.rand(logits.shape, device="cuda", generator=_gen("peaks", seed)) > 0.9995)
    return dict(kind="sample", args=(logits.to(torch.bfloat16).float(), pick([0.0, 0.7, 0.8, 1.0]), pick([0, 40, 50]).to(torch.int32), pick([0.9, 0.95, 1.0]), pick([0.0, 0.05]),
                                     torch.randint(0, 1 << 31, (n,), generator=g).to("cuda"), torch.randint(0, 2000, (n,), generator=g).to("cuda")))


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "serve":
        engine, out = state["engine"], []
        for i, entries in enumerate([state["first"]] + state["later"]):
            out.append(engine.replay(entries, end=state["keys"] if i == len(state["later"]) else ()))
        return out
    if kind == "step":
        model, batch = state["model"], state["batch"]
        hidden = model.forward_hidden(batch)
        if batch.is_decode:
            return dict(hidden=hidden, logits=model.full_logits(hidden))
        return dict(hidden=hidden, logits=model.full_logits(hidden[state["rows"]].contiguous()), cache=model.kv_cache)
    if kind == "experts":
        return state["layer"](state["x"])
    if kind == "image":
        return state["model"].forward(state["img"], state["txt"], state["sigma"], state["pooled"], state["img_ids"], state["txt_ids"], state["guidance"])
    if kind == "video":
        return state["model"].forward(state["latents"], state["timestep"], state["context"])
    return ops.sample_tokens(*state["args"])


# ------------------------------------------------------------------------------------------ least work
def _llm_work(case, cfg, spans, head_rows):
    """Weights once, cached rows read and written once, logits written; products of the tokens and the causal attention.
    ``spans``: (tokens held, new tokens) of every sequence."""
    h, d, m = cfg.hidden_size, cfg.head_dim, cfg.mla
    es = 1 if case["fp8"] else 2
    new = sum(q for _, q in spans)
    if m is None:
        lin = h * (cfg.q_size + 2 * cfg.kv_size) + h * cfg.q_size + 3 * h * cfg.ffn_size
        other, row, per_pair = 0, 2 * cfg.kv_size * 2, 4 * cfg.q_size
    else:
        lin = h * m.q_lora_rank + m.q_lora_rank * cfg.num_heads * (m.qk_nope_head_dim + m.qk_rope_head_dim) + h * cfg.num_heads * m.v_head_dim + 3 * h * cfg.ffn_size
        other = h * (m.kv_lora_rank + m.qk_rope_head_dim) + cfg.num_heads * (m.qk_nope_head_dim + m.v_head_dim) * m.kv_lora_rank
        row, per_pair = (m.kv_lora_rank + m.qk_rope_head_dim) * 2, 2 * cfg.num_heads * (2 * m.kv_lora_rank + m.qk_rope_head_dim)
    pairs = sum(q * c + q * (q + 1) // 2 for c, q in spans)
    head = cfg.vocab_size * h
    held = sum(c for c, _ in spans)
    return dict(bytes=case["layers"] * (lin * es + other * 2 + (held + new) * row) + head * 2 + new * h * 2 + head_rows * cfg.vocab_size * 2,
                flops=case["layers"] * (2 * (lin + other) * new + per_pair * pairs) + 2 * head * head_rows)


def work(case):
    kind = case["kind"]
    if kind == "serve":
        cfg, lens = _llm_config(case), _lengths(case)
        parts = [_llm_work(case, cfg, [(0, n) for n in lens], len(lens))]
        parts += [_llm_work(case, cfg, [(n + s, 1) for n in lens], len(lens)) for s in range(case["steps"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "step":
        held = _lengths(case)
        new = [1] * len(held) if case["decode"] else _queries(case)
        return _llm_work(case, _llm_config(case), list(zip(held, new)), len(held))
    if kind == "experts":
        cfg = llm.PRESETS[case["model"]]
        m, h, t = cfg.moe, cfg.hidden_size, case["tokens"]
        per, shared = 3 * h * m.expert_ffn, 3 * h * m.shared_ffn * m.num_shared_experts
        used = case["experts"] * (1 - (1 - m.top_k / case["experts"]) ** t)
        return dict(bytes=(used * per + shared) * (1 if case["fp8"] else 2) + case["experts"] * h * 2 + 2 * t * h * 2,
                    flops=2 * t * (m.top_k * per + shared + case["experts"] * h))
    if kind == "image":
        cfg = _flux_config(case)
        h, f, s_i, s_t = cfg.hidden_size, cfg.mlp_dim, case["height"] * case["width"], case["text"]
        s, block, one = s_i + s_t, 4 * h * h + 2 * h * f, 4 * h * h + 2 * h * f
        weights = case["double"] * (2 * block + 12 * h * h) + case["single"] * (one + 3 * h * h) + h * (cfg.context_dim + 5 * h + cfg.in_channels * 2)
        flops = 2 * s * (case["double"] * block + case["single"] * one) + (case["double"] + case["single"]) * 4 * s * s * h + 2 * s_t * cfg.context_dim * h + 4 * s_i * cfg.in_channels * h
        return dict(bytes=weights * (1 if case["fp8"] else 2) + 2 * (s_i * cfg.in_channels * 2 + s_t * cfg.context_dim), flops=flops)
    if kind == "video":
        cfg = _wan_config(case)
        h, f, s, l = cfg.hidden_size, cfg.ffn_size, case["frames"] * case["height"] * case["width"] // 4, cfg.text_len
        block = 6 * h * h + 2 * h * f
        flops = case["layers"] * (2 * s * block + 4 * l * h * h + 4 * s * s * h + 4 * s * l * h) + 4 * s * cfg.patch_dim * h
        return dict(bytes=(case["layers"] * (block + 2 * h * h) + 7 * h * h) * (1 if case["fp8"] else 2) + s * cfg.patch_dim * 6 + l * h * 2, flops=flops)
    return dict(bytes=case["rows"] * case["vocab"] * 4, flops=case["rows"] * case["vocab"] * 4)


def tolerance(case):
    """bf16 activations through a few layers; 8-bit activations turn a last-bit difference of a value into a step of theirs."""
    kind = case["kind"]
    if kind == "sample":
        return "exact"
    if kind == "serve":
        return dict(rel=0.03, max=0.5)
    return dict(rel=0.03 if case["fp8"] else 0.02, max=0.5)


# ------------------------------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    with torch.no_grad():
        return {"serve": _exact_serve, "step": _exact_step, "experts": _exact_experts, "image": _exact_image, "video": _exact_video, "sample": lambda c, s: None}[case["kind"]](case, seed)


def _mm(x, w, b=None, rows=16384):
    """x w^T + b, with the weight widened a part at a time."""
    y = torch.cat([x @ w[i:i + rows].double().t() for i in range(0, w.shape[0], rows)], -1)
    return y if b is None else y + b.double()


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def _ln(x, eps=1e-6):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rope(x, pos, theta, pairs):
    """x [T, heads, rot]; ``pairs``: neighbours turn together, else the two halves."""
    r = x.shape[-1]
    a = pos.double()[:, None] * theta ** (-torch.arange(0, r, 2, dtype=torch.float64, device=x.device) / r)
    return _turn(x, a.cos()[:, None], a.sin()[:, None], pairs)


def _turn(x, cos, sin, pairs):
    a, b = (x[..., 0::2], x[..., 1::2]) if pairs else x.chunk(2, -1)
    u, v = a * cos - b * sin, b * cos + a * sin
    return torch.stack([u, v], -1).flatten(-2) if pairs else torch.cat([u, v], -1)


def _attend(q, k, v, scale, first=None):
    """q [T, heads, d], k / v [S, kv heads, d]; query i sees keys up to ``first`` + i, or all of them."""
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    group, at = q.shape[1] // k.shape[1], torch.arange(k.shape[0], device=q.device)
    for h in range(q.shape[1]):
        for i in range(0, q.shape[0], 4096):
            s = q[i:i + 4096, h] @ k[:, h // group].t() * scale
            if first is not None:
                s.masked_fill_(at[None] > first + i + torch.arange(s.shape[0], device=q.device)[:, None], -math.inf)
            out[i:i + 4096, h] = torch.softmax(s, -1) @ v[:, h // group]
    return out


def _exact_layers(cfg, fp8, seed, x, spans, past):
    """Final-normed states. ``spans``: (tokens held, new tokens) per sequence, whose rows follow one another in x; ``past(layer,
    sequence)``: what the cache holds of them, as it is stored, or None."""
    t = lambda name: _llm_tensor(cfg, fp8, seed, name)
    pos = torch.cat([torch.arange(c, c + q, device=x.device) for c, q in spans])
    d, m, n = cfg.head_dim, cfg.mla, x.shape[0]
    for li in range(cfg.num_layers):
        p = f"model.layers.{li}."
        a = p + "self_attn."
        h = _rms(x, t(p + "input_layernorm.weight"), cfg.rms_eps)
        if m is None:
            q, k, v = (_mm(h, t(a + f"{s}_proj.weight"), t(a + f"{s}_proj.bias")).reshape(n, -1, d) for s in "qkv")
            q, k = _rope(q, pos, cfg.rope_theta, False), _rope(k, pos, cfg.rope_theta, False)
        else:
            q = _mm(_rms(_mm(h, t(a + "q_a_proj.weight")), t(a + "q_a_layernorm.weight"), cfg.rms_eps), t(a + "q_b_proj.weight")).reshape(n, cfg.num_heads, -1)
            q = torch.cat([q[..., :m.qk_nope_head_dim], _rope(q[..., m.qk_nope_head_dim:], pos, cfg.rope_theta, True)], -1)
            kv = _mm(h, t(a + "kv_a_proj_with_mqa.weight"))
            latent = _rms(kv[:, :m.kv_lora_rank], t(a + "kv_a_layernorm.weight"), cfg.rms_eps)
            turned = _rope(kv[:, None, m.kv_lora_rank:], pos, cfg.rope_theta, True)[:, 0]
            kv_b = t(a + "kv_b_proj.weight").double().reshape(cfg.num_heads, -1, m.kv_lora_rank)
            w_k, w_v = kv_b[:, :m.qk_nope_head_dim], kv_b[:, m.qk_nope_head_dim:]
        outs, at = [], 0
        for si, (c, w) in enumerate(spans):
            rows = slice(at, at + w)
            at += w
            old = past(li, si)
            if m is None:
                kk, vv = (k[rows], v[rows]) if old is None else (torch.cat([old[0], k[rows]]), torch.cat([old[1], v[rows]]))
                outs.append(_attend(q[rows], kk, vv, d ** -0.5, c).reshape(w, -1))
            else:
                row = torch.cat([latent[rows], turned[rows]], -1)
                row = row if old is None else torch.cat([old, row])
                lat, rot = row[:, :m.kv_lora_rank], row[:, m.kv_lora_rank:]
                # scores and values in latent space, which is the same sum
                ql = torch.cat([torch.einsum("thn,hnc->thc", q[rows][..., :m.qk_nope_head_dim], w_k), q[rows][..., m.qk_nope_head_dim:]], -1)
                o = _attend(ql, torch.cat([lat, rot], -1)[:, None], lat[:, None], (m.qk_nope_head_dim + m.qk_rope_head_dim) ** -0.5, c)
                outs.append(torch.einsum("thc,hvc->thv", o, w_v).reshape(w, -1))
        x = x + _mm(torch.cat(outs), t(a + "o_proj.weight"))
        h = _rms(x, t(p + "post_attention_layernorm.weight"), cfg.rms_eps)
        x = x + _mm(torch.nn.functional.silu(_mm(h, t(p + "mlp.gate_proj.weight"))) * _mm(h, t(p + "mlp.up_proj.weight")), t(p + "mlp.down_proj.weight"))
    return _rms(x, t("model.norm.weight"), cfg.rms_eps)


def _head(cfg, seed):
    return _llm_tensor(cfg, False, seed, "model.embed_tokens.weight" if cfg.tie_embeddings else "lm_head.weight")


def _exact_serve(case, seed):
    cfg, lens = _llm_config(case), _lengths(case)
    ids = _tokens(cfg, seed, len(lens), max(lens) + case["steps"])
    spans = [(0, n + case["steps"]) for n in lens]
    flat = torch.cat([ids[i, :q] for i, (_, q) in enumerate(spans)]).long().cuda()
    h = _exact_layers(cfg, case["fp8"], seed, _llm_tensor(cfg, case["fp8"], seed, "model.embed_tokens.weight")[flat].double(), spans, lambda li, si: None)
    starts = torch.tensor([0] + [q for _, q in spans]).cumsum(0)[:-1]
    w = _head(cfg, seed)
    return [_mm(h[(starts + torch.tensor(lens) - 1 + s).cuda()], w) for s in range(case["steps"] + 1)]


def _exact_step(case, seed):
    cfg, held = _llm_config(case), _lengths(case)
    new = [1] * len(held) if case["decode"] else _queries(case)
    table, pages = _pool_layout([a + b for a, b in zip(held, new)], seed)
    m = cfg.mla
    shape = (pages, PAGE, m.kv_lora_rank + m.qk_rope_head_dim) if m else (2, pages, cfg.num_kv_heads, PAGE, cfg.head_dim)
    g, pools = _gen("cache", seed), []

    def past(li, si):
        while len(pools) <= li:
            pools.append(torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, 1.0, generator=g))
        c = held[si]
        if c == 0:
            return None
        own = table[si, :(c + PAGE - 1) // PAGE].long().cuda()
        if m:
            return pools[li][own].reshape(-1, shape[-1])[:c].double()
        return [pools[li][j][own].transpose(1, 2).reshape(-1, cfg.num_kv_heads, cfg.head_dim)[:c].double() for j in (0, 1)]

    ids = _tokens(cfg, seed, sum(new)).long().cuda()
    h = _exact_layers(cfg, case["fp8"], seed, _llm_tensor(cfg, case["fp8"], seed, "model.embed_tokens.weight")[ids].double(), list(zip(held, new)), past)
    if case["decode"]:
        return dict(hidden=h, logits=_mm(h, _head(cfg, seed)))
    rows = torch.tensor(new).cumsum(0) - 1
    return dict(hidden=h, logits=_mm(h[rows.cuda()], _head(cfg, seed)), cache=None)


def _exact_experts(case, seed):
    cfg = llm.PRESETS[case["model"]]
    cfg = replace(cfg, moe=replace(cfg.moe, num_experts=case["experts"]))
    m, w = cfg.moe, _expert_weights(case, cfg, seed)
    x = w["x"].double()
    # the router's product is stored in the activation type, and the choice is made on what is stored
    s = torch.sigmoid(_mm(x, w["router"]).to(torch.bfloat16).double())
    c = s + w["bias"].double()
    groups = c.reshape(len(x), m.n_group, -1).topk(2, -1).values.sum(-1).topk(m.topk_group, -1).indices
    keep = torch.zeros(len(x), m.n_group, dtype=torch.bool, device=x.device).scatter_(1, groups, True)
    ids = c.masked_fill(~keep.repeat_interleave(m.num_experts // m.n_group, 1), -math.inf).topk(m.top_k, -1).indices
    wt = s.gather(1, ids)
    wt = wt / wt.sum(-1, keepdim=True) * m.routed_scaling_factor
    glu = lambda v: torch.nn.functional.silu(v.chunk(2, -1)[0]) * v.chunk(2, -1)[1]
    out = _mm(glu(_mm(x, w["shared_gate_up"])), w["shared_down"])
    gu, dn = w["gate_up"].reshape(m.num_experts, -1, cfg.hidden_size), w["down"].reshape(m.num_experts, cfg.hidden_size, -1)
    for e in range(m.num_experts):
        t, j = (ids == e).nonzero(as_tuple=True)
        if len(t):
            out.index_add_(0, t, wt[t, j][:, None] * _mm(glu(_mm(x[t], gu[e])), dn[e]))
    return out


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _sinusoid(t, dim):
    a = t.double()[:, None] * torch.exp(-math.log(10000.0) * torch.arange(dim // 2, dtype=torch.float64, device=t.device) / (dim // 2))
    return torch.cat([a.cos(), a.sin()], -1)


def _axes(ids, dims, theta):
    a = torch.cat([ids[:, i].double()[:, None] * theta ** (-torch.arange(0, d, 2, dtype=torch.float64, device=ids.device) / d) for i, d in enumerate(dims)], -1)
    return a.cos()[:, None], a.sin()[:, None]


def _exact_image(case, seed):
    cfg, silu = _flux_config(case), torch.nn.functional.silu
    x = _image_inputs(case, cfg, seed)
    t = lambda name: _flux_tensor(cfg, case["fp8"], seed, name)
    lin = lambda v, name: _mm(v, t(name + ".weight"), t(name + ".bias"))
    mlp = lambda v, name: lin(silu(lin(v, name + ".linear_1")), name + ".linear_2")
    e = "time_text_embed."
    temb = silu(mlp(_sinusoid(x["sigma"] * 1000, 256), e + "timestep_embedder") + mlp(_sinusoid(x["guidance"] * 1000, 256), e + "guidance_embedder")
                + mlp(x["pooled"].double(), e + "text_embedder"))
    s_t, n, d = case["text"], cfg.num_heads, cfg.head_dim
    cos, sin = _axes(torch.cat([x["txt_ids"], x["img_ids"]]), cfg.axes_dim, cfg.theta)
    img, txt = lin(x["img"][0].double(), "x_embedder"), lin(x["txt"][0].double(), "context_embedder")

    def heads(v, names, norms, rows):
        q, k, vv = (lin(v, name).reshape(len(v), n, d) for name in names)
        return (_turn(_rms(q, t(norms[0] + ".weight"), 1e-6), cos[rows], sin[rows], True), _turn(_rms(k, t(norms[1] + ".weight"), 1e-6), cos[rows], sin[rows], True), vv)

    for i in range(cfg.num_double_blocks):
        p = f"transformer_blocks.{i}."
        mi, mt = lin(temb, p + "norm1.linear").chunk(6, -1), lin(temb, p + "norm1_context.linear").chunk(6, -1)
        hi = heads(_ln(img) * (1 + mi[1]) + mi[0], [p + "attn.to_" + s for s in "qkv"], [p + "attn.norm_q", p + "attn.norm_k"], slice(s_t, None))
        ht = heads(_ln(txt) * (1 + mt[1]) + mt[0], [p + f"attn.add_{s}_proj" for s in "qkv"], [p + "attn.norm_added_q", p + "attn.norm_added_k"], slice(0, s_t))
        o = _attend(*(torch.cat([a, b]) for a, b in zip(ht, hi)), d ** -0.5).flatten(1)
        img, txt = img + mi[2] * lin(o[s_t:], p + "attn.to_out.0"), txt + mt[2] * lin(o[:s_t], p + "attn.to_add_out")
        img = img + mi[5] * lin(_gelu(lin(_ln(img) * (1 + mi[4]) + mi[3], p + "ff.net.0.proj")), p + "ff.net.2")
        txt = txt + mt[5] * lin(_gelu(lin(_ln(txt) * (1 + mt[4]) + mt[3], p + "ff_context.net.0.proj")), p + "ff_context.net.2")
    y = torch.cat([txt, img])
    for i in range(cfg.num_single_blocks):
        p = f"single_transformer_blocks.{i}."
        m = lin(temb, p + "norm.linear").chunk(3, -1)
        h = _ln(y) * (1 + m[1]) + m[0]
        o = _attend(*heads(h, [p + "attn.to_" + s for s in "qkv"], [p + "attn.norm_q", p + "attn.norm_k"], slice(None)), d ** -0.5).flatten(1)
        y = y + m[2] * lin(torch.cat([o, _gelu(lin(h, p + "proj_mlp"))], -1), p + "proj_out")
    scale, shift = lin(temb, "norm_out.linear").chunk(2, -1)
    return lin(_ln(y[s_t:]) * (1 + scale) + shift, "proj_out")[None]


def _exact_video(case, seed):
    cfg, silu = _wan_config(case), torch.nn.functional.silu
    x = _video_inputs(case, cfg, seed)
    t = lambda name: _wan_tensor(cfg, case["fp8"], seed, name)
    lin = lambda v, name: _mm(v, t(name + ".weight"), t(name + ".bias"))
    h, n, d, eps = cfg.hidden_size, cfg.num_heads, cfg.head_dim, cfg.eps
    text = lin(_gelu(lin(x["text"].double(), "text_embedding.0")), "text_embedding.2")
    grid = (case["frames"], case["height"] // 2, case["width"] // 2)
    z = x["latents"].double().reshape(cfg.in_channels, grid[0], grid[1], 2, grid[2], 2).permute(1, 2, 4, 0, 3, 5)
    y = lin(z.reshape(-1, cfg.patch_dim), "patch_embedding")
    s = len(y)
    if 4.0 * s * s * h * cfg.num_layers > 4e14:
        return None
    ids = torch.stack(torch.meshgrid(*(torch.arange(g, device="cuda") for g in grid), indexing="ij"), -1).reshape(-1, 3)
    cos, sin = _axes(ids, cfg.axes_dim, cfg.theta)
    e = lin(silu(lin(_sinusoid(x["timestep"].reshape(1), cfg.freq_dim), "time_embedding.0")), "time_embedding.2")
    e0 = lin(silu(e), "time_projection.1").reshape(6, h)
    for i in range(cfg.num_layers):
        p = f"blocks.{i}."
        m = t(p + "modulation").double().reshape(6, h) + e0
        v = _ln(y, eps) * (1 + m[1]) + m[0]
        q, k = (_turn(_rms(lin(v, p + f"self_attn.{c}"), t(p + f"self_attn.norm_{c}.weight"), eps).reshape(s, n, d), cos, sin, True) for c in "qk")
        y = y + m[2] * lin(_attend(q, k, lin(v, p + "self_attn.v").reshape(s, n, d), d ** -0.5).flatten(1), p + "self_attn.o")
        v = _ln(y, eps) * t(p + "norm3.weight").double() + t(p + "norm3.bias").double()
        q = _rms(lin(v, p + "cross_attn.q"), t(p + "cross_attn.norm_q.weight"), eps).reshape(s, n, d)
        k = _rms(lin(text, p + "cross_attn.k"), t(p + "cross_attn.norm_k.weight"), eps).reshape(-1, n, d)
        y = y + lin(_attend(q, k, lin(text, p + "cross_attn.v").reshape(-1, n, d), d ** -0.5).flatten(1), p + "cross_attn.o")
        v = _ln(y, eps) * (1 + m[4]) + m[3]
        y = y + m[5] * lin(_gelu(lin(v, p + "ffn.0")), p + "ffn.2")
    m = t("head.modulation").double().reshape(2, h) + e
    out = lin(_ln(y, eps) * (1 + m[1]) + m[0], "head.head").reshape(*grid, *cfg.patch, cfg.out_channels)
    return out.permute(6, 0, 3, 1, 4, 2, 5).reshape(cfg.out_channels, case["frames"], case["height"], case["width"])
