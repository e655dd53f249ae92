"""What this package is timed on: the work its users have it do, through its public entry points.

A case is one of these kinds:

attend    one new token for each of a batch of sequences: append to the fp8 cache and attention over it, in the two launches of
          decode_step_attention (a plug-in inside another engine calls exactly this once per layer and step)
fill      the rows of whole prompts: kv_append, then prefill_attention over the pages just written (one layer of a prefill pass)
decode    one decode step of a whole model: every slot one token at its own context, logits out, as a captured graph
prompts   prefill of a batch of prompts and the step that follows it: what a user waits for until the first token
feed      a portion of one sequence behind its context, logits of its last token back (a conversation's next turn, a replayed
          trace; a portion of one token is a decode step for a single user)

The models are the three of the registry: nanochat (fp8 cache, relu^2), Pudisun (gated linear and latent attention) and Rekudra
(gated delta rule and grouped attention, several streams), at the sizes of the benchmark and others of the same proportions
(width 64 per layer, heads of 128). Weights are random and scaled so that every branch adds about as much as the stream holds;
a context is already in the caches, as other turns left it there."""

import gc
import math

import torch
import torch.nn.functional as F

import nanochat_b200 as ncb
from nanochat_b200 import attention as ops
from nanochat_b200.decoder import Decoder, DecoderConfig, DecoderWeights
from nanochat_b200.hybrid import HybridConfig, HybridDecoder, HybridWeights

DEV, HEAD, VOCAB, F64 = "cuda", 128, 65536, torch.float64
LATENT, ROT, CONV, RANK_A = 512, 64, 4, 16
THETA, EPS = 10000.0, 1e-6
NANO_EPS = 1.1920928955078125e-07


def listed() -> list:
    return [
        # the smallest call: one user, one layer of a d20 model, a short conversation; two launches and their gaps
        {"name": "attend_one_short", "kind": "attend", "batch": 1, "heads": 10, "kv_heads": 10, "shortest": 512, "longest": 512,
         "window": 0},
        # the benchmark's default workload: a full batch of equal long contexts, four query heads to a key/value head
        {"name": "attend_64_long", "kind": "attend", "batch": 64, "heads": 32, "kv_heads": 8, "shortest": 8192, "longest": 8192,
         "window": 0},
        # the benchmark's ragged sweep, with an odd number of sequences
        {"name": "attend_ragged", "kind": "attend", "batch": 57, "heads": 32, "kv_heads": 8, "shortest": 512, "longest": 16384,
         "window": 0},
        # one layer of a long document's prefill at the d32 heads
        {"name": "fill_document", "kind": "fill", "prompts": 1, "heads": 16, "kv_heads": 4, "shortest": 8190, "longest": 8190},
        # the benchmark's small model: eight chats of a few hundred tokens
        {"name": "nanochat_decode", "kind": "decode", "model": "nanochat", "depth": 20, "kv_heads": 10, "batch": 8, "shortest": 512,
         "longest": 512, "dtype": "bf16"},
        {"name": "nanochat_prompts", "kind": "prompts", "model": "nanochat", "depth": 20, "kv_heads": 10, "batch": 8, "shortest": 512,
         "longest": 512, "dtype": "bf16"},
        {"name": "pudisun_prompts", "kind": "prompts", "model": "pudisun", "depth": 20, "kv_heads": 10, "batch": 8, "shortest": 512,
         "longest": 512, "dtype": "bf16"},
        {"name": "rekudra_prompts", "kind": "prompts", "model": "rekudra", "depth": 20, "kv_heads": 10, "batch": 8, "shortest": 512,
         "longest": 512, "dtype": "bf16"},
        # the benchmark's large models: a batch of 32 at contexts from a question to a long document
        {"name": "pudisun_decode_ragged", "kind": "decode", "model": "pudisun", "depth": 32, "kv_heads": 4, "batch": 32,
         "shortest": 256, "longest": 8192, "dtype": "bf16"},
        {"name": "rekudra_decode_ragged", "kind": "decode", "model": "rekudra", "depth": 32, "kv_heads": 4, "batch": 32,
         "shortest": 256, "longest": 8192, "dtype": "bf16"},
        # the next turn of a long conversation: a few thousand tokens behind a thousand already there
        {"name": "pudisun_long_turn", "kind": "feed", "model": "pudisun", "depth": 20, "kv_heads": 10, "context": 1000, "tokens": 3000,
         "dtype": "bf16"},
        # 32-bit runs exist to check other implementations against: a prompt of a few hundred tokens
        {"name": "rekudra_exact_turn", "kind": "feed", "model": "rekudra", "depth": 12, "kv_heads": 6, "context": 0, "tokens": 300,
         "dtype": "f32"},
    ]


def draw(rng) -> dict:
    def spread(low: int, high: int) -> int:
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["attend", "fill", "decode", "decode", "prompts", "prompts", "feed", "feed"])
    kv_heads, ratio = rng.choice([(10, 1), (4, 4), (8, 4), (6, 2), (16, 1), (2, 8)])
    if kind == "attend":
        batch = spread(1, 64)
        longest = spread(64, 16384 if batch * kv_heads <= 256 else 8192)
        return {"kind": kind, "batch": batch, "heads": kv_heads * ratio, "kv_heads": kv_heads, "shortest": spread(16, longest),
                "longest": longest, "window": rng.choice([0, 0, 0, 1024])}
    if kind == "fill":
        longest = spread(16, 8192)
        return {"kind": kind, "prompts": max(1, min(spread(1, 16), 8192 // longest)), "heads": kv_heads * ratio, "kv_heads": kv_heads,
                "shortest": max(2, longest // rng.randint(1, 4)), "longest": longest}
    model, dtype = rng.choice(["nanochat", "pudisun", "rekudra"]), "bf16"
    depth = 2 * rng.randint(4, 10)
    case = {"kind": kind, "model": model, "depth": depth, "kv_heads": rng.choice([depth // 2, 2 if depth % 4 == 0 else 3 if depth == 18 else 1])}
    if kind == "decode":
        longest = spread(64, 8192)
        case.update(batch=spread(1, 32), shortest=spread(16, longest), longest=longest)
    elif kind == "prompts":
        longest = spread(16, 2048)
        case.update(batch=max(1, min(spread(1, 16), 4096 // longest)), shortest=max(2, longest // rng.randint(1, 4)), longest=longest)
    else:
        if model != "nanochat" and rng.random() < 0.3:
            dtype = "f32"
        tokens = spread(1, 300 if dtype == "f32" else 4096)
        case.update(context=rng.choice([0, spread(1, 2000)]), tokens=tokens)
    case["dtype"] = dtype
    return case


def lengths(case: dict) -> list:
    """The sequences' lengths, from the shortest to the longest by equal factors."""
    count = case.get("batch", case.get("prompts"))
    low, high = case["shortest"], case["longest"]
    return [int(round(low * (high / low) ** (i / max(count - 1, 1)))) for i in range(count - 1)] + [high]


# ---- models ---------------------------------------------------------------------------------------------------------------


def up(n: int, multiple: int) -> int:
    return -(-n // multiple) * multiple


def config(case: dict) -> dict:
    """The model's config.json, as far as its numbers go."""
    depth, model = case["depth"], case["model"]
    C, H, G = 64 * depth, depth // 2, case["kv_heads"]
    if model == "nanochat":
        return {"num_hidden_layers": depth, "hidden_size": C, "num_attention_heads": H, "num_key_value_heads": G,
                "intermediate_size": 4 * C, "vocab_size": VOCAB, "rope_theta": THETA}
    mlp = {"ff": up(C * 12 // 5, 128), "kind": "dense"}
    if model == "pudisun":
        rot = {"base": THETA, "dims": ROT, "scaling": {"factor": 4.0, "fast": 32.0, "original": 4096, "slow": 1.0}}
        latent = {"dim": HEAD, "heads": H, "kv_rank": LATENT, "rot_dim": ROT, "vdim": HEAD, "scale": (HEAD + ROT) ** -0.5, "rot": rot}
        gla = {"dim": HEAD, "heads": (H + 1) // 2, "tau": 16.0, "vdim": 2 * HEAD}
        layers = [{"type": "latent_attention" if i % 4 else "gla", "mixer": latent if i % 4 else gla, "mlp": mlp} for i in range(depth)]
        return {"layers": layers, "width": C, "vocab": VOCAB, "norm": {"eps": EPS}, "residual_mult": 0.5, "logit_scale": 0.1}
    rot = {"base": 500000.0, "dims": ROT, "scaling": {"factor": 8.0, "high": 4.0, "low": 1.0, "original": 8192}}
    layers = []
    for i in range(depth):
        mixer = {"conv": CONV, "dim": HEAD, "heads": H, "kv_heads": G, "vdim": HEAD}
        if i % 2:
            mixer.update(rot=rot, scale=HEAD ** -0.5)
            if i % 4 == 3:
                mixer["kv_from"] = i - 2
        layers.append({"type": "attention" if i % 2 else "channel_delta", "mixer": mixer, "mlp": mlp})
    return {"layers": layers, "width": C, "vocab": VOCAB, "norm": {"eps": EPS}, "streams": 2, "embedding": {"scale": 1.0}}


def weights(case: dict, gen: torch.Generator) -> dict:
    """A checkpoint's tensors (bf16): products keep their input's size, what a branch adds is half of it, norms multiply by
    about one, decays reach from a few tokens to thousands."""
    cfg, model, C = config(case), case["model"], 64 * case["depth"]

    def w(*shape, scale=None, base=0.0):
        scale = shape[-1] ** -0.5 if scale is None else scale
        return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.bfloat16).mul_(scale).add_(base)

    if model == "nanochat":
        H, G, ff = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["intermediate_size"]
        state = {"model.embed_tokens.weight": w(VOCAB, C, scale=1.0), "lm_head.weight": w(VOCAB, C)}
        for i in range(case["depth"]):
            p = f"model.layers.{i}."
            state.update({p + "self_attn.q_proj.weight": w(H * HEAD, C), p + "self_attn.k_proj.weight": w(G * HEAD, C),
                          p + "self_attn.v_proj.weight": w(G * HEAD, C), p + "self_attn.o_proj.weight": w(C, H * HEAD),
                          p + "mlp.up_proj.weight": w(ff, C), p + "mlp.down_proj.weight": w(C, ff, scale=0.3 * ff ** -0.5),
                          p + "self_attn.q_norm_weight": w(HEAD, scale=0.1, base=1.0), p + "self_attn.k_norm_weight": w(HEAD, scale=0.1, base=1.0)})
        return state
    one = 1.0 if model == "pudisun" else 0.0  # Rekudra's norms multiply by one plus their weight
    state = {"embed": w(VOCAB, C, scale=1.0), "final.norm": w(C, scale=0.1, base=one)}
    if model == "rekudra":
        state["head"] = w(VOCAB, C)
    for i, entry in enumerate(cfg["layers"]):
        m, p = entry["mixer"], f"l{i}."
        H, D, V, ff = m["heads"], m["dim"], m["vdim"], entry["mlp"]["ff"]
        state.update({p + "norm1": w(C, scale=0.1, base=one), p + "norm2": w(C, scale=0.1, base=one), p + "mlp.gate": w(ff, C),
                      p + "mlp.up": w(ff, C), p + "mlp.down": w(C, ff), p + "mix.o": w(C, H * V, scale=0.5 * (H * V) ** -0.5)})
        if entry["type"] == "gla":
            shapes = {"q": (H * D, C), "k": (H * D, C), "v": (H * V, C), "g": (H * V, C), "a1": (RANK_A, C), "a2": (H * D, RANK_A)}
            state.update({p + "mix.a2.b": w(H * D, scale=1.0, base=2.0), p + "mix.norm": w(V, scale=0.1, base=1.0)})
        elif entry["type"] == "latent_attention":
            shapes = {"q": (H * (D + ROT), C), "dkv": (LATENT + ROT, C), "uk": (H * D, LATENT), "uv": (H * V, LATENT), "g": (H * V, C)}
            state.update({p + "mix.dkv.norm": w(LATENT, scale=0.1, base=1.0), p + "mix.sink": w(H, scale=1.0)})
        else:
            G, delta = m["kv_heads"], entry["type"] == "channel_delta"
            rows = {"q": (G if delta else H) * D, "k": G * D, "v": (H if delta else G) * V}
            rows = {"q": rows["q"]} if "kv_from" in m else rows
            shapes = {n: (count, C) for n, count in rows.items()}
            for n, count in rows.items():
                state[p + f"mix.{n}.conv"] = w(count, CONV, scale=0.2)
                state[p + f"mix.{n}.conv"][:, -1] += 1.0
            if delta:
                shapes.update({"b": (H, C), "a1": (HEAD, C), "a2": (H * D, HEAD), "g1": (HEAD, C), "g2": (H * V, HEAD)})
                state.update({p + "mix.A_log": w(H, scale=0.5), p + "mix.dt_bias": w(H * D, scale=1.0, base=-4.0), p + "mix.norm": w(V, scale=0.1, base=1.0)})
            else:
                shapes["g"] = (H, C)
        state.update({p + "mix." + n: w(*s) for n, s in shapes.items()})
        if model == "rekudra":
            for q in (1, 2):
                state.update({p + f"hc{q}.in": w(2, scale=0.05, base=0.5), p + f"hc{q}.out": w(2, scale=0.1, base=0.5),
                              p + f"hc{q}.mix": w(2, 2, scale=0.05) + torch.eye(2, device=DEV, dtype=torch.bfloat16)})
    return state


def quantised(x: torch.Tensor) -> tuple:
    """Rows (.., 128) -> (e4m3 bytes, fp32 scale): scale = amax / 448."""
    scale = x.abs().amax(-1).float() / 448.0
    return (x.float() / scale[..., None]).to(torch.float8_e4m3fn), scale


def context_of(case: dict, counts: list, gen: torch.Generator) -> list:
    """Per layer and slot what the caches hold of `counts` positions: a dict of tensors per layer, slots in front. nanochat's
    layers hold the same rows."""
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    most, B, cfg = max(max(counts), 1), len(counts), config(case)

    def rows(*shape, scale=1.0, kind=dtype):
        return torch.randn(*shape, generator=gen, device=DEV, dtype=kind).mul_(scale)

    if case["model"] == "nanochat":
        G = cfg["num_key_value_heads"]
        return [{"k": rows(B, G, most, HEAD), "v": rows(B, G, most, HEAD)}]
    found = []
    for entry in cfg["layers"]:
        m = entry["mixer"]
        H, D, V = m["heads"], m["dim"], m["vdim"]
        if entry["type"] == "gla":
            found.append({"state": rows(B, H, D, V, scale=3.0, kind=torch.float32)})
        elif entry["type"] == "latent_attention":
            found.append({"rows": rows(B, most, LATENT + ROT)})
        elif entry["type"] == "channel_delta":
            found.append({"state": rows(B, H, D, V, scale=0.3, kind=torch.float32), "ring": rows(B, CONV, 2 * m["kv_heads"] * D + H * V)})
        elif "kv_from" in m:
            found.append({"ring": rows(B, CONV, H * D)})
        else:
            G = m["kv_heads"]
            found.append({"rows": rows(B, G, most, D + V), "ring": rows(B, CONV, H * D + G * (D + V))})
    return found


def fill_caches(decoder, case: dict, counts: list, context: list) -> None:
    if case["model"] == "nanochat":
        first = decoder.caches[0]
        for slot, n in enumerate(counts):
            if n:
                (kb, ks), (vb, vs) = (quantised(context[0][name][slot, :, :n]) for name in "kv")
                first.write(slot, kb.view(torch.uint8), ks, vb.view(torch.uint8), vs)
        for cache in decoder.caches[1:]:
            cache.pages.copy_(first.pages)
        return
    for cache, held in zip(decoder.caches, context):
        parts = list(cache.parts)
        if "state" in held:
            parts[0].state.copy_(held["state"])
        if "rows" in held:
            n = held["rows"].shape[-2]
            parts[0].rows[..., :n, :].copy_(held["rows"])
        if "ring" in held:
            parts[-1].rows.copy_(held["ring"])


def decoder_of(case: dict, state: dict, slots: int, max_len: int):
    cfg = config(case)
    if case["model"] == "nanochat":
        cfg = DecoderConfig.from_exported(cfg, max_len)
        return Decoder(cfg, DecoderWeights.from_state_dict(state, cfg), slots)
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    cfg = (HybridConfig.from_pudisun if case["model"] == "pudisun" else HybridConfig.from_rekudra)(cfg, max_len)
    cfg.itemsize = dtype.itemsize
    return HybridDecoder(cfg, HybridWeights.from_state_dict(state, cfg, dtype), slots)


def captured_step(decoder, tokens: list, positions: list) -> tuple:
    """The decode step of slots 0 .. as a CUDA graph, longest sequences first: (graph, logits in the order of the slots)."""
    order = sorted(range(len(tokens)), key=lambda b: (-positions[b], b))
    dev_tokens = torch.tensor([tokens[b] for b in order], device=DEV)
    pos, slot_map = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([positions[b] for b in order], order))
    buf = decoder.step_buffers(len(tokens))
    decoder.chunk_pages = decoder.planned_chunk(positions, 1)
    idle = torch.full_like(pos, -1)
    decoder.run_step(dev_tokens, idle, slot_map, buf)  # first-use set-up outside the capture, every slot idle
    torch.cuda.synchronize()
    gc.collect()
    gc.disable()
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            decoder.run_step(dev_tokens, pos, slot_map, buf)
    finally:
        gc.enable()
        decoder.chunk_pages = 0
    return graph, buf["logits"], (dev_tokens, pos, slot_map, buf)


def updated(decoder) -> list:
    """The caches and states of a model whose caches hold floating numbers."""
    found = []
    for cache in decoder.caches:
        found += [part.state if hasattr(part, "state") else part.rows for part in getattr(cache, "parts", []) if hasattr(part, "state") or hasattr(part, "rows")]
    return found


# ---- one pass ---------------------------------------------------------------------------------------------------------------


def inputs(case: dict, seed: int) -> dict:
    """Everything random, in a fixed order."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    if case["kind"] in ("attend", "fill"):
        Hq, G, lens = case["heads"], case["kv_heads"], lengths(case)
        rows = len(lens) if case["kind"] == "attend" else sum(lens)
        made = {"lens": lens, "qkv": torch.randn(rows, (Hq + 2 * G) * HEAD, generator=gen, device=DEV, dtype=torch.bfloat16),
                "gains": torch.randn(2, HEAD, generator=gen, device=DEV).mul_(0.1).add_(1.0)}
        if case["kind"] == "attend":
            made["cached"] = [tuple(quantised(torch.randn(G, n, HEAD, generator=gen, device=DEV)) for _ in "kv") for n in lens]
        return made
    host = torch.Generator().manual_seed(seed)
    made = {"weights": weights(case, gen)}
    if case["kind"] == "feed":
        made["counts"], total = [case["context"]], [case["tokens"]]
    else:
        made["counts"], total = ([n - 1 for n in lengths(case)], [1] * case["batch"]) if case["kind"] == "decode" else ([0] * case["batch"], lengths(case))
    made["tokens"] = [torch.randint(0, VOCAB, (n,), generator=host).tolist() for n in total]
    if max(made["counts"]):
        made["context"] = context_of(case, made["counts"], gen)
    return made


@torch.no_grad()
def prepare(case: dict, seed: int) -> dict:
    made, kind = inputs(case, seed), case["kind"]
    if kind in ("attend", "fill"):
        lens, G = made["lens"], case["kv_heads"]
        cache = ncb.Fp8KVCache(len(lens), G, max(lens), device=DEV)
        state = {"case": case, "qkv": made["qkv"], "gains": made["gains"], "cache": cache, "rotary": ncb.rotary_table(max(lens), THETA, DEV)}
        if kind == "attend":
            for slot, ((kb, ks), (vb, vs)) in enumerate(made["cached"]):
                cache.write(slot, kb.view(torch.uint8), ks, vb.view(torch.uint8), vs)
            order = sorted(range(len(lens)), key=lambda b: -lens[b])  # a caller that knows the lengths lists the longest first
            state["pos"] = torch.tensor([lens[b] - 1 for b in order], dtype=torch.int32, device=DEV)
            state["slot_map"] = torch.tensor(order, dtype=torch.int32, device=DEV)
            state["chunk"] = ops.plan_chunk_pages(lens, G, max(lens), case["window"])
            need = ops.workspace_bytes(len(lens), case["heads"], G, max(lens), state["chunk"])
            state["workspace"] = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
            state["out"] = torch.empty((len(lens), case["heads"], HEAD), dtype=torch.bfloat16, device=DEV)
            return state
        slots = [s for s, n in enumerate(lens) for _ in range(n)]
        positions = [p for n in lens for p in range(n)]
        state["plan"] = ops.PrefillPlan(slots, positions, case["heads"], cache, DEV)
        state["pos"], state["slot_map"] = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in (positions, slots))
        return state
    counts, tokens = made["counts"], made["tokens"]
    longest = max(c + len(t) for c, t in zip(counts, tokens))
    decoder = decoder_of(case, made["weights"], len(tokens), longest + 64)
    state = {"case": case, "decoder": decoder, "tokens": tokens, "counts": counts}
    if kind == "feed":
        if len(tokens[0]) == 1:
            decoder.feed(0, tokens[0], counts[0], [0])  # captures the step, as serving does before its first request
    else:
        state["graph"], state["logits"], state["held"] = captured_step(
            decoder, [t[-1] for t in tokens], [c + len(t) - 1 for c, t in zip(counts, tokens)])
    if "context" in made:
        fill_caches(decoder, case, counts, made["context"])
    return state


@torch.no_grad()
def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "attend":
        cos, sin = state["rotary"]
        out = ops.decode_step_attention(state["qkv"], state["gains"][0], state["gains"][1], cos, sin, state["pos"], state["cache"],
                                        case["heads"], case["longest"], slot_map=state["slot_map"], window=case["window"],
                                        chunk_pages=state["chunk"], workspace=state["workspace"], out=state["out"])
        return {"out": out, "pages": state["cache"].pages}
    if kind == "fill":
        cos, sin = state["rotary"]
        q = ops.kv_append(state["qkv"], state["gains"][0], state["gains"][1], cos, sin, state["pos"], state["cache"], case["heads"],
                          slot_map=state["slot_map"])
        return {"q": q, "out": ops.prefill_attention(q, state["cache"], state["plan"]), "pages": state["cache"].pages}
    decoder, tokens = state["decoder"], state["tokens"]
    if kind == "feed":
        return {"logits": decoder.feed(0, tokens[0], state["counts"][0], [len(tokens[0]) - 1]), "caches": updated(decoder)}
    if kind == "prompts":
        decoder.prefill(tokens, list(range(len(tokens))))
    state["graph"].replay()
    return {"logits": state["logits"], "caches": updated(decoder) if kind == "prompts" else
            [part.state for cache in decoder.caches for part in getattr(cache, "parts", []) if hasattr(part, "state")]}


def work(case: dict) -> dict:
    if case["kind"] in ("attend", "fill"):
        Hq, G, lens = case["heads"], case["kv_heads"], lengths(case)
        if case["kind"] == "attend":
            span = sum(min(n, case["window"] or n) for n in lens)
            return {"bytes": span * G * 264 + len(lens) * HEAD * 2 * (2 * Hq + 2 * G), "flops": 4 * span * Hq * HEAD}
        rows = sum(lens)
        return {"bytes": rows * (HEAD * 2 * (3 * Hq + 2 * G) + 264 * G), "flops": 4 * HEAD * Hq * sum(n * (n + 1) // 2 for n in lens)}
    if case["kind"] == "feed":
        spans = [(case["context"], case["tokens"])]
    else:
        spans = [(n - 1, 1) if case["kind"] == "decode" else (0, n) for n in lengths(case)]
    rows, size = sum(n for _, n in spans), 2 if case["dtype"] == "bf16" else 4
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in spans)
    held, ends = sum(c for c, _ in spans), len(spans)  # what is read of contexts; rows whose logits are wanted
    C, cfg = 64 * case["depth"], config(case)
    params, attend, per_row, state_bytes, cache_bytes = 0, 0, 0, 0, 0  # per_row: a recurrent layer's operations
    if case["model"] == "nanochat":
        H, G = cfg["num_attention_heads"], cfg["num_key_value_heads"]
        params = case["depth"] * (C * HEAD * (2 * H + 2 * G) + 8 * C * C)
        attend, cache_bytes = case["depth"] * 4 * HEAD * H, case["depth"] * G * 264
    else:
        for entry in cfg["layers"]:
            m = entry["mixer"]
            H, D, V = m["heads"], m["dim"], m["vdim"]
            params += C * (3 * entry["mlp"]["ff"] + H * V)
            if entry["type"] == "gla":
                params += C * (2 * H * D + 2 * H * V + RANK_A) + RANK_A * H * D
                state_bytes += 8 * H * D * V
                per_row += 4 * H * D * V
            elif entry["type"] == "latent_attention":
                params += C * (H * (D + ROT) + LATENT + ROT + H * V) + LATENT * H * (D + V)
                attend += 2 * H * (D + ROT + V)
                cache_bytes += (LATENT + ROT) * size
            elif entry["type"] == "channel_delta":
                params += C * (2 * m["kv_heads"] * D + H * V + H + 2 * HEAD) + HEAD * H * (D + V)
                state_bytes += 8 * H * D * V
                per_row += 6 * H * D * V
            else:
                own = "kv_from" not in m
                params += C * (H * D + H + (m["kv_heads"] * (D + V) if own else 0))
                attend += 2 * H * (D + V)
                cache_bytes += m["kv_heads"] * (D + V) * size
    flops = (2 * params + per_row) * rows + 2 * VOCAB * C * ends + attend * pairs
    weight_bytes = size * (params + VOCAB * C)
    return {"bytes": weight_bytes + state_bytes * ends + cache_bytes * (held + rows) + ends * VOCAB * 4, "flops": flops}


def tolerance(case: dict):
    """About four times what one pass is off its value in 64 bits. Cache bytes are the same."""
    if case["kind"] in ("attend", "fill"):
        return {"rel": 1e-2, "max": 0.1}  # 0.0025 off
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-3}  # 1e-6 off
    return {"rel": 0.025, "max": 0.3} if case["model"] != "nanochat" else {"rel": 0.03, "max": 0.5}  # 0.006; 0.02 (fp8 keys and values)


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------------


def rms(x: torch.Tensor, eps: float) -> torch.Tensor:
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def turned(x: torch.Tensor, pos: torch.Tensor, freqs: torch.Tensor, factor: float = 1.0, sign: float = 1.0) -> torch.Tensor:
    """x [n, heads, dims]: dimension i of the first half of the rotated part turns with the same one of the second half."""
    half = freqs.numel()
    angle = pos.to(F64)[:, None, None] * freqs
    c, s = angle.cos() * factor, angle.sin() * (factor * sign)
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)


def plain_frequencies(dims: int, base: float) -> torch.Tensor:
    return base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device=DEV) / dims)


def frequencies64(rot: dict) -> tuple:
    f, s = plain_frequencies(rot["dims"], rot["base"]), rot["scaling"]
    if "low" in s:
        fits = s["original"] * f / (2.0 * math.pi)
        share = ((fits - s["low"]) / (s["high"] - s["low"])).clamp(0.0, 1.0)
        return f / s["factor"] * (1.0 - share) + f * share, 1.0

    def dim_of(turns: float) -> float:
        return rot["dims"] * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))

    lo, hi = max(math.floor(dim_of(s["fast"])), 0), min(math.ceil(dim_of(s["slow"])), rot["dims"] - 1)
    ramp = ((torch.arange(rot["dims"] // 2, dtype=F64, device=DEV) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def attended(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float, sink=None, window: int = 0) -> torch.Tensor:
    """q [n, H, D] of the last n positions, k [N, G, D], v [N, G, V] -> [n, H, V]; blocks of rows, so that scores stay small."""
    n, N, ratio = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    k, v = (t.repeat_interleave(ratio, 1).transpose(0, 1) for t in (k, v))
    out = torch.empty(n, q.shape[1], v.shape[-1], dtype=F64, device=DEV)
    at = torch.arange(N, device=DEV)
    for r in range(0, n, 512):
        rows = torch.arange(r, min(r + 512, n), device=DEV) + N - n
        score = q[r:r + 512].transpose(0, 1) @ k.transpose(1, 2) * scale
        hidden = at[None] > rows[:, None]
        if window:
            hidden |= at[None] <= rows[:, None] - window
        score.masked_fill_(hidden, -math.inf)
        if sink is not None:
            score = torch.cat([score, sink[:, None, None].expand(-1, score.shape[1], 1)], -1)
        out[r:r + 512] = (score.softmax(-1)[..., :N] @ v).transpose(0, 1)
    return out


def stored(x: torch.Tensor) -> torch.Tensor:
    """What the fp8 cache gives back for rows x."""
    b, s = quantised(x)
    return b.to(F64) * s.to(F64)[..., None]


class Rows64:
    """The rows of all sequences one after the other, and where each sequence's are."""

    def __init__(self, made: dict):
        self.counts, sizes = made["counts"], [len(t) for t in made["tokens"]]
        self.tokens = torch.tensor([t for ts in made["tokens"] for t in ts], device=DEV)
        ends = [sum(sizes[:i + 1]) for i in range(len(sizes))]
        self.spans = [slice(e - n, e) for e, n in zip(ends, sizes)]
        self.pos = torch.cat([torch.arange(c, c + n, device=DEV) for c, n in zip(self.counts, sizes)])
        self.last = torch.tensor(ends, device=DEV) - 1
        # [sequence, step] -> row, and which of them exist, for the recurrences
        steps = torch.arange(max(sizes), device=DEV)
        size = torch.tensor(sizes, device=DEV)[:, None]
        self.live = steps[None] < size
        self.row = (self.last[:, None] + 1 - size + steps[None]).clamp(max=len(self.tokens) - 1)


def convolved(x: torch.Tensor, w: torch.Tensor, rows: Rows64, ring) -> torch.Tensor:
    """x [rows, channels], w [channels, taps]; ring [slots, taps, channels]: position p's row at p % taps, of contexts only."""
    out = torch.zeros_like(x)
    for b, span in enumerate(rows.spans):
        c = rows.counts[b]
        before = [torch.zeros_like(x[:1]) if c - j < 0 or ring is None else ring[b, (c - j) % CONV][None].to(F64) for j in range(CONV - 1, 0, -1)]
        full = torch.cat([*before, x[span]])
        out[span] = sum(w[:, j] * full[j:j + span.stop - span.start] for j in range(CONV))
    return out


def recurrence(rows: Rows64, state: torch.Tensor, decay: torch.Tensor, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, beta=None) -> tuple:
    """state [slots, H, D, V]; decay, q, k [rows, H, D], v [rows, H, V] -> ([rows, H, V], the last states). With beta [rows, H] the
    delta rule, else a plain sum."""
    out = torch.zeros_like(v)
    for t in range(rows.row.shape[1]):
        live, at = rows.live[:, t], rows.row[:, t]
        new = decay[at][..., None] * state
        add = v[at] if beta is None else beta[at][..., None] * (v[at] - (new * k[at][..., None]).sum(-2))
        new = new + k[at][..., None] * add[..., None, :]
        state = torch.where(live[:, None, None, None], new, state)
        out[at[live]] = (new * q[at][..., None]).sum(-2)[live]
    return out, state


def unit(x: torch.Tensor) -> torch.Tensor:
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def nanochat64(case: dict, made: dict, rows: Rows64) -> dict:
    cfg, W = config(case), made["weights"]
    H, G = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    freqs, held = plain_frequencies(HEAD, THETA), None
    if "context" in made:
        held = {n: [stored(t[b, :, :c]).transpose(0, 1) for b, c in enumerate(rows.counts)] for n, t in made["context"][0].items()}
    h = rms(W["model.embed_tokens.weight"][rows.tokens].to(F64), NANO_EPS)
    for i in range(case["depth"]):
        w = {n[len(f"model.layers.{i}."):]: t.to(F64) for n, t in W.items() if n.startswith(f"model.layers.{i}.")}
        x = rms(h, NANO_EPS)
        q, k, v = ((x @ w[f"self_attn.{n}_proj.weight"].T).view(len(x), -1, HEAD) for n in "qkv")
        q, k = (turned(rms(t, NANO_EPS) * w[f"self_attn.{n}_norm_weight"], rows.pos, freqs, sign=-1.0) for n, t in (("q", q), ("k", k)))
        k, v = stored(k), stored(v)
        y = torch.empty(len(x), H * HEAD, dtype=F64, device=DEV)
        for b, span in enumerate(rows.spans):
            kb, vb = (t[span] if held is None else torch.cat([held[n][b], t[span]]) for n, t in (("k", k), ("v", v)))
            y[span] = attended(q[span], kb, vb, HEAD ** -0.5).flatten(1)
        h = h + y @ w["self_attn.o_proj.weight"].T
        h = h + F.relu(rms(h, NANO_EPS) @ w["mlp.up_proj.weight"].T).square() @ w["mlp.down_proj.weight"].T
    return {"logits": rms(h[rows.last], NANO_EPS) @ W["lm_head.weight"].to(F64).T, "caches": []}


def hybrid64(case: dict, made: dict, rows: Rows64) -> dict:
    cfg, W, rekudra = config(case), made["weights"], case["model"] == "rekudra"
    states, shared = [], {}
    embedded = W["embed"][rows.tokens].to(F64)
    x = torch.stack([embedded] * 2) if rekudra else embedded
    for i, entry in enumerate(cfg["layers"]):
        w = {n[len(f"l{i}."):]: t.to(F64) for n, t in W.items() if n.startswith(f"l{i}.")}
        m, mix, held = entry["mixer"], {n[4:]: t for n, t in w.items() if n.startswith("mix.")}, made["context"][i] if "context" in made else {}
        H, D, V, n = m["heads"], m["dim"], m["vdim"], len(rows.tokens)

        def branch(which: int, fn):
            if not rekudra:
                return x + cfg["residual_mult"] * fn(rms(x, EPS) * w[f"norm{which}"])
            read, write, mixed = (w[f"hc{which}.{part}"] for part in ("in", "out", "mix"))
            y = fn(rms(torch.einsum("s,snc->nc", read, x), EPS) * (1.0 + w[f"norm{which}"]))
            return torch.einsum("st,snc->tnc", mixed, x) + write[:, None, None] * y

        def fields(h: torch.Tensor, names: str) -> list:
            """Convolved projections; the ring holds them side by side."""
            found, at = [], 0
            for name in names:
                count = mix[name].shape[0]
                ring = held["ring"][..., at:at + count] if "ring" in held else None
                found.append(convolved(h @ mix[name].T, mix[name + ".conv"], rows, ring))
                at += count
            return found

        def start() -> torch.Tensor:
            return held["state"].to(F64) if "state" in held else torch.zeros(len(rows.counts), H, D, V, dtype=F64, device=DEV)

        def mixer(h: torch.Tensor) -> torch.Tensor:
            if entry["type"] == "gla":
                q, k, v = ((h @ mix[name].T).view(n, H, -1) for name in "qkv")
                decay = torch.sigmoid((h @ mix["a1"].T) @ mix["a2"].T + mix["a2.b"]) ** (1.0 / m["tau"])
                o, last = recurrence(rows, start(), decay.view(n, H, D), q * D ** -0.5, k, v)
                states.append(last)
                return ((rms(o, EPS) * mix["norm"]).flatten(1) * F.silu(h @ mix["g"].T)) @ mix["o"].T
            if entry["type"] == "latent_attention":
                freqs, factor = frequencies64(m["rot"])
                q, kv = (h @ mix["q"].T).view(n, H, D + ROT), h @ mix["dkv"].T
                q = torch.cat([q[..., :D], turned(q[..., D:], rows.pos, freqs, factor)], -1)
                kv = torch.cat([rms(kv[:, :LATENT], EPS) * mix["dkv.norm"], turned(kv[:, None, LATENT:], rows.pos, freqs, factor)[:, 0]], -1)
                out = torch.empty(n, H * V, dtype=F64, device=DEV)
                for b, span in enumerate(rows.spans):
                    full = torch.cat([held["rows"][b, :rows.counts[b]].to(F64), kv[span]]) if held else kv[span]
                    c = full[:, :LATENT]
                    k = torch.cat([(c @ mix["uk"].T).view(-1, H, D), full[:, None, LATENT:].expand(-1, H, -1)], -1)
                    out[span] = attended(q[span], k, (c @ mix["uv"].T).view(-1, H, V), m["scale"], mix["sink"]).flatten(1)
                return (out * torch.sigmoid(h @ mix["g"].T)) @ mix["o"].T
            G = m["kv_heads"]
            if entry["type"] == "channel_delta":
                q, k, v = (F.silu(t).view(n, -1, HEAD) for t in fields(h, "qkv"))
                q, k = ((unit(t) * s).repeat_interleave(H // G, 1) for t, s in ((q, D ** -0.5), (k, 1.0)))
                z = F.softplus((h @ mix["a1"].T) @ mix["a2"].T + mix["dt_bias"], threshold=50.0).view(n, H, D)
                o, last = recurrence(rows, start(), torch.exp(-mix["A_log"].exp()[:, None] * z), q, k, v, torch.sigmoid(h @ mix["b"].T))
                states.append(last)
                gate = torch.sigmoid((h @ mix["g1"].T) @ mix["g2"].T).view(n, H, V)
                return (rms(o, EPS) * mix["norm"] * gate).flatten(1) @ mix["o"].T
            freqs, _ = frequencies64(m["rot"])
            own = "kv_from" not in m
            q, *kv = fields(h, "qkv" if own else "q")
            q = rms(turned(q.view(n, H, D), rows.pos, freqs), EPS)
            if own:
                k, v = rms(turned(kv[0].view(n, G, D), rows.pos, freqs), EPS), kv[1].view(n, G, V)
                old = held["rows"].to(F64).transpose(1, 2) if "rows" in held else None
                shared[i] = [tuple(t[span] if old is None else torch.cat([part[b, :rows.counts[b]], t[span]])
                                   for t, part in ((k, None if old is None else old[..., :D]), (v, None if old is None else old[..., D:])))
                             for b, span in enumerate(rows.spans)]
            out = torch.empty(n, H, V, dtype=F64, device=DEV)
            for b, span in enumerate(rows.spans):
                out[span] = attended(q[span], *shared[m.get("kv_from", i)][b], m["scale"])
            return (out * torch.sigmoid(h @ mix["g"].T)[..., None]).flatten(1) @ mix["o"].T

        def feed_forward(h: torch.Tensor) -> torch.Tensor:
            gate = F.silu(h @ w["mlp.gate"].T) if rekudra else F.gelu(h @ w["mlp.gate"].T, approximate="tanh")
            return (gate * (h @ w["mlp.up"].T)) @ w["mlp.down"].T

        x = branch(1, mixer)
        x = branch(2, feed_forward)
    final = W["final.norm"].to(F64)
    if rekudra:
        logits = rms(x[:, rows.last].sum(0), EPS) * (1.0 + final) @ W["head"].to(F64).T
    else:
        logits = rms(x[rows.last], EPS) * final @ W["embed"].to(F64).T * cfg["logit_scale"]
    return {"logits": logits, "caches": states}


@torch.no_grad()
def exact(case: dict, seed: int):
    made, kind = inputs(case, seed), case["kind"]
    if kind in ("attend", "fill"):
        lens, H, G, x = made["lens"], case["heads"], case["kv_heads"], made["qkv"].to(F64)
        order = sorted(range(len(lens)), key=lambda b: -lens[b]) if kind == "attend" else list(range(len(lens)))
        sizes = [1 if kind == "attend" else lens[b] for b in order]
        pos = torch.cat([torch.arange(lens[b] - n, lens[b], device=DEV) for b, n in zip(order, sizes)])
        q, k, v = x.view(len(x), -1, HEAD).split([H, G, G], 1)
        freqs = plain_frequencies(HEAD, THETA)
        q, k = (turned(rms(t, NANO_EPS) * made["gains"][j].to(F64), pos, freqs, sign=-1.0) for j, t in ((0, q), (1, k)))
        k, v, out, at = stored(k), stored(v), torch.empty(len(x), H, HEAD, dtype=F64, device=DEV), 0
        for b, n in zip(order, sizes):
            span, kb, vb = slice(at, at + n), k[at:at + n], v[at:at + n]
            if kind == "attend":
                kb, vb = (torch.cat([(t.to(F64) * s.to(F64)[..., None]).transpose(0, 1)[:-1], new]) for (t, s), new in zip(made["cached"][b], (kb, vb)))
            out[span] = attended(q[span], kb, vb, HEAD ** -0.5, window=case.get("window", 0))
            at += n
        return {"out": out, "pages": None, **({"q": q} if kind == "fill" else {})}
    rows = Rows64(made)
    found = (nanochat64 if case["model"] == "nanochat" else hybrid64)(case, made, rows)
    ends = [c + len(t) for c, t in zip(made["counts"], made["tokens"])]
    order = sorted(range(len(ends)), key=lambda b: (-ends[b], b))
    found["logits"] = found["logits"][torch.tensor(order, device=DEV)]
    if kind == "decode":
        return found
    caches, states = [], iter(found["caches"])
    for entry in config(case).get("layers", []):  # as run() lists them: a state where there is one, rows and rings without
        kind_of, own = entry["type"], "kv_from" not in entry["mixer"]
        caches += {"gla": [0], "latent_attention": [None], "channel_delta": [0, None]}.get(kind_of, [None, None] if own else [None])
    return {"logits": found["logits"], "caches": [next(states) if c == 0 else None for c in caches]}
