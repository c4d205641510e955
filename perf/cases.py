"""Calls that a program serving one of this engine's decoders makes, at the sizes it makes them: what a change of speed is measured on.

Six kinds of case.  "llama": one engine step (`ModelRunner.step`) of a Llama decoder, a batch of single tokens, a portion of a prompt, or
both, from cached keys and values, in bfloat16 or in the true float32 path; its logits at the last place of every request.  "lasapel",
"lanirax": the layers of two other decoders, prompts (and, for Lasapel, single tokens) through `ModelRunner.forward` on a prepared step,
with the logits of every token and the recurrent states.  "gavodra": the two sublayers of a third one's routed layer, each on inputs of its
own (in a whole layer a last bit of the attention decides which of two nearly equal experts a token takes).  "sample": the device's top-k /
top-p sampler.

Everything is made from the seed on the GPU: weights N(0, 0.02) and norm weights N(1, 0.02) as the random-weights mode draws them, cached
keys, values and latent rows of the spread that such weights give, uniform token ids."""

from __future__ import annotations

import math
import struct

import torch

PAGE = 16
DEVICE = "cuda"

# The sizes of the Llama family that the benchmark serves (hidden, layers' heads, key/value heads, head size, feed-forward, rotary factor).
LLAMA = {
    "1b": dict(hidden=2048, heads=32, kv_heads=8, dim=64, ff=8192, factor=32.0, tied=True),
    "3b": dict(hidden=3072, heads=24, kv_heads=8, dim=128, ff=8192, factor=32.0, tied=True),
    "8b": dict(hidden=4096, heads=32, kv_heads=8, dim=128, ff=14336, factor=8.0, tied=False),
}


def listed():
    return [
        # One user, a short conversation: the smallest engine step, over half of the benchmark model's 16 layers.
        dict(name="decode_1", kind="llama", sizes="1b", layers=8, vocab=128256, dtype="bfloat16", decode=1, context=512, ragged=0.0, chunk=0, start=0),
        # The headline: eight users at 4,096 tokens of context, the whole model.
        dict(name="decode_8", kind="llama", sizes="1b", layers=16, vocab=128256, dtype="bfloat16", decode=8, context=4096, ragged=0.0, chunk=0, start=0),
        # A full batch of the 8B sizes at ragged long contexts (two of its layers: the others repeat them).
        dict(name="decode_32_long", kind="llama", sizes="8b", layers=2, vocab=32000, dtype="bfloat16", decode=32, context=8190, ragged=0.4, chunk=0, start=0),
        # The other headline: a prompt of 2,048 tokens, run whole through half of the layers.
        dict(name="prefill_2048", kind="llama", sizes="1b", layers=8, vocab=128256, dtype="bfloat16", decode=0, context=0, ragged=0.0, chunk=2048, start=0),
        # Continuous batching with chunked prefill at the 3B sizes: 39 users decode while a portion of a prompt runs, starting inside it.
        dict(name="mixed_512", kind="llama", sizes="3b", layers=4, vocab=32000, dtype="bfloat16", decode=39, context=2100, ragged=0.9, chunk=509, start=1024),
        # The true float32 path, which the logits are checked with: tokens one by one, and a prompt.
        dict(name="fp32_decode_8", kind="llama", sizes="1b", layers=4, vocab=32000, dtype="float32", decode=8, context=2048, ragged=0.3, chunk=0, start=0),
        dict(name="fp32_prefill_700", kind="llama", sizes="1b", layers=2, vocab=32000, dtype="float32", decode=0, context=0, ragged=0.0, chunk=700, start=0),
        # Lasapel: a layer with the decayed recurrence and one with attention over latents; a prompt, and eight users at 4,096 tokens.
        dict(name="lasapel_prompt", kind="lasapel", width=2048, prompts=1, tokens=2048, decode=0, context=0),
        dict(name="lasapel_decode_8", kind="lasapel", width=2048, prompts=0, tokens=0, decode=8, context=4096),
        # Lanirax: window attention beside the gated delta rule, two prompts of together an odd number of tokens.
        dict(name="lanirax_prompt", kind="lanirax", width=2048, prompts=2, tokens=1501),
        # Gavodra: attention with a distance bias, and 4 of 32 experts beside a shared one, over a prompt.
        dict(name="gavodra_prompt", kind="gavodra", width=2048, prompts=1, tokens=2048),
        # One token for each of 64 users with temperature, top-p and top-k, at the Llama vocabulary.
        dict(name="sample_64", kind="sample", rows=64, vocab=128256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["llama", "llama", "llama", "llama32", "lasapel", "lanirax", "gavodra", "sample"])
    if kind == "llama":
        sizes = rng.choice(["1b", "1b", "3b", "8b"])
        decode, chunk = rng.choice([(True, False), (True, False), (False, True), (True, True)])
        case = dict(kind="llama", sizes=sizes, layers=_log(rng, 2, {"1b": 8, "3b": 5, "8b": 3}[sizes]), vocab=rng.choice([32000, 128256]), dtype="bfloat16",
                    decode=0, context=0, ragged=0.0, chunk=0, start=0)
        if decode:
            case.update(decode=_log(rng, 1, 64), ragged=rng.choice([0.0, 0.4, 0.9]))
            case["context"] = _log(rng, 64, min(8192, 262144 // case["decode"]))
        if chunk:
            case.update(chunk=_log(rng, 16, 1024 if decode else 2048), start=rng.choice([0, 0, _log(rng, 16, 2048)]))
        return case
    if kind == "llama32":
        whole = rng.random() < 0.5
        case = dict(kind="llama", sizes=rng.choice(["1b", "1b", "3b"]), layers=1, vocab=32000, dtype="float32", decode=0, context=0, ragged=0.0, chunk=0, start=0)
        if whole:
            case["chunk"] = _log(rng, 17, 700)
        else:
            case.update(decode=_log(rng, 1, 16), context=_log(rng, 64, 2048), ragged=rng.choice([0.0, 0.5]), layers=rng.choice([1, 2, 3]))
        return case
    width = rng.choice([1024, 2048])
    if kind == "lasapel" and rng.random() < 0.5:
        return dict(kind="lasapel", width=width, prompts=0, tokens=0, decode=_log(rng, 1, 16), context=_log(rng, 64, 4096))
    if kind == "lasapel":
        return dict(kind="lasapel", width=width, prompts=rng.randint(1, 4), tokens=_log(rng, 128, 2048), decode=0, context=0)
    if kind in ("lanirax", "gavodra"):
        return dict(kind=kind, width=width, prompts=rng.randint(1, 4), tokens=_log(rng, 128, 2048))
    return dict(kind="sample", rows=_log(rng, 1, 64), vocab=rng.choice([32000, 50257, 128256]))


# ---- the requests of a case -----------------------------------------------------------------------------------------------------------


def _cut(total, parts):
    """`total` tokens in `parts` unequal portions of at least two."""
    weights = [3 + (5 * i) % 7 for i in range(parts)]
    sizes = [max(2, total * w // sum(weights)) for w in weights]
    sizes[0] += total - sum(sizes)
    return sizes


def _requests(case):
    """(tokens cached before, tokens now) of every request of the step."""
    if case["kind"] != "llama":
        one = [(case["context"] - 1, 1)] * case["decode"] if case.get("decode") else []
        return one + [(0, n) for n in (_cut(case["tokens"], case["prompts"]) if case["prompts"] else [])]
    out = []
    for i in range(case["decode"]):
        back = int(case["ragged"] * case["context"] * ((i * 37) % 101) / 101)
        out.append((max(1, case["context"] - back - 1), 1))
    if case["chunk"]:
        out.append((case["start"], case["chunk"]))
    return out


def _generator(seed, *what):
    g = torch.Generator(device=DEVICE)
    g.manual_seed((seed * 1000003 + sum((i + 1) * 7919 * (w + 1) for i, w in enumerate(what))) % (1 << 62))
    return g


def _tokens(case, seed, vocab):
    g = torch.Generator().manual_seed(seed * 17 + 3)
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for _, n in _requests(case)]


# ---- configurations and weights -------------------------------------------------------------------------------------------------------

MATRIX, NORM, OFFSET, GAIN, TAPS = (0.0, 0.02), (1.0, 0.02), (0.0, 0.1), (0.0, 1.0), (0.0, 0.5)
SMALL_VOCAB = 1024      # of the cases that ask for the logits of every token


def _llama(case):
    s, V, L = LLAMA[case["sizes"]], case["vocab"], case["layers"]
    H, d = s["hidden"], s["dim"]
    config = {
        "architectures": ["LlamaForCausalLM"], "hidden_size": H, "intermediate_size": s["ff"], "num_hidden_layers": L, "num_attention_heads": s["heads"],
        "num_key_value_heads": s["kv_heads"], "head_dim": d, "vocab_size": V, "rms_norm_eps": 1e-5, "rope_theta": 500000.0,
        "max_position_embeddings": 131072, "tie_word_embeddings": s["tied"],
        "rope_scaling": {"rope_type": "llama3", "factor": s["factor"], "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                         "original_max_position_embeddings": 8192}}
    t = {"model.embed_tokens.weight": ((V, H), MATRIX), "model.norm.weight": ((H,), NORM)}
    if not s["tied"]:
        t["lm_head.weight"] = ((V, H), MATRIX)
    for i in range(L):
        p = "model.layers.%d." % i
        t[p + "input_layernorm.weight"] = t[p + "post_attention_layernorm.weight"] = ((H,), NORM)
        t[p + "self_attn.q_proj.weight"] = ((s["heads"] * d, H), MATRIX)
        t[p + "self_attn.k_proj.weight"] = t[p + "self_attn.v_proj.weight"] = ((s["kv_heads"] * d, H), MATRIX)
        t[p + "self_attn.o_proj.weight"] = ((H, s["heads"] * d), MATRIX)
        t[p + "mlp.gate_proj.weight"] = t[p + "mlp.up_proj.weight"] = ((s["ff"], H), MATRIX)
        t[p + "mlp.down_proj.weight"] = ((H, s["ff"]), MATRIX)
    return config, t


def _lasapel(case):
    """The recurrent and the latent layer of the benchmark's Lasapel, without feed-forwards."""
    W, V = case["width"], SMALL_VOCAB
    H = W // 128
    lat = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 3 * W // 4, "kv_rank": 512, "scale": (128 + 64) ** -0.5,
           "rot": {"dims": 64, "base": 10000.0, "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    lin = {"heads": H, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - 3 * h / max(1, H - 1)) for h in range(H)]}
    config = {"architecture": "Lasapel", "vocab": V, "width": W, "norm": {"eps": 1e-6},
              "layers": [{"type": "lightning", "mixer": lin, "mlp": None}, {"type": "latent_attention", "mixer": lat, "mlp": None}]}
    t = {"embed": ((V, W), MATRIX), "head": ((V, W), MATRIX), "final.norm": ((W,), OFFSET)}
    for i in range(2):
        t["l%d.norm1" % i] = t["l%d.norm1b" % i] = ((W,), OFFSET)
        t["l%d.ls1" % i] = ((W,), NORM)
        t["l%d.mix.o" % i] = ((W, H * 128), MATRIX)
    for n in "qkvg":
        t["l0.mix." + n] = ((H * 128, W), MATRIX)
    t["l0.mix.norm"] = ((H * 128,), NORM)
    p, r = "l1.mix.", lat["q_rank"]
    t.update({p + "dq": ((r, W), MATRIX), p + "dq.norm": ((r,), NORM), p + "uq": ((H * 192, r), MATRIX), p + "dkv": ((576, W), MATRIX), p + "dkv.norm": ((512,), NORM),
              p + "uk": ((H * 128, 512), MATRIX), p + "uv": ((H * 128, 512), MATRIX), p + "sink": ((H,), GAIN)})
    return config, t


def _lanirax(case):
    """A parallel layer of the benchmark's Lanirax: a window of 1,024 over heads of 64, and the delta rule over heads of 128 x 128."""
    W, V = case["width"], SMALL_VOCAB
    rot = {"dims": 48, "base": 10000.0, "scaling": {"factor": 4.0, "original": 8192, "fast": 16.0, "slow": 2.0}}
    left = {"heads": W // 64, "kv_heads": W // 256, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": 1024}, "rot": rot}
    right = {"heads": W // 128, "kv_heads": W // 256, "dim": 128, "vdim": 128, "conv": 4}
    config = {"architecture": "Lanirax", "vocab": V, "width": W, "norm": {"eps": 1e-5}, "postln_alpha": 2.0,
              "layers": [{"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": None}]}
    t = {"embed": ((V, W), MATRIX), "embed.norm": ((W,), NORM), "head": ((V, W), MATRIX), "final.norm": ((W,), NORM), "l0.norm1": ((W,), NORM)}
    p = "l0.mix.left."
    t.update({p + "q": ((W, W), MATRIX), p + "k": ((W // 4, W), MATRIX), p + "sink": ((W // 64,), GAIN), p + "o": ((W, W), MATRIX), p + "out": ((W,), NORM)})
    p, H, qk = "l0.mix.right.", right["heads"], right["kv_heads"] * 128
    t.update({p + "q": ((qk, W), MATRIX), p + "k": ((qk, W), MATRIX), p + "v": ((W, W), MATRIX), p + "g": ((W, W), MATRIX), p + "o": ((W, W), MATRIX),
              p + "q.conv": ((qk, 4), TAPS), p + "k.conv": ((qk, 4), TAPS), p + "v.conv": ((W, 4), TAPS), p + "b": ((H, W), MATRIX), p + "a": ((H, W), MATRIX),
              p + "A_log": ((H,), OFFSET), p + "dt_bias": ((H,), OFFSET), p + "norm": ((128,), NORM), p + "out": ((W,), NORM)})
    return config, t


def _gavodra(case):
    """A routed layer of the benchmark's Gavodra."""
    W, V, E = case["width"], SMALL_VOCAB, 32
    H, ff = W // 64, W // 2
    mix = {"heads": H, "kv_heads": H // 4, "dim": 64, "vdim": 64, "scale": 0.125, "bias_max": 128, "v_mix": False, "bias_rows": 48}
    moe = {"kind": "moe", "expert": {"ff": ff, "limit": 7.0}, "router": {"experts": E, "top": 4, "scale": 2.5}, "shared": {"ff": ff, "limit": 7.0}}
    config = {"architecture": "Gavodra", "vocab": V, "width": W, "norm": {"eps": 1e-5}, "residual_mult": 0.5, "embedding": {"scale": 8.0}, "logit_scale": 0.5,
              "logit_softcap": 30.0, "layers": [{"type": "attention", "mixer": mix, "mlp": moe}]}
    t = {"embed": ((V, W), MATRIX), "final.norm": ((W,), NORM), "l0.norm1": ((W,), NORM), "l0.norm2": ((W,), NORM)}
    p = "l0.mix."
    t.update({p + "q": ((W, W), MATRIX), p + "k": ((W // 4, W), MATRIX), p + "v": ((W // 4, W), MATRIX), p + "o": ((W, W), MATRIX), p + "g": ((H, W), MATRIX),
              p + "q.norm": ((64,), NORM), p + "k.norm": ((64,), NORM), p + "rel": ((48, H), OFFSET)})
    p = "l0.mlp."
    for q in ["e%d." % e for e in range(E)] + ["shared."]:
        t.update({p + q + "gate": ((ff, W), MATRIX), p + q + "up": ((ff, W), MATRIX), p + q + "down": ((W, ff), MATRIX)})
    t.update({p + "router": ((E, W), MATRIX), p + "correction": ((E,), OFFSET), p + "shared.sg": ((1, W), MATRIX)})
    return config, t


MODELS = {"llama": _llama, "lasapel": _lasapel, "lanirax": _lanirax, "gavodra": _gavodra}


def _weights(case, seed):
    """The configuration, and the tensors as a checkpoint stores them."""
    config, shapes = MODELS[case["kind"]](case)
    g, dtype = _generator(seed, 1), torch.float32 if case.get("dtype") == "float32" else torch.bfloat16
    return config, {n: (torch.randn(shape, generator=g, device=DEVICE) * std + mean).to(dtype) for n, (shape, (mean, std)) in shapes.items()}


def _cached_rows(case, seed, b, layer):
    """What request b has in a layer's cache, in the order of its tokens: keys and values [tokens, heads, dim] (Llama), or latent rows."""
    n, g = _requests(case)[b][0], _generator(seed, 2, b, layer)
    if case["kind"] == "lasapel":
        return torch.randn((n, 576), generator=g, device=DEVICE).to(torch.bfloat16)
    s = LLAMA[case["sizes"]]
    kv = 0.02 * math.sqrt(s["hidden"]) * torch.randn((2, n, s["kv_heads"], s["dim"]), generator=g, device=DEVICE)
    return kv if case["dtype"] == "float32" else kv.to(torch.bfloat16)


def _inputs(case, seed):
    """What the sublayers of a Gavodra layer read: rows of the residual stream, once for each."""
    x = torch.randn((2, case["tokens"], case["width"]), generator=_generator(seed, 5), device=DEVICE)
    return (0.6 * x).to(torch.bfloat16).unbind(0)


def _cached_states(case, seed):
    """The recurrent states of Lasapel's requests that decode, [requests, heads, value, key]."""
    H = case["width"] // 128
    return torch.randn((case["decode"], H, 128, 128), generator=_generator(seed, 3), device=DEVICE)


# ---- what is timed --------------------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    from rust_llm_inference_server_b200.cache import CacheStorage, make_cache_manager, plan_groups
    from rust_llm_inference_server_b200.engine import ModelRunner, StepEntry
    from rust_llm_inference_server_b200.models import build_model
    from rust_llm_inference_server_b200.weights.safetensors_io import Checkpoint

    config, tensors = _weights(case, seed)
    model = build_model(config, case.get("dtype", "bfloat16"))
    model.load(Checkpoint(tensors=tensors))
    del tensors
    requests = _requests(case)
    longest = max(s + n for s, n in requests)
    groups = plan_groups(model.cache_slot_specs, PAGE)
    for group in groups:
        group.num_pages = sum(-(-(s + n) // PAGE) for s, n in requests) + 1
    cache = make_cache_manager(groups, len(requests))
    storage = CacheStorage(groups, model.call_state_specs, len(requests), model.dtype, model.device)
    runner = ModelRunner(model, cache, storage, max_seq_len=longest)
    slots = [cache.acquire_state_slot(b) for b in range(len(requests))]
    for upto in range(4 * PAGE, longest + 4 * PAGE, 4 * PAGE):      # requests that grow side by side: their pages lie among each other
        for b, (s, n) in enumerate(requests):
            if upto - 4 * PAGE < s + n and not cache.reserve(b, min(upto, s + n)):
                raise RuntimeError("the pool is too small")
    every = case["kind"] != "llama"
    entries = [StepEntry(b, tokens, s, list(range(n)) if every else [n - 1])
               for b, (tokens, (s, n)) in enumerate(zip(_tokens(case, seed, model.spec.vocab_size), requests))]
    step = runner.prepare(entries)
    step.materialize()
    for layer in range(len(model.cache_slot_specs)):
        rows = storage.layer_cache(layer)
        for b, (s, _) in enumerate(requests):
            if rows is None or s == 0:
                continue
            pages = step.block_tables[rows.group][b, :-(-s // PAGE)].long()
            kept = _cached_rows(case, seed, b, layer)
            for pool, x in zip((rows.k, rows.v), (kept[:, None],) if case["kind"] == "lasapel" else kept):
                padded = x.new_zeros((len(pages) * PAGE,) + tuple(x.shape[1:]))
                padded[:s] = x
                pool[pages] = padded.view(len(pages), PAGE, *x.shape[1:]).transpose(1, 2)
    if every and slots != sorted(slots):
        raise RuntimeError("requests are expected in the order of their state slots")
    state = dict(runner=runner, entries=entries, step=step if every else None, storage=storage)
    if case["kind"] == "gavodra":
        state.update(block=model.blocks[0], inputs=_inputs(case, seed))
    if case.get("decode") and not case.get("chunk"):        # a serving process has recorded the graph of a decode shape long ago
        for _ in range(runner.GRAPH_AFTER_STEPS + 1):
            run(state)
    if case["kind"] == "lasapel" and case["decode"]:        # (the steps above have moved the states on)
        storage.states[0].copy_(_cached_states(case, seed))
    return state


def _bits(x):
    return struct.unpack("<i", struct.pack("<f", x))[0]


def _prepare_sample(case, seed):
    """Logits as a model gives them, and per row a temperature, top-p or top-k or both, and a uniform number of 53 bits."""
    g, R = _generator(seed, 4), case["rows"]
    logits = 3.0 * torch.randn((R, case["vocab"]), generator=g, device=DEVICE)
    u = torch.randint(0, 1 << 31, (R, 2), generator=g, device=DEVICE, dtype=torch.int64)
    rows = [[_bits(1.0 / (0.7, 0.8, 1.0)[r % 3]), (0, 50, 0, 40)[r % 4], _bits((0.9, 1.0, 0.95, 0.9)[r % 4])] for r in range(R)]
    params = torch.cat([torch.tensor(rows, dtype=torch.int64, device=DEVICE), u[:, :1], u[:, 1:] >> 10], dim=1).to(torch.int32)
    return dict(logits=logits, params=params.contiguous())


def run(state):
    if "logits" in state:
        from rust_llm_inference_server_b200 import ops
        return ops.sample_filtered(state["logits"], state["params"])
    if state["step"] is None:
        return state["runner"].step(state["entries"])
    if "block" in state:
        (a, b), block, step, storage = state["inputs"], state["block"], state["step"], state["storage"]
        return {"attention": block.mixer.forward(a, step, storage.layer_cache(0), None), "experts": block.feed_forward.forward(b, step)}
    out = {"logits": state["runner"].forward(state["step"])}
    for i, s in enumerate(state["storage"].states):
        if s is not None:
            out["state%d" % i] = s
    return out


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 0.0}
    config, shapes = MODELS[case["kind"]](case)
    requests, size = _requests(case), 4 if case.get("dtype") == "float32" else 2
    T = sum(n for _, n in requests)
    numbers = lambda names: sum(math.prod(shapes[n][0]) for n in names)
    experts = [n for n in shapes if ".mlp.e" in n and n.split(".")[2][1:].isdigit()]
    embed = [n for n in shapes if "embed" in n]
    head = embed if not any(n in shapes for n in ("head", "lm_head.weight")) else [n for n in shapes if n in ("head", "lm_head.weight")]
    dense = numbers(n for n in shapes if n not in experts and n not in embed and n not in head)
    wanted = len(requests) if case["kind"] == "llama" else T if case["kind"] != "gavodra" else 0
    V = config.get("vocab") or config["vocab_size"]
    per_pair = numbers(experts) / 32
    flops = 2.0 * T * dense + 2.0 * wanted * numbers(head) + 2.0 * T * 4 * per_pair
    bytes_ = size * (dense + (numbers(head) if wanted else 0) + min(32, 4 * T) * per_pair) + 4.0 * wanted * V
    window = 1024 if case["kind"] == "lanirax" else 1 << 40
    seen = sum(min(s + i + 1, window) for s, n in requests for i in range(n))
    if case["kind"] == "llama":
        s = LLAMA[case["sizes"]]
        row = 2 * s["kv_heads"] * s["dim"] * case["layers"] * size
        return {"bytes": bytes_ + row * sum(a + n for a, n in requests), "flops": flops + 4.0 * seen * s["heads"] * s["dim"] * case["layers"]}
    W = case["width"]
    if case["kind"] == "lasapel":
        state = len(requests) * W // 128 * 128 * 128 * 4
        return {"bytes": bytes_ + (2 if case["decode"] else 1) * state + 576 * size * sum(a + n for a, n in requests),
                "flops": flops + 4.0 * T * W * 128 + 2.0 * seen * (W // 128) * (576 + 512)}
    if case["kind"] == "lanirax":
        return {"bytes": bytes_ + len(requests) * W * 128 * 4, "flops": flops + 4.0 * seen * W + 8.0 * T * W * 128}
    return {"bytes": bytes_ + (4 * W + W // 2) * T * size, "flops": flops + 4.0 * seen * W}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"      # token ids by integer arithmetic on the same 32-bit exponentials
    if case.get("dtype") == "float32":
        return {"rel": 4e-5}
    # Off 64 bits by 0.017 to 0.023 after 16 Llama layers and by 0.010 to 0.013 after 2 to 5, by 0.002 to 0.005 after the others' one or two.
    return {"rel": 0.03 if case["kind"] == "llama" else 0.012}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------------------


def exact(case, seed):
    if case["kind"] == "sample":
        return None
    config, tensors = _weights(case, seed)
    w = lambda n: tensors[n].double()
    tokens = [torch.tensor(t, device=DEVICE) for t in _tokens(case, seed, config.get("vocab") or config["vocab_size"])]
    return EXACT[case["kind"]](case, seed, config, w, tokens)


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(q, k, v, start, scale, window=None, bias=None, sink=None):
    """q [n, H, d] at positions start.., k and v [start + n, G, .]: causal attention, a group of query heads at a time."""
    n, H, _ = q.shape
    G, per = k.shape[1], H // k.shape[1]
    back = (start + torch.arange(n, device=DEVICE))[:, None] - torch.arange(k.shape[0], device=DEVICE)[None, :]
    hidden = (back < 0) | (back >= (window or 1 << 40))
    out = torch.empty((n, H, v.shape[2]), dtype=torch.float64, device=DEVICE)
    for g in range(G):
        hs = slice(g * per, (g + 1) * per)
        s = torch.einsum("nhd,kd->hnk", q[:, hs], k[:, g]) * scale
        if bias is not None:
            s = s + bias[back.clamp(min=0)][:, :, hs].permute(2, 0, 1)
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:        # one more term of the denominator
            s = torch.cat([s, sink[hs][:, None, None].expand(-1, n, 1)], dim=2)
        p = torch.softmax(s, dim=2)[:, :, :k.shape[0]]
        out[:, hs] = torch.einsum("hnk,kd->nhd", p, v[:, g])
    return out


def _exact_llama(case, seed, config, w, tokens):
    s, eps = LLAMA[case["sizes"]], config["rms_norm_eps"]
    d, H, G = s["dim"], s["heads"], s["kv_heads"]
    f = 500000.0 ** (-torch.arange(0, d, 2, dtype=torch.float64, device=DEVICE) / d)
    turns = 8192 * f / (2 * math.pi)        # over the original context: slow frequencies are divided, those between blended
    smooth = ((turns - 1.0) / (4.0 - 1.0)).clamp(0.0, 1.0)
    f = f * smooth + f / s["factor"] * (1.0 - smooth)
    requests = _requests(case)
    at = [slice(e - n, e) for (_, n), e in zip(requests, torch.tensor([n for _, n in requests]).cumsum(0).tolist())]
    angle = torch.cat([torch.arange(a, a + n, dtype=torch.float64, device=DEVICE) for a, n in requests])[:, None] * f
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def rotate(x):
        a, b = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)

    x = w("model.embed_tokens.weight")[torch.cat(tokens)]
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        h = _unit(x, eps) * w(p + "input_layernorm.weight")
        q = rotate((h @ w(p + "self_attn.q_proj.weight").T).view(-1, H, d))
        k = rotate((h @ w(p + "self_attn.k_proj.weight").T).view(-1, G, d))
        v = (h @ w(p + "self_attn.v_proj.weight").T).view(-1, G, d)
        o = []
        for b, (a, n) in enumerate(requests):
            kept = _cached_rows(case, seed, b, i).double()
            o.append(_attend(q[at[b]], torch.cat([kept[0], k[at[b]]]), torch.cat([kept[1], v[at[b]]]), a, d ** -0.5))
        x = x + torch.cat(o).flatten(1) @ w(p + "self_attn.o_proj.weight").T
        h = _unit(x, eps) * w(p + "post_attention_layernorm.weight")
        x = x + (_silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    x = _unit(x[torch.tensor([a.stop - 1 for a in at], device=DEVICE)], eps) * w("model.norm.weight")
    return x @ w("model.embed_tokens.weight" if s["tied"] else "lm_head.weight").T


def _yarn(rot):
    """Frequencies of the rotated pairs, blended by how often they turn over the original context, and the factor on cos and sin."""
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEVICE)
    f = base ** (-2.0 * i / dims)
    pair = lambda turns: dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(pair(sc["fast"])), 0), min(math.ceil(pair(sc["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _exact_lasapel(case, seed, config, w, tokens):
    eps, requests, H = 1e-6, _requests(case), case["width"] // 128
    lin, lat = (layer["mixer"] for layer in config["layers"])
    zero = lambda x, name: _unit(x, eps) * (1.0 + w(name))
    decay = torch.tensor(lin["decay"], dtype=torch.float64, device=DEVICE)[:, None, None]
    f, mult = _yarn(lat["rot"])
    first = _cached_states(case, seed).double() if case["decode"] else None
    outs, states = [], []
    for b, (start, n) in enumerate(requests):
        x = w("embed")[tokens[b]]
        h = zero(x, "l0.norm1")
        q, k, v = (_silu(h @ w("l0.mix." + m).T).view(n, H, 128) for m in "qkv")
        S = first[b] if first is not None else torch.zeros((H, 128, 128), dtype=torch.float64, device=DEVICE)     # [head, value, key]
        o = torch.empty_like(v)
        for t in range(n):
            S = decay * S + v[t, :, :, None] * k[t, :, None, :]
            o[t] = (S @ q[t, :, :, None])[..., 0]
        states.append(S)
        y = (_unit(o.flatten(1), eps) * w("l0.mix.norm") * torch.sigmoid(h @ w("l0.mix.g").T)) @ w("l0.mix.o").T
        x = x + w("l0.ls1") * zero(y, "l0.norm1b")
        h, p = zero(x, "l1.norm1"), "l1.mix."
        angle = torch.arange(start, start + n, dtype=torch.float64, device=DEVICE)[:, None] * f
        cos, sin = angle.cos() * mult, angle.sin() * mult
        turn = lambda z, c, s: torch.cat([z[..., :32] * c - z[..., 32:] * s, z[..., 32:] * c + z[..., :32] * s], dim=-1)
        z = h @ w(p + "dkv").T
        rows = torch.cat([_unit(z[:, :512], eps) * w(p + "dkv.norm"), turn(z[:, 512:], cos, sin)], dim=1)
        rows = torch.cat([_cached_rows(case, seed, b, 1).double(), rows])
        q = ((_unit(h @ w(p + "dq").T, eps) * w(p + "dq.norm")) @ w(p + "uq").T).view(n, H, 192)
        folded = torch.einsum("nhd,hdr->nhr", q[..., :128], w(p + "uk").view(H, 128, 512))
        q = torch.cat([folded, turn(q[..., 128:], cos[:, None], sin[:, None])], dim=2)
        a = _attend(q, rows[:, None], rows[:, None, :512], start, lat["scale"], sink=w(p + "sink"))
        y = torch.einsum("nhr,hdr->nhd", a, w(p + "uv").view(H, 128, 512)).flatten(1) @ w(p + "o").T
        outs.append(zero(x + w("l1.ls1") * zero(y, "l1.norm1b"), "final.norm") @ w("head").T)
    return {"logits": torch.cat(outs), "state0": torch.stack(states)}


def _exact_lanirax(case, seed, config, w, tokens):
    eps = 1e-5
    left, right = (config["layers"][0]["mixer"][m] for m in ("left", "right"))
    H, G = right["heads"], right["kv_heads"]
    freqs, mult = _yarn(left["rot"])
    outs, states = [], []
    for ids in tokens:
        n = len(ids)
        x = _unit(w("embed")[ids], eps) * w("embed.norm")
        p = "l0.mix.left."
        angle = torch.arange(n, dtype=torch.float64, device=DEVICE)[:, None] * freqs
        cos, sin = angle.cos()[:, None] * mult, angle.sin()[:, None] * mult

        def turned(z):
            u, v = z[..., 0:48:2], z[..., 1:48:2]
            return _unit(torch.cat([torch.stack([u * cos - v * sin, v * cos + u * sin], dim=-1).flatten(-2), z[..., 48:]], dim=-1), eps)

        q, k = (x @ w(p + "q").T).view(n, -1, 64), (x @ w(p + "k").T).view(n, -1, 64)
        a = _attend(turned(q), turned(k), k, 0, 0.125, window=1024, sink=w(p + "sink")).flatten(1) @ w(p + "o").T
        p = "l0.mix.right."

        def conv(m):
            z = torch.cat([torch.zeros((3, w(p + m).shape[0]), dtype=torch.float64, device=DEVICE), x @ w(p + m).T])
            return _silu(sum(z[j:j + n] * w(p + m + ".conv")[:, j] for j in range(4))).view(n, -1, 128), z[n:]

        (q, tail_q), (k, tail_k), (v, tail_v) = conv("q"), conv("k"), conv("v")
        q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * 128 ** -0.5).repeat_interleave(H // G, dim=1)
        k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)
        beta = torch.sigmoid(x @ w(p + "b").T)
        decay = torch.exp(-torch.exp(w(p + "A_log")) * torch.nn.functional.softplus(x @ w(p + "a").T + w(p + "dt_bias")))
        S = torch.zeros((H, 128, 128), dtype=torch.float64, device=DEVICE)         # [head, value, key]
        o = torch.empty_like(v)
        for t in range(n):
            S = decay[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + u[:, :, None] * k[t][:, None, :]
            o[t] = (S @ q[t][:, :, None])[..., 0]
        b = ((_unit(o, eps) * w(p + "norm")).flatten(1) * _silu(x @ w(p + "g").T)) @ w(p + "o").T
        mixed = 0.5 * (_unit(a, eps) * w("l0.mix.left.out") + _unit(b, eps) * w(p + "out"))
        x = _unit(2.0 * x + mixed, eps) * w("l0.norm1")
        outs.append((_unit(x, eps) * w("final.norm")) @ w("head").T)
        # the state ends in the convolutions' last three inputs
        states.append(torch.cat([S.flatten(), torch.cat([tail_q, tail_k, tail_v], dim=1).flatten()]))
    return {"logits": torch.cat(outs), "state0": torch.stack(states)}


def _exact_gavodra(case, seed, config, w, tokens):
    eps, rows, far = 1e-5, 48, 128.0
    a, x = (t.double() for t in _inputs(case, seed))
    outs = []
    for h in a.split([len(t) for t in tokens]):
        n, p = len(h), "l0.mix."
        q, k = (_unit((h @ w(p + m).T).view(n, -1, 64), eps) * w(p + m + ".norm") for m in "qk")
        v = (h @ w(p + "v").T).view(n, -1, 64)
        log_rows = lambda i: int(math.log(i / (rows // 2)) / math.log(far / (rows // 2)) * (rows - rows // 2))
        bucket = [i if i < rows // 2 else min(rows - 1, rows // 2 + log_rows(i)) for i in range(n)]
        o = _attend(q, k, v, 0, 0.125, bias=w(p + "rel")[torch.tensor(bucket, device=DEVICE)])
        outs.append((o * torch.sigmoid(h @ w(p + "g").T)[:, :, None]).flatten(1) @ w(p + "o").T)
    p = "l0.mlp."

    def unit(h, m):
        g, u = (h @ w(p + m + "gate").T).clamp(max=7.0), (h @ w(p + m + "up").T).clamp(-7.0, 7.0)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + m + "down").T

    scores = torch.sigmoid(x @ w(p + "router").T)
    chosen = torch.topk(scores + w(p + "correction"), 4, dim=1).indices
    y = torch.sigmoid(x @ w(p + "shared.sg").T) * unit(x, "shared.")
    for e in range(32):
        t = (chosen == e).any(dim=1).nonzero()[:, 0]
        y[t] += 2.5 * scores[t, e:e + 1] * unit(x[t], "e%d." % e)
    return {"attention": torch.cat(outs), "experts": y}


EXACT = {"llama": _exact_llama, "lasapel": _exact_lasapel, "lanirax": _exact_lanirax, "gavodra": _exact_gavodra}
