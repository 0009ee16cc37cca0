"""Cases whose speed is followed from change to change: what users of the framework have it do, through the classes they hold.

* `train`: one optimizer step of a `DecoderTrainer` (GPT-J, GPT-2 and Llama blocks; micro-batches of forward and backward
  passes, fp32 gradient means, AdamW on fp32 masters). Widths, heads, feed-forwards, vocabularies and sequence lengths are those
  of the named shapes of `DecoderConfig`; two layers stand for the stack, which repeats them.
* `int4`: one `DecoderGenerator.generate` call: prefill of equal prompts, then greedy decoding with 4-bit weights.
* `serve`: a `SequenceGenerator` with a Dunelix or Zirunex model. `generate`: greedy continuation of a batch of prompts.
  `prompts`: long prompts of unequal length through `step`, the logits of the last token of each. `sample`: a caller that
  chooses every token itself from the logits that `step` returns.

Served models are held by a program once for all requests, so `prepare` keeps the handle of the latest case; prompts come from
the seed. A trainer belongs to its state: a step changes its weights. Heads of served models favour one next token clearly, as
trained ones do, so that the rounding of the last bit does not decide what is generated.
"""
import json
import math

import numpy as np
import torch

# ---------------------------------------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------------------------------------


def _train(family, hidden, heads, ffn, vocab, seq, micro_batches, micro_batch_size, recompute, rotary=0, layers=2):
    return dict(kind="train", family=family, layers=layers, hidden=hidden, heads=heads, rotary=rotary, ffn=ffn, vocab=vocab,
                seq=seq, micro_batches=micro_batches, micro_batch_size=micro_batch_size, recompute=recompute)


def _int4(hidden, heads, ffn, vocab, layers, batch, prompt, new, rotary=64):
    return dict(kind="int4", hidden=hidden, heads=heads, rotary=rotary, ffn=ffn, vocab=vocab, layers=layers, batch=batch,
                prompt=prompt, new=new)


def _serve(model, mode, width, ff, heads, kv_heads, layers, window, batch, prompt, new, vocab=32000, dtype="bfloat16"):
    return dict(kind="serve", model=model, mode=mode, dtype=dtype, width=width, ff=ff, heads=heads, kv_heads=kv_heads,
                layers=layers, window=window, batch=batch, prompt=prompt, new=new, vocab=vocab)


def listed():
    return [
        # the smallest training step: a model for tests and debugging, where launches and host work count
        dict(_train("gptj", 256, 4, 512, 1024, 128, 2, 1, True, rotary=32), name="train_tiny"),
        # GPT-2 small: several sequences per micro-batch, biases everywhere, a vocabulary of 50257
        dict(_train("gpt2", 768, 12, 3072, 50257, 1024, 2, 4, False), name="train_gpt2"),
        # Llama-2-7B layers, recomputing the blocks in the backward pass (the trainer's default)
        dict(_train("llama", 4096, 32, 11008, 32000, 2048, 2, 1, True, rotary=128), name="train_llama"),
        # GPT-J-6B layers without recomputation, the headline configuration; the largest step
        dict(_train("gptj", 4096, 16, 16384, 50400, 2048, 4, 1, False, rotary=64), name="train_gptj"),
        # int4 generation at the batch of the headline decoding benchmark
        dict(_int4(4096, 16, 16384, 50400, 4, 16, 512, 32), name="int4_batch16"),
        # one user, an odd prompt length: latency
        dict(_int4(2048, 16, 8192, 50400, 4, 1, 61, 64), name="int4_single"),
        # long prompts of unequal lengths; recurrent layers and differential attention
        dict(_serve("dunelix", "prompts", 4096, 11008, 32, 8, "rrar", 8192, 4, 2048, 0), name="dunelix_prompts"),
        # a batch of short prompts, mostly decoding
        dict(_serve("dunelix", "generate", 4096, 11008, 32, 8, "rrar", 8192, 16, 128, 32), name="dunelix_generate"),
        # documents of several thousand tokens with windows next to the first tokens
        dict(_serve("zirunex", "prompts", 4096, 11008, 32, 8, "aaaa", 1024, 2, 4096, 0), name="zirunex_prompts"),
        # a larger batch of users than one tile of the decoding products holds
        dict(_serve("zirunex", "generate", 2048, 5632, 16, 4, "aaaa", 256, 40, 64, 32), name="zirunex_generate"),
        # one user whose program samples on the host: a portion of one token and its logits per call
        dict(_serve("zirunex", "sample", 2048, 5632, 16, 4, "aaaa", 256, 1, 33, 16), name="zirunex_sample"),
        # a float32 model, for results without the rounding of 16-bit operands
        dict(_serve("dunelix", "generate", 1024, 2816, 8, 2, "rrar", 8192, 4, 200, 16, dtype="float32"), name="dunelix_float32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_once(rng):
    kind = rng.choice(["train", "train", "int4", "serve", "serve", "serve"])
    if kind == "train":
        family = rng.choice(["gptj", "gpt2", "llama"])
        dim = {"gptj": rng.choice([64, 256]), "gpt2": 64, "llama": 128}[family]
        heads = max(1, _log(rng, 256, 4096) // dim)
        hidden = heads * dim
        seq = 2 * _log(rng, 64, 1024)
        size = _log(rng, 1, max(1, 4096 // seq))
        return _train(family, hidden, heads, 8 * int(hidden * rng.uniform(2, 4) / 8), _log(rng, 1000, 50400), seq, rng.randint(2, 4),
                      size, rng.random() < 0.5, rotary={"gptj": dim // 2 if dim == 64 else 64, "gpt2": 0, "llama": dim}[family])
    if kind == "int4":
        dim = rng.choice([128, 256])
        heads = _log(rng, 1024, 4096) // dim
        hidden = heads * dim
        return _int4(hidden, heads, 64 * int(hidden * rng.uniform(2, 4) / 64), 2 * _log(rng, 500, 25200), rng.randint(1, 4),
                     _log(rng, 1, 16), _log(rng, 16, 512), _log(rng, 8, 64))
    model, mode = rng.choice(["dunelix", "zirunex"]), rng.choice(["generate", "prompts", "sample"])
    groups, kv_heads = rng.choice([1, 2, 4]), rng.choice([2, 4, 8])
    width = 128 * max(8, min(32, int(groups * kv_heads * rng.choice([1, 1.5, 2]))))
    dtype = "float32" if mode == "generate" and rng.random() < 0.2 else "bfloat16"
    if dtype == "float32":
        width, groups, kv_heads = 1024, 4, 2
    layers = ("a" if model == "zirunex" else rng.choice(["r", "a"])) + "".join(
        "a" if model == "zirunex" else rng.choice("ra") for _ in range(rng.randint(1, 3)))
    if "a" not in layers:
        layers = layers[:-1] + "a"
    batch = {"generate": _log(rng, 1, 4 if dtype == "float32" else 48), "prompts": _log(rng, 1, 8), "sample": _log(rng, 1, 4)}[mode]
    prompt = {"generate": _log(rng, 8, 256), "prompts": _log(rng, 300, 8192 // batch if batch > 2 else 4096),
              "sample": _log(rng, 8, 256)}[mode]
    new = {"generate": _log(rng, 8, 64), "prompts": 0, "sample": _log(rng, 4, 16)}[mode]
    return _serve(model, mode, width, 8 * int(width * rng.uniform(2, 3) / 8), groups * kv_heads, kv_heads, layers,
                  _log(rng, 64, 8192), batch, prompt, new, vocab=8 * _log(rng, 500, 4000), dtype=dtype)


def draw(rng):
    top = [work(c) for c in listed() if c["name"] == "train_gptj"][0]
    while True:
        case = _draw_once(rng)
        w = work(case)
        if w["flops"] <= top["flops"] and w["bytes"] <= top["bytes"]:
            return case


def _lengths(case):
    """Prompt lengths of the requests: fixed by the case, up to a quarter shorter than the longest."""
    n = case["prompt"]
    return [n - (i * 7919) % max(1, n // 4) for i in range(case["batch"])]


# ---------------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------------


def _matrices(case):
    """Weights of one layer's products, by layer."""
    if case["kind"] == "serve":
        C, F, H, G = case["width"], case["ff"], case["heads"], case["kv_heads"]
        att = C * (H + 2 * G + H) * 128 + (C * H * 128 if case["model"] == "zirunex" else 0)
        return [(4 * C * C if k == "r" else att) + 3 * C * F for k in case["layers"]]
    h, f = case["hidden"], case["ffn"]
    return [4 * h * h + (3 if case.get("family") == "llama" else 2) * h * f] * case["layers"]


def _pairs(n, window):
    """Visible (query, key) pairs of a causal sequence with a window."""
    w = min(n, window) if window else n
    return n * w - w * (w - 1) / 2


def work(case):
    body = sum(_matrices(case))
    if case["kind"] == "train":
        rows = case["micro_batch_size"] * case["seq"] * case["micro_batches"]
        params = body + 2 * case["vocab"] * case["hidden"]
        attention = 2 * 2 * case["hidden"] * case["seq"] / 2 * rows * case["layers"]  # scores and their product, forward
        # per parameter: master, both moments read and written, the 16-bit weight read and written, the gradient written
        return {"bytes": 32.0 * params, "flops": 6.0 * (params - case["vocab"] * case["hidden"]) * rows + 3.5 * attention}
    B = case["batch"]
    lengths = [case["prompt"]] * B if case["kind"] == "int4" else _lengths(case)
    rows, new = sum(lengths), case["new"]
    width = case["hidden"] if case["kind"] == "int4" else case["width"]
    if case["kind"] == "int4":
        per_weight, layers, kv, window, heads_dim = 0.5 + 4 / 64, case["layers"], 2 * width, 0, width
    else:
        per_weight = 4.0 if case["dtype"] == "float32" else 2.0
        layers, window = case["layers"].count("a"), case["window"] if case["model"] == "zirunex" else 0
        kv, heads_dim = 2 * case["kv_heads"] * 128, case["heads"] * 128
    cache_byte = 4 if case.get("dtype") == "float32" else 2
    head = case["vocab"] * width
    seen = sum(min(n, window + 4) if window else n for n in lengths)
    flops = 2.0 * rows * body + 4.0 * heads_dim * layers * sum(_pairs(n, window) for n in lengths) + 2.0 * B * head * max(1, new)
    flops += 2.0 * B * max(0, new - 1) * body
    passes = max(1, new)
    return {"bytes": passes * per_weight * (body + head) + max(0, new - 1) * layers * kv * seen * cache_byte, "flops": flops}


# ---------------------------------------------------------------------------------------------------------------------------
# weights and inputs
# ---------------------------------------------------------------------------------------------------------------------------


class _Draws:
    """Normal tensors on the GPU, one after another from a seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, *shape, std=1.0, mean=0.0):
        return torch.empty(shape, device="cuda").normal_(mean, std, generator=self.gen)

    def tokens(self, vocab, *shape):
        """Ids with the frequencies of a text's words: about 1 / rank."""
        u = torch.empty(shape, dtype=torch.float64, device="cuda").uniform_(0.0, 1.0, generator=self.gen)
        return (vocab ** u - 1).int().clamp(0, vocab - 1).cpu()


def _peaked(embed, std):
    """Head rows `(vocab, width)` that favour one next token after every token, and that next token by token."""
    V = embed.shape[0]
    order = torch.randperm(V, generator=torch.Generator().manual_seed(V))
    following = torch.empty(V, dtype=torch.long)
    following[order] = order.roll(-1)
    head = torch.empty_like(embed)
    head[following.to(embed.device)] = embed * std
    return head, following


def _train_weights(case, seed):
    """fp32 masters by name. Norms and biases are those of a model that has been trained for a while: not ones and zeros."""
    n, h, f = _Draws(seed), case["hidden"], case["ffn"]
    out = {"embedding.wte.weight": n(case["vocab"], h, std=0.02)}
    back = 0.02 / math.sqrt(2 * case["layers"])

    def norm(name):
        out[name + ".weight"] = n(h, std=0.1, mean=1.0)
        if case["family"] != "llama":
            out[name + ".bias"] = n(h, std=0.05)

    if case["family"] == "gpt2":
        out["embedding.wpe.weight"] = n(case["seq"], h, std=0.02)
    for i in range(case["layers"]):
        p = f"layer{i}."
        norm(p + "ln_1")
        out[p + "attention.qkv.weight"], out[p + "attention.out.weight"] = n(h, 3 * h, std=0.02), n(h, h, std=back)
        if case["family"] == "gpt2":
            out[p + "attention.qkv.bias"], out[p + "attention.out.bias"] = n(3 * h, std=0.05), n(h, std=0.05)
        if case["family"] != "gptj":
            norm(p + "ln_2")
        if case["family"] == "llama":
            out[p + "mlp.gate.weight"], out[p + "mlp.up.weight"] = n(h, f, std=0.02), n(h, f, std=0.02)
        else:
            out[p + "mlp.fc_in.weight"], out[p + "mlp.fc_in.bias"] = n(h, f, std=0.02), n(f, std=0.05)
            out[p + "mlp.fc_out.bias"] = n(h, std=0.05)
        out[p + "mlp.fc_out.weight"] = n(f, h, std=back)
    norm("head.ln_f")
    out["head.lm_head.weight"] = n(h, case["vocab"], std=2.5 * h ** -0.5)  # logits as spread as a trained model's
    if case["family"] == "gptj":
        out["head.lm_head.bias"] = n(case["vocab"], std=0.05)
    return out


def _train_tokens(case, seed):
    return _Draws(seed + 1).tokens(case["vocab"], case["micro_batches"], 1, case["micro_batch_size"], case["seq"] + 1)


def _quantise(w):
    """4-bit codes in groups of 64 inputs of `w (out, in)`, with an fp16 scale and zero point per group."""
    g = w.reshape(w.shape[0], -1, 64)
    lo, hi = g.amin(-1, keepdim=True), g.amax(-1, keepdim=True)
    scale = (hi - lo) / 15
    return ((g - lo) / scale).round().clamp(0, 15), scale.half(), lo.half()


def _int4_weights(case):
    """Dense fp32 weights by name; matrices `(out, in)`. One model per case, as a program holds it."""
    n, h, f, V = _Draws(case["hidden"] + case["vocab"]), case["hidden"], case["ffn"], case["vocab"]
    wte = n(V, h).bfloat16()
    head, following = _peaked(wte.float(), h ** -0.5)
    out = {"wte": wte, "lm_head": head, "lm_head.bias": n(V, std=0.1), "ln_f": (n(h, std=0.1, mean=1.0), n(h, std=0.1))}
    for i in range(case["layers"]):
        out[f"{i}.ln"] = (n(h, std=0.1, mean=1.0), n(h, std=0.1))
        out[f"{i}.w1"], out[f"{i}.w2"] = n(3 * h + f, h, std=1.5 * h ** -0.5), n(h, h + f, std=0.3 * (h + f) ** -0.5)
        out[f"{i}.b1"], out[f"{i}.b2"] = n(3 * h + f, std=0.1), n(h, std=0.1)
        out[f"{i}.b1"][:3 * h] = 0
    return out, following


def _serve_config(case):
    mlp = {"ff": case["ff"], "kind": "dense"}
    if case["model"] == "zirunex":
        layer = {"type": "attention", "mlp": dict(mlp, limit=7.0),
                 "mixer": {"heads": case["heads"], "kv_heads": case["kv_heads"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                           "mask": {"size": case["window"], "keep_first": 4}}}
        return {"architecture": "Zirunex", "vocab": case["vocab"], "width": case["width"], "norm": {"eps": 1e-6},
                "embedding": {"scale": 8.0}, "layers": [layer] * len(case["layers"])}
    gru = {"type": "mingru", "mixer": {"width": case["width"]}, "mlp": mlp}
    att = {"type": "attention", "mlp": mlp,
           "mixer": {"heads": case["heads"], "kv_heads": case["kv_heads"], "dim": 64, "vdim": 128, "diff": 0.5, "scale": 0.125,
                     "mask": {"size": case["window"]},
                     "rot": {"base": 500000.0, "dims": 64,
                             "scaling": {"factor": 16.0, "low": 1.0, "high": 4.0, "original": 4096}}}}
    return {"architecture": "Dunelix", "vocab": case["vocab"], "width": case["width"], "norm": {"eps": 1e-6}, "residual_mult": 0.5,
            "layers": [{"r": gru, "a": att}[k] for k in case["layers"]]}


def _serve_checkpoint(case):
    """Checkpoint tensors by name (matrices in the model's type, vectors in fp32), and the next token by token."""
    n, C, F, H, G = _Draws(case["width"] + case["vocab"]), case["width"], case["ff"], case["heads"], case["kv_heads"]
    zirunex = case["model"] == "zirunex"
    dt = getattr(torch, case["dtype"])
    embed = n(case["vocab"], C, std=0.125 if zirunex else 1.0).to(dt)
    head, following = _peaked(embed.float(), (8.0 if zirunex else 1.0) * C ** -0.5)
    out = {"embed": embed, "head": head}

    def norm(name):
        if zirunex:
            out[name] = n(C, std=0.2)
        else:
            out.update({name: n(C, std=0.1, mean=1.0), name + ".b": n(C, std=0.1), name + ".alpha": torch.tensor(0.5, device="cuda")})

    for i, kind in enumerate(case["layers"]):
        p = f"l{i}.mix."
        norm(f"l{i}.norm1")
        if kind == "r":
            out.update({p + k: n(C, C, std=C ** -0.5) for k in "zxgo"})
            out[p + "z.b"], out[p + "x.b"] = n(C, mean=-3.0), n(C, std=0.1)
        else:
            d = 128 if zirunex else 2 * 64
            out[p + "q"], out[p + "k"] = n(H * d, C, std=C ** -0.5), n(G * d, C, std=C ** -0.5)
            out[p + "v"], out[p + "o"] = n(G * 128, C, std=C ** -0.5), n(C, H * 128, std=(H * 128) ** -0.5)
            if zirunex:
                out[p + "g"] = n(H * 128, C, std=2 * C ** -0.5)
                out[p + "q.norm"], out[p + "k.norm"] = n(128, std=0.2, mean=1.6), n(128, std=0.2, mean=1.2)
            else:
                out.update({p + k: n(64, std=0.1) for k in ("lq1", "lk1", "lq2", "lk2")})
        if not zirunex:
            norm(f"l{i}.norm2")
        out[f"l{i}.mlp.gate"], out[f"l{i}.mlp.up"] = n(F, C, std=C ** -0.5), n(F, C, std=C ** -0.5)
        out[f"l{i}.mlp.down"] = n(C, F, std=F ** -0.5)
    norm("final.norm")
    return {k: v.to(dt) if v.dim() == 2 else v for k, v in out.items()}, following


def _prompts(case, seed):
    n = _Draws(seed)
    lengths = [case["prompt"]] * case["batch"] if case["kind"] == "int4" else _lengths(case)
    return [n.tokens(case["vocab"], k) for k in lengths]


# ---------------------------------------------------------------------------------------------------------------------------
# states and passes
# ---------------------------------------------------------------------------------------------------------------------------

_held = {}  # the served model of the latest case


def _handle(case, make):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _held:
        _held.clear()
        torch.cuda.empty_cache()
        _held[key] = make(case)
    return _held[key]


def _make_int4(case):
    from popxl_addons_b200.models.decoder import DecoderConfig
    from popxl_addons_b200.models.generator import DecoderGenerator, interleave_scale_zero

    cfg = DecoderConfig(family="gptj", layers=case["layers"], hidden=case["hidden"], heads=case["heads"],
                        head_dim=case["hidden"] // case["heads"], rotary_dim=case["rotary"], ffn=case["ffn"],
                        vocab_size=case["vocab"], seq_len=case["prompt"] + case["new"])
    gen = DecoderGenerator(cfg, case["batch"], case["prompt"], case["new"], device="cuda")
    weights, _ = _int4_weights(case)

    def put(var, value):
        t = gen.session._vars[var][0]
        t.view(torch.int16 if t.dtype == torch.uint16 else t.dtype).copy_(value.reshape(t.shape))

    def put_linear(q, w, bias):
        codes, scale, zero = _quantise(w)
        c = codes.int().reshape(*codes.shape[:2], -1, 4)
        word = (c[..., 0] << 12) | (c[..., 1] << 8) | (c[..., 2] << 4) | c[..., 3]
        put(q.packed, torch.where(word > 32767, word - 65536, word).to(torch.int16))
        put(q.scale, scale)
        put(q.zero, zero)
        put(q.sz, interleave_scale_zero(scale, zero))
        put(q.bias, bias)

    put(gen.wte, weights["wte"])
    put_linear(gen.head, weights["lm_head"], weights["lm_head.bias"])
    for var, value in zip(gen.ln_f, weights["ln_f"]):
        put(var, value)
    for i, L in enumerate(gen.layers):
        put(L["ln_w"], weights[f"{i}.ln"][0])
        put(L["ln_b"], weights[f"{i}.ln"][1])
        put_linear(L["w1"], weights[f"{i}.w1"], weights[f"{i}.b1"])
        put_linear(L["w2"], weights[f"{i}.w2"], weights[f"{i}.b2"])
    return gen


def _make_serve(case):
    from popxl_addons_b200.models.registry import architecture
    from popxl_addons_b200.models.sequence_generator import SequenceGenerator

    config = _serve_config(case)
    arch = architecture(config["architecture"])
    gen = SequenceGenerator(arch.model(arch.config(config), case["dtype"]), batch=case["batch"],
                            max_seq=case["prompt"] + max(1, case["new"]), max_new_tokens=max(1, case["new"]), device="cuda")
    return gen.load_checkpoint(_serve_checkpoint(case)[0])


def _make_train(case, seed):
    from popxl_addons_b200.models.decoder import DecoderConfig
    from popxl_addons_b200.models.trainer import DecoderTrainer

    cfg = DecoderConfig(family=case["family"], layers=case["layers"], hidden=case["hidden"], heads=case["heads"],
                        head_dim=case["hidden"] // case["heads"], rotary_dim=case["rotary"], ffn=case["ffn"],
                        vocab_size=case["vocab"], seq_len=case["seq"])
    trainer = DecoderTrainer(cfg, case["micro_batches"], case["micro_batch_size"], device="cuda", recompute=case["recompute"])
    held, weights = trainer.session._vars, trainer.weights.to_dict()
    for name, value in _train_weights(case, seed).items():
        held[trainer.master[name]][0].copy_(value)
        held[weights[name]][0].copy_(value)
    gradients = {v.name.replace(".grad.accum.", "."): held[v][0] for v in trainer.ir.initial_values if ".grad.accum." in v.name}
    masters = {name: held[v][0] for name, v in trainer.master.items()}
    return trainer, {"gradients": gradients, "weights": masters}


def prepare(case, seed):
    if case["kind"] == "train":
        trainer, buffers = _make_train(case, seed)
        return {"case": case, "trainer": trainer, "buffers": buffers, "tokens": _train_tokens(case, seed).pin_memory()}
    prompts = _prompts(case, seed)
    if case["kind"] == "int4":
        gen = _handle(case, _make_int4)
        caches = [gen.session._vars[L[k]][0] for L in gen.layers for k in ("k", "v")]
        return {"case": case, "gen": gen, "prompt": torch.stack(prompts).pin_memory(), "caches": caches}
    gen = _handle(case, _make_serve)
    last = case["layers"].rindex("a")
    names = {"v": f"{'l' if case['model'] == 'zirunex' else 'run'}{last}.v"}
    if case["batch"] <= 20:
        names["k"] = names["v"][:-1] + "k"
        if "r" in case["layers"]:
            names["state"] = f"run{case['layers'].rindex('r')}.state"
    held = {k: gen.session._vars[gen._vars[name]][0] for k, name in names.items()}
    return {"case": case, "gen": gen, "prompts": [p.tolist() for p in prompts], "held": held}


def _slot_state(state, slots, positions):
    """What the last layers hold for every request: its positions of the caches, its recurrent state."""
    return {k: [t[s] if k == "state" else t[s][..., :n, :] for s, n in zip(slots, positions)] for k, t in state["held"].items()}


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        return {"loss": state["trainer"].step(state["tokens"]), **state["buffers"]}
    if case["kind"] == "int4":
        return {"tokens": state["gen"].generate(state["prompt"]), "caches": state["caches"]}
    gen, prompts, new = state["gen"], state["prompts"], case["new"]
    lengths = [len(p) for p in prompts]
    if case["mode"] == "generate":
        slots = gen._free[::-1]  # requests take slots from the end of the list
        tokens = gen.generate(prompts, new)
        return {"tokens": np.stack(tokens), "held": _slot_state(state, slots, [n + new - 1 for n in lengths])}
    for r in range(len(prompts)):
        gen.admit(r)
    logits = [gen.step(dict(enumerate(prompts)), {r: [n - 1] for r, n in enumerate(lengths)})]
    tokens = []
    for k in range(new):
        tokens.append([int(np.argmax(logits[-1][r][0])) for r in range(len(prompts))])
        if k + 1 < new:
            logits.append(gen.step({r: [t] for r, t in enumerate(tokens[-1])}, {r: [0] for r in range(len(prompts))}))
    held = _slot_state(state, [gen.slots[r] for r in range(len(prompts))], [n + max(0, new - 1) for n in lengths])
    for r in reversed(range(len(prompts))):
        gen.release(r)
    out = {"logits": np.stack([np.concatenate([at[r] for r in range(len(prompts))]) for at in logits]), "held": held}
    if tokens:
        out["tokens"] = np.array(tokens)
    return out


def tolerance(case):
    """Bounds for another implementation with the same operand types, from the distance to `exact`: 16-bit operands put the
    gradients up to 1.4e-2, the caches of int4 models 1.0e-2 and those of served models 5.5e-3 away from it, float32 ones 2e-6.
    Tokens are chosen with a wide lead."""
    if case["kind"] == "serve":
        return {"rel": 1e-5 if case["dtype"] == "float32" else 0.02, "max": 1e-3 if case["dtype"] == "float32" else 0.5, "differ": 0.0}
    return {"rel": 0.03, "max": 0.9, "differ": 0.0}


# ---------------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------------


def _layer_norm(x, w, b, eps=1e-5):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, eps)


def _rms_norm(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rotate(x, angle):
    """Rotate the leading pairs of `x (..., tokens, dim)` by `angle (tokens, pairs)`."""
    r = 2 * angle.shape[1]
    a, b, c, s = x[..., 0:r:2], x[..., 1:r:2], torch.cos(angle), torch.sin(angle)
    return torch.cat([torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2), x[..., r:]], -1)


def _angles(n, dims, base=10000.0):
    f = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device="cuda") / dims)
    return torch.outer(torch.arange(n, dtype=torch.float64, device="cuda"), f)


def _causal(n):
    i = torch.arange(n, device="cuda")
    return i[:, None] >= i[None, :]


def _decoder_attention(qkv, heads, rotary):
    """Causal attention on packed projections `(batch, tokens, 3 * width)`; also the rotated keys and the values."""
    B, n, w = qkv.shape
    q, k, v = qkv.reshape(B, n, 3, heads, -1).permute(2, 0, 3, 1, 4)
    if rotary:
        a = _angles(n, rotary)
        q, k = _rotate(q, a), _rotate(k, a)
    s = (q @ k.transpose(-1, -2)) / math.sqrt(q.shape[-1])
    out = torch.softmax(s.masked_fill(~_causal(n), float("-inf")), -1) @ v
    return out.transpose(1, 2).reshape(B, n, w // 3), k, v


def _train_loss(case, w, tokens):
    inp, labels = tokens[:, :-1].long(), tokens[:, 1:].long()
    x = w["embedding.wte.weight"][inp]
    if case["family"] == "gpt2":
        x = x + w["embedding.wpe.weight"]

    def norm(name, x):
        if case["family"] == "llama":
            return _rms_norm(x, w[name + ".weight"], 1e-5)
        return _layer_norm(x, w[name + ".weight"], w[name + ".bias"])

    def linear(x, name):
        y = x @ w[name + ".weight"]
        return y + w[name + ".bias"] if name + ".bias" in w else y

    for i in range(case["layers"]):
        p = f"layer{i}."
        h = norm(p + "ln_1", x)
        a = linear(_decoder_attention(linear(h, p + "attention.qkv"), case["heads"], case["rotary"])[0], p + "attention.out")
        if case["family"] != "gptj":
            x = x + a
            h = norm(p + "ln_2", x)
        if case["family"] == "llama":
            z = torch.nn.functional.silu(linear(h, p + "mlp.gate")) * linear(h, p + "mlp.up")
        else:
            z = torch.nn.functional.gelu(linear(h, p + "mlp.fc_in"), approximate="tanh" if case["family"] == "gpt2" else "none")
        y = linear(z, p + "mlp.fc_out")
        x = x + a + y if case["family"] == "gptj" else x + y
    logits = linear(norm("head.ln_f", x), "head.lm_head")
    return torch.nn.functional.cross_entropy(logits.reshape(-1, case["vocab"]), labels.reshape(-1))


def _exact_train(case, seed):
    masters = _train_weights(case, seed)
    w = {k: v.bfloat16().double().requires_grad_() for k, v in masters.items()}
    tokens = _train_tokens(case, seed).cuda()
    losses = []
    for m in range(case["micro_batches"]):
        loss = _train_loss(case, w, tokens[m, 0])
        (loss / case["micro_batches"]).backward()
        losses.append(loss.item())
    new = {}
    for k, v in masters.items():  # first AdamW step: both moments start from zero
        g, v = w[k].grad, v.double()
        new[k] = v - 1e-4 * (g / (g.abs() + 1e-5) + (0.01 * v if v.dim() > 1 else 0))
    return {"loss": float(np.mean(losses)), "gradients": {k: t.grad for k, t in w.items()}, "weights": new}


def _continued(case, seed, following):
    """Prompts with the tokens that follow them, `max(1, new) - 1` of which the model reads."""
    out = []
    for p in _prompts(case, seed):
        p = p.tolist()
        for _ in range(max(0, case["new"] - 1)):
            p.append(int(following[p[-1]]))
        out.append(p)
    return out


def _exact_int4(case, seed):
    weights, following = _int4_weights(case)

    def dense(w):
        codes, scale, zero = _quantise(w)
        return (codes.double() * scale.double() + zero.double()).reshape(w.shape)

    def vector(v):
        return v.bfloat16().double()

    new, h, S = case["new"], case["hidden"], case["prompt"] + case["new"]
    tokens = torch.tensor(_continued(case, seed, following), device="cuda")
    x, caches = weights["wte"].double()[tokens], []
    for i in range(case["layers"]):
        hn = _layer_norm(x, *(vector(v) for v in weights[f"{i}.ln"]))
        y = hn @ dense(weights[f"{i}.w1"]).T + vector(weights[f"{i}.b1"])
        a, k, v = _decoder_attention(y[..., :3 * h], case["heads"], case["rotary"])
        caches += [torch.nn.functional.pad(t, (0, 0, 0, S - t.shape[2])) for t in (k, v)]
        z = torch.nn.functional.gelu(y[..., 3 * h:])
        x = x + torch.cat([a, z], -1) @ dense(weights[f"{i}.w2"]).T + vector(weights[f"{i}.b2"])
    hn = _layer_norm(x[:, case["prompt"] - 1:], *(vector(v) for v in weights["ln_f"]))
    logits = hn @ dense(weights["lm_head"]).T + vector(weights["lm_head.bias"])
    return {"tokens": logits.argmax(-1).int().reshape(case["batch"], new), "caches": caches}


def _window(n, window):
    i = torch.arange(n, device="cuda")
    return _causal(n) & ((i[:, None] - i[None, :] < window) | (i[None, :] < 4))


def _zirunex_layer(case, W, p, x):
    H, G, n = case["heads"], case["kv_heads"], x.shape[0]
    h = _rms_norm(x, 1 + W[p + "norm1"], 1e-6)
    m = p + "mix."
    q = _rms_norm((h @ W[m + "q"].T).reshape(n, G, H // G, 128), W[m + "q.norm"], 1e-6)
    k = _rms_norm((h @ W[m + "k"].T).reshape(n, G, 128), W[m + "k.norm"], 1e-6)
    v = (h @ W[m + "v"].T).reshape(n, G, 128)
    mask, heads = _window(n, case["window"]), []
    for g in range(G):
        s = (q[:, g].transpose(0, 1) @ k[:, g].T * 128 ** -0.5).masked_fill(~mask, float("-inf"))
        s = torch.cat([s, torch.zeros_like(s[..., :1])], -1)  # the sink
        heads.append(torch.softmax(s, -1)[..., :-1] @ v[:, g])
    o = torch.stack(heads, 0).permute(2, 0, 1, 3).reshape(n, H * 128) * torch.sigmoid(h @ W[m + "g"].T)
    gate, up = (h @ W[p + "mlp.gate"].T).clamp(max=7.0), (h @ W[p + "mlp.up"].T).clamp(-7.0, 7.0)
    y = (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ W[p + "mlp.down"].T
    return x + o @ W[m + "o"].T + y, {"k": k.transpose(0, 1), "v": v.transpose(0, 1)}


def _dunelix_norm(W, name, x):
    return torch.tanh(W[name + ".alpha"] * x) * W[name] + W[name + ".b"]


def _dunelix_angles(n):
    """Frequencies of base 500000 over 64 features, long wavelengths slowed as the configuration says."""
    a = _angles(n, 64, 500000.0)
    f = a[1] if n > 1 else _angles(2, 64, 500000.0)[1]
    turns = 4096 * f / (2 * math.pi)
    blend = ((turns - 1.0) / 3.0).clamp(0, 1)
    return a * ((1 - blend) / 16.0 + blend)


def _dunelix_layer(case, W, p, kind, x):
    H, G, n = case["heads"], case["kv_heads"], x.shape[0]
    h, m, held = _dunelix_norm(W, p + "norm1", x), p + "mix.", {}
    if kind == "r":
        z, u = torch.sigmoid(h @ W[m + "z"].T + W[m + "z.b"]), h @ W[m + "x"].T + W[m + "x.b"]
        c = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
        s, states = torch.zeros_like(c[0]), []
        for keep, add in zip((1 - z).unbind(), c.unbind()):
            s = torch.addcmul(add, keep, s)
            states.append(s)
        held["state"] = s
        y = torch.stack(states) * torch.nn.functional.silu(h @ W[m + "g"].T)
    else:
        a = _dunelix_angles(n)
        q = _rotate((h @ W[m + "q"].T).reshape(n, H, 2, 64).permute(1, 2, 0, 3), a)
        k = _rotate((h @ W[m + "k"].T).reshape(n, G, 2, 64).permute(1, 2, 0, 3), a)
        v = (h @ W[m + "v"].T).reshape(n, G, 128).transpose(0, 1)
        lam = torch.exp((W[m + "lq1"] * W[m + "lk1"]).sum()) - torch.exp((W[m + "lq2"] * W[m + "lk2"]).sum()) + 0.5
        i = torch.arange(n, device="cuda") // case["window"]
        mask, heads = _causal(n) & (i[:, None] == i[None, :]), []
        for j in range(H):
            g = j // (H // G)
            s = (q[j] @ k[g].transpose(-1, -2) * 0.125).masked_fill(~mask, float("-inf"))
            both = torch.softmax(s, -1) @ v[g]
            heads.append(_rms_norm(both[0] - lam * both[1], 0.5, 1e-6))
        y = torch.cat(heads, -1)
        held.update(k=k, v=v)
    x = x + 0.5 * y @ W[m + "o"].T
    h = _dunelix_norm(W, p + "norm2", x)
    z = torch.nn.functional.silu(h @ W[p + "mlp.gate"].T) * (h @ W[p + "mlp.up"].T)
    return x + 0.5 * z @ W[p + "mlp.down"].T, held


def _exact_serve(case, seed):
    ckpt, following = _serve_checkpoint(case)
    W = {k: v.double() for k, v in ckpt.items()}
    zirunex, new = case["model"] == "zirunex", case["new"]
    logits, held = [], {"k": [], "v": [], "state": []}
    for tokens, n in zip(_continued(case, seed, following), _lengths(case)):
        x = W["embed"][torch.tensor(tokens, device="cuda")] * (8.0 if zirunex else 1.0)
        last = {}
        for i, kind in enumerate(case["layers"]):
            x, now = _zirunex_layer(case, W, f"l{i}.", x) if zirunex else _dunelix_layer(case, W, f"l{i}.", kind, x)
            last.update(now)
        x = x[n - 1:]
        x = _rms_norm(x, 1 + W["final.norm"], 1e-6) if zirunex else _dunelix_norm(W, "final.norm", x)
        logits.append(x @ W["head"].T)
        for k, t in last.items():
            held[k].append(t)
    if case["batch"] > 20:
        held = {"v": held["v"]}
    elif not held["state"]:
        del held["state"]
    logits = torch.stack(logits)  # (requests, tokens, vocab)
    tokens = logits.argmax(-1).int()
    if case["mode"] == "generate":
        return {"tokens": tokens, "held": held}
    out = {"logits": logits.transpose(0, 1), "held": held}
    if new:
        out["tokens"] = tokens.T.contiguous().long()
    return out


def exact(case, seed):
    with torch.set_grad_enabled(case["kind"] == "train"):
        return {"train": _exact_train, "int4": _exact_int4, "serve": _exact_serve}[case["kind"]](case, seed)
