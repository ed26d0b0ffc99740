"""The work by which this library's speed is judged: prompt steps, one-token steps, short generations and sampling.

A case is a dict of plain values.  `path` says what one pass does:

* "prompt": every sequence reads its tokens in one `Engine.step` and gives the logits of its last `want` places; with
  `cached` > 0 the sequences hold that many positions already (a long prompt read in pieces) and are rewound afterwards.
* "decode": sequences that hold a prompt are stepped `steps` times by a decode runner, one token each, and rewound.
* "generate": slots are opened, prompts read, `steps` one-token steps run, slots closed: one batch of the generation loop
  with given tokens in the place of picked ones.
* "sample": one token for each row of logits.

Sizes are those of the benchmark (`bench.py`): the three Llama shapes, and the layer sizes of the other decoders.  The
wider shapes run with fewer layers than the models have: their layers are alike.  Decoders that may route tokens to
experts have dense feed-forwards here, as in the benchmark's comparisons: at 16 bits a near tie between two experts goes
either way in two correct implementations, and logits can then not be compared.

`exact` gives every case's logits in 64-bit arithmetic by plain whole-sequence formulas, without the library.
"""
import math

import torch

LLAMA = {
    "1b": dict(hidden=2048, heads=32, kv=8, ff=8192, vocab=128256, factor=32.0, tied=True),
    "3b": dict(hidden=3072, heads=24, kv=8, ff=8192, vocab=128256, factor=32.0, tied=True),
    "8b": dict(hidden=4096, heads=32, kv=8, ff=14336, vocab=128256, factor=8.0, tied=False),
}
NAVALORN = {
    "w2048": dict(width=2048, heads=16, dim=128, rot=64, vdim=128, kv_rank=512, q_rank=1536, ff=8192, vocab=32000),
    "w2048_small": dict(width=2048, heads=32, dim=64, rot=32, vdim=64, kv_rank=256, q_rank=768, ff=8192, vocab=32000),
}
VAVUPEL = {
    "w2048": dict(width=2048, heads=16, dim=128, rot=64, vdim=128, kv_rank=512, window=1024, ret_heads=16, ret_dim=128, ret_vdim=128,
                  ff=8192, buckets=65521, vocab=32000),
    "w2048_odd": dict(width=2048, heads=32, dim=64, rot=32, vdim=40, kv_rank=256, window=500, ret_heads=12, ret_dim=96, ret_vdim=64,
                      ff=6144, buckets=40009, vocab=32000),
}
SOFOPEL = {
    "w2048": dict(width=2048, heads=16, kv=4, dim=64, vdim=128, chunk=1024, win_heads=16, win_kv=4, win_dim=128, win_vdim=128,
                  window=1024, keep_first=64, lin_heads=16, lin_dim=128, lin_vdim=128, ff=8192, vocab=32000),
    "w2048_odd": dict(width=2048, heads=24, kv=4, dim=40, vdim=56, chunk=500, win_heads=20, win_kv=5, win_dim=96, win_vdim=40,
                      window=500, keep_first=20, lin_heads=12, lin_dim=96, lin_vdim=64, ff=6144, vocab=32000),
}
BAROVIK = {
    "w2048": dict(width=2048, heads=32, kv=8, dim=64, vdim=64, chunk=8192, ff=8192, ssm_heads=64, ssm_dim=64, state=128, groups=8,
                  vocab=32000),
    "w2048_odd": dict(width=2048, heads=32, kv=8, dim=64, vdim=40, chunk=1000, ff=8192, ssm_heads=64, ssm_dim=40, state=96, groups=4,
                      vocab=32000),
}
SIZES = {"llama": LLAMA, "navalorn": NAVALORN, "vavupel": VAVUPEL, "sofopel": SOFOPEL, "barovik": BAROVIK}
DEVICE = "cuda:0"


def _case(name, model, size, layers, dtype, path, seqs, shortest, longest, cached=0, want=1, steps=0):
    return dict(name=name, model=model, size=size, layers=layers, dtype=dtype, path=path, seqs=seqs, shortest=shortest, longest=longest,
                cached=cached, want=want, steps=steps)


def listed():
    return [
        # one user at a keyboard, the smallest model: the shortest step there is, launches and latency
        _case("llama_1b_decode_1", "llama", "1b", 16, "bfloat16", "decode", 1, 200, 200, steps=1),
        # a server's batch of 64 with unequal contexts (the benchmark's 1B workload)
        _case("llama_1b_decode_64", "llama", "1b", 16, "bfloat16", "decode", 64, 133, 2043, steps=4),
        # the benchmark's headline: batch 8 behind 2,000-token contexts at the 8B layer sizes
        _case("llama_8b_decode_8", "llama", "8b", 8, "bfloat16", "decode", 8, 2000, 2000, steps=4),
        # the same model's prompt step
        _case("llama_8b_prompt_2048", "llama", "8b", 8, "bfloat16", "prompt", 1, 2048, 2048, want=16),
        # a long prompt read in pieces: the last 4,096 tokens of 16,384 (the benchmark's 3B workload)
        _case("llama_3b_prompt_at_12288", "llama", "3b", 14, "bfloat16", "prompt", 1, 4096, 4096, cached=12288, want=16),
        # the true 32-bit path (checking another program's numbers): three unequal prompts, and a few sequences stepped
        _case("llama_1b_float32_prompt", "llama", "1b", 16, "float32", "prompt", 3, 100, 301, want=16),
        _case("llama_1b_float32_decode_4", "llama", "1b", 16, "float32", "decode", 4, 300, 700, steps=4),
        # the decoder with a latent cache reads a prompt
        _case("navalorn_prompt_2048", "navalorn", "w2048", 4, "bfloat16", "prompt", 1, 2048, 2048, want=16),
        # retention and windowed latent attention with looped layers: a batch of short requests, prompt and answer
        _case("vavupel_generate_8", "vavupel", "w2048", 4, "bfloat16", "generate", 8, 150, 410, steps=24),
        # difference of maps, windowed attention and decays per key channel: unequal prompts at the odd sizes
        _case("sofopel_prompts_odd", "sofopel", "w2048_odd", 4, "bfloat16", "prompt", 3, 501, 1203, want=16),
        # the hybrid decoder (capped attention, state-space layers) reads a prompt
        _case("barovik_prompt_2048", "barovik", "w2048", 4, "bfloat16", "prompt", 1, 2048, 2048, want=16),
        # sampling at the command line's defaults for a server's batch
        dict(name="sample_64", path="sample", rows=64, vocab=128256, temperature=0.7, top_k=40, top_p=0.9),
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    def spread(lo, hi):
        a, b = log_int(lo, hi), log_int(lo, hi)
        return min(a, b), max(a, b)

    kind = rng.choice(["decode", "decode", "prompt", "prompt", "piece", "float32", "other", "other", "generate", "sample"])
    if kind == "sample":
        c = dict(path="sample", rows=log_int(1, 64), vocab=rng.choice([128256, 32000, log_int(2000, 150000)]),
                 temperature=round(rng.uniform(0.3, 1.3), 2), top_k=rng.choice([0, 40, log_int(2, 500)]), top_p=rng.choice([1.0, 0.9, 0.95]))
        return c
    if kind == "decode":
        size = rng.choice(["1b", "1b", "3b", "8b"])
        lo, hi = spread(17, 3000)
        c = _case("", "llama", size, {"1b": 16, "3b": 14, "8b": 8}[size], "bfloat16", "decode", log_int(1, 64), lo, hi, steps=rng.randint(1, 4))
    elif kind == "prompt":
        size = rng.choice(["1b", "3b", "8b"])
        n = rng.randint(1, 4)
        lo, hi = spread(16, 3000 // n)
        c = _case("", "llama", size, {"1b": 16, "3b": 14, "8b": 8}[size], "bfloat16", "prompt", n, lo, hi, want=rng.randint(1, 16))
    elif kind == "piece":
        size = rng.choice(["1b", "3b"])
        n = log_int(100, 3000)
        c = _case("", "llama", size, 10, "bfloat16", "prompt", 1, n, n, cached=log_int(200, 12000), want=rng.randint(1, 16))
    elif kind == "float32":
        if rng.random() < 0.5:
            n = rng.randint(1, 4)
            lo, hi = spread(16, 800 // n)
            c = _case("", "llama", "1b", rng.choice([8, 16]), "float32", "prompt", n, lo, hi, want=rng.randint(1, 16))
        else:
            lo, hi = spread(17, 1500)
            c = _case("", "llama", "1b", rng.choice([8, 16]), "float32", "decode", log_int(1, 16), lo, hi, steps=rng.randint(1, 4))
    elif kind == "other":
        model = rng.choice(["navalorn", "vavupel", "sofopel", "barovik"])
        n = rng.randint(1, 4)
        lo, hi = spread(60, 3000 // n)
        c = _case("", model, rng.choice(sorted(SIZES[model])), 4, "bfloat16", "prompt", n, lo, hi, want=rng.randint(1, 16))
    else:
        model = rng.choice(["navalorn", "vavupel", "sofopel", "barovik"])
        lo, hi = spread(20, 500)
        c = _case("", model, rng.choice(sorted(SIZES[model])), 4, "bfloat16", "generate", log_int(1, 16), lo, hi, steps=rng.randint(4, 24))
    c["want"] = min(c["want"], c["shortest"])
    del c["name"]
    return c


# ---- configurations -------------------------------------------------------------------------------------------------
def config(case):
    z, n = SIZES[case["model"]][case["size"]], case["layers"]
    if case["model"] == "llama":
        return {"architectures": ["LlamaForCausalLM"], "hidden_size": z["hidden"], "num_hidden_layers": n, "num_attention_heads": z["heads"],
                "num_key_value_heads": z["kv"], "head_dim": z["hidden"] // z["heads"], "intermediate_size": z["ff"], "vocab_size": z["vocab"],
                "max_position_embeddings": 131072, "rope_theta": 500000.0,
                "rope_scaling": {"rope_type": "llama3", "factor": z["factor"], "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                                 "original_max_position_embeddings": 8192},
                "rms_norm_eps": 1e-5, "tie_word_embeddings": z["tied"]}
    top = {"architecture": case["model"].capitalize(), "width": z["width"], "vocab": z["vocab"], "norm": {"eps": 1e-5}}
    mlp = {"kind": "dense", "ff": z["ff"]}
    if case["model"] == "navalorn":
        mixer = {"heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot"], "vdim": z["vdim"], "kv_rank": z["kv_rank"], "q_rank": z["q_rank"],
                 "scale": (z["dim"] + z["rot"]) ** -0.5,
                 "rot": {"base": 10000.0, "dims": z["rot"], "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        return dict(top, layers=[{"type": "latent_attention", "mixer": mixer, "mlp": mlp}] * n)
    if case["model"] == "vavupel":
        latent = {"type": "latent_attention", "mlp": mlp, "mixer": {
            "heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot"], "vdim": z["vdim"], "kv_rank": z["kv_rank"],
            "scale": (z["dim"] + z["rot"]) ** -0.5, "mask": {"size": z["window"]}, "rot": {"base": 10000.0, "dims": z["rot"]}}}
        retention = {"type": "retention", "mlp": mlp, "mixer": {
            "heads": z["ret_heads"], "dim": z["ret_dim"], "vdim": z["ret_vdim"], "rot": {"base": 10000.0, "dims": z["ret_dim"]},
            "decay": [1.0 - 2.0 ** -(1 + 7 * h / (z["ret_heads"] - 1)) for h in range(z["ret_heads"])]}}
        return dict(top, logit_softcap=30.0, embedding={"scale": 1.0, "bigram": {"buckets": z["buckets"], "mul_prev": 31, "mul_cur": 7}},
                    loop={"start": 1, "stop": 3, "times": 2}, layers=[retention, latent] * (n // 2))
    if case["model"] == "sofopel":
        mlp = dict(mlp, limit=7.0)
        maps = {"type": "attention", "mlp": mlp, "mixer": {
            "heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["vdim"], "scale": z["dim"] ** -0.5, "diff": 0.3, "conv": 4,
            "mask": {"size": z["chunk"]}, "rot": {"base": 500000.0, "dims": z["dim"] // 2}}}
        windowed = {"type": "attention_2", "mlp": mlp, "mixer": {
            "heads": z["win_heads"], "kv_heads": z["win_kv"], "dim": z["win_dim"], "vdim": z["win_vdim"], "scale": z["win_dim"] ** -0.5,
            "mask": {"size": z["window"], "keep_first": z["keep_first"]},
            "rot": {"base": 500000.0, "dims": z["win_dim"], "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
        linear = {"type": "gla", "mlp": mlp, "mixer": {"heads": z["lin_heads"], "dim": z["lin_dim"], "vdim": z["lin_vdim"], "tau": 16.0}}
        return dict(top, embedding={"scale": 1.0}, residual_mult=0.5, loop={"start": 1, "stop": 3, "times": 2},
                    layers=[maps, windowed, linear, windowed])
    attention = {"type": "attention", "mlp": mlp, "mixer": {
        "heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["vdim"], "scale": z["dim"] ** -0.5, "softcap": 30.0,
        "mask": {"size": z["chunk"]}, "v_mix": True}}
    ssm = {"type": "mamba2", "mlp": mlp, "mixer": {
        "heads": z["ssm_heads"], "vdim": z["ssm_dim"], "state": z["state"], "groups": z["groups"], "conv": 4, "norm_groups": z["groups"]}}
    return dict(top, embedding={"scale": 1.0}, layers=[attention, ssm] * (n // 2))


def runs_of(cfg):
    """The layers in the order they run, each with whether a pass over a loop starts there."""
    n, loop = len(cfg["layers"]), cfg.get("loop")
    if not loop:
        return [(i, False) for i in range(n)]
    body = [(i, i == loop["start"]) for i in range(loop["start"], loop["stop"])]
    return [(i, False) for i in range(loop["start"])] + body * loop["times"] + [(i, False) for i in range(loop["stop"], n)]


# ---- inputs ---------------------------------------------------------------------------------------------------------
def weights(case, seed):
    """name -> tensor: matrices of 1 / sqrt(inputs), so that what a layer adds is of the size of what it reads."""
    dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    out = {}

    def put(name, *shape, std=None, mean=0.0):
        std = std if std is not None else 1.0 / math.sqrt(shape[-1])
        out[name] = torch.empty(shape, dtype=dtype, device=DEVICE).normal_(mean, std, generator=gen)

    def norm(name, n, spread=0.1):
        put(name, n, std=spread, mean=1.0)

    def tanh_norm(name, n, alpha):
        norm(name, n)
        put(name + ".b", n, std=0.1)
        put(name + ".alpha", std=0.05, mean=alpha)

    cfg = config(case)
    if case["model"] == "llama":
        d, hd, ff = cfg["hidden_size"], cfg["head_dim"], cfg["intermediate_size"]
        put("model.embed_tokens.weight", cfg["vocab_size"], d, std=1.0 if not cfg["tie_word_embeddings"] else 1.0 / math.sqrt(d))
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            norm(p + "input_layernorm.weight", d)
            norm(p + "post_attention_layernorm.weight", d)
            put(p + "self_attn.q_proj.weight", cfg["num_attention_heads"] * hd, d)
            put(p + "self_attn.k_proj.weight", cfg["num_key_value_heads"] * hd, d)
            put(p + "self_attn.v_proj.weight", cfg["num_key_value_heads"] * hd, d)
            put(p + "self_attn.o_proj.weight", d, cfg["num_attention_heads"] * hd)
            put(p + "mlp.gate_proj.weight", ff, d)
            put(p + "mlp.up_proj.weight", ff, d)
            put(p + "mlp.down_proj.weight", d, ff)
        norm("model.norm.weight", d)
        if not cfg["tie_word_embeddings"]:
            put("lm_head.weight", cfg["vocab_size"], d)
        return out
    d, model = cfg["width"], case["model"]
    put("embed", cfg["vocab"], d, std=1.0)
    if model == "navalorn":
        norm("embed.norm", d)
        norm("final.norm", d)
    elif model == "vavupel":
        put("bigram", cfg["embedding"]["bigram"]["buckets"] + 1, d, std=0.7)
        tanh_norm("embed.norm", d, 0.6)
        tanh_norm("final.norm", d, 0.4)
        put("loop.in", d, 2 * d)
    else:
        norm("final.norm", d)
    if model != "navalorn":
        put("head", cfg["vocab"], d)
    for i, layer in enumerate(cfg["layers"]):
        p, x, m, ff = f"l{i}.", f"l{i}.mix.", layer["mixer"], layer["mlp"]["ff"]
        H, n, mv = m["heads"], m.get("dim"), m["vdim"]
        G = m.get("kv_heads", H)
        if model == "vavupel":
            tanh_norm(p + "norm1", d, 0.6)
            tanh_norm(p + "norm1b", d, 0.9)
            tanh_norm(p + "norm2", d, 0.6)
            tanh_norm(p + "norm2b", d, 0.9)
        else:
            norm(p + "norm1", d)
            if model != "sofopel":
                norm(p + "norm2", d)
        if model in ("sofopel", "barovik"):
            put(p + "mlp.gate", ff, d)
        put(p + "mlp.up", ff, d)
        put(p + "mlp.down", d, ff)
        if model == "navalorn":
            put(p + "mlp.up.b", ff, std=0.3)
            put(p + "mlp.down.b", d, std=0.3)
        if layer["type"] == "latent_attention":
            r, rank = m["rot_dim"], m["kv_rank"]
            if model == "navalorn":
                put(x + "dq", m["q_rank"], d)
                norm(x + "dq.norm", m["q_rank"])
                put(x + "uq", H * (n + r), m["q_rank"])
            else:
                put(x + "q", H * (n + r), d)
                put(x + "sink", H, std=1.0)
                put(x + "g", H, d)
            put(x + "dkv", rank + r, d)
            norm(x + "dkv.norm", rank)
            put(x + "uk", H * n, rank)
            put(x + "uv", H * mv, rank)
            put(x + "o", d, H * mv)
        elif layer["type"] == "mamba2":
            N, groups = m["state"], m["groups"]
            inner = H * mv
            put(x + "in", 2 * inner + 2 * groups * N + H, d)
            put(x + "conv", inner + 2 * groups * N, m["conv"], std=0.5)
            put(x + "conv.b", inner + 2 * groups * N, std=0.2)
            put(x + "dt_bias", H, std=0.5, mean=-1.0)
            put(x + "A_log", H, std=0.5, mean=-0.5)
            put(x + "D", H, std=0.5, mean=1.0)
            norm(x + "norm", inner)
            put(x + "o", d, inner)
        elif layer["type"] in ("retention", "gla"):
            put(x + "q", H * n, d)
            put(x + "k", H * n, d)
            put(x + "v", H * mv, d)
            put(x + "g", H * mv, d)
            put(x + "o", d, H * mv)
            if layer["type"] == "gla":
                put(x + "a1", 16, d)
                put(x + "a2", H * n, 16)
                put(x + "a2.b", H * n, std=1.0, mean=1.0)
                norm(x + "norm", mv, 0.2)
        else:
            two = 2 if model == "sofopel" and layer["type"] == "attention" else 1
            put(x + "q", H * two * n, d)
            put(x + "k", G * two * n, d)
            put(x + "v", G * mv, d)
            put(x + "o", d, H * mv)
            if model == "barovik":
                put(x + "sink", H, std=1.0)
                put(x + "vmix", std=0.2, mean=0.4)
            elif two == 2:
                for t, c in (("q", H * 2 * n), ("k", G * 2 * n), ("v", G * mv)):
                    put(x + t + ".conv", c, m["conv"], std=0.6)
                for t in ("lq1", "lk1", "lq2", "lk2"):
                    put(x + t, n, std=0.6 / n ** 0.25)
            else:
                norm(x + "q.norm", n, 0.2)
                norm(x + "k.norm", n, 0.2)
                put(x + "g", H, d)
    return out


def lengths(case):
    """The prompts' lengths: evenly spread over the case's range, in a mixed order."""
    n, lo, hi = case["seqs"], case["shortest"], case["longest"]
    spread = [lo + (hi - lo) * i // max(1, n - 1) for i in range(n)] if n > 1 else [hi]
    step = next(s for s in range(max(1, int(n * 0.6)), 2 * n + 2) if math.gcd(s, n) == 1)
    return [spread[i * step % n] for i in range(n)]


def token_lists(case, seed):
    """Every sequence's tokens: what is cached, the prompt, and the tokens of the one-token steps."""
    gen = torch.Generator()
    gen.manual_seed(seed * 7919 + 1)
    vocab = SIZES[case["model"]][case["size"]]["vocab"]
    return [torch.randint(0, vocab, (case["cached"] + n + case["steps"],), generator=gen).tolist() for n in lengths(case)]


def _logits(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    return torch.empty((case["rows"], case["vocab"]), device=DEVICE).normal_(0.0, 2.5, generator=gen)


class State:
    pass


def prepare(case, seed):
    import ghost_infer_b200 as gi
    s = State()
    s.case = case
    if case["path"] == "sample":
        from ghost_infer_b200.sampling import DeviceSampler
        s.logits, s.ids = _logits(case, seed), list(range(case["rows"]))
        s.sampler = DeviceSampler(gi.SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=seed), DEVICE)
        s.sampler.start(case["rows"])
        return s
    model = gi.Model.from_config_dict(config(case)).bind(weights(case, seed), case["dtype"], DEVICE)
    s.tokens = token_lists(case, seed)
    longest = max(len(t) for t in s.tokens)
    llm = gi.LLM(model, max_tokens=sum(len(t) + 64 for t in s.tokens), max_slots=case["seqs"], max_seq_len=longest + 64)
    s.engine, s.cache = llm.engine, llm.cache
    s.slots = s.runner = None
    if case["path"] == "generate":
        return s
    s.held = [case["cached"] + (n if case["path"] == "decode" else 0) for n in lengths(case)]
    if max(s.held) > 0:      # what the sequences hold already
        s.slots = [s.cache.open_slot() for _ in s.tokens]
        for slot, tokens, n in zip(s.slots, s.tokens, s.held):
            s.engine.step([gi.StepEntry(slot, tokens[:n])])
    if case["path"] == "decode":
        s.runner = s.engine.decoder(s.slots)
    return s


def run(s):
    from ghost_infer_b200 import StepEntry
    case = s.case
    if case["path"] == "sample":
        return s.sampler.pick_device(s.logits, s.ids)
    slots = s.slots if s.slots is not None else [s.cache.open_slot() for _ in s.tokens]
    steps, out = case["steps"], []
    if case["path"] == "decode":
        runner = s.runner
    else:
        entries = []
        for slot, tokens in zip(slots, s.tokens):
            part = tokens[case["cached"]:len(tokens) - steps]
            entries.append(StepEntry(slot, part, range(len(part) - case["want"], len(part))))
        out.append(s.engine.step(entries))
        runner = s.engine.decoder(slots) if steps else None
    for k in range(steps):
        # the runner's logits are a buffer that its next step writes again
        out.append(runner.forward(tokens=[t[len(t) - steps + k] for t in s.tokens]).clone())
    if slots is s.slots:
        for slot, n in zip(slots, s.held):
            s.cache.truncate(slot, n)
    else:
        for slot in slots:
            s.cache.close_slot(slot)
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _per_layer(layer, model, width):
    """(weights of one run of a layer, multiply-adds per query and visible key, numbers cached per position, visible
    positions at most, numbers of per-sequence state, multiply-adds per token on that state)."""
    m, ff = layer["mixer"], layer["mlp"]["ff"]
    H, n, mv = m["heads"], m.get("dim"), m["vdim"]
    G = m.get("kv_heads", H)
    params = (3 if model in ("sofopel", "barovik") else 2) * ff * width
    span = (m.get("mask") or {}).get("size") or 1 << 30
    if layer["type"] == "latent_attention":
        r, rank = m["rot_dim"], m["kv_rank"]
        query = width * m["q_rank"] + m["q_rank"] * H * (n + r) if "q_rank" in m else width * H * (n + r)
        # keys and values of every head out of the latents once per token, then plain attention
        return params + query + width * (rank + r) + rank * H * (n + mv) + width * H * mv, H * (n + r + mv), rank + r, span, 0, 0
    if layer["type"] == "mamba2":
        inner, N, groups = H * mv, m["state"], m["groups"]
        return params + (2 * inner + 2 * groups * N + H) * width + width * inner, 0, 0, 0, H * mv * N, 2 * H * mv * N
    if layer["type"] in ("retention", "gla"):
        return params + (2 * H * n + 3 * H * mv) * width, 0, 0, 0, H * n * mv, 2 * H * n * mv
    two = 2 if model == "sofopel" and layer["type"] == "attention" else 1
    return params + (H * two * n + G * two * n + G * mv + H * mv) * width, H * two * (n + mv), G * (two * n + mv), span, 0, 0


def work(case):
    if case["path"] == "sample":
        return {"bytes": 4.0 * case["rows"] * (case["vocab"] + 1), "flops": 2.0 * case["rows"] * case["vocab"]}
    cfg, size = config(case), 2 if case["dtype"] == "bfloat16" else 4
    if case["model"] == "llama":
        d, hd, H, G = cfg["hidden_size"], cfg["head_dim"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        layers = [(d * (2 * H + 2 * G) * hd + 3 * d * cfg["intermediate_size"], H * 2 * hd, G * 2 * hd, 1 << 30, 0, 0)] * cfg["num_hidden_layers"]
        vocab, extra = cfg["vocab_size"], 0
    else:
        d, vocab = cfg["width"], cfg["vocab"]
        layers = [_per_layer(cfg["layers"][i], case["model"], d) for i, _ in runs_of(cfg)]
        extra = sum(2 * d * d for _, starts in runs_of(cfg) if starts) if case["model"] == "vavupel" else 0
    linear = sum(a[0] for a in layers) + extra
    ns, steps = lengths(case), case["steps"]
    passes = []                                        # (tokens, first position) of every sequence, per pass over the weights
    if case["path"] != "decode":
        passes.append([(n, case["cached"]) for n in ns])
    start = 0 if case["path"] == "prompt" else 1
    passes += [[(1, n + k) for n in ns] for k in range(steps if start else 0)]
    total = {"bytes": 0.0, "flops": 0.0}
    for k, seqs in enumerate(passes):
        tokens = sum(n for n, _ in seqs)
        rows = len(seqs) * (case["want"] if k == 0 and case["path"] != "decode" else 1)
        total["bytes"] += size * (linear + vocab * d + tokens * d) + 4.0 * rows * vocab
        total["flops"] += 2.0 * tokens * linear + 2.0 * rows * vocab * d
        for _, per_key, cached, span, state, per_token in layers:
            total["bytes"] += size * cached * sum(min(p, span) + n for n, p in seqs) + 8.0 * state * len(seqs)
            total["flops"] += 2.0 * per_token * tokens
            for n, p in seqs:
                whole = max(0, min(n, span - p))       # queries that see everything before them
                total["flops"] += 2.0 * per_key * (whole * p + whole * (whole + 1) / 2.0 + (n - whole) * span) if span else 0.0
    return total


def tolerance(case):
    """About four times the distance from 64-bit arithmetic that was measured; for 16-bit paths the roundings of weights,
    activations and cache through all layers, for the 32-bit path the order of its sums."""
    if case["path"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": 0.03 if case["model"] == "llama" else 0.025}


# ---- the same in 64 bits, by plain formulas over whole sequences ----------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, eps):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(z):
    return z * torch.sigmoid(z)


def _frequencies(dims, base, scaling):
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64)
    if not scaling:
        return f, 1.0

    def pair_of(turns):
        return dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    lo, hi = max(math.floor(pair_of(scaling["fast"])), 0), min(math.ceil(pair_of(scaling["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return ramp * f / scaling["factor"] + (1.0 - ramp) * f, 0.1 * math.log(scaling["factor"]) + 1.0


def _llama_frequencies(hd, theta, sc):
    f = [theta ** (-2.0 * i / hd) for i in range(hd // 2)]
    out = []
    for v in f:
        wave, orig = 2.0 * math.pi / v, sc["original_max_position_embeddings"]
        low, high = sc["low_freq_factor"], sc["high_freq_factor"]
        if wave > orig / low:
            v = v / sc["factor"]
        elif wave >= orig / high:
            s = (orig / wave - low) / (high - low)
            v = (1.0 - s) * v / sc["factor"] + s * v
        out.append(v)
    return torch.tensor(out, dtype=torch.float64)


def _turn(x, cos, sin, layout):
    """x [T, heads..., n]; cos and sin [T, pairs] turn the first 2 * pairs numbers: halves or neighbours."""
    half = cos.shape[1]
    shape = (x.shape[0],) + (1,) * (x.dim() - 2) + (half,)
    c, s = cos.view(shape), sin.view(shape)
    out = x.clone()
    ia, ib = (slice(0, half), slice(half, 2 * half)) if layout == "half" else (slice(0, 2 * half, 2), slice(1, 2 * half, 2))
    a, b = x[..., ia], x[..., ib]
    out[..., ia], out[..., ib] = a * c - b * s, b * c + a * s
    return out


def _angles(pos, rot):
    f, mag = _frequencies(rot["dims"], rot["base"], rot.get("scaling"))
    ang = pos.double()[:, None] * f.to(pos.device)[None, :]
    return torch.cos(ang) * mag, torch.sin(ang) * mag


def _attend(q, k, v, scale, window=None, keep_first=0, chunk=None, cap=None, sink=None):
    """q [T, H, n], k [T, G, n], v [T, G, m] of one sequence; `sink`: a term exp(sink_h) of the denominator alone."""
    T, H, _ = q.shape
    G = k.shape[1]
    kk, vv = (t.repeat_interleave(H // G, 1).transpose(0, 1) for t in (k, v))
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    for r in range(0, T, 1024):
        e = min(T, r + 1024)
        i, j = torch.arange(r, e, device=q.device)[:, None], torch.arange(e, device=q.device)[None, :]
        seen = j <= i
        if window:
            seen &= (i - j < window) | (j < keep_first)
        if chunk:
            seen &= i // chunk == j // chunk
        s = q[r:e].transpose(0, 1) @ kk[:, :e].transpose(1, 2) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s.masked_fill_(~seen, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[:, None, None])
        p = torch.exp(s - top)
        below = p.sum(-1, keepdim=True)
        if sink is not None:
            below = below + torch.exp(sink[:, None, None] - top)
        out[r:e] = ((p / below) @ vv[:, :e]).transpose(0, 1)
    return out


def _short_conv(u, w):
    """y[t, c] = sum_j w[c, j] u[t - taps + 1 + j, c], zeros before the start."""
    taps = w.shape[1]
    padded = torch.cat([torch.zeros((taps - 1, u.shape[1]), dtype=u.dtype, device=u.device), u])
    return sum(padded[j:j + u.shape[0]] * w[:, j] for j in range(taps))


def _walk(q, k, v, keep):
    """S <- keep_t S + k_t v_t^T, o_t = S^T q_t; q, k [T, H, n], v [T, H, m], keep [T, H, n or 1]."""
    T, H, n = k.shape
    S = torch.zeros((H, n, v.shape[2]), dtype=q.dtype, device=q.device)
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    for t in range(T):
        S = keep[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out[t] = (S * q[t][:, :, None]).sum(1)
    return out


def _each(spans, f, *rows):
    """f over every sequence's rows, put together again."""
    return torch.cat([f(*(r[a:b] for r in rows)) for a, b in spans])


def exact(case, seed):
    if case["path"] == "sample":
        return None
    if case["dtype"] == "bfloat16" and case["model"] == "llama" and case["cached"] > 0 and case["cached"] + case["longest"] > 20000:
        return None
    stored, cfg, model = weights(case, seed), config(case), case["model"]
    W = lambda name: stored[name].double()                      # noqa: E731
    lin = lambda x, name: x @ stored[name].double().T           # noqa: E731
    lists = token_lists(case, seed)
    spans, at = [], 0
    for t in lists:
        spans.append((at, at + len(t)))
        at += len(t)
    ids = torch.tensor([i for t in lists for i in t], device=DEVICE)
    pos = torch.cat([torch.arange(b - a, device=DEVICE) for a, b in spans])
    if model == "llama":
        eps, H, G, hd = cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
        # the definition's angles are 32-bit products of a 32-bit table
        f = _llama_frequencies(hd, cfg["rope_theta"], cfg["rope_scaling"]).float().to(DEVICE)
        ang = (pos.float()[:, None] * f[None, :]).double()
        cos, sin = torch.cos(ang), torch.sin(ang)
        x = stored["model.embed_tokens.weight"][ids].double()
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = _rms(x, eps) * W(p + "input_layernorm.weight")
            q, k, v = (lin(h, p + f"self_attn.{t}_proj.weight").view(at, -1, hd) for t in "qkv")
            q, k = _turn(q, cos, sin, "half"), _turn(k, cos, sin, "half")
            a = _each(spans, lambda q, k, v: _attend(q, k, v, hd ** -0.5), q, k, v)
            x = x + lin(a.reshape(at, H * hd), p + "self_attn.o_proj.weight")
            h = _rms(x, eps) * W(p + "post_attention_layernorm.weight")
            x = x + lin(_silu(lin(h, p + "mlp.gate_proj.weight")) * lin(h, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
        x = _rms(x, eps) * W("model.norm.weight")
        head = "model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"
    else:
        x, head = _exact_other(model, cfg, stored, W, lin, ids, pos, spans)
    steps, want, out = case["steps"], case["want"], []
    pick = []
    if case["path"] != "decode":
        pick.append([r for a, b in spans for r in range(b - steps - want, b - steps)])
    pick += [[b - steps + k for _, b in spans] for k in range(steps)]
    for rows in pick:
        z = x[torch.tensor(rows, device=DEVICE)] @ W(head).T
        cap = cfg.get("logit_softcap")
        out.append(cap * torch.tanh(z / cap) if cap else z)
    return out


def _exact_other(model, cfg, stored, W, lin, ids, pos, spans):
    """The last norm's rows and the name of the output matrix, for the decoders other than Llama."""
    eps, T = cfg["norm"]["eps"], len(ids)

    def tanh_norm(x, name):
        return torch.tanh(W(name + ".alpha") * x) * W(name) + W(name + ".b")

    def each(f, *rows):
        return _each(spans, f, *rows)

    x = stored["embed"][ids].double()
    if model == "navalorn":
        x = _layer_norm(x, W("embed.norm"), eps)
    elif model == "vavupel":
        b = cfg["embedding"]["bigram"]
        before = torch.cat([ids[:1], ids[:-1]])
        rows = torch.where(pos == 0, torch.full_like(ids, b["buckets"]), (before * b["mul_prev"] + ids * b["mul_cur"]) % b["buckets"])
        x = tanh_norm(x + stored["bigram"][rows].double(), "embed.norm")
    x0, first_values = x, None
    for i, starts_pass in runs_of(cfg):
        layer, p = cfg["layers"][i], f"l{i}."
        m, mix = layer["mixer"], p + "mix."
        H, n, mv = m["heads"], m.get("dim"), m["vdim"]
        if starts_pass and model == "vavupel":
            x = lin(torch.cat([x, x0], 1), "loop.in")
        h = tanh_norm(x, p + "norm1") if model == "vavupel" else _layer_norm(x, W(p + "norm1"), eps) if model == "navalorn" else _rms(x, eps) * W(p + "norm1")
        if layer["type"] == "latent_attention":
            r, rank = m["rot_dim"], m["kv_rank"]
            cq = _rms(lin(h, mix + "dq"), eps) * W(mix + "dq.norm") if model == "navalorn" else h
            q = lin(cq, mix + ("uq" if model == "navalorn" else "q")).view(T, H, n + r)
            down = lin(h, mix + "dkv")
            c = _rms(down[:, :rank], eps) * W(mix + "dkv.norm")
            cos, sin = _angles(pos, m["rot"])
            q = torch.cat([q[..., :n], _turn(q[..., n:], cos, sin, "adjacent")], -1)
            k_rot = _turn(down[:, rank:], cos, sin, "adjacent")
            k = torch.cat([lin(c, mix + "uk").view(T, H, n), k_rot[:, None, :].expand(T, H, r)], -1)
            v = lin(c, mix + "uv").view(T, H, mv)
            window, sink = (m.get("mask") or {}).get("size"), W(mix + "sink") if model == "vavupel" else None
            y = each(lambda q, k, v: _attend(q, k, v, m["scale"], window=window, sink=sink), q, k, v)
            if model == "vavupel":
                y = y * torch.sigmoid(lin(h, mix + "g"))[:, :, None]
            y = lin(y.reshape(T, H * mv), mix + "o")
        elif layer["type"] == "mamba2":
            N, groups = m["state"], m["groups"]
            inner = H * mv
            proj = lin(h, mix + "in")
            z, xbc, dt = proj[:, :inner], proj[:, inner:2 * inner + 2 * groups * N], proj[:, 2 * inner + 2 * groups * N:]
            w, bias = W(mix + "conv"), W(mix + "conv.b")
            xbc = _silu(each(lambda u: _short_conv(u, w) + bias, xbc))
            u = xbc[:, :inner].reshape(T, H, mv)
            B, C = (xbc[:, a:a + groups * N].reshape(T, groups, N).repeat_interleave(H // groups, 1) for a in (inner, inner + groups * N))
            dt = torch.nn.functional.softplus(dt + W(mix + "dt_bias"))
            keep = torch.exp(-torch.exp(W(mix + "A_log")) * dt)[:, :, None]
            y = each(_walk, C, B, dt[:, :, None] * u, keep) + W(mix + "D")[:, None] * u
            y = y.reshape(T, inner) * _silu(z)
            y = _rms(y.view(T, m["norm_groups"], -1), eps).reshape(T, inner) * W(mix + "norm")
            y = lin(y, mix + "o")
        elif layer["type"] in ("retention", "gla"):
            q, k, v = (lin(h, mix + t).view(T, H, -1) for t in "qkv")
            if layer["type"] == "retention":
                cos, sin = _angles(pos, m["rot"])
                q, k = _turn(q, cos, sin, "half"), _turn(k, cos, sin, "half") * n ** -0.5
                keep = torch.tensor(m["decay"], dtype=torch.float64, device=x.device)[None, :, None].expand(T, H, 1)
            else:
                q = q * n ** -0.5
                z = lin(lin(h, mix + "a1"), mix + "a2") + W(mix + "a2.b")
                keep = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).view(T, H, n)
            o = _rms(each(_walk, q, k, v, keep), eps)
            if layer["type"] == "gla":
                o = o * W(mix + "norm")
            y = lin(o.reshape(T, H * mv) * _silu(lin(h, mix + "g")), mix + "o")
        elif model == "barovik":
            G = m["kv_heads"]
            q, k = lin(h, mix + "q").view(T, H, n), lin(h, mix + "k").view(T, G, n)
            v = lin(h, mix + "v")
            if first_values is None:
                first_values = v
            else:
                lam = W(mix + "vmix")
                v = (1.0 - lam) * v + lam * first_values
            sink = W(mix + "sink")
            y = each(lambda q, k, v: _attend(q, k, v, m["scale"], chunk=m["mask"]["size"], cap=m["softcap"], sink=sink), q, k, v.view(T, G, mv))
            y = lin(y.reshape(T, H * mv), mix + "o")
        elif layer["type"] == "attention":                     # the difference of two maps
            G, parts = m["kv_heads"], []
            for t in "qkv":
                w = W(mix + t + ".conv")
                parts.append(each(lambda u: _short_conv(u, w), lin(h, mix + t)))
            cos, sin = _angles(pos, m["rot"])
            q, k = _turn(parts[0].view(T, H, 2, n), cos, sin, "adjacent"), _turn(parts[1].view(T, G, 2, n), cos, sin, "adjacent")
            v = parts[2].view(T, G, mv)
            lam = torch.exp(W(mix + "lq1") @ W(mix + "lk1")) - torch.exp(W(mix + "lq2") @ W(mix + "lk2")) + m["diff"]
            a, b = (each(lambda q, k, v: _attend(q, k, v, m["scale"], chunk=m["mask"]["size"]), q[:, :, j], k[:, :, j], v) for j in (0, 1))
            y = lin((_rms(a - lam * b, eps) * (1.0 - m["diff"])).reshape(T, H * mv), mix + "o")
        else:                                                  # a window that keeps first positions, a one in the denominator
            G = m["kv_heads"]
            q, k, v = lin(h, mix + "q").view(T, H, n), lin(h, mix + "k").view(T, G, n), lin(h, mix + "v").view(T, G, mv)
            cos, sin = _angles(pos, m["rot"])
            q, k = _turn(_rms(q, eps) * W(mix + "q.norm"), cos, sin, "half"), _turn(_rms(k, eps) * W(mix + "k.norm"), cos, sin, "half")
            zero = torch.zeros((H,), dtype=torch.float64, device=x.device)
            y = each(lambda q, k, v: _attend(q, k, v, m["scale"], window=m["mask"]["size"], keep_first=m["mask"]["keep_first"], sink=zero), q, k, v)
            y = lin((y * torch.sigmoid(lin(h, mix + "g"))[:, :, None]).reshape(T, H * mv), mix + "o")
        if model == "sofopel":
            limit = layer["mlp"]["limit"]
            g, u = lin(h, p + "mlp.gate").clamp(max=limit), lin(h, p + "mlp.up").clamp(-limit, limit)
            x = x + cfg["residual_mult"] * (y + lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), p + "mlp.down"))
        elif model == "vavupel":
            x = x + tanh_norm(y, p + "norm1b")
            x = x + tanh_norm(lin(lin(tanh_norm(x, p + "norm2"), p + "mlp.up").clamp(min=0.0) ** 2, p + "mlp.down"), p + "norm2b")
        elif model == "navalorn":
            x = x + y
            up = lin(_layer_norm(x, W(p + "norm2"), eps), p + "mlp.up") + W(p + "mlp.up.b")
            x = x + lin(up.clamp(min=0.0) ** 2, p + "mlp.down") + W(p + "mlp.down.b")
        else:
            x = x + y
            h = _rms(x, eps) * W(p + "norm2")
            gate = torch.nn.functional.gelu(lin(h, p + "mlp.gate"), approximate="tanh")
            x = x + lin(gate * lin(h, p + "mlp.up"), p + "mlp.down")
    if model == "vavupel":
        return tanh_norm(x, "final.norm"), "head"
    if model == "navalorn":
        return _layer_norm(x, W("final.norm"), eps), "embed"
    return _rms(x, eps) * W("final.norm"), "head"
