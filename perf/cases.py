"""What a user has this engine do, as cases that can be timed and checked.

A pass is what a program does that drives the step function itself (``Engine.forward``, the entry point that the trace replay and
any scheduler of one's own stand on): requests that already hold a context bring their next token, new requests are opened and bring
their prompts, cut as they come into steps of mixed work; then the new requests go on for some steps, a token at a time, and are
closed. The logits of all steps are kept and come back as one tensor. Token ids are given (as in scoring or in a replay), so a pass can be repeated.

Models: the layers of the Llama-3.1-8B preset (8 of its 32, with the whole vocabulary), of the Llama-3.2-3B preset in 32 bits (2 of its
28), and the six other designs at the larger size at which the benchmark sets them beside the Llama decoder (width 2048, six layers or
runs). Two of these have a dense feed-forward, or none, in the place of their mixture: their routers stand behind a norm that gives
every layer's output the same weight as the stream, so an expert that wins by a rounding changes a token's logits by a third, and two
correct 16-bit runs would not be comparable. The mixtures are measured in the Nidilix and the Tutizen design.

``exact`` states every design once more in float64, on whole sequences, from the formulas.
"""

import math

import torch

F64 = torch.float64
PAGE = 16


# ------------------------------------------------------------------------------------------------------------------- the models
def _llama(name, layers):
    from stride_b200 import preset
    return dict(preset(name), num_hidden_layers=layers)


def _nidilix():
    latent = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "rot": {"base": 10000.0, "dims": 64}, "scale": 192 ** -0.5}
    mlp = {"kind": "moe", "router": {"experts": 32, "top": 4}, "expert": {"ff": 768}, "shared": {"ff": 1024}}
    recurrent = {"type": "rglru", "mixer": {"width": 2560, "blocks": 10, "conv": 4}, "mlp": mlp}
    return {"architecture": "Nidilix", "width": 2048, "vocab": 32000, "residual_mult": 0.5, "norm": {"eps": 1e-6}, "token_side": {"dim": 128},
            "layers": [recurrent, recurrent, {"type": "latent_attention", "mixer": latent, "mlp": mlp},
                       recurrent, recurrent, {"type": "latent_attention", "mixer": dict(latent, kv_from=2), "mlp": mlp}]}


def _migelix():
    rot = {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 4096, "fast": 16.0, "slow": 2.0}}
    heads = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024}}
    right = {"heads": 16, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 128}
    mlp = {"kind": "dense", "ff": 5504}
    kinds = [{"type": "parallel", "mixer": {"left": dict(heads, rot=rot), "right": right, "left_scale": 0.7, "right_scale": 1.2}, "mlp": mlp},
             {"type": "wkv", "mixer": {"heads": 32, "dim": 64, "decay_rank": 64}, "mlp": mlp},
             {"type": "attention", "mixer": dict(heads, softcap=30.0, rot={"base": 500000.0, "dims": 128}), "mlp": mlp}]
    return {"architecture": "Migelix", "width": 2048, "vocab": 32000, "norm": {"eps": 1e-6}, "logit_softcap": 30.0, "layers": kinds * 2}


def _tutizen():
    heads = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    dense = {"kind": "dense", "ff": 5504, "limit": 7.0}
    moe = {"kind": "moe", "expert": {"ff": 1024, "limit": 7.0}, "shared": {"ff": 1408, "limit": 7.0},
           "router": {"experts": 32, "top": 4, "scale": 2.5, "groups": {"count": 8, "keep": 4}}}
    layers = [{"type": "attention", "mixer": dict(heads, kv_from=i - 1) if i % 2 else heads, "mlp": moe if i % 2 else dense} for i in range(6)]
    return {"architecture": "Tutizen", "width": 2048, "vocab": 32000, "norm": {"eps": 1e-6}, "residual_mult": 0.7, "layers": layers}


def _netusun():
    latent = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 768, "scale": 192 ** -0.5,
              "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}}}
    heads = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "conv": 4, "mask": {"size": 1024}, "softcap": 30.0}
    mlp = {"kind": "dense", "ff": 5504}
    layers = [{"type": "latent_attention", "mixer": latent, "mlp": mlp}, {"type": "attention", "mixer": heads, "mlp": mlp},
              {"type": "mlstm", "mixer": {"heads": 16, "dim": 128, "vdim": 128, "gate_cap": 15.0}, "mlp": mlp},
              {"type": "attention", "mixer": heads, "mlp": mlp}]
    return {"architecture": "Netusun", "width": 2048, "vocab": 32000, "norm": {"eps": 1e-6}, "layers": layers,
            "loop": {"start": 0, "stop": 2, "times": 2}}


def _dopudra():
    memory = {"heads": 16, "dim": 128, "vdim": 128}
    left = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "conv": 4, "bias_max": 256, "buckets": 32,
            "q_temp": {"coef": 0.1, "every": 512}}
    mlp = {"kind": "dense", "ff": 8256}
    fading = {"type": "lightning", "mixer": dict(memory, decay=[1.0 - 2.0 ** (-2.0 - 8.0 * h / 16) for h in range(16)]), "mlp": mlp}
    both = {"type": "parallel", "mixer": {"left": left, "right": dict(memory, tau=16.0, decay_rank=16), "left_scale": 1.0, "right_scale": 1.0}, "mlp": mlp}
    return {"architecture": "Dopudra", "width": 2048, "vocab": 32000, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0}, "streams": 4,
            "max_positions": 8192, "layers": [fading, fading, both] * 2}


def _negotar():
    attention = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0, "v_mix": True,
                 "rot": {"base": 500000.0, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    memory = {"heads": 64, "vdim": 64, "groups": 8, "state": 128, "conv": 4, "norm_groups": 8}
    return {"architecture": "Negotar", "width": 2048, "vocab": 32000, "norm": {"eps": 1e-6}, "logit_scale": 0.5,
            "layers": [{"type": "mamba2", "mixer": memory, "mlp": None}, {"type": "attention", "mixer": attention, "mlp": None}] * 3}


MODELS = {"llama-8b": lambda: _llama("llama3.1-8b", 8), "llama-3b-f32": lambda: _llama("llama3.2-3b", 2), "nidilix": _nidilix,
          "migelix": _migelix, "tutizen": _tutizen, "netusun": _netusun, "dopudra": _dopudra, "negotar": _negotar}


# -------------------------------------------------------------------------------------------------------------------- the cases
def _case(model, standing=0, context=0, ragged=False, prompts=0, tokens=0, rows=1, steps=0, name=None):
    """``standing`` requests of ``context`` tokens (ragged: down to half of it) bring their next token; ``prompts`` new requests bring
    ``tokens`` tokens in all, with logits for the last ``rows`` of each, and then go on for ``steps`` steps."""
    c = {"model": model, "standing": standing, "context": context, "ragged": ragged, "prompts": prompts, "tokens": tokens, "rows": rows, "steps": steps}
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one user, a short conversation: latency of a single token
        _case("llama-8b", 1, 2048, name="llama_decode_1x2048"),
        # the headline of this repository's benchmark: eight users with long contexts
        _case("llama-8b", 8, 8192, name="llama_decode_8x8192"),
        # a busy server: requests of every length, a batch that is no power of two
        _case("llama-8b", 57, 1500, ragged=True, name="llama_decode_57_ragged"),
        # the first token of a prompt that fills the step's token budget
        _case("llama-8b", prompts=1, tokens=2048, name="llama_prompt_2048"),
        # continuous batching: three prompts come in beside nineteen running requests
        _case("llama-8b", 19, 900, ragged=True, prompts=3, tokens=1003, name="llama_mixed"),
        # the 32-bit path, which the 16-bit one is checked with: two prompts and what follows them
        _case("llama-3b-f32", prompts=2, tokens=301, steps=3, name="llama_f32"),
        # a long prompt into recurrent layers, latent attention and a mixture
        _case("nidilix", prompts=1, tokens=2048, rows=32, name="nidilix_prompt_2048"),
        # several prompts into the delta rule, the decayed memory and windowed attention, and the tokens after them
        _case("migelix", prompts=3, tokens=1750, steps=4, name="migelix_3_requests"),
        # eight short questions, answered by a model with routed experts: decode of a batch
        _case("tutizen", prompts=8, tokens=531, rows=4, steps=12, name="tutizen_8_requests"),
        # scoring the end of a long text with latent and windowed attention and the matrix LSTM
        _case("netusun", prompts=1, tokens=1999, rows=32, name="netusun_score_1999"),
        # five requests through fading memories and copies of the stream
        _case("dopudra", prompts=5, tokens=1201, steps=6, name="dopudra_5_requests"),
        # two prompts into state space layers, and a few tokens
        _case("negotar", prompts=2, tokens=1503, steps=3, name="negotar_2_requests"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.5:
        kind = rng.choice(["decode", "decode", "prompt", "mixed", "f32"])
        if kind == "decode":
            n = _log(rng, 1, 64)
            return _case("llama-8b", n, _log(rng, 64, min(8192, 65536 // n)), ragged=rng.random() < 0.6)
        if kind == "prompt":
            n = _log(rng, 1, 8)
            return _case("llama-8b", prompts=n, tokens=_log(rng, 12 * n, 2048))
        if kind == "mixed":
            n = _log(rng, 1, 32)
            return _case("llama-8b", n, _log(rng, 64, 2048), ragged=True, prompts=rng.randint(1, 4), tokens=_log(rng, 64, 2048 - n))
        return _case("llama-3b-f32", prompts=rng.randint(1, 3), tokens=_log(rng, 20, 300), steps=rng.randint(0, 3))
    model = rng.choice(["nidilix", "migelix", "tutizen", "netusun", "dopudra", "negotar"])
    n = _log(rng, 1, 8)
    if rng.random() < 0.5:
        return _case(model, prompts=n, tokens=_log(rng, 48 * n, 2048), rows=max(8, 32 // n), steps=0)
    return _case(model, prompts=n, tokens=_log(rng, 16 * n, 640), rows=4, steps=rng.randint(4, 12))


def _contexts(case):
    n, c = case["standing"], case["context"]
    return [max(2, c - (c // 2) * ((7 * i) % n) // n) if case["ragged"] else c for i in range(n)]


def _lengths(case):
    """Prompt lengths: between once and twice a common measure, adding up to ``tokens``."""
    n, total = case["prompts"], case["tokens"]
    if not n:
        return []
    parts = [n + (3 * i) % n if n % 3 else n + i for i in range(n)]
    lengths = [max(1, total * p // sum(parts)) for p in parts]
    lengths[-1] += total - sum(lengths)
    return lengths


def _tokens(case, seed, vocab):
    """Token ids of every request: its context or its prompt, and what follows."""
    g = torch.Generator().manual_seed(int(seed) * 2 + 1)
    lengths = _contexts(case) + [n + case["steps"] for n in _lengths(case)]
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for n in lengths]


def _dtype(case):
    return "float32" if case["model"].endswith("f32") else "bfloat16"


class _State:
    pass


def prepare(case, seed):
    from stride_b200 import Engine
    config = MODELS[case["model"]]()
    vocab = config.get("vocab", config.get("vocab_size"))
    s = _State()
    s.case, s.next_key, s.tokens = case, 1000, _tokens(case, seed, vocab)
    pages = sum(-(-len(t) // PAGE) + 1 for t in s.tokens)
    s.engine = Engine(config=config, random_weights=seed, dtype=_dtype(case), block_size=PAGE, num_blocks=pages + 160, max_batch_seqs=64)
    # the running requests' contexts, in portions as they fit the token budget
    work, room = [], 2048
    for key in range(case["standing"]):
        tokens, at = s.tokens[key], 0
        s.engine.cache.open(key, "user")
        if not s.engine.cache.ensure(key, len(tokens), 0):
            raise RuntimeError("the page pool is too small")
        while at < len(tokens) - 1:
            n = min(room, len(tokens) - 1 - at)
            work.append((key, tokens[at:at + n], at, []))
            at, room = at + n, room - n
            if room == 0:
                s.engine.forward(work)
                work, room = [], 2048
    if work:
        s.engine.forward(work)
    return s


def run(s):
    case, engine = s.case, s.engine
    first = case["standing"]
    work = [(key, [s.tokens[key][-1]], len(s.tokens[key]) - 1, [0]) for key in range(first)]
    new = []
    for i, n in enumerate(_lengths(case)):
        key = s.next_key + i
        engine.cache.open(key, "user")
        if not engine.cache.ensure(key, n + case["steps"], 0):
            raise RuntimeError("the page pool is too small")
        new.append((key, s.tokens[first + i], n))
        work.insert(i, (key, s.tokens[first + i][:n], 0, list(range(max(0, n - case["rows"]), n))))
    s.next_key += len(new)
    logits = engine.forward(work)
    if case["steps"]:
        steps = [logits.clone()]                # a view that the next step reuses
        for step in range(case["steps"]):
            steps.append(engine.forward([(key, [tokens[n + step]], n + step, [0]) for key, tokens, n in new]).clone())
        logits = torch.cat(steps)
    for key, _tokens_of, _n in new:
        engine.cache.close(key)
    return logits


# ------------------------------------------------------------------------------------------------- tensors, work and tolerances
def _tensors(cfg):
    """Matrices of a model by name: shape. (Vectors are ones everywhere, as the engine's random weights have them.)"""
    t = {}
    if "architectures" in cfg:
        h, hd, ff = cfg["hidden_size"], cfg["head_dim"], cfg["intermediate_size"]
        t["model.embed_tokens.weight"] = (cfg["vocab_size"], h)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for n, rows in (("q", cfg["num_attention_heads"]), ("k", cfg["num_key_value_heads"]), ("v", cfg["num_key_value_heads"])):
                t[f"{p}self_attn.{n}_proj.weight"] = (rows * hd, h)
            t[p + "self_attn.o_proj.weight"] = (h, cfg["num_attention_heads"] * hd)
            t.update({p + "mlp.gate_proj.weight": (ff, h), p + "mlp.up_proj.weight": (ff, h), p + "mlp.down_proj.weight": (h, ff)})
        if not cfg["tie_word_embeddings"]:
            t["lm_head.weight"] = (cfg["vocab_size"], h)
        return t
    W, V, design = cfg["width"], cfg["vocab"], cfg["architecture"]
    t["embed"] = (V, W)
    if design in ("Nidilix", "Tutizen", "Dopudra"):
        t["head"] = (V, W)
    if design == "Dopudra":
        t["pos"] = (cfg["max_positions"], W)
    if design == "Netusun":
        t["loop.in"] = (W, 2 * W)
    side = cfg.get("token_side", {}).get("dim")
    if side:
        t["side.embed"] = (V, side * len(cfg["layers"]))

    def heads(p, m, values=True, keys=True):
        t[p + "q"], t[p + "o"] = (m["heads"] * m["dim"], W), (W, m["heads"] * m["vdim"])
        if keys:
            t[p + "k"] = (m["kv_heads"] * m["dim"], W)
        if keys and values:
            t[p + "v"] = (m["kv_heads"] * m["vdim"], W)

    def memory(p, m, gate=True):
        for n, rows in (("q", m["dim"]), ("k", m["dim"]), ("v", m["vdim"])):
            t[p + n] = (m["heads"] * rows, W)
        if gate:
            t[p + "g"] = (m["heads"] * m["vdim"], W)
        t[p + "o"] = (W, m["heads"] * m["vdim"])

    for i, layer in enumerate(cfg["layers"]):
        p, m, kind, mlp = f"l{i}.mix.", layer["mixer"], layer["type"], layer["mlp"]
        if kind == "rglru":
            bw = m["width"] // m["blocks"]
            t.update({p + "y": (m["width"], W), p + "x": (m["width"], W), p + "o": (W, m["width"]), p + "conv": (m["width"], m["conv"])})
            t.update({p + "ra": (m["blocks"], bw, bw), p + "ri": (m["blocks"], bw, bw)})
        elif kind == "latent_attention":
            H, wide = m["heads"], m["dim"] + m["rot_dim"]
            t.update({p + "uk": (H * m["dim"], m["kv_rank"]), p + "uv": (H * m["vdim"], m["kv_rank"]), p + "o": (W, H * m["vdim"])})
            if "q_rank" in m:
                t.update({p + "dq": (m["q_rank"], W), p + "uq": (H * wide, m["q_rank"]), p + "g": (H * m["vdim"], W)})
            else:
                t.update({p + "q": (H * wide, W), p + "g": (H, W)})
            if "kv_from" not in m:
                t[p + "dkv"] = (m["kv_rank"] + m["rot_dim"], W)
        elif kind == "wkv":
            n = m["heads"] * m["dim"]
            t.update({p + k: (n, W) for k in "rkvg"})
            t.update({p + "w1": (m["decay_rank"], W), p + "w2": (n, m["decay_rank"]), p + "o": (W, n)})
        elif kind == "mlstm":
            memory(p, m)
            t.update({p + "i": (m["heads"], W), p + "f": (m["heads"], W)})
        elif kind == "lightning":
            memory(p, m)
        elif kind == "mamba2":
            inner = m["heads"] * m["vdim"]
            t.update({p + "in": (2 * inner + 2 * m["groups"] * m["state"] + m["heads"], W), p + "o": (W, inner)})
        elif kind == "parallel" and design == "Migelix":
            r = m["right"]
            heads(p + "left.", m["left"], values=False)
            memory(p + "right.", r, gate=False)
            q = p + "right."
            t.update({q + "b": (r["heads"], W), q + "a1": (r["decay_rank"], W), q + "a2": (r["heads"] * r["dim"], r["decay_rank"]),
                      q + "g1": (r["gate_rank"], W), q + "g2": (r["heads"] * r["vdim"], r["gate_rank"])})
        elif kind == "parallel":
            r = m["right"]
            heads(p + "left.", m["left"])
            memory(p + "right.", r)
            t.update({p + "right.a1": (r["decay_rank"], W), p + "right.a2": (r["heads"] * r["dim"], r["decay_rank"])})
        else:
            heads(p, m, values=design != "Migelix", keys="kv_from" not in m)
            if design == "Migelix":
                t[p + "g"] = (m["heads"] * m["vdim"], W)
            if design == "Tutizen":
                t[p + "g"] = (m["heads"], W)
        p = f"l{i}.mlp."
        gated = design not in ("Nidilix", "Dopudra")

        def unit(q, ff):
            if gated:
                t[q + "gate"] = (ff, W)
            t[q + "up"], t[q + "down"] = (ff, W), (W, ff)

        if mlp and mlp["kind"] == "moe":
            t[p + "router"] = (mlp["router"]["experts"], W)
            for e in range(mlp["router"]["experts"]):
                unit(f"{p}e{e}.", mlp["expert"]["ff"])
            unit(p + "shared.", mlp["shared"]["ff"])
            if design == "Tutizen":
                t[p + "shared.sg"] = (1, W)
        elif mlp:
            unit(p, mlp["ff"])
        if side:
            t.update({f"l{i}.side.gate": (side, W), f"l{i}.side.proj": (W, side)})
    return t


def _runs(cfg):
    """Layers in the order in which they run."""
    n, loop = cfg.get("num_hidden_layers") or len(cfg["layers"]), cfg.get("loop")
    if not loop:
        return list(range(n))
    return list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], n))


def _kept(cfg):
    """For every run of a layer: what attention keeps a token (numbers), what its scores and sums cost a (query, key) pair
    (multiply-adds), the window, what its memory holds a request (numbers), and the multiply-adds of a token in it."""
    out = []
    for i in _runs(cfg):
        if "architectures" in cfg:
            hd = cfg["head_dim"]
            out.append((2 * cfg["num_key_value_heads"] * hd, 2 * cfg["num_attention_heads"] * hd, 0, 0, 0))
            continue
        m, kind = cfg["layers"][i]["mixer"], cfg["layers"][i]["type"]
        a, r = (m["left"], m["right"]) if kind == "parallel" else (m, m)
        keep = pair = window = held = token = 0
        if kind in ("attention", "parallel"):
            keep, pair = a["kv_heads"] * (a["dim"] + a["vdim"]), a["heads"] * (a["dim"] + a["vdim"])
            window = (a.get("mask") or {}).get("size", 0)
        if kind == "latent_attention":
            keep, pair = m["kv_rank"] + m["rot_dim"], m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        if kind == "rglru":
            held, token = m["width"], 4 * m["width"]
        elif kind == "mamba2":
            held = m["heads"] * m["vdim"] * m["state"]
            token = 2 * held
        elif kind not in ("attention", "latent_attention"):
            held = r["heads"] * r["dim"] * r.get("vdim", r["dim"])
            token = (3 if kind == "parallel" and "kv_heads" in r else 2) * held
        out.append((keep, pair, window, held, token))
    return out


def _calls(case):
    """(new tokens, tokens before them) of every request, for every step of a pass."""
    lengths = _lengths(case)
    calls = [[(n, 0) for n in lengths] + [(1, c - 1) for c in _contexts(case)]]
    return calls + [[(1, n + s) for n in lengths] for s in range(case["steps"])]


def work(case):
    cfg = MODELS[case["model"]]()
    item = 4 if _dtype(case) == "float32" else 2
    tensors, runs, kept = _tensors(cfg), _runs(cfg), _kept(cfg)
    V, W = tensors["model.embed_tokens.weight" if "architectures" in cfg else "embed"]
    total_bytes = total_flops = 0.0
    for number, call in enumerate(_calls(case)):
        tokens = sum(n for n, _c in call)
        rows = sum(min(n, case["rows"]) if not c else 1 for n, c in call) if number == 0 else len(call)
        weights = float(V * W)                                                      # the head, or the table that stands for it
        flops = 2.0 * rows * V * W
        for name, shape in tensors.items():
            if "layers." not in name and not (name[0] == "l" and name[1].isdigit()) and name != "loop.in":
                continue
            size = float(math.prod(shape))
            if "layers" in cfg and name != "loop.in":
                layer = cfg["layers"][int(name[1:name.index(".")])]
                times = sum(1 for r in runs if r == int(name[1:name.index(".")]))
                part = name.split(".")[2]
                if part[0] == "e" and part[1:].isdigit():                           # an expert: read if one token of the step takes it
                    share = layer["mlp"]["router"]["top"] / layer["mlp"]["router"]["experts"]
                    weights += size * (1.0 - (1.0 - share) ** tokens)
                    flops += 2.0 * tokens * size * share
                    continue
                weights, flops = weights + size, flops + 2.0 * tokens * size * times / (shape[0] if len(shape) == 3 else 1)
            else:
                times = cfg["loop"]["times"] if name == "loop.in" else 1
                weights, flops = weights + size, flops + 2.0 * tokens * size * times
        moved = 0.0
        for keep, pair, window, held, token in kept:
            for n, c in call:
                reach = min(c, window - 1) if window else c
                moved += (n + reach) * keep * item + (held * 4 * (2 if c else 1))
                pairs = n * reach + n * (n + 1) / 2 if not window or n + reach <= window else n * (reach + min(n, window)) / 2
                flops += 2.0 * pairs * pair + 2.0 * n * token
        total_bytes += weights * item + moved + rows * V * 4.0 + tokens * (W * item + 4)
        total_flops += flops
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    # 32-bit: sums of 3,072 and 8,192 terms in another order, three orders of magnitude above one rounding. 16-bit: every product's
    # result is rounded to 8 bits, and six to eight layers of them carry the roundings on; prompts cut in other places (other kernels,
    # other orders of the sums) moved the logits by 0.002 to 0.007.
    return {"rel": 1e-5} if _dtype(case) == "float32" else {"rel": 0.025, "max": 0.5}


# ------------------------------------------------------------------------------------------------------- the designs in float64
def _fnv(name):
    h = 0xCBF29CE484222325
    for b in name.encode():
        h = ((h ^ b) * 0x100000001B3) & 0xFFFFFFFFFFFFFFFF
    return h


class _Weights:
    """The engine's seeded random weights: N(0, 0.02), every tensor from a generator of its own, as stored in the model's element type."""

    def __init__(self, cfg, seed, dtype):
        self.shapes, self.seed, self.dtype, self.kept = _tensors(cfg), int(seed), dtype, {}

    def __getitem__(self, name):
        t = self.kept.get(name)
        if t is None:
            g = torch.Generator(device="cuda")
            g.manual_seed((_fnv(name) ^ (self.seed * 0x9E3779B97F4A7C15)) & 0x7FFFFFFFFFFFFFFF)
            t = (torch.randn(self.shapes[name], generator=g, dtype=torch.float32, device="cuda") * 0.02).to(self.dtype).to(F64)
            self.kept[name] = t
        return t


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _angles(T, rot):
    """Angles [T, dims / 2] and the factor on cos and sin of a rotation with or without rescaled frequencies."""
    dims, base, sc = rot["dims"], float(rot["base"]), rot.get("scaling")
    f, factor = [base ** (-2.0 * i / dims) for i in range(dims // 2)], 1.0
    if sc and "fast" in sc:
        at = lambda turns: dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f, factor = [x / sc["factor"] * r + x * (1.0 - r) for x, r in zip(f, ramp)], 0.1 * math.log(sc["factor"]) + 1.0
    elif sc:
        for i, x in enumerate(f):
            wave = 2.0 * math.pi / x
            s = min(max((sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"]), 0.0), 1.0)
            f[i] = (1.0 - s) * x / sc["factor"] + s * x
    return torch.arange(T, dtype=F64, device="cuda")[:, None] * torch.tensor(f, dtype=F64, device="cuda"), factor


def _turn(x, angles, factor=1.0, neighbours=False):
    """x [T, heads, n]: the first 2 x (number of angles) entries turn, pairwise or half against half."""
    n = angles.shape[1]
    c, s = (angles.cos() * factor)[:, None, :], (angles.sin() * factor)[:, None, :]
    out = x.clone()
    a, b = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if neighbours else (slice(0, n), slice(n, 2 * n))
    u, v = x[..., a], x[..., b]
    out[..., a], out[..., b] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, first=0, window=0, cap=None, sink=None, slopes=None, table=None):
    """q [n, H, D] of the queries from position ``first`` on, k and v [T, G, .] from position 0 on."""
    n, H, _ = q.shape
    T, G, _ = k.shape
    k, v = (t.transpose(0, 1).repeat_interleave(H // G, 0) for t in (k, v))
    out = []
    for a in range(0, n, 512):
        i = torch.arange(first + a, first + min(n, a + 512), device="cuda")
        end = int(i[-1]) + 1
        j = torch.arange(end, device="cuda")
        s = (q[a:a + 512].transpose(0, 1) @ k[:, :end].transpose(1, 2)) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        far = i[:, None] - j[None, :]
        if slopes is not None:
            s = s - slopes[:, None, None] * far
        if table is not None:
            s = s + table[:, far.clamp(min=0)]
        seen = (far >= 0) & (far < window) if window else far >= 0
        s = s.masked_fill(~seen, float("-inf"))
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = top.clamp(min=sink)
        e = torch.exp(s - top)
        den = e.sum(-1, keepdim=True) + (torch.exp(sink - top) if sink is not None else 0.0)
        out.append(((e / den) @ v[:, :end]).transpose(0, 1))
    return torch.cat(out)


def _conv(u, taps):
    """A causal convolution whose taps are all one (vectors) or given."""
    T, n = u.shape[0], taps if isinstance(taps, int) else taps.shape[1]
    padded = torch.cat([torch.zeros(n - 1, u.shape[1], dtype=F64, device="cuda"), u])
    return sum(padded[j:j + T] * (1.0 if isinstance(taps, int) else taps[:, j]) for j in range(n))


def _scan(keep, k, v, q, bonus=False, beta=None):
    """A matrix memory a head: S <- keep S + k v^T, o = S^T q; keep [T, H, D] or [T, H, 1]. ``bonus``: o is read before the decay with
    the token's own term; ``beta``: the delta rule, which writes beta (v - S^T k) behind the decay."""
    T, H, D = k.shape
    S = torch.zeros(H, D, v.shape[2], dtype=F64, device="cuda")
    out = torch.empty(T, H, v.shape[2], dtype=F64, device="cuda")
    for t in range(T):
        if bonus:
            S2 = S + k[t][:, :, None] * v[t][:, None, :]
            out[t] = (S2 * q[t][:, :, None]).sum(1)
            S = keep[t][:, :, None] * S + (S2 - S)
            continue
        S = keep[t][:, :, None] * S
        new = v[t] if beta is None else beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
        S = S + k[t][:, :, None] * new[:, None, :]
        out[t] = (S * q[t][:, :, None]).sum(1)
    return out


def _mixture(h, w, p, ids, weights, unit):
    out = torch.zeros_like(h)
    for e in ids.unique().tolist():
        rows, which = (ids == e).nonzero(as_tuple=True)
        out[rows] += weights[rows, which][:, None] * unit(h[rows], f"{p}e{e}.")
    return out


def _forward_llama(cfg, w, tokens, rows):
    eps, hd, H, G = cfg["rms_norm_eps"], cfg["head_dim"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
    T, sc = len(tokens), cfg["rope_scaling"]
    # the table's angles are float32 products of float32 frequencies by definition
    f = 1.0 / (cfg["rope_theta"] ** (torch.arange(0, hd, 2, dtype=torch.float32) / hd))
    wave = 2 * math.pi / f
    s = ((sc["original_max_position_embeddings"] / wave - sc["low_freq_factor"]) / (sc["high_freq_factor"] - sc["low_freq_factor"])).clamp(0.0, 1.0)
    f = (1 - s) * (f / sc["factor"]) + s * f
    angles = torch.outer(torch.arange(T, dtype=torch.float32), f).cuda().to(F64)
    x = w["model.embed_tokens.weight"][torch.tensor(tokens, device="cuda")]
    last = cfg["num_hidden_layers"] - 1
    for i in range(last + 1):
        p = f"model.layers.{i}."
        h = _unit(x, eps)
        k = _turn((h @ w[p + "self_attn.k_proj.weight"].T).view(T, G, hd), angles)
        v = (h @ w[p + "self_attn.v_proj.weight"].T).view(T, G, hd)
        start = 0 if i < last else min(rows)                    # the last layer: only the wanted end of the sequence
        h, x = h[start:], x[start:]
        q = _turn((h @ w[p + "self_attn.q_proj.weight"].T).view(T - start, H, hd), angles[start:])
        x = x + _attend(q, k, v, hd ** -0.5, first=start).reshape(T - start, -1) @ w[p + "self_attn.o_proj.weight"].T
        for a in range(0, x.shape[0], 2048):
            h = _unit(x[a:a + 2048], eps)
            x[a:a + 2048] += (_silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    return _unit(x[[r - min(rows) for r in rows]], eps) @ w["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"].T


def _latent(h, w, p, m, eps, kept, neighbours):
    T, H, D, R, DV = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"]
    angles, factor = _angles(T, m["rot"])
    if kept is None:
        d = h @ w[p + "dkv"].T
        kept = _unit(d[:, :m["kv_rank"]], eps), _turn(d[:, None, m["kv_rank"]:], angles, factor, neighbours)
    c, shared = kept
    q = (_unit(h @ w[p + "dq"].T, eps) @ w[p + "uq"].T if "q_rank" in m else h @ w[p + "q"].T).view(T, H, D + R)
    q = torch.cat([q[..., :D], _turn(q[..., D:], angles, factor, neighbours)], -1)
    k = torch.cat([(c @ w[p + "uk"].T).view(T, H, D), shared.expand(T, H, R)], -1)
    o = _attend(q, k, (c @ w[p + "uv"].T).view(T, H, DV), m["scale"], sink=1.0 if "q_rank" in m else None)
    gate = torch.sigmoid(h @ w[p + "g"].T)
    return (o * gate.view(T, H, -1)).reshape(T, H * DV) @ w[p + "o"].T, kept


def _forward_nidilix(cfg, w, tokens, rows):
    eps, mult, n, kept = cfg["norm"]["eps"], cfg["residual_mult"], cfg["token_side"]["dim"], {}
    ids = torch.tensor(tokens, device="cuda")
    T, x = len(tokens), w["embed"][ids]
    norm = lambda x: torch.tanh(x) + 1.0                                                                       # noqa: E731
    unit = lambda h, p: torch.relu(h @ w[p + "up"].T) ** 2 @ w[p + "down"].T                                   # noqa: E731
    for i, layer in enumerate(cfg["layers"]):
        p, m, h = f"l{i}.mix.", layer["mixer"], norm(x)
        if layer["type"] == "rglru":
            B = m["blocks"]
            y = _gelu(h @ w[p + "y"].T + 1.0)
            u = _conv(h @ w[p + "x"].T + 1.0, w[p + "conv"]) + 1.0
            r, g = (torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(T, B, -1), w[p + k]).reshape(T, -1) + 1.0) for k in ("ra", "ri"))
            a = torch.exp(-8.0 * r * math.log1p(math.e))
            add, S, out = torch.sqrt(1.0 - a * a) * g * u, torch.zeros_like(u[0]), torch.empty_like(u)
            for t in range(T):
                S = a[t] * S + add[t]
                out[t] = S
            x = x + mult * ((out * y) @ w[p + "o"].T)
        else:
            y, kept[i] = _latent(h, w, p, m, eps, kept.get(m.get("kv_from")), True)
            x = x + mult * y
        p, h, router = f"l{i}.mlp.", norm(x), layer["mlp"]["router"]
        z, chosen = (h @ w[p + "router"].T + 1.0).topk(router["top"], -1)
        x = x + mult * (_mixture(h, w, p, chosen, torch.softmax(z, -1), unit) + unit(h, p + "shared."))
        g = _gelu(x @ w[f"l{i}.side.gate"].T) * w["side.embed"][ids][:, i * n:(i + 1) * n]
        x = x + mult * _unit(g @ w[f"l{i}.side.proj"].T, eps)
    return norm(x[rows]) @ w["head"].T


def _forward_migelix(cfg, w, tokens, rows):
    eps, T = cfg["norm"]["eps"], len(tokens)
    x = w["embed"][torch.tensor(tokens, device="cuda")]
    norm = lambda x: _unit(x, eps) * 2.0                                                                       # noqa: E731

    def attention(h, p, m, bias, sink):
        q, k = (h @ w[p + "q"].T + bias).view(T, m["heads"], -1), (h @ w[p + "k"].T + bias).view(T, m["kv_heads"], -1)
        angles, factor = _angles(T, m["rot"])
        return _attend(_turn(q, angles, factor, True), _turn(k, angles, factor, True), k, m["scale"], window=m["mask"]["size"],
                       cap=m.get("softcap"), sink=sink).reshape(T, -1)

    for i, layer in enumerate(cfg["layers"]):
        p, m, h = f"l{i}.mix.", layer["mixer"], norm(x)
        if layer["type"] == "parallel":
            left = attention(h, p + "left.", m["left"], 1.0, 1.0) @ w[p + "left.o"].T
            r, p = m["right"], p + "right."
            q, k, v = (_silu(_conv(h @ w[p + n].T, r["conv"])).view(T, r["heads"], -1) for n in "qkv")
            q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * r["dim"] ** -0.5
            k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            keep = torch.exp(-math.e * torch.nn.functional.softplus(h @ w[p + "a1"].T @ w[p + "a2"].T + 1.0)).view(T, r["heads"], -1)
            o = _unit(_scan(keep, k, v, q, beta=torch.sigmoid(h @ w[p + "b"].T)), eps).reshape(T, -1)
            right = (o * torch.sigmoid(h @ w[p + "g1"].T @ w[p + "g2"].T)) @ w[p + "o"].T
            x = x + m["left_scale"] * left + m["right_scale"] * right
        elif layer["type"] == "wkv":
            prev = torch.cat([torch.zeros_like(h[:1]), h[:-1]])         # every mix is wholly the token before: its factors are one
            r, k, v = ((prev @ w[p + n].T).view(T, m["heads"], -1) for n in "rkv")
            keep = torch.exp(-torch.exp(torch.tanh(prev @ w[p + "w1"].T) @ w[p + "w2"].T + 1.0)).view(T, m["heads"], -1)
            x = x + (_unit(_scan(keep, k, v, r, bonus=True), eps).reshape(T, -1) * _silu(prev @ w[p + "g"].T)) @ w[p + "o"].T
        else:
            x = x + (attention(h, p, m, 0.0, None) * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T
        p, h = f"l{i}.mlp.", norm(x)
        x = x + (_gelu(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T
    z = norm(x[rows]) @ w["embed"].T
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def _forward_tutizen(cfg, w, tokens, rows):
    eps, mult, W, T, kept = cfg["norm"]["eps"], cfg["residual_mult"], cfg["width"], len(tokens), {}
    a = torch.arange(T, dtype=F64, device="cuda")[:, None] * 10000.0 ** (-2.0 * torch.arange(W // 2, dtype=F64, device="cuda") / W)
    x = w["embed"][torch.tensor(tokens, device="cuda")] + torch.stack([a.sin(), a.cos()], -1).reshape(T, W)

    def unit(h, p, limit=7.0):
        g, u = (h @ w[p + "gate"].T).clamp(max=limit), (h @ w[p + "up"].T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[p + "down"].T

    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        H = m["heads"]
        if "kv_from" not in m:
            kept[i] = tuple(_unit((x @ w[p + n].T + 1.0).view(T, m["kv_heads"], -1), eps) for n in "kv")
        k, v = kept[m.get("kv_from", i)]
        slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=F64, device="cuda") / H)
        o = _attend(_unit((x @ w[p + "q"].T + 1.0).view(T, H, -1), eps), k, v, m["scale"], slopes=slopes)
        x = x + mult * _unit((o * torch.sigmoid(x @ w[p + "g"].T)[:, :, None]).reshape(T, -1) @ w[p + "o"].T + 1.0, eps)
        p = f"l{i}.mlp."
        if mlp["kind"] == "dense":
            y = unit(x, p)
        else:
            r = mlp["router"]
            s = torch.sigmoid(x @ w[p + "router"].T)
            groups = (s + 1.0).view(T, r["groups"]["count"], -1)
            best = groups.topk(2, -1)[0].sum(-1).topk(r["groups"]["keep"], -1)[1]
            allowed = torch.zeros_like(groups[..., 0], dtype=torch.bool).scatter(1, best, True)
            chosen = groups.masked_fill(~allowed[..., None], float("-inf")).reshape(T, -1).topk(r["top"], -1)[1]
            weights = s.gather(1, chosen)
            y = _mixture(x, w, p, chosen, weights / (weights.sum(-1, keepdim=True) + 1e-20) * r["scale"], unit)
            y = y + torch.sigmoid(x @ w[p + "shared.sg"].T) * unit(x, p + "shared.")
        x = x + mult * _unit(y, eps)
    return _unit(x[rows], eps) @ w["head"].T


def _forward_netusun(cfg, w, tokens, rows):
    eps, T, loop = cfg["norm"]["eps"], len(tokens), cfg["loop"]
    x = x0 = w["embed"][torch.tensor(tokens, device="cuda")]
    for i in _runs(cfg):
        if i == loop["start"]:
            x = torch.cat([x, x0], -1) @ w["loop.in"].T + 1.0
        p, m, h = f"l{i}.mix.", cfg["layers"][i]["mixer"], _unit(x, eps)
        kind, H = cfg["layers"][i]["type"], m["heads"]
        if kind == "latent_attention":
            y, _kept_here = _latent(h, w, p, m, eps, None, False)
        elif kind == "attention":
            q, k, v = (_conv(h @ w[p + n].T, m["conv"]) for n in "qkv")
            q, k, v = _unit(q.view(T, H, -1), eps), _unit(k.view(T, m["kv_heads"], -1), eps), v.view(T, m["kv_heads"], -1)
            y = _attend(q, k, v, m["scale"], window=m["mask"]["size"], cap=m["softcap"], sink=0.0).reshape(T, -1) @ w[p + "o"].T
        else:
            q, k, v = ((h @ w[p + n].T).view(T, H, -1) for n in "qkv")
            q, cap = q * m["dim"] ** -0.5, m["gate_cap"]
            gi, gf = (cap * torch.tanh((h @ w[p + n].T + 1.0) / cap) for n in "if")
            lf = torch.nn.functional.logsigmoid(gf)
            tops, top = [], torch.zeros(H, dtype=F64, device="cuda")
            for t in range(T):
                tops.append(torch.maximum(lf[t] + top, gi[t]))
                top = tops[-1]
            tops = torch.stack(tops)
            before = torch.cat([torch.zeros_like(tops[:1]), tops[:-1]])
            keep, take = torch.exp(lf + before - tops)[..., None], torch.exp(gi - tops)[..., None]
            o = _scan(keep, k * take, torch.cat([v, torch.ones_like(v[..., :1])], -1), q)          # the last column is the norm's sum
            o = o[..., :-1] / (torch.maximum(o[..., -1:].abs(), torch.exp(-tops)[..., None]) + 1e-6)
            y = (_unit(o, eps).reshape(T, -1) * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T
        x = x + _unit(y, eps)
        p, h = f"l{i}.mlp.", _unit(x, eps)
        x = x + _unit((_silu(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T, eps)
    return _unit(x[rows], eps) @ w["embed"].T


def _forward_dopudra(cfg, w, tokens, rows):
    eps, T = cfg["norm"]["eps"], len(tokens)
    x = w["embed"][torch.tensor(tokens, device="cuda")] * cfg["embedding"]["scale"] + w["pos"][:T]
    X = x[None].repeat(cfg["streams"], 1, 1)                    # every number of the reads, mixes and writes is one
    for i, layer in enumerate(cfg["layers"]):
        p, m, h = f"l{i}.mix.", layer["mixer"], _unit(X.sum(0), eps)
        if layer["type"] == "lightning":
            q, k, v = (_silu(h @ w[p + n].T).view(T, m["heads"], -1) for n in "qkv")
            keep = torch.tensor(m["decay"], dtype=F64, device="cuda")[None, :, None].expand(T, -1, 1)
            y = (_unit(_scan(keep, k, v, q).reshape(T, -1), eps) * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T
        else:
            a, q = m["left"], p + "left."
            Q, K, V = (_conv(h @ w[q + n].T, a["conv"]) for n in "qkv")
            Q, K, V = _unit(Q, eps).view(T, a["heads"], -1), _unit(K, eps).view(T, a["kv_heads"], -1), V.view(T, a["kv_heads"], -1)
            grow = torch.tensor([1.0 + a["q_temp"]["coef"] * math.log((t + 1) // a["q_temp"]["every"] + 1) for t in range(T)], dtype=F64, device="cuda")
            # a learned number a bucket of distances; a vector, hence one, for all of them
            table = torch.ones(a["heads"], T, dtype=F64, device="cuda")
            left = _attend(Q * grow[:, None, None], K, V, a["scale"], table=table).reshape(T, -1) @ w[q + "o"].T
            r, q = m["right"], p + "right."
            Q, K, V = ((h @ w[q + n].T).view(T, r["heads"], -1) for n in "qkv")
            keep = (torch.sigmoid(h @ w[q + "a1"].T @ w[q + "a2"].T + 1.0) ** (1.0 / r["tau"])).view(T, r["heads"], -1)
            o = _unit(_scan(keep, K, V, Q / math.sqrt(r["dim"])), eps).reshape(T, -1) * _silu(h @ w[q + "g"].T)
            y = m["left_scale"] * left + m["right_scale"] * (o @ w[q + "o"].T)
        X = X.sum(0, keepdim=True) + y[None].expand(cfg["streams"], -1, -1)
        p, h = f"l{i}.mlp.", _unit(X.sum(0), eps)
        X = X.sum(0, keepdim=True) + (torch.relu(h @ w[p + "up"].T) ** 2 @ w[p + "down"].T)[None].expand(cfg["streams"], -1, -1)
    return _unit(X.sum(0)[rows], eps) @ w["head"].T


def _forward_negotar(cfg, w, tokens, rows):
    eps, T, values = cfg["norm"]["eps"], len(tokens), None
    x = w["embed"][torch.tensor(tokens, device="cuda")]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H = m["heads"]
        if layer["type"] == "mamba2":
            inner, GN = H * m["vdim"], m["groups"] * m["state"]
            z, u, dt = torch.split(x @ w[p + "in"].T, [inner, inner + 2 * GN, H], 1)
            u, dt = _silu(_conv(u, m["conv"]) + 1.0), torch.nn.functional.softplus(dt + 1.0)
            v = u[:, :inner].reshape(T, H, -1)
            k, q = (t.reshape(T, m["groups"], -1).repeat_interleave(H // m["groups"], 1) for t in (u[:, inner:inner + GN], u[:, inner + GN:]))
            y = (_scan(torch.exp(-math.e * dt)[..., None], k, v * dt[..., None], q) + v).reshape(T, inner) * _silu(z)
            y = _unit(y.view(T, m["norm_groups"], -1), eps).reshape(T, inner) @ w[p + "o"].T
        else:
            q, k, v = ((x @ w[p + n].T + 1.0).view(T, n_heads, -1) for n, n_heads in (("q", H), ("k", m["kv_heads"]), ("v", m["kv_heads"])))
            values = v if values is None else values                    # the share of the first layer's values is one
            angles, _factor = _angles(T, m["rot"])
            y = _attend(_unit(_turn(q, angles), eps), _unit(_turn(k, angles), eps), values, m["scale"], cap=m["softcap"]).reshape(T, -1) @ w[p + "o"].T
        x = x + 2.0 * _unit(y, eps)
    return 2.0 * _unit(x[rows], eps) @ w["embed"].T * cfg["logit_scale"]


_FORWARD = {"nidilix": _forward_nidilix, "migelix": _forward_migelix, "tutizen": _forward_tutizen, "netusun": _forward_netusun,
            "dopudra": _forward_dopudra, "negotar": _forward_negotar}


def exact(case, seed):
    cfg = MODELS[case["model"]]()
    vocab = cfg.get("vocab", cfg.get("vocab_size"))
    w = _Weights(cfg, seed, getattr(torch, _dtype(case)))
    forward = _FORWARD.get(case["model"], _forward_llama)
    tokens = _tokens(case, seed, vocab)
    first, prompts, steps = [], [], [[] for _ in range(case["steps"])]
    for ids in tokens[:case["standing"]]:
        first.append(forward(cfg, w, ids, [len(ids) - 1]))
    for ids, n in zip(tokens[case["standing"]:], _lengths(case)):
        rows = list(range(max(0, n - case["rows"]), n + case["steps"]))
        z = forward(cfg, w, ids, rows)
        prompts.append(z[:z.shape[0] - case["steps"]])
        for s in range(case["steps"]):
            steps[s].append(z[z.shape[0] - case["steps"] + s][None])
    return torch.cat(prompts + first + [row for rows in steps for row in rows])
