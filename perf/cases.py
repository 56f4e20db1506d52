"""The work this library is used for, as cases that can be timed and compared.

A case is one pass of a user's program over a model that it holds: whole requests through ``Model.step`` (prompts, then
tokens one at a time), single-token steps on sequences that are already long, whole prompts alone, or ``Model.generate``.
Weights are random at the sizes of this repository's configurations; tokens are uniform.  Sequences of a case have
lengths spread evenly between ``low`` and ``high``.

``exact`` states the same models in 64 bits with plain torch: whole sequences, no cache.  The designs with a learned
router are left out: a tie between two experts that rounding breaks the other way changes a whole row, so their logits
cannot be compared by an error norm (Lilupel's mixtures, whose experts hang on the token id, run the same grouped
products).
"""
import math

import torch

PHI2 = dict(architectures=["PhiForCausalLM"], model_type="phi", num_hidden_layers=32, hidden_size=2560,
            num_attention_heads=32, num_key_value_heads=32, intermediate_size=10240, vocab_size=51200,
            partial_rotary_factor=0.4, rope_theta=10000.0, layer_norm_eps=1e-5, hidden_act="gelu_new",
            qk_layernorm=False, tie_word_embeddings=False, max_position_embeddings=2048, initializer_range=0.02)
PHI15 = dict(PHI2, num_hidden_layers=24, hidden_size=2048, intermediate_size=8192, partial_rotary_factor=0.5)
TINY = dict(PHI2, num_hidden_layers=2, hidden_size=64, num_attention_heads=4, num_key_value_heads=4, intermediate_size=256,
            vocab_size=512, partial_rotary_factor=0.5, max_position_embeddings=128)
PHIS = {"phi-2": PHI2, "phi-1.5": PHI15, "tiny-phi": TINY}


def listed():
    return [
        # the smallest call: a model of a few hundred kilobytes in 32 bits, sampled; launches and the host are all there is
        dict(name="tiny generate", model="tiny-phi", dtype="float32", what="generate", batch=3, low=5, high=32, steps=16),
        # one user, one short question, the first tokens of the answer
        dict(name="short request", model="phi-1.5", dtype="bfloat16", what="request", batch=1, low=37, high=37, steps=12),
        # one long conversation going on
        dict(name="decode 1", model="phi-2", dtype="bfloat16", what="decode", batch=1, low=2040, high=2040, steps=4),
        # a few long conversations going on together
        dict(name="decode 8", model="phi-2", dtype="bfloat16", what="decode", batch=8, low=1900, high=2040, steps=4),
        # a server's full batch, conversations of every age
        dict(name="decode 64", model="phi-2", dtype="bfloat16", what="decode", batch=64, low=16, high=1024, steps=4),
        # one document as long as the model takes
        dict(name="prompt 2048", model="phi-2", dtype="bfloat16", what="prompt", batch=1, low=2048, high=2048, steps=0),
        # unequal prompts that arrive together
        dict(name="prompts ragged", model="phi-2", dtype="bfloat16", what="prompt", batch=16, low=16, high=1536, steps=0),
        # a small batch of requests from prompt to answer
        dict(name="requests", model="phi-1.5", dtype="bfloat16", what="request", batch=12, low=5, high=700, steps=12),
        # the true 32-bit path: a check of another implementation, a model whose weights were trained in 32 bits
        dict(name="requests fp32", model="phi-1.5", dtype="float32", what="request", batch=4, low=16, high=300, steps=6),
        # the other designs' mechanisms at a real model's layer sizes: matrix and selective-scan recurrences, attention
        # with mixed heads beside a gated linear memory, a loop
        dict(name="recurrent requests", model="vopedra-2048", dtype="bfloat16", what="request", batch=4, low=64, high=1000, steps=8),
        # state-space layers, windowed attention beside a retention, mixtures of experts: one long document
        dict(name="state-space document", model="lilupel-2048", dtype="bfloat16", what="request", batch=1, low=2047, high=2047, steps=4),
        # attention through a latent, chunked attention beside a gated recurrence, several residual streams
        dict(name="latent requests", model="nakurax-1024", dtype="bfloat16", what="request", batch=8, low=33, high=900, steps=8),
    ]


def draw(rng):
    def spread(a, b):
        return max(a, min(b, int(round(math.exp(rng.uniform(math.log(a), math.log(b + 0.999)))))))

    what = rng.choice(["request", "request", "decode", "prompt", "generate"])
    model = rng.choice({"decode": ["phi-2", "phi-1.5"], "generate": ["tiny-phi"], "prompt": ["phi-2", "phi-1.5"]}.get(
        what, ["phi-2", "phi-1.5", "phi-1.5", "vopedra-1024", "vopedra-2048", "lilupel-1024", "lilupel-2048", "nakurax-1024", "nakurax-2048"]))
    if what == "generate":
        low = spread(1, 40)
        return dict(model=model, dtype="float32", what=what, batch=spread(1, 8), low=low, high=spread(low, 80), steps=rng.randint(4, 40))
    dtype = "float32" if model == "phi-1.5" and rng.random() < 0.3 else "bfloat16"
    steps = {"request": spread(2, 16), "decode": rng.randint(2, 6), "prompt": 0}[what]
    most = 1200 if dtype == "float32" else 8000 if what != "decode" else 32000      # positions in all
    longest = 2048 - steps if what != "decode" else 2040
    batch = spread(1, 64 if what == "decode" and dtype == "bfloat16" else 16)
    high = spread(8, min(longest, max(8, most // batch)))
    return dict(model=model, dtype=dtype, what=what, batch=batch, low=spread(1, high) if batch > 1 else high, high=high, steps=steps)


# ---------------------------------------------------------------------------
# models: sizes and weights
# ---------------------------------------------------------------------------
def _config(case):
    name = case["model"]
    if name in PHIS:
        return dict(PHIS[name], torch_dtype=case["dtype"])
    design, width = name.rsplit("-", 1)
    width = int(width)
    heads, ff, hd = width // 64, 5504 * width // 2048, 64
    base = dict(vocab=32000, width=width, norm={"eps": 1e-6}, torch_dtype=case["dtype"], initializer_range=0.02)
    if design == "vopedra":
        mlp = {"kind": "dense", "ff": ff}
        mlstm = {"type": "mlstm", "mixer": {"heads": heads // 4, "dim": 2 * hd, "vdim": 4 * hd, "gate_cap": 15.0}, "mlp": mlp}
        mamba = {"type": "mamba1", "mixer": {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "conv": 4}, "mlp": mlp}
        pair = {"type": "parallel", "mlp": mlp, "mixer": {
            "left": {"heads": heads, "kv_heads": heads // 4, "dim": hd, "vdim": hd, "rot": {"dims": hd // 2, "base": 10000.0}, "scale": hd ** -0.5},
            "right": {"heads": heads, "dim": hd // 2, "vdim": hd}}}
        return dict(base, architecture="Vopedra", layers=[mlstm, mamba, pair, mlstm, mamba, pair], loop={"start": 1, "stop": 5, "times": 2})
    if design == "lilupel":
        moe = {"kind": "moe", "expert": {"ff": ff // 4 // 64 * 64}, "router": {"experts": 32, "top": 4}}
        ssd = {"type": "mamba2", "mlp": moe, "mixer": {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}}
        pair = {"type": "parallel", "mlp": moe, "mixer": {
            "left": {"heads": heads, "kv_heads": heads // 4, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": {"size": 512},
                     "rot": {"dims": hd, "base": 10000.0}},
            "right": {"heads": heads // 2, "dim": hd, "vdim": 2 * hd, "decay": [1.0 - 2.0 ** (-5 - i % 4) for i in range(heads // 2)],
                      "rot": {"dims": hd, "base": 1000000.0}},
            "left_scale": 1.0, "right_scale": 1.0}}
        return dict(base, architecture="Lilupel", layers=[ssd, ssd, pair, ssd, dict(pair, weights_of=2)] + [ssd, ssd, pair, ssd, dict(pair, weights_of=7)])
    latent = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 3 * ff // 2 // 64 * 64},
              "mixer": {"heads": heads, "dim": hd, "vdim": hd, "kv_rank": 256, "scale": hd ** -0.5}}
    pair = {"type": "parallel", "mlp": latent["mlp"], "mixer": {
        "left": {"heads": heads, "kv_heads": heads // 4, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": {"size": 512},
                 "rot": {"dims": hd, "base": 500000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}},
        "right": {"width": 5 * width // 4, "blocks": 10, "conv": 4}, "left_scale": 1.0, "right_scale": 1.0}}
    return dict(base, architecture="Nakurax", streams=4, embedding={"scale": 1.0}, layers=[latent, pair, latent, latent, pair],
                loop={"start": 0, "stop": 5, "times": 2})


def _shapes(cfg):
    """Tensor name -> (shape, (mean, spread) of a normal distribution, or how else it is drawn)."""
    s = {}
    gamma, small, wide = (1.0, 0.1), (0.0, 0.1), (0.0, 1.0)

    def mat(name, *shape):
        s[name] = (shape, (0.0, shape[-1] ** -0.5))

    if "model_type" in cfg:
        W, F, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
        both = [("model.final_layernorm", None), ("lm_head", (V, W))]
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            both += [(p + "input_layernorm", None), (p + "mlp.fc1", (F, W)), (p + "mlp.fc2", (W, F))]
            both += [(p + "self_attn." + n, (W, W)) for n in ("q_proj", "k_proj", "v_proj", "dense")]
        s["model.embed_tokens.weight"] = ((V, W), (0.0, 0.02))
        for n, shape in both:
            s[n + ".weight"] = (shape, (0.0, 0.02)) if shape else ((W,), (1.0, 0.02))
            s[n + ".bias"] = ((shape[0],) if shape else (W,), (0.0, 0.02))
        return s
    W, V, design = cfg["width"], cfg["vocab"], cfg["architecture"]
    s["embed"], s["final.norm"] = ((V, W), wide), ((W,), small if design == "Lilupel" else gamma)
    if design != "Lilupel":
        mat("head", V, W)
    if design == "Vopedra":
        s["embed.norm"], s["loop.step"] = ((W,), gamma), ((cfg["loop"]["times"], W), small)
    for i, L in enumerate(cfg["layers"]):
        if L.get("weights_of", i) != i:
            continue
        p, m = f"l{i}.", L["mixer"]
        q = p + "mix."
        F = L["mlp"].get("ff")
        for n in ("norm1", "norm2"):           # (Lilupel norms what a sublayer adds, by one plus its weights: small additions)
            s[p + n] = ((W,), (-0.7, 0.1) if design == "Lilupel" else gamma)
        if design == "Nakurax":
            S = cfg["streams"]
            for n in ("hc1", "hc2"):
                s[f"{p}{n}.in"], s[f"{p}{n}.out"], s[f"{p}{n}.mix"] = ((S,), (1.0 / S, 0.1 / S)), ((S,), gamma), ((S, S), "near identity")
            mat(p + "mlp.up", F, W), mat(p + "mlp.down", W, F)
        elif design == "Vopedra":
            mat(p + "mlp.gate", F, W), mat(p + "mlp.up", F, W), mat(p + "mlp.down", W, F)
        else:
            F, E = L["mlp"]["expert"]["ff"], L["mlp"]["router"]["experts"]
            s[p + "mlp.table"] = ((V, L["mlp"]["router"]["top"]), E)
            for e in range(E):
                mat(f"{p}mlp.e{e}.gate", F, W), mat(f"{p}mlp.e{e}.up", F, W), mat(f"{p}mlp.e{e}.down", W, F)
        if L["type"] == "mlstm":
            H, D, Vd = m["heads"], m["dim"], m["vdim"]
            mat(q + "q", H * D, W), mat(q + "k", H * D, W), mat(q + "v", H * Vd, W), mat(q + "g", H * Vd, W)
            mat(q + "i", H, W), mat(q + "f", H, W), mat(q + "o", W, H * Vd)
            s[q + "norm"], s[q + "i.b"], s[q + "f.b"] = ((H * Vd,), gamma), ((H,), wide), ((H,), (4.0, 1.0))
        elif L["type"] == "mamba1":
            C, N, R, K = m["inner"], m["state"], m["dt_rank"], m["conv"]
            mat(q + "in", 2 * C, W), mat(q + "conv", C, K), mat(q + "x", R + 2 * N, C), mat(q + "dt", C, R), mat(q + "o", W, C)
            s[q + "conv.b"], s[q + "dt.b"], s[q + "A_log"], s[q + "D"] = ((C,), small), ((C,), (-4.0, 1.0)), ((C, N), "states"), ((C,), gamma)
        elif L["type"] == "mamba2":
            H, N, G = m["heads"], m["state"], m["groups"]
            C = H * m["vdim"]
            mat(q + "in", 2 * C + 2 * G * N + H, W), mat(q + "conv", C + 2 * G * N, m["conv"]), mat(q + "o", W, C)
            s[q + "conv.b"], s[q + "dt_bias"], s[q + "A_log"] = ((C + 2 * G * N,), small), ((H,), (-3.0, 1.0)), ((H,), (1.0, 0.7))
            s[q + "D"], s[q + "norm"] = ((H,), gamma), ((C,), gamma)
        elif L["type"] == "latent_attention":
            H, D, R = m["heads"], m["dim"], m["kv_rank"]
            mat(q + "q", H * D, W), mat(q + "dkv", R, W), mat(q + "uk", H * D, R), mat(q + "uv", H * m["vdim"], R), mat(q + "o", W, H * m["vdim"])
            s[q + "dkv.norm"] = ((R,), gamma)
        else:
            a, r = m["left"], m["right"]
            H, G, D, Vd = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
            for n, rows, cols in (("q", H * D, W), ("k", G * D, W), ("v", G * Vd, W), ("o", W, H * Vd)):
                mat(f"{q}left.{n}", rows, cols)
                if design == "Lilupel":
                    s[f"{q}left.{n}.b"] = ((rows,), small)
            q2 = q + "right."
            if design == "Vopedra":
                s[q + "left.q.norm"], s[q + "left.k.norm"], s[q + "left.talk"] = ((H * D,), gamma), ((G * D,), gamma), ((H, H), "near identity")
                s[q + "left.out"], s[q2 + "out"], s[q2 + "norm"] = ((W,), gamma), ((W,), gamma), ((r["vdim"],), gamma)
                H, D, Vd = r["heads"], r["dim"], r["vdim"]
                mat(q2 + "q", H * D, W), mat(q2 + "f", H * D, W), mat(q2 + "v", H * Vd, W), mat(q2 + "o", W, H * Vd)
                s[q2 + "f.b"], s[q2 + "lower"] = ((H * D,), wide), ((H * D,), "share")
            elif design == "Lilupel":
                s[q + "left.sink"] = ((H,), wide)
                H, D, Vd = r["heads"], r["dim"], r["vdim"]
                mat(q2 + "q", H * D, W), mat(q2 + "k", H * D, W), mat(q2 + "v", H * Vd, W), mat(q2 + "g", H * Vd, W), mat(q2 + "o", W, H * Vd)
            else:
                C, B, n = r["width"], r["blocks"], r["width"] // r["blocks"]
                mat(q2 + "y", C, W), mat(q2 + "x", C, W), mat(q2 + "conv", C, r["conv"]), mat(q2 + "ra", B, n, n), mat(q2 + "ri", B, n, n), mat(q2 + "o", W, C)
                for k in ("y.b", "x.b", "conv.b"):
                    s[q2 + k] = ((C,), small)
                s[q2 + "ra.b"], s[q2 + "ri.b"], s[q2 + "lam"] = ((B, n), wide), ((B, n), wide), ((C,), (-5.0, 1.0))
    return s


def _weights(case, seed):
    """Tensor name -> tensor on the GPU, in the type a model file of this case's type holds."""
    cfg = _config(case)
    stored = getattr(torch, case["dtype"])
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    out = {}
    for name, (shape, how) in _shapes(cfg).items():
        if isinstance(how, int):               # a row of different experts for every token id
            out[name] = torch.rand((shape[0], how), generator=g, device="cuda").argsort(-1)[:, :shape[1]].to(torch.int32).contiguous()
            continue
        z = torch.randn(shape, generator=g, device="cuda", dtype=stored if len(shape) > 1 and isinstance(how, tuple) else torch.float32)
        if how == "share":
            z = torch.sigmoid(z + 2.0)
        elif how == "near identity":
            z = torch.eye(shape[0], device="cuda") + 0.1 * z
        elif how == "states":
            z = torch.log(torch.arange(1, shape[1] + 1, device="cuda").float()) + 0.1 * z
        else:
            z = z.mul_(how[1]).add_(how[0])
        out[name] = z.to(stored)
    return out


def _lengths(case):
    n, low, high = case["batch"], case["low"], case["high"]
    if n == 1:
        return [high]
    even = [low + (high - low) * i // (n - 1) for i in range(n)]
    return [even[(i * 7 + 3) % n] for i in range(n)] if n % 7 else even


def _tokens(case, seed):
    """The prompts, and the tokens fed behind them: [step][sequence]."""
    cfg = _config(case)
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    g = torch.Generator().manual_seed(7919 * seed + 5)
    prompts = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in _lengths(case)]
    return prompts, torch.randint(0, vocab, (case["steps"], case["batch"]), generator=g).tolist()


# ---------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    from gopherllm_b200.api import LoadInfo, Model, build_model
    from gopherllm_b200.cache.sequence_cache import SequenceCache
    from gopherllm_b200.config.registry import architecture_from_config
    from gopherllm_b200.engine.step import Engine
    from gopherllm_b200.weights.loader import resident_dtype, tensor_table

    # a model as load() leaves it, with weights drawn on the GPU
    cfg, dtype, device = _config(case), getattr(torch, case["dtype"]), torch.device("cuda:0")
    arch = architecture_from_config(cfg)
    typed = arch.config_class.from_dict(cfg)
    net = build_model(arch, typed)
    table = tensor_table(net.parameters(), arch.tensor_names(typed))
    drawn = _weights(case, seed)
    net.load({key: drawn[name].to(resident_dtype(spec, dtype, dtype, dtype)).contiguous() for name, (key, spec) in table.items()})
    del drawn
    prompts, fed = _tokens(case, seed)
    longest = min(net.spec.max_positions, -(-(max(map(len, prompts)) + case["steps"] + 1) // 64) * 64)
    room = sum(-(-(len(p) + case["steps"] + 1) // 64) * 64 for p in prompts)
    cache = SequenceCache(net.cache_requests(), room, longest, dtype, device, max_slots=case["batch"])
    info = LoadInfo("random", arch.name, case["dtype"], 0.0, 0, net.weight_bytes(), cache.bytes(), room)
    model = Model(arch, typed, Engine(net, cache, dtype, device), info)
    state = dict(case=case, model=model, prompts=prompts, fed=fed)
    if case["what"] == "decode":
        slots = state["slots"] = [model.open_sequence() for _ in prompts]
        for i in range(0, len(prompts), 8):
            model.step(list(zip(slots, prompts))[i:i + 8])
    return state


def run(state):
    case, model, prompts, fed = state["case"], state["model"], state["prompts"], state["fed"]
    if case["what"] == "generate":
        # answers with the default sampling, and the logits of every place of the prompts (what they score)
        answers = model.generate(prompts, max_tokens=case["steps"], temperature=0.7, top_k=40, top_p=0.9, repeat_penalty=1.1,
                                 seed=11, stop_tokens=())
        slots = [model.open_sequence() for _ in prompts]
        scores = model.step(list(zip(slots, prompts)), [list(range(len(p))) for p in prompts])
        for s in slots:
            model.close_sequence(s)
        return {"tokens": torch.tensor([a.tokens for a in answers]), "scores": scores}
    if case["what"] == "decode":
        slots = state["slots"]
        out = [model.step([(s, [t]) for s, t in zip(slots, row)]) for row in fed]
        for s, p in zip(slots, prompts):               # the next continuation starts from the same place
            model.engine.cache.commit(s, len(p))
        return out
    slots = [model.open_sequence() for _ in prompts]
    out = [model.step(list(zip(slots, prompts)))]
    for row in fed:
        out.append(model.step([(s, [t]) for s, t in zip(slots, row)]))
    for s in slots:
        model.close_sequence(s)
    return out


def work(case):
    """Every matrix once a step (of the experts, those that tokens can choose), every cached key and value that is seen once,
    the logits; two operations for a weight and a token, and for a key's and a value's element and a query."""
    cfg = _config(case)
    size = 4 if case["dtype"] == "float32" else 2
    lens, steps = _lengths(case), case["steps"]
    order = _order(cfg)
    layers = [0.0] * (max(order) + 1)                   # numbers in a layer's matrices that one token meets
    experts = [0.0] * (max(order) + 1)                  # numbers in all of a layer's experts
    phi = "model_type" in cfg
    vocab, width = (cfg["vocab_size"], cfg["hidden_size"]) if phi else (cfg["vocab"], cfg["width"])
    for name, (shape, how) in _shapes(cfg).items():
        if len(shape) < 2 or not isinstance(how, tuple) or name.startswith(("embed", "head", "lm_head", "loop", "model.embed")):
            continue
        i = int(name.split(".")[2]) if phi else int(name.split(".")[0][1:])
        if ".mlp.e" in name:
            experts[i] += math.prod(shape)
        else:
            layers[i] += math.prod(shape)
    share = 4 / 32
    attends = sum(1 for i in order if phi or cfg["layers"][i]["type"] in ("parallel", "latent_attention"))
    near = 0 if phi or cfg["architecture"] == "Vopedra" else 512
    held = 2 * width if phi else width // 2 if cfg["architecture"] != "Nakurax" else 256

    def step(new, cached):
        T = sum(new)
        touched = min(1.0, share * T)
        weights = sum(layers) + sum(experts) * touched + vocab * width
        flops = 2.0 * T * sum(layers[i] + share * experts[i] for i in order) + 2.0 * len(new) * vocab * width
        nbytes = weights * size + 4.0 * vocab * len(new)
        for n, c in zip(new, cached):
            seen = sum(min(c + j + 1, near or c + n) for j in ([0, n - 1] if n > 1 else [0])) / (2 if n > 1 else 1)
            flops += 4.0 * n * seen * width * attends
            nbytes += (min(c, near or c) + n) * held * size * attends
        return nbytes, flops

    parts = []
    if case["what"] != "decode":
        parts.append(step(lens, [0] * len(lens)))
    if case["what"] == "generate":
        parts.append(parts[0])
    for j in range(steps):
        parts.append(step([1] * len(lens), [n + j for n in lens]))
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    """Four times the relative error against ``exact`` that was measured: 3.2e-6 in 32 bits, 0.005 in bfloat16 for Phi and
    Nakurax, 0.0074 for the designs with long recurrences.  ``max``: eight standard deviations of that."""
    if case["dtype"] == "float32":
        return {"rel": 1.3e-5, "max": 1e-4, "differ": 0.01}
    return {"rel": 0.02, "max": 0.16} if case["model"].startswith(("phi", "nakurax")) else {"rel": 0.03, "max": 0.24}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    cfg, w = _config(case), _weights(case, seed)
    prompts, fed = _tokens(case, seed)
    rows = []
    with torch.no_grad():
        if case["what"] == "generate":
            return {"tokens": None, "scores": torch.cat([_logits(cfg, w, p, range(len(p))) for p in prompts])}
        for b, p in enumerate(prompts):
            first = len(p) - (case["what"] != "decode")        # the first place whose logits come back
            whole = p + [row[b] for row in fed]
            rows.append(_logits(cfg, w, whole, range(first, len(whole))))
    return [torch.stack([r[j] for r in rows]) for j in range(len(rows[0]))]


def _order(cfg):
    """The layer whose weights each layer run uses, in the order of the runs."""
    if "model_type" in cfg:
        return list(range(cfg["num_hidden_layers"]))
    own = [L.get("weights_of", i) for i, L in enumerate(cfg["layers"])]
    loop = cfg.get("loop") or {"start": 0, "stop": 0, "times": 1}
    return own[:loop["start"]] + own[loop["start"]:loop["stop"]] * loop["times"] + own[loop["stop"]:]


def _logits(cfg, w, tokens, places):
    places = torch.tensor(list(places), device="cuda")
    ids = torch.tensor(tokens, device="cuda")
    W = lambda name: w[name].double()  # noqa: E731
    return {"Vopedra": _vopedra, "Lilupel": _lilupel, "Nakurax": _nakurax}.get(cfg.get("architecture"), _phi)(cfg, W, ids, places)


def _rms(x, weight, eps):
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return x if weight is None else x * weight


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _silu(z):
    return z * torch.sigmoid(z)


def _rotate(x, dims, base, scaling=None, neighbours=False):
    """x [T, heads, dim], by position and base^(-2i / dims); pairs are dims i and i + dims / 2, or 2i and 2i + 1."""
    freq = float(base) ** (-2.0 * torch.arange(dims // 2, device=x.device).double() / dims)
    if scaling:
        wave = 2.0 * math.pi / freq
        s = ((scaling["original"] / wave - scaling["low"]) / (scaling["high"] - scaling["low"])).clamp(0.0, 1.0)
        freq = (1.0 - s) * freq / scaling["factor"] + s * freq
    angle = torch.arange(len(x), device=x.device).double()[:, None, None] * freq
    c, s = torch.cos(angle), torch.sin(angle)
    turned = x[..., :dims]
    if neighbours:
        a, b = turned[..., 0::2], turned[..., 1::2]
        return torch.cat([torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2), x[..., dims:]], -1)
    a, b = turned.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)


def _attention(q, k, v, scale, window=0, chunk=0, sink=None, talk=None):
    """q [T, H, D], k and v [T, G, D]: causal softmax attention, each key/value head for H / G query heads."""
    T, H = q.shape[:2]
    k, v = (t.repeat_interleave(H // t.shape[1], 1) for t in (k, v))
    at = torch.arange(T, device=q.device)
    seen = at[:, None] >= at
    if window:
        seen &= at[:, None] - at < window
    if chunk:
        seen &= at[:, None] // chunk == at // chunk
    if talk is None and T * T * H > 1 << 26:               # a few heads at a time
        n = max(1, (1 << 26) // (T * T))
        return torch.cat([_attention(q[:, h:h + n], k[:, h:h + n], v[:, h:h + n], scale, window, chunk, None if sink is None else sink[h:h + n])
                          for h in range(0, H, n)], 1)
    p = (torch.einsum("ihd,jhd->hij", q, k) * scale).masked_fill(~seen, -math.inf)
    if sink is None:
        p = torch.softmax(p, -1)
    else:
        p = torch.softmax(torch.cat([p, sink[:, None, None].expand(H, T, 1)], -1), -1)[..., :T]
    if talk is not None:
        p = torch.einsum("hg,gij->hij", talk, p)
    return torch.einsum("hij,jhd->ihd", p, v)


def _conv(x, taps, bias):
    """A causal filter over the tokens, channel by channel; the last tap weighs the current token."""
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    return sum(padded[j:j + len(x)] * taps[:, j] for j in range(n)) + bias


def _scan(keep, add, read):
    """S <- keep_t S + add_t, token by token; read(t, S) of each."""
    S = torch.zeros_like(add(0))
    out = []
    for t in range(len(keep)):
        S = keep[t] * S + add(t)
        out.append(read(t, S))
    return torch.stack(out)


def _phi(cfg, W, ids, places):
    H, eps = cfg["num_attention_heads"], cfg["layer_norm_eps"]
    T, width = len(ids), cfg["hidden_size"]
    hd = width // H
    lin = lambda x, n: x @ W(n + ".weight").T + W(n + ".bias")  # noqa: E731
    norm = lambda x, n: torch.nn.functional.layer_norm(x, (width,), W(n + ".weight"), W(n + ".bias"), eps)  # noqa: E731
    x = W("model.embed_tokens.weight")[ids]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        n = norm(x, p + "input_layernorm")
        q, k, v = (lin(n, f"{p}self_attn.{c}_proj").view(T, H, hd) for c in "qkv")
        rot = int(cfg["partial_rotary_factor"] * hd)
        q, k = _rotate(q, rot, cfg["rope_theta"]), _rotate(k, rot, cfg["rope_theta"])
        a = _attention(q, k, v, hd ** -0.5).reshape(T, width)
        x = x + lin(a, p + "self_attn.dense") + lin(_gelu(lin(n, p + "mlp.fc1")), p + "mlp.fc2")
    return lin(norm(x[places], "model.final_layernorm"), "lm_head")


def _vopedra(cfg, W, ids, places):
    eps, T = cfg["norm"]["eps"], len(ids)

    def mlstm(h, p, m):
        H, D, V, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = (h @ W(p + n).T for n in "qkv")
        q, k, v = q.view(T, H, D) * D ** -0.5, k.view(T, H, D), v.view(T, H, V)
        take = cap * torch.tanh((h @ W(p + "i").T + W(p + "i.b")) / cap)
        keep = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ W(p + "f").T + W(p + "f.b")) / cap))
        top, tops = torch.zeros_like(take[0]), []
        for t in range(T):
            top = torch.maximum(keep[t] + top, take[t])
            tops.append(top)
        tops = torch.stack(tops)
        before = torch.cat([torch.zeros_like(tops[:1]), tops[:-1]])
        keep, take = torch.exp(keep + before - tops)[:, :, None, None], torch.exp(take - tops)[:, :, None, None]
        v1 = torch.cat([v, v.new_ones(T, H, 1)], -1)                # the last column is the normaliser
        y = _scan(keep, lambda t: take[t] * k[t, :, :, None] * v1[t, :, None, :], lambda t, S: torch.einsum("hd,hdv->hv", q[t], S))
        y = y[..., :V] / (torch.maximum(y[..., V:].abs(), torch.exp(-tops)[..., None]) + 1e-6)
        y = _rms(y, None, eps).reshape(T, H * V) * W(p + "norm") * torch.sigmoid(h @ W(p + "g").T)
        return y @ W(p + "o").T

    def mamba1(h, p, m):
        C, N, R = m["inner"], m["state"], m["dt_rank"]
        x, z = (h @ W(p + "in").T).chunk(2, -1)
        x = _silu(_conv(x, W(p + "conv"), W(p + "conv.b")))
        dt, B, Cm = (x @ W(p + "x").T).split([R, N, N], -1)
        dt = torch.nn.functional.softplus(dt @ W(p + "dt").T + W(p + "dt.b"))
        rate = -torch.exp(W(p + "A_log"))
        S, y = torch.zeros_like(rate), []
        for t in range(T):
            S = torch.exp(dt[t][:, None] * rate) * S + (dt[t] * x[t])[:, None] * B[t]
            y.append(S @ Cm[t])
        return ((torch.stack(y) + W(p + "D") * x) * _silu(z)) @ W(p + "o").T

    def pair(h, p, m):
        a, r = m["left"], m["right"]
        H, G, D = a["heads"], a["kv_heads"], a["dim"]
        q = _rms(h @ W(p + "left.q").T, W(p + "left.q.norm"), eps).view(T, H, D)
        k = _rms(h @ W(p + "left.k").T, W(p + "left.k.norm"), eps).view(T, G, D)
        q, k = (_rotate(u, a["rot"]["dims"], a["rot"]["base"]) for u in (q, k))
        left = _attention(q, k, (h @ W(p + "left.v").T).view(T, G, -1), a["scale"], talk=W(p + "left.talk")).reshape(T, -1) @ W(p + "left.o").T
        p, H, D, V = p + "right.", r["heads"], r["dim"], r["vdim"]
        q, v = _silu(h @ W(p + "q").T).view(T, H, D), (h @ W(p + "v").T).view(T, H, V)
        f = (W(p + "lower") + (1.0 - W(p + "lower")) * torch.sigmoid(h @ W(p + "f").T + W(p + "f.b"))).view(T, H, D, 1)
        y = _scan(f, lambda t: (1.0 - f[t]) * v[t, :, None, :], lambda t, S: torch.einsum("hd,hdv->hv", q[t], S))
        right = _rms(y, W(p + "norm"), eps).reshape(T, H * V) @ W(p + "o").T
        q = p[:-6]
        return 0.5 * (_rms(left, W(q + "left.out"), eps) + _rms(right, W(q + "right.out"), eps))

    mixers = {"mlstm": mlstm, "mamba1": mamba1, "parallel": pair}
    x = x0 = _rms(W("embed")[ids], W("embed.norm"), eps)
    loop, passes = cfg["loop"], 0
    for n, i in enumerate(_order(cfg)):
        if i == loop["start"] and loop["start"] <= n < loop["start"] + (loop["stop"] - loop["start"]) * loop["times"]:
            x = x + (x0 if passes else 0.0) + W("loop.step")[passes]
            passes += 1
        L, p = cfg["layers"][i], f"l{i}."
        y = mixers[L["type"]](_rms(x, W(p + "norm1"), eps), p + "mix.", L["mixer"])
        h = _rms(x, W(p + "norm2"), eps)
        x = x + y + (_gelu(h @ W(p + "mlp.gate").T) * (h @ W(p + "mlp.up").T)) @ W(p + "mlp.down").T
    return _rms(x[places], W("final.norm"), eps) @ W("head").T


def _lilupel(cfg, W, ids, places):
    eps, T = cfg["norm"]["eps"], len(ids)

    def mamba2(h, p, m):
        H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        C = H * P
        z, xbc, dt = (h @ W(p + "in").T).split([C, C + 2 * G * N, H], -1)
        x, B, Cm = _silu(_conv(xbc, W(p + "conv"), W(p + "conv.b"))).split([C, G * N, G * N], -1)
        x = x.view(T, H, P)
        B, Cm = (u.view(T, G, N).repeat_interleave(H // G, 1) for u in (B, Cm))
        dt = torch.nn.functional.softplus(dt + W(p + "dt_bias"))
        keep = torch.exp(-torch.exp(W(p + "A_log")) * dt)[:, :, None, None]
        xd = x * dt[..., None]
        y = _scan(keep, lambda t: B[t, :, :, None] * xd[t, :, None, :], lambda t, S: torch.einsum("hn,hnp->hp", Cm[t], S))
        y = (y + W(p + "D")[:, None] * x).reshape(T, C) * _silu(z)
        y = _rms(y.view(T, m["norm_groups"], -1), None, eps).reshape(T, C) * W(p + "norm")
        return y @ W(p + "o").T

    def pair(h, p, m):
        a, r = m["left"], m["right"]
        q, k, v = (h @ W(f"{p}left.{n}").T + W(f"{p}left.{n}.b") for n in "qkv")
        q, k = (_rms(_rotate(u.view(T, -1, a["dim"]), a["rot"]["dims"], a["rot"]["base"]), None, eps) for u in (q, k))
        y = _attention(q, k, v.view(T, a["kv_heads"], -1), a["scale"], window=a["mask"]["size"], sink=W(p + "left.sink"))
        left = y.reshape(T, -1) @ W(p + "left.o").T + W(p + "left.o.b")
        p, H = p + "right.", r["heads"]
        q, k = (_rotate((h @ W(p + n).T).view(T, H, -1), r["rot"]["dims"], r["rot"]["base"]) for n in "qk")
        k, v = k * r["dim"] ** -0.5, (h @ W(p + "v").T).view(T, H, -1)
        decay = torch.tensor(r["decay"], device=h.device).double()[:, None, None].expand(T, H, 1, 1)
        y = _scan(decay, lambda t: k[t, :, :, None] * v[t, :, None, :], lambda t, S: torch.einsum("hd,hdv->hv", q[t], S))
        right = (_rms(y, None, eps).reshape(T, -1) * _silu(h @ W(p + "g").T)) @ W(p + "o").T
        return m["left_scale"] * left + m["right_scale"] * right

    x = W("embed")[ids]
    for run, i in enumerate(_order(cfg)):
        L, p = cfg["layers"][run], f"l{i}."
        y = (mamba2 if L["type"] == "mamba2" else pair)(x, p + "mix.", L["mixer"])
        x = x + _rms(y, 1.0 + W(p + "norm1"), eps)
        table, y = W(p + "mlp.table")[ids], torch.zeros_like(x)
        for e in range(L["mlp"]["router"]["experts"]):
            rows = (table == e).any(-1).nonzero()[:, 0]
            h, q = x[rows], f"{p}mlp.e{e}."
            y[rows] += (_silu(h @ W(q + "gate").T) * (h @ W(q + "up").T)) @ W(q + "down").T / table.shape[1]
        x = x + _rms(y, 1.0 + W(p + "norm2"), eps)
    return _rms(x[places], 1.0 + W("final.norm"), eps) @ W("embed").T


def _nakurax(cfg, W, ids, places):
    eps, T = cfg["norm"]["eps"], len(ids)

    def latent(h, p, m):
        H = m["heads"]
        c = _rms(h @ W(p + "dkv").T, W(p + "dkv.norm"), eps)
        q, k, v = (u.view(T, H, -1) for u in (h @ W(p + "q").T, c @ W(p + "uk").T, c @ W(p + "uv").T))
        return _attention(q, k, v, m["scale"]).reshape(T, -1) @ W(p + "o").T

    def pair(h, p, m):
        a, r = m["left"], m["right"]
        q, k, v = ((h @ W(f"{p}left.{n}").T).view(T, -1, a["dim"]) for n in "qkv")
        q, k = (_rotate(u, a["rot"]["dims"], a["rot"]["base"], a["rot"]["scaling"], neighbours=True) for u in (q, k))
        left = _attention(q, k, v, a["scale"], chunk=a["mask"]["size"]).reshape(T, -1) @ W(p + "left.o").T
        p, B = p + "right.", r["blocks"]
        u = _conv(h @ W(p + "x").T + W(p + "x.b"), W(p + "conv"), W(p + "conv.b"))
        gates = [torch.sigmoid(torch.einsum("tbn,bmn->tbm", u.view(T, B, -1), W(p + n)) + W(p + n + ".b")).reshape(T, -1) for n in ("ra", "ri")]
        log_a = -8.0 * gates[0] * torch.nn.functional.softplus(W(p + "lam"))
        add = torch.sqrt(-torch.expm1(2.0 * log_a)) * gates[1] * u
        S = _scan(torch.exp(log_a), lambda t: add[t], lambda t, S: S)
        right = (S * _gelu(h @ W(p + "y").T + W(p + "y.b"))) @ W(p + "o").T
        return m["left_scale"] * left + m["right_scale"] * right

    def connected(X, p, sublayer):
        y = sublayer(torch.einsum("s,stw->tw", W(p + "in"), X))
        return torch.einsum("sr,stw->rtw", W(p + "mix"), X) + W(p + "out")[:, None, None] * y

    X = (W("embed")[ids] * cfg["embedding"]["scale"]).expand(cfg["streams"], -1, -1)
    for i in _order(cfg):
        L, p = cfg["layers"][i], f"l{i}."
        mix = latent if L["type"] == "latent_attention" else pair
        X = connected(X, p + "hc1.", lambda u: mix(_rms(u, W(p + "norm1"), eps), p + "mix.", L["mixer"]))
        X = connected(X, p + "hc2.", lambda u: torch.relu(_rms(u, W(p + "norm2"), eps) @ W(p + "mlp.up").T) ** 2 @ W(p + "mlp.down").T)
    return _rms(X[:, places].sum(0), W("final.norm"), eps) @ W("head").T
