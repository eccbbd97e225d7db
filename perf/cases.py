"""The passes that this library's speed is judged by: prompt steps, decode steps and whole generation calls.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) a model with random weights, its engine, and the tokens of the pass
    run(state)          one pass through the public entry points
    work(case)          the bytes and operations a pass cannot do without
    tolerance(case)     how far another correct implementation may be off
    exact(case, seed)   the pass's logits in 64 bits, in plain torch

A case has a `kind`:

  decode    one step of a `DecodeSession`: every sequence goes on by one token from a context it already holds.  The
            step is repeated at the same position (a position computed again leaves the cache as it was).
  prompts   one `Engine.step` that brings whole prompts of unequal lengths, taken into free slots and given back
            afterwards; with `continuing`, that many sequences in the middle of their answers go on by one token in the
            same step, as when requests join a running batch.  Logits are wanted at each sequence's last token.
  generate  `Model.generate_ids` from host lists to host lists, and `Model.get_logits` of every prompt.

Models are GPT-2 in its four sizes and three of the other designs in the two sizes that bench.py uses for them: Kotisun
(windowed attention beside a state-space recurrence, a residual in streams, looped layers), Pelenex (three recurrences
with a matrix state per head, routed experts) and Kuvusun (latent attention, routed experts).
"""
from __future__ import annotations

import math
import types

import numpy as np
import torch
import torch.nn.functional as F

from vlrf_b200 import Model, SamplingParams
from vlrf_b200.config import load_preset
from vlrf_b200.engine import BuildOptions, Engine, StepEntry, parse_dtype
from vlrf_b200.engine.decode import DecodeSession
from vlrf_b200.registry import parse_config
from vlrf_b200.weights.spec import check_tensors

DEVICE = "cuda"


# ---- the cases --------------------------------------------------------------------------------------------------------

def listed() -> list:
    return [
        # one user typing: the fewest bytes a step can have, so launches and latencies count
        dict(name="gpt2 decode 1", kind="decode", model="gpt2", dtype="bfloat16", batch=1, shortest=200, longest=200),
        # the batch of the headline benchmark, sequences of unequal age
        dict(name="gpt2 decode 8", kind="decode", model="gpt2", dtype="bfloat16", batch=8, shortest=380, longest=660),
        # a full server: the cache is most of the traffic
        dict(name="gpt2 decode 64", kind="decode", model="gpt2", dtype="bfloat16", batch=64, shortest=100, longest=900),
        # the largest preset: weights are most of the traffic
        dict(name="gpt2-xl decode 8", kind="decode", model="gpt2-xl", dtype="bfloat16", batch=8, shortest=400, longest=640),
        # two long prompts, the shape of the headline prompt benchmark
        dict(name="gpt2 prompts 2048", kind="prompts", model="gpt2", dtype="bfloat16", lengths="1024,1024", continuing=0, context=0),
        # requests of odd lengths that join three sequences in the middle of their answers, on the largest preset
        dict(name="gpt2-xl prompts joining", kind="prompts", model="gpt2-xl", dtype="bfloat16", lengths="1013,517,389,97,31",
             continuing=3, context=300),
        # a whole call in 32 bits with sampling as a user leaves it: prompts and tokens in host memory
        dict(name="gpt2 generate float32", kind="generate", model="gpt2", dtype="float32", lengths="143,61,29,7", new_tokens=24,
             temperature=0.8, top_k=50, top_p=0.9, repetition_penalty=1.0, no_repeat_ngram=0),
        # long prompts through a recurrence beside windowed attention
        dict(name="kotisun-s prompts 2048", kind="prompts", model="kotisun-s", dtype="bfloat16", lengths="1024,1024", continuing=0,
             context=0),
        # the same design at its larger size, answering
        dict(name="kotisun-m decode 8", kind="decode", model="kotisun-m", dtype="bfloat16", batch=8, shortest=500, longest=1200),
        # three kinds of recurrence and routed experts over ragged prompts
        dict(name="pelenex-m prompts ragged", kind="prompts", model="pelenex-m", dtype="bfloat16", lengths="777,650,411,90", continuing=0,
             context=0),
        # their states and experts at a medium batch
        dict(name="pelenex-s decode 32", kind="decode", model="pelenex-s", dtype="bfloat16", batch=32, shortest=150, longest=800),
        # latent attention and routed experts, answering
        dict(name="kuvusun-s decode 16", kind="decode", model="kuvusun-s", dtype="bfloat16", batch=16, shortest=300, longest=1000),
    ]


def _log_int(rng, low: int, high: int) -> int:
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng) -> dict:
    kind = rng.choice(["decode", "decode", "decode", "prompts", "prompts", "prompts", "generate"])
    if kind == "generate":
        lengths = [_log_int(rng, 1, 150) for _ in range(rng.randint(1, 4))]
        return dict(kind=kind, model="gpt2", dtype="float32", lengths=",".join(map(str, lengths)), new_tokens=rng.randint(4, 24),
                    temperature=rng.choice([0.0, 0.8, 1.1]), top_k=rng.choice([0, 50, 7]), top_p=rng.choice([1.0, 0.9]),
                    repetition_penalty=rng.choice([1.0, 1.0, 1.2]), no_repeat_ngram=rng.choice([0, 0, 3]))
    model = rng.choice(["gpt2", "gpt2", "gpt2-medium", "gpt2-large", "gpt2-xl", "kotisun-s", "kotisun-m", "pelenex-s", "pelenex-m",
                        "kuvusun-s", "kuvusun-m"])
    dtype = "float32" if model == "gpt2" and rng.random() < 0.15 else "bfloat16"
    big = model in ("gpt2-large", "gpt2-xl") or model.endswith("-m")
    most = 1000 if model.startswith("gpt2") else 1400
    if kind == "decode":
        batch = _log_int(rng, 1, 16 if big or dtype == "float32" else 64)
        longest = _log_int(rng, 8, most)
        return dict(kind=kind, model=model, dtype=dtype, batch=batch, shortest=rng.randint(max(1, longest // 4), longest), longest=longest)
    left, lengths = (400 if dtype == "float32" else 1500 if big else 2048), []
    for _ in range(rng.randint(1, 6)):
        n = min(_log_int(rng, 2, most), left)
        if n > 0:
            lengths.append(n)
            left -= n
    continuing = rng.choice([0, 0, 1, 5])
    return dict(kind=kind, model=model, dtype=dtype, lengths=",".join(map(str, lengths)), continuing=continuing,
                context=_log_int(rng, 20, 500) if continuing else 0)


# ---- configurations (the sizes of the presets and of bench.py's designs) --------------------------------------------------

KOTISUN = {
    "s": dict(width=1024, heads=16, kv_heads=4, dim=64, vdim=96, window=512, rot=32, r_heads=32, r_vdim=64, state=64, groups=4,
              norm_groups=4, ff=2816),
    "m": dict(width=2048, heads=16, kv_heads=2, dim=128, vdim=128, window=1024, rot=64, r_heads=32, r_vdim=128, state=128, groups=8,
              norm_groups=8, ff=5632),
}
PELENEX = {
    "s": dict(width=1024, heads=16, kv_heads=4, dim=64, window=512, keep=64, decayed=(16, 64, 128), stabilized=(8, 64, 256),
              delta=(8, 4, 128, 128), ff=2816, experts=16, top=2, expert_ff=1024, shared_ff=1024),
    "m": dict(width=2048, heads=16, kv_heads=2, dim=128, window=1024, keep=128, decayed=(32, 128, 128), stabilized=(16, 128, 256),
              delta=(32, 16, 128, 128), ff=5632, experts=32, top=4, expert_ff=1408, shared_ff=2816),
}
KUVUSUN = {
    "s": dict(width=1024, heads=16, dim=64, rot=32, vdim=64, kv_rank=256, q_rank=384, ff=4096, experts=16, top=2, expert_ff=1024,
              shared_ff=1024),
    "m": dict(width=2048, heads=16, dim=128, rot=64, vdim=128, kv_rank=512, q_rank=768, ff=8192, experts=32, top=4, expert_ff=1408,
              shared_ff=2816),
}
VOCAB = 32000


def _moe(z: dict) -> dict:
    return {"kind": "moe", "expert": {"ff": z["expert_ff"]}, "router": {"experts": z["experts"], "top": z["top"]},
            "shared": {"ff": z["shared_ff"]}}


def _config(model: str) -> dict:
    if model.startswith("gpt2"):
        return load_preset(model)
    design, size = model.split("-")
    if design == "kotisun":
        z = KOTISUN[size]
        left = {"heads": z["heads"], "kv_heads": z["kv_heads"], "dim": z["dim"], "vdim": z["vdim"], "scale": z["dim"] ** -0.5,
                "mask": {"size": z["window"]}, "rot": {"base": 10000.0, "dims": z["rot"], "scaling": {"factor": 2.0}}}
        right = {"heads": z["r_heads"], "vdim": z["r_vdim"], "state": z["state"], "groups": z["groups"], "conv": 4,
                 "norm_groups": z["norm_groups"]}
        layer = {"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 0.7, "right_scale": 0.7},
                 "mlp": {"kind": "dense", "ff": z["ff"]}}
        return {"architecture": "Kotisun", "vocab": VOCAB, "width": z["width"], "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
                "streams": 4, "loop": {"start": 1, "stop": 2, "times": 2}, "logit_softcap": 30.0, "layers": [layer] * 3}
    if design == "pelenex":
        z = PELENEX[size]
        left = {"heads": z["heads"], "kv_heads": z["kv_heads"], "dim": z["dim"], "vdim": z["dim"], "scale": z["dim"] ** -0.5,
                "mask": {"size": z["window"], "keep_first": z["keep"]}}
        (gh, gk, gv), (lh, lk, lv), (dh, dg, dk, dv) = z["decayed"], z["stabilized"], z["delta"]
        dense = {"kind": "dense", "ff": z["ff"]}
        lstm = {"type": "mlstm", "mixer": {"heads": lh, "dim": lk, "vdim": lv, "gate_cap": 15.0}, "mlp": _moe(z)}
        side = {"type": "parallel", "mixer": {"left": left, "right": {"heads": gh, "dim": gk, "vdim": gv, "tau": 16.0}}, "mlp": dense}
        delta = {"type": "channel_delta", "mixer": {"heads": dh, "kv_heads": dg, "dim": dk, "vdim": dv, "conv": 4}, "mlp": dense}
        return {"architecture": "Pelenex", "vocab": VOCAB, "width": z["width"], "norm": {"eps": 1e-5, "groups": 4}, "logit_softcap": 30.0,
                "layers": [side, lstm, delta, lstm]}
    z = KUVUSUN[size]
    first = {"type": "latent_attention", "mixer": {"heads": z["heads"], "dim": z["dim"], "vdim": z["vdim"], "kv_rank": z["kv_rank"],
                                                   "q_rank": z["q_rank"], "scale": z["dim"] ** -0.5}}
    second = {"heads": z["heads"], "dim": z["dim"], "vdim": z["vdim"], "kv_rank": z["kv_rank"], "rot_dim": z["rot"],
              "rot": {"base": 10000.0, "dims": z["rot"]}, "scale": (z["dim"] + z["rot"]) ** -0.5}
    layers = [dict(first, mlp={"kind": "dense", "ff": z["ff"]}), {"type": "latent_attention_2", "mixer": second, "mlp": _moe(z)},
              {"type": "latent_attention_2", "mixer": dict(second, kv_from=1), "mlp": _moe(z)}, dict(first, mlp=_moe(z))]
    return {"architecture": "Kuvusun", "vocab": VOCAB, "width": z["width"], "norm": {"eps": 1e-5, "groups": 4}, "layers": layers}


# ---- weights and tokens, from the seed alone --------------------------------------------------------------------------------

def _draw_weights(config: dict, seed: int, dtype: torch.dtype, device) -> dict:
    """Random weights by tensor name, matrices in `dtype`, vectors in float32.  Scales keep every sublayer's output near
    that of its input; gates, decays and steps are spread so that some heads forget within a few tokens and others keep
    hundreds.  Routers decide clearly, as trained ones do: a token's embedding has a part along the directions of the
    experts it belongs to, and the experts' shares of the vocabulary are even."""
    arch, cfg = parse_config(config)
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    width = config.get("n_embd", config.get("width"))
    moe = next((layer["mlp"] for layer in config.get("layers", []) if layer["mlp"]["kind"] == "moe"), None)
    toward = None
    if moe is not None:
        toward = torch.randn((moe["router"]["experts"], width), generator=gen, device=device)
        toward /= toward.norm(dim=1, keepdim=True)
    out = {}
    for spec in arch.weight_spec(cfg):
        name, shape, last = spec.name, spec.drawn_shape, spec.name.rsplit(".", 1)[-1]
        t = torch.randn(shape, generator=gen, device=device)
        if config.get("model_type") == "gpt2":
            if spec.kind == "vector":
                t = 1.0 + 0.1 * t if last == "weight" else 0.05 * t
            elif name in ("wte.weight", "wpe.weight"):
                t = t * (0.05 if name == "wte.weight" else 0.02)
            else:
                t = t * (0.8 / shape[0] ** 0.5)                   # (stored [in, out])
        elif last == "router":
            layer = int(name.split(".")[0][1:])
            t = 0.3 * toward.roll(layer, 0) + t * (0.05 / shape[-1] ** 0.5)
        elif name == "embed":
            if toward is not None:
                mine = torch.rand((shape[0], len(toward)), generator=gen, device=device).topk(moe["router"]["top"], dim=1).indices
                for j in range(mine.shape[1]):
                    t += 16.0 * toward[mine[:, j]]
        elif ".hc" in name:
            streams = config["streams"]
            t = {"in": 1.0 / streams + 0.2 * t, "out": 1.0 + 0.3 * t}.get(last) if last != "mix" else torch.eye(streams, device=device) + 0.15 * t
        elif last == "dt_bias":
            t = -2.0 + 1.0 * t.clamp(-2.0, 2.0)
        elif last == "A_log":
            t = -0.2 + 0.8 * t.clamp(-2.5, 1.5)
        elif last == "conv":
            t = t / shape[-1] ** 0.5
        elif name.endswith(".f.b"):
            t = 3.0 + t
        elif name.endswith(".a2.b"):
            t = 1.0 + 1.5 * t
        elif last == "b" and name.endswith("router.b"):
            t = 0.1 * t
        elif name.endswith(".i.b"):
            pass
        elif last == "b" and spec.kind == "vector":
            t = 0.3 * t
        elif spec.kind == "vector":
            t = 1.0 + 0.1 * t
        else:
            t = t / shape[-1] ** 0.5
        out[name] = t if spec.kind == "vector" else t.to(dtype)
    return out


def _decoder(case: dict, seed: int):
    config, dtype = _config(case["model"]), parse_dtype(case["dtype"])
    arch, cfg = parse_config(config)
    weights = check_tensors(_draw_weights(config, seed, dtype, DEVICE), arch.weight_spec(cfg), source="drawn weights")
    return arch.build(cfg, weights, BuildOptions(dtype=dtype, device=torch.device(DEVICE, 0)))


def _contexts(case: dict) -> list:
    """How many tokens each sequence of a decode step holds: spread between the shortest and the longest.  (A context one
    token short of a whole block is made one shorter: the step would give back a window's oldest block at its end, and
    could then not be repeated.)"""
    low, high, n = case["shortest"], case["longest"], case["batch"]
    lens = [high - int(round((high - low) * ((0.618034 * i) % 1.0))) for i in range(n)]
    return [c - 1 if (c + 2) % 64 == 0 and c > 1 else c for c in lens]


def _tokens(case: dict, seed: int) -> tuple:
    """(contexts that the cache already holds, the tokens that the pass brings), one int32 array per sequence."""
    vocab = _config(case["model"]).get("vocab_size", VOCAB)
    rng = np.random.default_rng(seed)
    ids = lambda n: rng.integers(0, vocab, n).astype(np.int32)   # noqa: E731
    if case["kind"] == "decode":
        held = [ids(n) for n in _contexts(case)]
        return held, [ids(1) for _ in held]
    lengths = [int(n) for n in case["lengths"].split(",")]
    held = [ids(0) for _ in lengths] + [ids(case["context"]) for _ in range(case.get("continuing", 0))]
    return held, [ids(n) for n in lengths] + [ids(1) for _ in range(case.get("continuing", 0))]


# ---- a pass -----------------------------------------------------------------------------------------------------------------

def prepare(case: dict, seed: int):
    decoder = _decoder(case, seed)
    held, brought = _tokens(case, seed)
    state = types.SimpleNamespace(case=case)
    blocks = sum(64 * -(-(len(h) + len(b) + case.get("new_tokens", 1)) // 64) for h, b in zip(held, brought))
    if case["kind"] == "generate":
        state.model = Model(decoder, max_tokens=blocks, n_slots=len(brought))
        state.prompts = [b.tolist() for b in brought]
        state.params = SamplingParams(max_new_tokens=case["new_tokens"], temperature=case["temperature"], top_k=case["top_k"],
                                      top_p=case["top_p"], repetition_penalty=case["repetition_penalty"],
                                      no_repeat_ngram_size=case["no_repeat_ngram"], stop_token_ids=(), seed=seed)
        return state
    engine = state.engine = Engine(decoder, max_tokens=blocks, n_slots=len(held))
    state.slots = [engine.start_sequence() if len(h) else None for h in held]
    waiting = [i for i, h in enumerate(held) if len(h)]
    while waiting:                                   # the contexts, a few thousand tokens a step
        some, total = [], 0
        while waiting and (not some or total + len(held[waiting[0]]) <= 4096):
            total += len(held[waiting[0]])
            some.append(waiting.pop(0))
        engine.step([StepEntry(state.slots[i], held[i], []) for i in some])
    state.held = [len(h) for h in held]
    if case["kind"] == "decode":
        state.tokens = torch.from_numpy(np.concatenate(brought)).to(DEVICE)
        state.session = DecodeSession(engine, state.slots)
        state.session.reserve_ahead(1)
        run(state)                                   # (the session captures its step when it first runs)
    else:
        state.brought = brought
    engine.check_device_errors()
    return state


def _rewind(state) -> None:
    for slot, n in zip(state.slots, state.held):
        if n:
            state.engine.cache.lengths[slot] = n


def run(state):
    if state.case["kind"] == "generate":
        results = state.model.generate_ids(state.prompts, state.params)
        return {"tokens": [np.asarray(r.new_tokens, dtype=np.int64) for r in results],
                "logits": [state.model.get_logits(p) for p in state.prompts]}
    if state.case["kind"] == "decode":
        state.session.set_tokens(state.tokens)
        logits = state.session.step(advance_on_device=False)
        _rewind(state)
        return logits
    engine = state.engine
    slots = [engine.start_sequence() if s is None else s for s in state.slots]
    logits = engine.step([StepEntry(s, toks, [len(toks) - 1]) for s, toks in zip(slots, state.brought)])
    for s, kept in zip(slots, state.slots):
        if kept is None:
            engine.end_sequence(s)
    _rewind(state)
    return logits


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------------

def _attention_layers(config: dict) -> list:
    """(heads, numbers of a query and a value that a pair costs, numbers kept per token, window or 0) of every attention that
    runs in a pass."""
    if config.get("model_type") == "gpt2":
        dim = config["n_embd"] // config["n_head"]
        return [(config["n_head"], 2 * dim, 2 * config["n_embd"], 0)] * config["n_layer"]
    out = []
    for layer in _scheduled(config):
        m = layer["mixer"]
        if layer["type"].startswith("latent"):
            kept = m["kv_rank"] + m.get("rot_dim", 0)
            out.append((m["heads"], m["dim"] + m.get("rot_dim", 0) + m["vdim"], kept, 0))
        elif layer["type"] == "parallel":
            a = m["left"]
            out.append((a["heads"], a["dim"] + a["vdim"], a["kv_heads"] * (a["dim"] + a["vdim"]), a["mask"]["size"]))
    return out


def _scheduled(config: dict) -> list:
    layers, loop = config["layers"], config.get("loop")
    if not loop:
        return layers
    a, b, k = loop["start"], loop["stop"], loop["times"]
    return layers[:a] + layers[a:b] * k + layers[b:]


def _states(config: dict) -> list:
    """Numbers in the recurrent state of every layer that has one."""
    out = []
    for layer in _scheduled(config) if "layers" in config else []:
        m = layer["mixer"].get("right", layer["mixer"])
        if layer["type"] in ("parallel", "mlstm", "channel_delta"):
            out.append(m["heads"] * m["vdim"] * m.get("state", m.get("dim", 0)))
    return out


def _one_step(case: dict, held: list, brought: list) -> dict:
    config = _config(case["model"])
    arch, cfg = parse_config(config)
    size = 4 if case["dtype"] == "float32" else 2
    tokens, wanted = sum(brought), len(brought)
    layer_runs = {}
    if "loop" in config:
        layer_runs = {i: config["loop"]["times"] for i in range(config["loop"]["start"], config["loop"]["stop"])}
    moe = next((layer["mlp"] for layer in config.get("layers", []) if layer["mlp"]["kind"] == "moe"), None)
    share_read = share_used = 1.0
    if moe is not None:
        experts, top = moe["router"]["experts"], moe["router"]["top"]
        share_read = 1.0 - (1.0 - top / experts) ** tokens
        share_used = top / experts
    nbytes = flops = 0.0
    for spec in arch.weight_spec(cfg):
        n = float(np.prod(spec.drawn_shape))
        if spec.kind == "vector":
            nbytes += 4 * n
        elif spec.name in ("wte.weight", "embed", "wpe.weight", "head"):
            if spec.name in ("wte.weight", "head") or (spec.name == "embed" and config.get("architecture") == "Kuvusun"):
                nbytes += size * n                                       # the head
                flops += 2 * n * wanted
            if spec.name != "head":
                nbytes += size * spec.drawn_shape[-1] * tokens           # rows of an embedding
        else:
            expert = ".mlp.e" in spec.name
            times = layer_runs.get(int(spec.name.split(".")[0][1:]), 1) if spec.name.startswith("l") else 1
            nbytes += size * n * (share_read if expert else 1.0)
            flops += 2 * n * tokens * times * (share_used if expert else 1.0)
    for heads, per_pair, kept, window in _attention_layers(config):
        for h, b in zip(held, brought):
            seen = lambda p: min(p + 1, window) if window else p + 1     # noqa: E731
            flops += 2 * heads * per_pair * sum(seen(p) for p in range(h, h + b))
            nbytes += size * kept * ((min(h, window) if window else h) + b)
    for n in _states(config):
        nbytes += 4 * n * sum((2 if h else 1) for h in held)
        flops += 4 * n * tokens
    nbytes += 4 * _vocab(config) * wanted
    return {"bytes": nbytes, "flops": flops}


def _vocab(config: dict) -> int:
    return config.get("vocab_size", config.get("vocab"))


def work(case: dict) -> dict:
    if case["kind"] == "decode":
        held = _contexts(case)
        return _one_step(case, held, [1] * len(held))
    lengths = [int(n) for n in case["lengths"].split(",")]
    if case["kind"] == "prompts":
        return _one_step(case, [0] * len(lengths) + [case["context"]] * case["continuing"], lengths + [1] * case["continuing"])
    total = _one_step(case, [0] * len(lengths), lengths)
    steps = [_one_step(case, [n + i for n in lengths], [1] * len(lengths)) for i in range(case["new_tokens"] - 1)]
    scored = [_one_step(case, [0], [n]) for n in lengths]
    return {k: total[k] + sum(s[k] for s in steps) + sum(s[k] for s in scored) for k in ("bytes", "flops")}


def tolerance(case: dict) -> dict:
    """About four times what passes were off `exact` when measured: 1.1e-6 to 1.5e-6 in float32; in bfloat16 0.0031 to
    0.0034 for GPT-2 and 0.0038 to 0.0089 for the designs, whose recurrences and experts add to it.  (A token of a random
    stream may flip where two probabilities touch.)"""
    if case["dtype"] == "float32":
        return {"rel": 6e-6, "max": 6e-5, "differ": 0.01}
    return {"rel": 0.015, "max": 0.08} if case["model"].startswith("gpt2") else {"rel": 0.03, "max": 0.2}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------------

def _over_rms(x, eps, groups=1):
    parts = x.reshape(*x.shape[:-1], groups, x.shape[-1] // groups)
    return (parts / torch.sqrt((parts * parts).mean(-1, keepdim=True) + eps)).reshape(x.shape)


def _attend(scores, v, window=0, keep=0):
    """scores [B, H, T, T], v [B, H, T, n] -> [B, T, H·n]; query i sees keys j <= i, with a window those less than `window`
    back and the first `keep`."""
    T = scores.shape[-1]
    i, j = torch.arange(T, device=v.device)[:, None], torch.arange(T, device=v.device)[None, :]
    seen = j <= i
    if window:
        seen &= (i - j < window) | (j < keep)
    p = torch.softmax(scores.masked_fill(~seen, -math.inf), dim=-1)
    return (p @ v).transpose(1, 2).flatten(2)


def _rotate(x, base, dims, factor=1.0):
    """x [B, T, H, n]: entry i of the first `dims` pairs with entry i + dims/2."""
    half = dims // 2
    freq = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims) / factor
    t = (torch.arange(x.shape[1], dtype=torch.float64, device=x.device)[:, None] * freq)[:, None, :]
    a, b = x[..., :half], x[..., half:dims]
    return torch.cat([a * t.cos() - b * t.sin(), b * t.cos() + a * t.sin(), x[..., dims:]], dim=-1)


class _Weights:
    """Weights by name, widened when they are used."""

    def __init__(self, tensors: dict):
        self.tensors = tensors

    def __getitem__(self, name):
        return self.tensors[name].double()

    def __contains__(self, name):
        return name in self.tensors


def _gated(h, w, p, act):
    return (act(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T


def _gpt2(config, w, ids, last):
    B, T = ids.shape
    d, H, eps = config["n_embd"], config["n_head"], config["layer_norm_epsilon"]
    norm = lambda x, p: F.layer_norm(x, (d,), w[p + ".weight"], w[p + ".bias"], eps)   # noqa: E731
    x = w["wte.weight"][ids] + w["wpe.weight"][:T]
    for i in range(config["n_layer"]):
        p = f"h.{i}."
        qkv = norm(x, p + "ln_1") @ w[p + "attn.c_attn.weight"] + w[p + "attn.c_attn.bias"]
        q, k, v = (t.reshape(B, T, H, d // H).transpose(1, 2) for t in qkv.split(d, dim=-1))
        x = x + _attend(q @ k.transpose(-1, -2) * (d // H) ** -0.5, v) @ w[p + "attn.c_proj.weight"] + w[p + "attn.c_proj.bias"]
        h = F.gelu(norm(x, p + "ln_2") @ w[p + "mlp.c_fc.weight"] + w[p + "mlp.c_fc.bias"], approximate="tanh")
        x = x + h @ w[p + "mlp.c_proj.weight"] + w[p + "mlp.c_proj.bias"]
    return norm(x[torch.arange(B, device=x.device), last], "ln_f") @ w["wte.weight"].T


def _kotisun(config, w, ids, last):
    B, T = ids.shape
    eps, cap = config["norm"]["eps"], config["logit_softcap"]

    def attention(h, p, m):
        H, G = m["heads"], m["kv_heads"]
        q, k, v = ((h @ w[p + n].T + w[p + n + ".b"]).reshape(B, T, heads, size)
                   for n, heads, size in (("q", H, m["dim"]), ("k", G, m["dim"]), ("v", G, m["vdim"])))
        q, k = (_rotate(t, m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"]["factor"]) for t in (q, k))
        k, v = (t.repeat_interleave(H // G, dim=2).transpose(1, 2) for t in (k, v))
        return _attend(q.transpose(1, 2) @ k.transpose(-1, -2) * m["scale"], v, m["mask"]["size"]) @ w[p + "o"].T

    def recurrence(h, p, m):
        H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        z, u, dt = (h @ w[p + "in"].T).split([H * P, H * P + 2 * G * N, H], dim=-1)
        taps = w[p + "conv"]
        u = F.silu(F.conv1d(F.pad(u.transpose(1, 2), (taps.shape[1] - 1, 0)), taps[:, None], w[p + "conv.b"], groups=taps.shape[0])
                   .transpose(1, 2))
        v, b, c = u.split([H * P, G * N, G * N], dim=-1)
        v, dt = v.reshape(B, T, H, P), F.softplus(dt + w[p + "dt_bias"])
        b, c = (t.reshape(B, T, G, N).repeat_interleave(H // G, dim=2) for t in (b, c))
        keep, fed = torch.exp(-torch.exp(w[p + "A_log"]) * dt), dt[..., None] * b
        S, y = torch.zeros(B, H, N, P, dtype=h.dtype, device=h.device), torch.empty_like(v)
        for t in range(T):
            S = keep[:, t, :, None, None] * S + fed[:, t, :, :, None] * v[:, t, :, None, :]
            y[:, t] = (S * c[:, t, :, :, None]).sum(2)
        y = (y + w[p + "D"][:, None] * v).flatten(2) * F.silu(z)
        return (_over_rms(y, eps, m["norm_groups"]) * w[p + "norm"]) @ w[p + "o"].T

    def sublayer(xs, p, norm, fn):
        y = fn(_over_rms(torch.einsum("s,sbtd->btd", w[p + "in"], xs), eps) * w[norm])
        return torch.einsum("sj,sbtd->jbtd", w[p + "mix"], xs) + w[p + "out"][:, None, None, None] * y

    order = list(range(len(config["layers"])))
    a, b, k = (config["loop"][n] for n in ("start", "stop", "times"))
    xs = (w["embed"][ids] * config["embedding"]["scale"])[None].repeat(config["streams"], 1, 1, 1)
    for i in order[:a] + order[a:b] * k + order[b:]:
        p, m = f"l{i}.", config["layers"][i]["mixer"]
        xs = sublayer(xs, p + "hc1.", p + "norm1", lambda h: m["left_scale"] * attention(h, p + "mix.left.", m["left"])
                      + m["right_scale"] * recurrence(h, p + "mix.right.", m["right"]))
        xs = sublayer(xs, p + "hc2.", p + "norm2", lambda h: _gated(h, w, p + "mlp.", torch.relu))
    x = xs.sum(0)[torch.arange(B, device=ids.device), last]
    return cap * torch.tanh((_over_rms(x, eps) * w["final.norm"]) @ w["head"].T / cap)


def _pelenex(config, w, ids, last):
    B, T = ids.shape
    eps, groups, cap, d = config["norm"]["eps"], config["norm"]["groups"], config["logit_softcap"], config["width"]
    heads = lambda t, H: t.reshape(B, T, H, -1)   # noqa: E731

    def side_by_side(h, p, m):
        a, r = m["left"], m["right"]
        H, G = a["heads"], a["kv_heads"]
        q, k = heads(h @ w[p + "left.q"].T, H), heads(h @ w[p + "left.k"].T, G)
        v, k = k, _over_rms(k, eps)
        k, v = (t.repeat_interleave(H // G, dim=2).transpose(1, 2) for t in (k, v))
        pos = torch.arange(T, dtype=h.dtype, device=h.device)
        slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=h.dtype, device=h.device) / H)
        s = _over_rms(q, eps).transpose(1, 2) @ k.transpose(-1, -2) * a["scale"] - slopes[:, None, None] * (pos[:, None] - pos)
        left = _attend(s, v, a["mask"]["size"], a["mask"]["keep_first"]) @ w[p + "left.o"].T
        p += "right."
        H = r["heads"]
        q, k, v = heads(h @ w[p + "q"].T, H) * r["dim"] ** -0.5, heads(h @ w[p + "k"].T, H), heads(h @ w[p + "v"].T, H)
        alpha = heads(torch.exp(F.logsigmoid((h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "a2.b"]) / r["tau"]), H)
        S, y = torch.zeros(B, H, r["dim"], r["vdim"], dtype=h.dtype, device=h.device), torch.empty_like(v)
        for t in range(T):
            S = alpha[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None, :]
            y[:, t] = (S * q[:, t, :, :, None]).sum(2)
        y = (_over_rms(y, eps) * w[p + "norm"]).flatten(2) * F.silu(h @ w[p + "g"].T)
        right, p = y @ w[p + "o"].T, p[:-6]
        return 0.5 * (_over_rms(left, eps) * w[p + "left.out"] + _over_rms(right, eps) * w[p + "right.out"])

    def mlstm(h, p, m):
        H, limit = m["heads"], m["gate_cap"]
        q, k, v = heads(h @ w[p + "q"].T, H) * m["dim"] ** -0.5, heads(h @ w[p + "k"].T, H), heads(h @ w[p + "v"].T, H)
        capped = lambda z: limit * torch.tanh(z / limit)   # noqa: E731
        log_i, log_f = capped(h @ w[p + "i"].T + w[p + "i.b"]), F.logsigmoid(capped(h @ w[p + "f"].T + w[p + "f.b"]))
        S, n = torch.zeros(B, H, m["dim"], m["vdim"], dtype=h.dtype, device=h.device), torch.zeros_like(k[:, 0])
        top, y = torch.zeros_like(log_i[:, 0]), torch.empty_like(v)
        for t in range(T):
            new = torch.maximum(log_f[:, t] + top, log_i[:, t])
            keep, take = torch.exp(log_f[:, t] + top - new), torch.exp(log_i[:, t] - new)[..., None] * k[:, t]
            S = keep[..., None, None] * S + take[..., None] * v[:, t, :, None, :]
            n, top = keep[..., None] * n + take, new
            den = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
            y[:, t] = (S * q[:, t, :, :, None]).sum(2) / den[..., None]
        return (_over_rms(y, eps).flatten(2) * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T

    def channel_delta(h, p, m):
        H, G = m["heads"], m["kv_heads"]

        def conv(n):
            u, taps = (h @ w[p + n].T).transpose(1, 2), w[p + n + ".conv"]
            return F.silu(F.conv1d(F.pad(u, (taps.shape[1] - 1, 0)), taps[:, None], groups=taps.shape[0]).transpose(1, 2))
        unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)   # noqa: E731
        q, k = (unit(heads(conv(n), G)).repeat_interleave(H // G, dim=2) for n in ("q", "k"))
        q, v, beta = q * m["dim"] ** -0.5, heads(conv("v"), H), torch.sigmoid(h @ w[p + "b"].T)
        keep = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * F.softplus(heads((h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "dt_bias"], H)))
        S, y = torch.zeros(B, H, m["dim"], m["vdim"], dtype=h.dtype, device=h.device), torch.empty_like(v)
        for t in range(T):
            S = keep[:, t, :, :, None] * S
            u = beta[:, t, :, None] * (v[:, t] - (S * k[:, t, :, :, None]).sum(2))
            S = S + k[:, t, :, :, None] * u[:, :, None, :]
            y[:, t] = (S * q[:, t, :, :, None]).sum(2)
        y = (_over_rms(y, eps) * w[p + "norm"]).flatten(2)
        return (y * torch.sigmoid((h @ w[p + "g1"].T) @ w[p + "g2"].T)) @ w[p + "o"].T

    def experts(h, p, ml):
        z = h @ w[p + "router"].T
        chosen = z.topk(ml["router"]["top"], dim=-1).indices
        y = _gated(h, w, p + "shared.", F.silu)
        for e in range(ml["router"]["experts"]):
            mine = (chosen == e).any(-1)
            y[mine] += _gated(h[mine] * torch.sigmoid(z[mine][:, e:e + 1]), w, p + f"e{e}.", F.silu)
        return y

    pos = torch.arange(T, dtype=torch.float64, device=ids.device)[:, None]
    ang = pos * 10000.0 ** (-torch.arange(0, d, 2, dtype=torch.float64, device=ids.device) / d)
    x = w["embed"][ids] + torch.stack([ang.sin(), ang.cos()], dim=-1).flatten(1)
    mixers = {"parallel": side_by_side, "mlstm": mlstm, "channel_delta": channel_delta}
    for i, layer in enumerate(config["layers"]):
        p, ml = f"l{i}.", layer["mlp"]
        h = _over_rms(x, eps, groups) * w[p + "norm1"]
        x = x + mixers[layer["type"]](h, p + "mix.", layer["mixer"])
        x = x + (_gated(h, w, p + "mlp.", F.silu) if ml["kind"] == "dense" else experts(h, p + "mlp.", ml))
    x = x[torch.arange(B, device=ids.device), last]
    return cap * torch.tanh((_over_rms(x, eps, groups) * w["final.norm"]) @ w["head"].T / cap)


def _kuvusun(config, w, ids, last):
    B, T = ids.shape
    eps, groups = config["norm"]["eps"], config["norm"]["groups"]
    norm = lambda x, name: _over_rms(x, eps, groups) * w[name]   # noqa: E731

    def attention(x, p, m, kept):
        H, n, R = m["heads"], m["dim"], m.get("rot_dim", 0)
        q = (_over_rms(x @ w[p + "dq"].T, eps) * w[p + "dq.norm"]) @ w[p + "uq"].T if "q_rank" in m else x @ w[p + "q"].T
        q = q.reshape(B, T, H, n + R)
        c, r = kept
        k, v = ((c @ w[p + u].T).reshape(B, T, H, -1).transpose(1, 2) for u in ("uk", "uv"))
        s = q[..., :n].transpose(1, 2) @ k.transpose(-1, -2)
        if R:
            s = s + _rotate(q[..., n:], m["rot"]["base"], m["rot"]["dims"]).transpose(1, 2) @ r.permute(0, 2, 3, 1)
        y = _attend(s * m["scale"], v)
        if p + "g" in w:
            y = y * torch.sigmoid(x @ w[p + "g"].T)
        return y @ w[p + "o"].T

    def experts(h, p, ml):
        z = h @ w[p + "router"].T + w[p + "router.b"]
        best = z.topk(ml["router"]["top"], dim=-1)
        share = torch.zeros_like(z).scatter_(-1, best.indices, torch.softmax(best.values, dim=-1))
        y = _gated(h, w, p + "shared.", F.silu) * torch.sigmoid(h @ w[p + "shared.sg"].T)
        for e in range(ml["router"]["experts"]):
            mine = share[..., e] > 0
            y[mine] += share[mine][:, e:e + 1] * _gated(h[mine], w, p + f"e{e}.", F.silu)
        return y

    x = norm(w["embed"][ids], "embed.norm")
    rows = {}
    for i, layer in enumerate(config["layers"]):
        p, m, ml = f"l{i}.", layer["mixer"], layer["mlp"]
        if "kv_from" not in m:
            proj = x @ w[p + "mix.dkv"].T
            r = _rotate(proj[..., None, m["kv_rank"]:], m["rot"]["base"], m["rot"]["dims"]) if m.get("rot_dim") else None
            rows[i] = (_over_rms(proj[..., :m["kv_rank"]], eps) * w[p + "mix.dkv.norm"], r)
        x = x + norm(attention(x, p + "mix.", m, rows[m.get("kv_from", i)]), p + "norm1")
        y = (torch.relu(x @ w[p + "mlp.up"].T) ** 2) @ w[p + "mlp.down"].T if ml["kind"] == "dense" else experts(x, p + "mlp.", ml)
        x = x + norm(y, p + "norm2")
    return norm(x[torch.arange(B, device=ids.device), last], "final.norm") @ w["embed"].T


FORWARD = {"gpt2": _gpt2, "kotisun": _kotisun, "pelenex": _pelenex, "kuvusun": _kuvusun}


def exact(case: dict, seed: int):
    config = _config(case["model"])
    w = _Weights(_draw_weights(config, seed, parse_dtype(case["dtype"]), DEVICE))
    held, brought = _tokens(case, seed)
    whole = [np.concatenate(pair) for pair in zip(held, brought)]
    forward = FORWARD[case["model"].split("-")[0]]
    order = sorted(range(len(whole)), key=lambda i: len(whole[i]))
    logits = [None] * len(whole)
    while order:                                     # sequences of like lengths together, padded behind their ends
        some = [order.pop()]
        longest = len(whole[some[0]])
        while order and (len(some) + 1) * longest <= 8192:
            some.append(order.pop())
        ids = np.zeros((len(some), longest), dtype=np.int64)
        for row, i in enumerate(some):
            ids[row, :len(whole[i])] = whole[i]
        last = torch.tensor([len(whole[i]) - 1 for i in some], device=DEVICE)
        for i, row in zip(some, forward(config, w, torch.from_numpy(ids).to(DEVICE), last)):
            logits[i] = row
    if case["kind"] == "generate":
        return {"tokens": None, "logits": logits}
    return torch.stack(logits)
