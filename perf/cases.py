"""The work that users have the engine do, as cases that can be timed and compared: prompts, traces of prompts and
single tokens, and whole generations, for the seven architectures at the layer sizes that `bench.py` measures, with
random weights (the Qwen3 models with fewer layers than the published ones, the others with six).

A case is one of two kinds:

  replay     the step function under `Engine` and `bin/trace_run`: `build`, then one step that brings `count` prompts
             and `steps` steps that bring one known token for each; the logits of every prompt's last token and of every
             later token come back. With `steps` = 0 it is a prompt's computation; with more, teacher-forced scoring.
  generate   `Engine.generate`: `count` prompts in, `tokens` greedily chosen tokens out for each, decode steps replayed
             from CUDA graphs. No prefix cache: every pass computes its prompts. The tokens come back, and what the
             engine's cache and its matrix states hold afterwards.

`length` is the longest prompt's length; with `ragged` the others are shorter, down to a fraction of it. The weights keep
the distributions of trained models where the path's numbers depend on them: tables large against the sublayers' outputs, a next
token that stands clear of the others, decays near one.
"""
from __future__ import annotations

import math
import re

import torch

DEVICE = "cuda:0"
PAGE = 64
RARE = 1000                                     # prompts hold tokens from here on, as the benchmark's do


# ---------------------------------------------------------------- models
def _qwen3(layers, hidden, heads, kv_heads, ff, vocab=151936, tied=False):
    return {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": layers, "hidden_size": hidden,
            "num_attention_heads": heads, "num_key_value_heads": kv_heads, "head_dim": 128, "intermediate_size": ff,
            "vocab_size": vocab, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": tied,
            "max_position_embeddings": 40960}


def _model(architecture, width, layers, **more):
    return {"architecture": architecture, "width": width, "vocab": 32768, "norm": {"eps": 1e-6}, "layers": layers, **more}


def _rulorax(width, heads, rank, rot, dim, dense_ff, experts, top, ff, shared):
    def mixer(i):
        m = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": dim, "kv_rank": rank, "rot": {"base": 10000.0, "dims": rot},
             "scale": (dim + rot) ** -0.5}
        return dict(m, kv_from=i - 1) if i % 2 else m
    moe = {"kind": "moe", "router": {"experts": experts, "top": top, "scale": 1.0}, "expert": {"ff": ff}, "shared": {"ff": shared}}
    return _model("Rulorax", width, [{"type": "latent_attention", "mixer": mixer(i),
                                      "mlp": moe if i else {"kind": "dense", "ff": dense_ff}} for i in range(6)], streams=4)


def _decays(heads):
    return [1 - 2.0 ** (-5 - h % 6) for h in range(heads)]


YARN = {"factor": 16.0, "original": 4096, "fast": 32.0, "slow": 1.0}


def _kasovik(width, heads, kv_heads, window, ff):
    left = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "mask": {"size": window}, "scale": 128 ** -0.5}
    right = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    parallel = {"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}, "mlp": mlp}
    retention = {"type": "retention", "mlp": mlp, "mixer": {"heads": heads, "dim": 128, "vdim": 128, "decay": _decays(heads),
                                                            "rot": {"base": 1000000.0, "dims": 128}}}
    return _model("Kasovik", width, [dict(retention if i % 3 == 2 else parallel) for i in range(6)],
                  embedding={"scale": 1.0, "bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}})


def _tilarax(width, heads, kv_heads, chunk, ff, memory_dim):
    attention = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "mask": {"size": chunk},
                 "rot": {"base": 10000.0, "dims": 64}, "scale": 128 ** -0.5, "v_mix": True}
    memory = {"heads": 8, "dim": memory_dim, "vdim": 2 * memory_dim, "gate_cap": 15.0}
    moe = {"kind": "moe", "router": {"experts": 32, "top": 4}, "expert": {"ff": ff // 4}}
    return _model("Tilarax", width, [{"type": "mlstm" if i % 2 else "attention", "mixer": memory if i % 2 else attention,
                                      "mlp": moe if i else {"kind": "dense", "ff": ff}} for i in range(6)])


def _vobosun(width, heads, kv_heads, ff, rank):
    attention = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                 "rot": {"base": 1000000.0, "dims": 128, "scaling": {"factor": 8.0}}}
    delta = {"heads": heads, "dim": 128, "decay_rank": rank}
    moe = {"kind": "moe", "router": {"experts": 28, "identity": 4, "top": 4, "groups": {"count": 8, "keep": 4}},
           "expert": {"ff": ff // 4}, "shared": {"ff": ff // 4}}
    return _model("Vobosun", width, [{"type": "attention" if i % 3 else "general_delta", "mixer": attention if i % 3 else delta,
                                      "mlp": moe if i % 2 else {"kind": "dense", "ff": ff}} for i in range(6)])


def _gegunex(width, heads, kv_heads, window, ff, low_rank):
    latent = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": width * 3 // 8, "kv_rank": 512,
              "mask": {"size": window}, "scale": 192 ** -0.5, "rot": {"base": 1000000.0, "dims": 64, "scaling": YARN}}
    delta = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": low_rank, "gate_rank": low_rank}
    lightning = {"heads": heads, "dim": 128, "vdim": 128, "decay": _decays(heads)}
    moe = {"kind": "moe", "router": {"experts": 32, "top": 4}, "expert": {"ff": ff // 4, "limit": 7.0}}
    turns = [("channel_delta", delta), ("latent_attention", latent), ("lightning", lightning)]
    return _model("Gegunex", width, [{"type": turns[i % 3][0], "mixer": turns[i % 3][1], "mlp": moe} for i in range(6)],
                  residual_mult=0.5, logit_softcap=30.0)


def _bukuvik(width, heads, kv_heads, window, ff, groups):
    two_maps = {"heads": heads, "kv_heads": kv_heads, "dim": 64, "vdim": 128, "scale": 0.125, "softcap": 50.0, "diff": 0.5,
                "mask": {"size": window}, "rot": {"base": 1000000.0, "dims": 32}}
    left = {"heads": heads, "kv_heads": kv_heads, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
            "mask": {"size": window, "keep_first": 16}, "rot": {"base": 1000000.0, "dims": 128, "scaling": YARN}}
    right = {"heads": 2 * heads, "groups": groups, "state": 128, "vdim": 64, "conv": 4, "norm_groups": groups}
    mlp = {"kind": "dense", "ff": ff}
    parallel = {"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": mlp}
    return _model("Bukuvik", width, [{"type": "attention", "mixer": two_maps, "mlp": mlp} if i % 3 == 2 else parallel
                                     for i in range(6)], residual_mult=0.5, embedding={"scale": width ** 0.5})


# The sizes of the benchmark: of each design the layers of a model of about 1.5 billion parameters ("base", "lite") and a second
# size (the larger ones have the width of the 8-billion-parameter model).
MODELS = {
    "qwen3 0.6b": _qwen3(28, 1024, 16, 8, 3072, tied=True),
    "qwen3 8b": _qwen3(12, 4096, 32, 8, 12288),
    "rulorax lite": _rulorax(2048, 16, 512, 64, 128, 10944, 64, 6, 1408, 2816),
    "rulorax small": _rulorax(2560, 40, 256, 32, 64, 6400, 32, 4, 1024, 2048),
    "kasovik base": _kasovik(2048, 16, 4, 1024, 6144),
    "kasovik wide": _kasovik(4096, 32, 8, 2048, 12288),
    "tilarax base": _tilarax(2048, 16, 4, 1024, 6144, 128),
    "tilarax wide": _tilarax(4096, 32, 8, 2048, 12288, 256),
    "vobosun base": _vobosun(2048, 16, 4, 6144, 64),
    "vobosun wide": _vobosun(4096, 32, 8, 12288, 128),
    "gegunex base": _gegunex(2048, 16, 4, 1024, 6144, 64),
    "gegunex wide": _gegunex(4096, 32, 8, 2048, 12288, 128),
    "bukuvik base": _bukuvik(2048, 16, 4, 1024, 9216, 4),
    "bukuvik wide": _bukuvik(4096, 32, 8, 2048, 18432, 8),
}


# ---------------------------------------------------------------- cases
def _replay(name, model, count, length, ragged=False, steps=0, dtype="bfloat16"):
    return {"name": name, "kind": "replay", "model": model, "dtype": dtype, "count": count, "length": length, "ragged": ragged,
            "steps": steps}


def _generate(name, model, count, length, tokens, ragged=False):
    return {"name": name, "kind": "generate", "model": model, "dtype": "bfloat16", "count": count, "length": length,
            "ragged": ragged, "tokens": tokens}


def listed() -> list[dict]:
    return [
        # one short question to a small model: every step is launches and latency
        _generate("small model, one request", "qwen3 0.6b", 1, 32, 16),
        # the reference's benchmark: a batch of requests, decoding behind prompts
        _generate("decode, batch 8", "qwen3 8b", 8, 1024, 96),
        # a loaded server: many short requests of different lengths
        _generate("decode, batch 48, ragged", "qwen3 8b", 48, 300, 32, ragged=True),
        # a prompt of the benchmark's length
        _replay("prompt of 2,048 tokens", "qwen3 8b", 1, 2048),
        # teacher-forced scoring of several texts of odd lengths, tokens one by one behind them
        _replay("trace, ragged", "qwen3 0.6b", 5, 701, ragged=True, steps=6),
        # the same in true 32-bit, which traces are checked with
        _replay("trace, 32-bit", "qwen3 0.6b", 2, 333, ragged=True, steps=4, dtype="float32"),
        # prompts of the other designs, one long or several ragged ones
        _replay("latent attention, prompt", "rulorax lite", 1, 2048),
        _replay("delta rule and retention, prompt", "kasovik base", 1, 2048),
        _replay("mixed heads and memory, prompts", "tilarax base", 3, 1111, ragged=True),
        _replay("delta, latent and lightning, prompts", "gegunex base", 2, 1500, ragged=True),
        # and their decoding
        _generate("general delta, batch 8", "vobosun base", 8, 256, 64),
        _generate("state space, one request", "bukuvik wide", 1, 700, 64),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    design = rng.choice(["qwen3 0.6b", "qwen3 8b", "qwen3 8b"] + [m for m in MODELS if not m.startswith("qwen3")])
    kind = rng.choice(["replay", "generate"])
    count = _log(rng, 1, 12)
    # the tokens of all prompts together stay under the largest listed case's, of the wider models under half of them
    room = 2048 if design.endswith("wide") else 4096
    length = _log(rng, 17, max(64, min(3000, room // count)))
    if kind == "generate":
        return {k: v for k, v in _generate("", design, count, length, _log(rng, 4, 64), rng.random() < 0.5).items() if k != "name"}
    dtype = "float32" if design == "qwen3 0.6b" and rng.random() < 0.4 else "bfloat16"
    if dtype == "float32":
        length = max(17, length // 4)
    return {k: v for k, v in _replay("", design, count, length, rng.random() < 0.6, rng.choice([0, 0, 1, 3]), dtype).items()
            if k != "name"}


def _lengths(case) -> list[int]:
    n, c = case["length"], case["count"]
    return [n - (n * 3 * i) // (4 * c) if case["ragged"] else n for i in range(c)]


def _prompts(case, seed) -> list[list[int]]:
    """The prompts; of a replay with the tokens that follow one by one."""
    cfg = MODELS[case["model"]]
    g = torch.Generator().manual_seed(seed * 7 + 3)
    more = case.get("steps", 0)
    return [torch.randint(RARE, cfg.get("vocab_size", cfg.get("vocab")) - 128, (n + more,), generator=g).tolist() for n in _lengths(case)]


# ---------------------------------------------------------------- weights
#: What is not drawn as the package's random source draws it: (end of the stored name, factor, added). Projections that
#: end a sublayer are small against the stream, decays lie near one.
SHAPED = [("o_proj.weight", 0.4, 0.0), ("down_proj.weight", 0.4, 0.0), (".o", 0.4, 0.0), (".down", 0.4, 0.0), (".dt_bias", 8.0, -4.0),
          (".w0", 8.0, -3.0), (".f.b", 4.0, 3.0), ("bigram", 2.0, 0.0)]
#: Factors on the embedding's table, by design: with norms on the sublayers' outputs these have a size of one.
TABLE = {"Tilarax": 20.0, "Vobosun": 20.0, "Bukuvik": 1.0}
#: How much of an expert's weights is its own: experts that were copies of one feed-forward when their training began. (With
#: nothing in common, one token whose choice is a near tie decides how far two runs in bfloat16 are apart.)
OWN = 0.02


def _source(case, seed):
    from holon_b200.weights import RandomSource

    class Source(RandomSource):
        def tensors(self):
            table, common = None, {}
            for name, x in super().tensors():
                factor, add = next(((f, a) for end, f, a in SHAPED if name.endswith(end)), (1.0, 0.0))
                if name == "embed":
                    factor = TABLE.get(self._config["architecture"], 5.0)
                elif name == "model.embed_tokens.weight":
                    factor = 10.0 if self._config["tie_word_embeddings"] else 40.0
                expert = re.sub(r"\.e\d+\.", ".common.", name)
                if expert != name:
                    if expert not in common:
                        g = torch.Generator(device=self.device).manual_seed(seed * 1009 + len(common))
                        common[expert] = torch.randn(x.shape, generator=g, device=self.device).mul_(self.STD_MATRIX)
                    x = x.float().mul_(OWN).add_(common[expert], alpha=(1 - OWN ** 2) ** 0.5).mul_(factor).to(self.dtype)
                    factor = 1.0
                if factor != 1.0 or add:
                    x = (x.float() * factor + add).to(self.dtype)
                if name in ("embed", "model.embed_tokens.weight"):
                    table = x
                if name in ("head", "lm_head.weight"):           # the token that follows in the table stands clear
                    x = (table.float().roll(-1, 0).mul(self.STD_MATRIX * 5 / table[:256].float().std())).to(self.dtype)
                yield name, x

    return Source(MODELS[case["model"]], seed=seed, device=DEVICE, dtype=getattr(torch, case["dtype"]))


# ---------------------------------------------------------------- what a user's program does
def prepare(case, seed):
    prompts, tokens = _prompts(case, seed), case.get("tokens", 0)
    longest = max(map(len, prompts)) + tokens + 1
    room = -(-longest // PAGE) * PAGE
    if case["kind"] == "generate":
        from holon_b200 import Engine, EngineConfig, SamplingParams
        engine = Engine(EngineConfig(model="random weights", device=DEVICE, dtype=case["dtype"], page_size=PAGE,
                                     max_seqs=case["count"], max_model_len=room, max_step_tokens=4096, prefix_cache=False,
                                     state_memory=3 << 29, seed=0), source=_source(case, seed))
        return {"engine": engine, "prompts": prompts, "params": SamplingParams(temperature=0.0, max_tokens=tokens, ignore_eos=True)}
    from holon_b200.engine import build
    with torch.inference_mode():
        built = build(_source(case, seed), dtype=case["dtype"], device=DEVICE, page_size=PAGE, max_seqs=case["count"],
                      max_model_len=room, max_step_tokens=max(case["count"], sum(_lengths(case))),
                      pages=case["count"] * (room // PAGE))
    return {"built": built, "prompts": prompts, "lengths": _lengths(case), "steps": case["steps"]}


def run(state):
    if "engine" in state:
        engine = state["engine"]
        tokens = engine.generate(state["prompts"], state["params"])
        cache = engine.built.cache
        return {"tokens": torch.tensor(tokens), "pages": [g.kv[:, :-1] for g in cache.groups],
                "states": [t[:-1] for _, t in sorted(cache.slot_states.items())]}
    from holon_b200.engine import StepEntry
    cache, runner, out = state["built"].cache, state["built"].runner, []
    with torch.inference_mode():
        slots = [cache.admit() for _ in state["prompts"]]
        at = [0] * len(slots)
        for step in range(1 + state["steps"]):
            entries = []
            for i, (slot, ids, n) in enumerate(zip(slots, state["prompts"], state["lengths"])):
                brought = ids[:n] if step == 0 else ids[at[i]:at[i] + 1]
                cache.reserve(slot, at[i] + len(brought))
                entries.append(StepEntry(slot, brought, at[i], [len(brought) - 1]))
                at[i] += len(brought)
            out.append(runner.step(entries))
        for slot in slots:
            cache.release(slot)
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def work(case) -> dict:
    """Bytes: every weight once a step (of the experts those that some token chooses on average), a row of the cache per token
    written once and read once by every later token's step, matrix states read and written; logits written. Flops: products,
    attention's scores and sums, three multiply-adds a state's element and token."""
    cfg = MODELS[case["model"]]
    item = 2 if case["dtype"] == "bfloat16" else 4
    lengths, later = _lengths(case), case.get("steps", max(0, case.get("tokens", 1) - 1))
    dense, moe, kv, pair, state = 0, [], 0, 0, 0
    for layer in _layers(cfg):
        dense += layer["dense"]
        kv, pair, state = kv + layer["kv"], pair + layer["pair"], state + layer["state"]
        if layer["experts"]:
            moe.append(layer)
    vocab, width = cfg.get("vocab_size", cfg.get("vocab")), cfg.get("hidden_size", cfg.get("width"))
    total = {"bytes": 0.0, "flops": 0.0}
    for step in range(1 + later):
        n = sum(lengths) if step == 0 else case["count"]
        rows = case["count"]
        total["bytes"] += item * (dense + vocab * width) + 4 * rows * vocab + n * (kv * item + width * item)
        total["flops"] += 2.0 * n * dense + 2.0 * rows * vocab * width + 6.0 * n * state
        total["bytes"] += 8.0 * rows * state * (step > 0) + 4.0 * rows * state * (step == 0)
        for e in moe:
            total["bytes"] += item * e["expert"] * e["experts"] * (1 - (1 - e["top"] / e["experts"]) ** n)
            total["flops"] += 2.0 * n * e["expert"] * e["top"]
        for m in lengths:
            seen = m * (m + 1) / 2 if step == 0 else m + step
            total["flops"] += 2.0 * pair * seen
            total["bytes"] += kv * item * (m + step) * (step > 0)
    return total


def _layers(cfg):
    """Per layer: parameters that every token uses, numbers a token leaves in the cache, multiply-adds a query and key pair,
    numbers of a matrix state, parameters of an expert, experts and how many of them a token chooses."""
    if "architectures" in cfg:
        h, d, a, k, f = (cfg[x] for x in ("hidden_size", "head_dim", "num_attention_heads", "num_key_value_heads", "intermediate_size"))
        one = {"dense": (2 * a + 2 * k) * d * h + 3 * f * h, "kv": 2 * k * d, "pair": 2 * a * d, "state": 0, "experts": 0}
        return [one] * cfg["num_hidden_layers"]
    out, w = [], cfg["width"]
    glu = {"Bukuvik": 2, "Tilarax": 2, "Vobosun": 2}.get(cfg["architecture"], 3)
    for layer in cfg["layers"]:
        one = {"dense": 0, "kv": 0, "pair": 0, "state": 0, "experts": 0}
        m, mlp = layer["mixer"], layer["mlp"]
        for part in ([m["left"], m["right"]] if layer["type"] == "parallel" else [m]):
            heads, dim, vdim = part["heads"], part.get("dim", part.get("state")), part.get("vdim", part.get("dim"))
            kvh = part.get("kv_heads", part.get("groups", heads))
            one["dense"] += w * heads * vdim * 2
            if "kv_rank" in part:
                rank, rot = part["kv_rank"], part["rot_dim"]
                one["dense"] += w * (rank + rot) * ("kv_from" not in part) + heads * rank * (dim + vdim)
                one["dense"] += part.get("q_rank", w) * heads * (dim + rot) + part.get("q_rank", 0) * w
                one["kv"] += (rank + rot) * ("kv_from" not in part)
                one["pair"] += heads * (dim + rot + vdim)
            elif "mask" in part or layer["type"] == "attention":
                maps = 2 if "diff" in part else 1
                one["dense"] += w * (heads + kvh) * dim * maps + w * kvh * vdim
                one["kv"] += kvh * (dim * maps + vdim)
                one["pair"] += heads * (dim + vdim) * maps
            else:
                one["dense"] += w * (2 * kvh * dim + heads * vdim)
                one["state"] += heads * dim * vdim
        if mlp["kind"] == "dense":
            one["dense"] += glu * w * mlp["ff"]
        else:
            r, per = mlp["router"], 2 if cfg["architecture"] == "Rulorax" else 3
            one.update(experts=r["experts"], top=r["top"], expert=per * w * mlp["expert"]["ff"])
            one["dense"] += w * r["experts"] + per * w * (mlp.get("shared") or {"ff": 0})["ff"]
        out.append(one)
    return out


def tolerance(case) -> dict:
    """Measured against `exact` and against runs with products summed in another order. 32-bit logits are 2.2e-6 from `exact`;
    bfloat16 logits 0.002 to 0.018 (deepest where norms stand on the sublayers' outputs), their largest difference 0.04; the
    cache's pages 0.007, with single small numbers as far apart as their size. Greedy tokens stand clear of the next best."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 4e-4}
    return {"rel": 0.03, "max": 0.99 if case["kind"] == "generate" else 0.2, "differ": 0.002}


# ---------------------------------------------------------------- the same in 64 bits, written out plainly
def exact(case, seed):
    """Every design over whole sequences [sequence, token, channel], without cache or batch layout. Of a generation the tokens
    (the cache's pages and states are this engine's own layout)."""
    weights = dict(_source(case, seed).tensors())
    plain = Plain(MODELS[case["model"]], weights)
    prompts, lengths = _prompts(case, seed), _lengths(case)
    if case["kind"] == "replay":
        x = plain.trunk(prompts)
        return [plain.logits(torch.stack([x[i, n - 1 + s] for i, n in enumerate(lengths)])) for s in range(1 + case["steps"])]
    found = [[] for _ in prompts]
    for _ in range(case["tokens"]):              # (the rest is guessed to go on as the last pair of tokens does)
        full = []
        for p, f in zip(prompts, found):
            a, b = ([*p, *f])[-2:]
            step = 0 if a == b and f else 1 if f and b == a + 1 else 0
            full.append([*p, *f, *((b + step * (k + 1)) % plain.vocab for k in range(case["tokens"] - len(f)))])
        x = plain.trunk([f[:-1] for f in full])
        best = [plain.logits(x[i, n - 1:n - 1 + case["tokens"]]).argmax(-1).tolist() for i, n in enumerate(lengths)]
        if all(b == f[n:] for b, f, n in zip(best, full, lengths)):
            break
        for i, (b, f, n) in enumerate(zip(best, full, lengths)):
            same = next((k for k in range(case["tokens"]) if b[k] != f[n + k]), case["tokens"] - 1)
            found[i] = b[:same + 1]
    return {"tokens": torch.tensor(best), "pages": None, "states": None}


def _rms(x, eps, weight=1.0):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, rot, neighbours=False):
    """x [sequence, token, head, channel]: pairs of the first rot["dims"] channels turned by position times frequency, halves
    or neighbours paired; a scaling of a factor alone stretches all frequencies, one with an original length is YaRN's."""
    dims, base, s, size = rot["dims"], float(rot["base"]), rot.get("scaling"), 1.0
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    f = base ** (-2.0 * i / dims)
    if s and "original" in s:
        pair = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))    # noqa: E731
        low, high = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), dims - 1)
        ramp = ((i - low) / max(high - low, 0.001)).clamp(0, 1)
        f, size = f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1
    elif s:
        f = f / s["factor"]
    angle = torch.arange(x.shape[1], dtype=torch.float64, device=x.device)[:, None, None] * f
    cos, sin, rest = angle.cos() * size, angle.sin() * size, x[..., dims:]
    a, b = (x[..., 0:dims:2], x[..., 1:dims:2]) if neighbours else (x[..., :dims // 2], x[..., dims // 2:dims])
    u, v = a * cos - b * sin, b * cos + a * sin
    return torch.cat((torch.stack((u, v), -1).flatten(-2) if neighbours else torch.cat((u, v), -1), rest), -1)


def _seen(t, mask, device, blocks=False):
    i, j = torch.arange(t, device=device)[:, None], torch.arange(t, device=device)[None, :]
    seen = j <= i
    if mask and blocks:
        return seen & (i // mask["size"] == j // mask["size"])
    return seen & ((i - j < mask["size"]) | (j < mask.get("keep_first", 0))) if mask else seen


def _weights_of_keys(q, k, scale, seen, cap=None, sink=None):
    """Softmax weights [head, query, key] of one sequence, q and k [token, head, channel]."""
    k = k.repeat_interleave(q.shape[1] // k.shape[1], 1)
    s = torch.einsum("qhd,khd->hqk", q, k) * scale
    s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(~seen, -math.inf)
    if sink is None:
        return torch.softmax(s, -1)
    return torch.softmax(torch.cat((s, sink[:, None, None].expand(-1, s.shape[1], 1)), -1), -1)[..., :-1]


def _attend(q, k, v, *options, **more):
    """q, k, v [sequence, token, head, channel] -> [sequence, token, head, channel]."""
    v = v.repeat_interleave(q.shape[2] // v.shape[2], 2)
    return torch.stack([torch.einsum("hqk,khd->qhd", _weights_of_keys(a, b, *options, **more), c) for a, b, c in zip(q, k, v)])


def _convolve(x, taps):
    n, t = taps.shape[1], x.shape[1]
    x = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return sum(x[:, j:j + t] * taps[:, j] for j in range(n))


def _linear_scan(decay, k, v, q):
    """S <- decay S + k v', o = S' q; k, q [sequence, token, head, key], v [..., value], decay broadcast against k."""
    s, out = k.new_zeros(*k.shape[:1], *k.shape[2:], v.shape[-1]), []
    decay = decay.expand(k.shape)
    for t in range(k.shape[1]):
        s = decay[:, t, ..., None] * s + k[:, t, ..., None] * v[:, t, :, None, :]
        out.append(torch.einsum("bhkv,bhk->bhv", s, q[:, t]))
    return torch.stack(out, 1)


class Plain:
    def __init__(self, cfg, weights) -> None:
        self.cfg, self.stored = cfg, weights
        self.name = cfg.get("architecture", "Qwen3")
        self.eps = cfg["rms_norm_eps"] if self.name == "Qwen3" else cfg["norm"]["eps"]
        self.vocab = cfg.get("vocab_size", cfg.get("vocab"))

    def w(self, name):
        return self.stored[name].double()

    def mul(self, x, name):
        y = x @ self.w(name).T
        return y + self.w(name + ".b") if name + ".b" in self.stored else y

    def heads(self, x, name, n):
        return self.mul(x, name).unflatten(-1, (n, -1))

    # ------------------------------------------------------------ layers
    def trunk(self, sequences):
        """The normed rows [sequence, token, channel] ahead of the head; shorter sequences are followed by zeros."""
        t = max(map(len, sequences))
        ids = torch.tensor([s + [0] * (t - len(s)) for s in sequences], device=DEVICE)
        return getattr(self, self.name.lower())(ids)

    def logits(self, rows):
        table = next(n for n in ("lm_head.weight", "head", "embed", "model.embed_tokens.weight") if n in self.stored)
        rows = torch.cat([rows @ part.double().T for part in self.stored[table].split(16384)], -1)
        cap = self.cfg.get("logit_softcap")
        return cap * torch.tanh(rows / cap) if cap else rows

    def qwen3(self, ids):
        c, eps = self.cfg, self.eps
        x, seen = self.w("model.embed_tokens.weight")[ids], _seen(ids.shape[1], None, DEVICE)
        rot = {"dims": c["head_dim"], "base": c["rope_theta"]}
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h, a = _rms(x, eps, self.w(p + "input_layernorm.weight")), p + "self_attn."
            q, k, v = (self.heads(h, f"{a}{n}_proj.weight", c[m]) for n, m in
                       (("q", "num_attention_heads"), ("k", "num_key_value_heads"), ("v", "num_key_value_heads")))
            q, k = (_turn(_rms(y, eps, self.w(f"{a}{n}_norm.weight")), rot) for y, n in ((q, "q"), (k, "k")))
            x = x + self.mul(_attend(q, k, v, c["head_dim"] ** -0.5, seen).flatten(2), a + "o_proj.weight")
            h, m = _rms(x, eps, self.w(p + "post_attention_layernorm.weight")), p + "mlp."
            x = x + self.mul(_silu(self.mul(h, m + "gate_proj.weight")) * self.mul(h, m + "up_proj.weight"), m + "down_proj.weight")
        return _rms(x, eps, self.w("model.norm.weight"))

    def rulorax(self, ids):
        eps, x = self.eps, self.w("embed")[ids]
        xs, latents = torch.stack([x] * self.cfg["streams"]), {}
        for i, layer in enumerate(self.cfg["layers"]):
            m, p = layer["mixer"], f"l{i}."
            for part in "12":
                h = _rms(torch.einsum("s,s...->...", self.w(f"{p}hc{part}.in"), xs), eps, self.w(p + "norm" + part))
                if part == "1":
                    if "kv_from" not in m:
                        latents[i] = self.latent(h, p + "mix.", m, neighbours=False)
                    y = self.latent_attention(h, self.heads(h, p + "mix.q", m["heads"]), latents[m.get("kv_from", i)], p + "mix.", m, False)
                    y = self.mul(y * torch.sigmoid(self.mul(h, p + "mix.g")), p + "mix.o")
                else:
                    y = self.ff(h, p + "mlp.", layer["mlp"])
                xs = torch.einsum("st,s...->t...", self.w(f"{p}hc{part}.mix"), xs) + self.w(f"{p}hc{part}.out")[:, None, None, None] * y
        return _rms(xs.sum(0), eps, self.w("final.norm"))

    def latent(self, h, p, m, neighbours):
        d = self.mul(h, p + "dkv")
        return _rms(d[..., :m["kv_rank"]], self.eps, self.w(p + "dkv.norm")), _turn(d[..., None, m["kv_rank"]:], m["rot"], neighbours)

    def latent_attention(self, h, q, latent, p, m, neighbours, sink=None):
        c, turned = latent
        q = torch.cat((q[..., :m["dim"]], _turn(q[..., m["dim"]:], m["rot"], neighbours)), -1)
        k = self.heads(c, p + "uk", m["heads"])
        k = torch.cat((k, turned.expand(*k.shape[:3], -1)), -1)
        seen = _seen(h.shape[1], m.get("mask"), h.device)
        return _attend(q, k, self.heads(c, p + "uv", m["heads"]), m["scale"], seen, sink=sink).flatten(2)

    def kasovik(self, ids):
        eps, b = self.eps, self.cfg["embedding"]["bigram"]
        before = torch.nn.functional.pad(ids[:, :-1], (1, 0))
        pair = (before * b["mul_prev"] + ids * b["mul_cur"]) % b["buckets"]
        pair[:, 0] = b["buckets"]
        x = self.w("embed")[ids] * self.cfg["embedding"]["scale"] + self.stored["bigram"][pair].double()
        for i, layer in enumerate(self.cfg["layers"]):
            m, p, mlp = layer["mixer"], f"l{i}.mix.", f"l{i}.mlp."
            h = _rms(x, eps, self.w(f"l{i}.norm1"))
            if layer["type"] == "retention":
                q, k, v = (self.heads(h, p + n, m["heads"]) for n in "qkv")
                y = _linear_scan(torch.tensor(m["decay"], dtype=torch.float64, device=DEVICE)[:, None],
                                 _turn(k, m["rot"]) * m["dim"] ** -0.5, v, _turn(q, m["rot"]))
                y = self.mul(_rms(y, eps).flatten(2) * _silu(self.mul(h, p + "g")), p + "o")
            else:
                a = m["left"]
                q, k = self.heads(h, p + "left.q", a["heads"]), self.heads(h, p + "left.k", a["kv_heads"])
                y = _attend(_rms(q, eps), _rms(k, eps), k, a["scale"], _seen(h.shape[1], a["mask"], h.device), sink=self.w(p + "left.sink"))
                y = m["left_scale"] * self.mul(y.flatten(2), p + "left.o") + m["right_scale"] * self.delta(h, p + "right.", m["right"])
            limit = layer["mlp"]["limit"]
            g, u = self.mul(h, mlp + "gate").clamp(max=limit), self.mul(h, mlp + "up").clamp(-limit, limit)
            x = x + y + self.mul(g * torch.sigmoid(1.702 * g) * (u + 1), mlp + "down")
        return _rms(x, eps, self.w("final.norm"))

    def delta(self, h, p, m):
        heads, kvh, dim, eps = m["heads"], m["kv_heads"], m["dim"], self.eps
        q, k, v = (_silu(_convolve(self.mul(h, p + n), self.w(f"{p}{n}.conv"))).unflatten(-1, (g, -1))
                   for n, g in (("q", kvh), ("k", kvh), ("v", heads)))
        q, k = (y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (q, k))
        q, k = (y.repeat_interleave(heads // kvh, 2) for y in (q * dim ** -0.5, k))
        beta = torch.sigmoid(self.mul(h, p + "b"))[..., None]
        a = (self.mul(self.mul(h, p + "a1"), p + "a2") + self.w(p + "dt_bias")).unflatten(-1, (heads, dim))
        keep = torch.exp(-torch.exp(self.w(p + "A_log"))[:, None] * torch.nn.functional.softplus(a, threshold=1e9))
        s, out = h.new_zeros(h.shape[0], heads, dim, v.shape[-1]), []
        for t in range(h.shape[1]):
            s = keep[:, t, ..., None] * s
            u = beta[:, t] * (v[:, t] - torch.einsum("bhkv,bhk->bhv", s, k[:, t]))
            s = s + k[:, t, ..., None] * u[:, :, None]
            out.append(torch.einsum("bhkv,bhk->bhv", s, q[:, t]))
        gate = torch.sigmoid(self.mul(self.mul(h, p + "g1"), p + "g2"))
        return self.mul(_rms(torch.stack(out, 1), eps, self.w(p + "norm")).flatten(2) * gate, p + "o")

    def tilarax(self, ids):
        eps, x = self.eps, self.w("embed")[ids]
        out = lambda y, name: _rms(y, eps) * (1 + self.w(name))                                  # noqa: E731
        history, first = [x], None
        for i, layer in enumerate(self.cfg["layers"]):
            m, p = layer["mixer"], f"l{i}.mix."
            if layer["type"] == "attention":
                q, k, v = (self.heads(x, p + n, m[g]) for n, g in (("q", "heads"), ("k", "kv_heads"), ("v", "kv_heads")))
                q, k = (_turn(_rms(y, eps, self.w(f"{p}{n}.norm")), m["rot"], True) for y, n in ((q, "q"), (k, "k")))
                v = v if first is None else torch.lerp(v, first, self.w(p + "vmix"))
                first = v if first is None else first
                q, seen = q * self.w(p + "temp")[:, None], _seen(x.shape[1], m["mask"], x.device, blocks=True)
                vs = v.repeat_interleave(m["heads"] // m["kv_heads"], 2)
                y = torch.stack([torch.einsum("hqk,khd->qhd", torch.einsum("hg,gqk->hqk", self.w(p + "talk"),
                                              _weights_of_keys(a, b, m["scale"], seen)), c) for a, b, c in zip(q, k, vs)])
                y = self.mul(y.flatten(2), p + "o")
            else:
                y = self.mlstm(x, p, m)
            x = x + out(y, f"l{i}.norm1")
            x = x + out(self.ff(x, f"l{i}.mlp.", layer["mlp"]), f"l{i}.norm2")
            history.append(x)
            x = sum(c * y for c, y in zip(self.w(f"l{i}.dwa"), history))
        return out(x, "final.norm")

    def mlstm(self, x, p, m):
        heads, dim, cap = m["heads"], m["dim"], float(m["gate_cap"])
        q, k, v = (self.heads(x, p + n, heads) for n in "qkv")
        q = q * dim ** -0.5
        gi, gf = (cap * torch.tanh(self.mul(x, p + n) / cap) for n in "if")
        gf = torch.nn.functional.logsigmoid(gf)
        s, n, top, out = x.new_zeros(x.shape[0], heads, dim, v.shape[-1]), x.new_zeros(x.shape[0], heads, dim), x.new_zeros(x.shape[0], heads), []
        for t in range(x.shape[1]):
            new = torch.maximum(gf[:, t] + top, gi[:, t])
            keep, take = torch.exp(gf[:, t] + top - new)[..., None], torch.exp(gi[:, t] - new)[..., None] * k[:, t]
            s, n, top = keep[..., None] * s + take[..., None] * v[:, t, :, None], keep * n + take, new
            below = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
            out.append(torch.einsum("bhkv,bhk->bhv", s, q[:, t]) / below[..., None])
        y = _rms(torch.stack(out, 1), self.eps).flatten(2) * self.w(p + "norm")
        return self.mul(y * torch.sigmoid(self.mul(x, p + "g")), p + "o")

    def vobosun(self, ids):
        x = self.w("embed")[ids]
        norm = lambda y, n: torch.tanh(self.w(n + ".alpha") * y) * self.w(n) + self.w(n + ".b")      # noqa: E731
        for i, layer in enumerate(self.cfg["layers"]):
            m, l, p = layer["mixer"], f"l{i}.", f"l{i}.mix."                                   # noqa: E741
            h = norm(x, l + "norm1")
            h = torch.lerp(h, torch.nn.functional.pad(h[:, :-1], (0, 0, 1, 0)), self.w(l + "shift"))
            if layer["type"] == "attention":
                q, k, v = (self.heads(h, p + n, m[g]) for n, g in (("q", "heads"), ("k", "kv_heads"), ("v", "kv_heads")))
                y = self.mul(_attend(_turn(q, m["rot"]), _turn(k, m["rot"]), v, m["scale"], _seen(h.shape[1], None, h.device)).flatten(2), p + "o")
            else:
                y = self.general_delta(h, p, m)
            x = x + norm(y, l + "norm1b")
            x = x + norm(self.ff(norm(x, l + "norm2"), l + "mlp.", layer["mlp"]), l + "norm2b")
        return norm(x, "final.norm")

    def general_delta(self, h, p, m):
        heads = m["heads"]
        r, k, v = (self.heads(h, p + n, heads) for n in "rkv")
        low = self.mul(torch.tanh(self.mul(h, p + "w1")), p + "w2") + self.w(p + "w0")
        keep = torch.exp(-math.exp(-0.5) * torch.sigmoid(low)).unflatten(-1, (heads, -1))
        unit = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        drop = torch.sigmoid(self.mul(h, p + "a")).unflatten(-1, (heads, -1)) * unit
        s, out = h.new_zeros(h.shape[0], heads, m["dim"], m["dim"]), []
        for t in range(h.shape[1]):
            old = torch.einsum("bhkv,bhk->bhv", s, unit[:, t])
            s = keep[:, t, ..., None] * s - drop[:, t, ..., None] * old[:, :, None] + k[:, t, ..., None] * v[:, t, :, None]
            out.append(torch.einsum("bhkv,bhk->bhv", s, r[:, t]))
        y = _rms(torch.stack(out, 1), self.eps).flatten(2) * self.w(p + "norm")
        return self.mul(y * torch.sigmoid(self.mul(h, p + "g")), p + "o")

    def gegunex(self, ids):
        eps, x, mult = self.eps, self.w("embed")[ids], self.cfg["residual_mult"]

        def norm(y, name):
            y = y - y.mean(-1, keepdim=True)
            return _rms(y, eps, self.w(name))

        for i, layer in enumerate(self.cfg["layers"]):
            m, p = layer["mixer"], f"l{i}.mix."
            h = norm(x, f"l{i}.norm1")
            if layer["type"] == "channel_delta":
                y = self.delta(h, p, m)
            elif layer["type"] == "latent_attention":
                q = self.heads(_rms(self.mul(h, p + "dq"), eps, self.w(p + "dq.norm")), p + "uq", m["heads"])
                y = self.mul(self.latent_attention(h, q, self.latent(h, p, m, True), p, m, True, self.w(p + "sink")), p + "o")
            else:
                q, k, v = (_silu(self.heads(h, p + n, m["heads"])) for n in "qkv")
                y = _linear_scan(torch.tensor(m["decay"], dtype=torch.float64, device=DEVICE)[:, None], k, v, q).flatten(2)
                y = self.mul(_rms(y, eps, self.w(p + "norm")) * torch.sigmoid(self.mul(h, p + "g")), p + "o")
            x = x + mult * y
            x = x + mult * self.ff(norm(x, f"l{i}.norm2"), f"l{i}.mlp.", layer["mlp"])
        return norm(x, "final.norm")

    def bukuvik(self, ids):
        eps, mult = self.eps, self.cfg["residual_mult"]
        x = self.w("embed")[ids] * self.cfg["embedding"]["scale"]
        for i, layer in enumerate(self.cfg["layers"]):
            m, l, p = layer["mixer"], f"l{i}.", f"l{i}.mix."                                   # noqa: E741
            if layer["type"] == "attention":
                y = self.two_maps(x, p, m)
            else:
                y = 0.5 * (_rms(self.kept_window(x, p + "left.", m["left"]), eps, self.w(p + "left.out"))
                           + _rms(self.state_space(x, p + "right.", m["right"]), eps, self.w(p + "right.out")))
            x = x + mult * _rms(y, eps, self.w(l + "norm1")) * self.w(l + "ls1")
            y = self.mul(torch.relu(self.mul(x, l + "mlp.up")) ** 2, l + "mlp.down")
            x = x + mult * _rms(y, eps, self.w(l + "norm2")) * self.w(l + "ls2")
        return _rms(x, eps, self.w("final.norm"))

    def two_maps(self, x, p, m):
        eps, d, seen = self.eps, m["diff"], _seen(x.shape[1], m["mask"], x.device)
        q, k = (self.heads(x, p + n, m[g]).unflatten(-1, (2, -1)) for n, g in (("q", "heads"), ("k", "kv_heads")))
        q, k = (_rms(y, eps, self.w(f"{p}{n}.norm")) for y, n in ((q, "q"), (k, "k")))
        v = self.heads(x, p + "v", m["kv_heads"])
        a, b = (_attend(_turn(q[..., j, :], m["rot"]), _turn(k[..., j, :], m["rot"]), v, m["scale"], seen, cap=m["softcap"]) for j in (0, 1))
        lam = torch.exp(self.w(p + "lq1") @ self.w(p + "lk1")) - torch.exp(self.w(p + "lq2") @ self.w(p + "lk2")) + d
        return self.mul((_rms(a - lam * b, eps) * (1 - d)).flatten(2) * torch.sigmoid(self.mul(x, p + "g")), p + "o")

    def kept_window(self, x, p, m):
        q, k, v = (self.heads(x, p + n, m[g]) for n, g in (("q", "heads"), ("k", "kv_heads"), ("v", "kv_heads")))
        q, k = (_rms(_turn(y, m["rot"]), self.eps) for y in (q, k))
        y = _attend(q, k, v, m["scale"], _seen(x.shape[1], m["mask"], x.device))
        return self.mul(y.flatten(2) * torch.sigmoid(self.mul(x, p + "g")), p + "o")

    def state_space(self, x, p, m):
        heads, groups, n, inner = m["heads"], m["groups"], m["state"], m["heads"] * m["vdim"]
        z, mixed, dt = self.mul(x, p + "in").split([inner, inner + 2 * groups * n, heads], -1)
        mixed = _silu(_convolve(mixed, self.w(p + "conv")) + self.w(p + "conv.b"))
        v, k, q = mixed.split([inner, groups * n, groups * n], -1)
        v, (k, q) = v.unflatten(-1, (heads, -1)), (y.unflatten(-1, (groups, -1)).repeat_interleave(heads // groups, 2) for y in (k, q))
        dt = torch.nn.functional.softplus(dt + self.w(p + "dt_bias"), threshold=1e9)[..., None]
        y = _linear_scan(torch.exp(-torch.exp(self.w(p + "A_log"))[:, None] * dt), dt * k, v, q) + self.w(p + "D")[:, None] * v
        y = _rms((y.flatten(2) * _silu(z)).unflatten(-1, (m["norm_groups"], -1)), self.eps).flatten(2) * self.w(p + "norm")
        return self.mul(y, p + "o")

    # ------------------------------------------------------------ feed-forwards
    def unit(self, h, p, mlp):
        """Gated, plain or clamped, as the design has them."""
        if self.name == "Gegunex":
            g, u = self.mul(h, p + "gate").clamp(max=mlp["expert"]["limit"]), self.mul(h, p + "up")
            return self.mul(g * torch.sigmoid(1.702 * g) * (u.clamp(-mlp["expert"]["limit"], mlp["expert"]["limit"]) + 1), p + "down")
        if p + "gate" in self.stored:
            return self.mul(_silu(self.mul(h, p + "gate")) * self.mul(h, p + "up"), p + "down")
        up = self.mul(h, p + "up")
        if self.name == "Tilarax":
            return self.mul(torch.nn.functional.gelu(up, approximate="tanh"), p + "down")
        if self.name == "Vobosun":
            a, b = torch.nn.functional.softplus(self.w(p + "act"))
            return self.mul(torch.where(up > 0, a * up * up + up / 2, (0.5 + b) * (torch.expm1(up.clamp(max=0)) - up) + up / 2), p + "down")
        return self.mul(torch.relu(up) ** 2, p + "down")

    def ff(self, h, p, mlp):
        if mlp["kind"] == "dense":
            return self.unit(h, p, mlp)
        r, rows = mlp["router"], h.flatten(0, 1)
        z, real = self.mul(rows, p + "router"), r["experts"]
        score = torch.sigmoid(z) if self.name == "Gegunex" else torch.softmax(z, -1)
        choice = z
        if self.name == "Vobosun":
            choice = score + self.w(p + "correction")
            by_group = choice.unflatten(-1, (r["groups"]["count"], -1))
            kept = torch.zeros_like(by_group[..., 0], dtype=torch.bool).scatter(-1, by_group.amax(-1).topk(r["groups"]["keep"], -1).indices, True)
            choice = by_group.masked_fill(~kept[..., None], -math.inf).flatten(-2)
        chosen = choice.topk(r["top"], -1).indices
        share = score.gather(-1, chosen)
        if self.name == "Tilarax":
            share = torch.softmax(z.gather(-1, chosen), -1)
        elif self.name == "Vobosun":
            share = share / (share.sum(-1, keepdim=True) + 1e-20)
        out = torch.zeros_like(rows)
        for e in range(z.shape[-1]):
            at, place = (chosen == e).nonzero(as_tuple=True)
            if at.numel():
                g, y = share[at, place][:, None], rows[at]
                if self.name == "Gegunex":
                    out[at] += self.unit(g * y, f"{p}e{e}.", mlp)
                else:
                    out[at] += g * (y if e >= real else self.unit(y, f"{p}e{e}.", mlp))
        if mlp.get("shared"):
            y = self.unit(rows, p + "shared.", mlp)
            out = out + (torch.sigmoid(self.mul(rows, p + "shared.sg")) * y if self.name == "Rulorax" else y)
        return out.unflatten(0, h.shape[:2])
