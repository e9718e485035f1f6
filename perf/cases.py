"""The work that programs have this library do, as cases that can be timed and checked one by one.

Two kinds of case:

* `model`: a whole GPT-2 decode step through `Engine.step`, logits out.  After every pass the lengths go back to where they
  were (`CacheBank.commit`), as in a program that scores several next tokens after the same prompts.
* `layers`: the layers of a plan on a step's rows, `block.forward(ctx, stream, entry, owns)`, recorded once as a CUDA graph
  and replayed, as the engine records and replays its steps.  The rows are a 32-bit residual stream; what comes out is the
  stream behind the layers, the cache pages they filed and the per-sequence states they left.

The sizes are those of `bench.py` (GPT-2 small to XL; the other designs at GPT-2's small and medium width) and of the tests.
"""
from __future__ import annotations

import json
import math
import tempfile
from pathlib import Path

import torch

import burn_transformers_b200 as bt
from burn_transformers_b200.weights.safetensors_io import write_file

F64 = torch.float64
EPS = 1e-5
VOCAB = 50257          # of whole models; a layer's engine is built with a vocabulary of 64 that no pass touches
SIZES = {"small": (768, 12), "medium": (1024, 16), "large": (1280, 20), "xl": (1600, 25)}       # width, heads
DESIGNS = ("sovozen", "gokezen", "rakarax", "visadra", "zatinex")


# ---- the cases ---------------------------------------------------------------------------------------------------

def listed():
    def layers(name, design, size, seqs, shortest, longest, past=0, new=0, dtype="bfloat16"):
        return {"name": name, "kind": "layers", "design": design, "size": size, "dtype": dtype, "seqs": seqs,
                "shortest": shortest, "longest": longest, "past": past, "new": new}

    return [
        # one user at a prompt: the library's smallest call, all latency
        {"name": "gpt2_small_decode_1", "kind": "model", "size": "small", "seqs": 1, "shortest": 511, "longest": 511},
        # the library's headline: a handful of conversations of unequal lengths, one token each
        {"name": "gpt2_small_decode_8", "kind": "model", "size": "small", "seqs": 8, "shortest": 203, "longest": 901},
        # a serving batch of the largest model: a layer of GPT-2 XL, one token for each of 64 sequences
        layers("gpt2_xl_decode_64", "gpt2", "xl", 64, 250, 510, past=1, new=1),
        # prompts of ordinary length arriving together
        layers("gpt2_small_prompts_2x1024", "gpt2", "small", 2, 1024, 1024),
        # the largest step: a full batch of long prompts through a layer of the largest model
        layers("gpt2_xl_prompts_16x1024", "gpt2", "xl", 16, 1024, 1024),
        # prompts brought in portions (`prefill_chunk_size`), behind unequal beginnings
        layers("gpt2_medium_portions_8x129", "gpt2", "medium", 8, 17, 771, past=1, new=129),
        # the true 32-bit path (reference checks, evaluation), odd lengths
        layers("gpt2_small_prompts_f32", "gpt2", "small", 3, 37, 499, dtype="float32"),
        # a latent attention with sink and gate, and a decayed linear attention
        layers("sovozen_medium_prompts_2x1024", "sovozen", "medium", 2, 1024, 1024),
        # a windowed attention beside a matrix memory, routed experts with a shared one
        layers("gokezen_medium_prompts_2x1024", "gokezen", "medium", 2, 1024, 1024),
        # a talking attention behind a convolution beside a selective scan; unequal prompts
        layers("rakarax_small_prompts_ragged", "rakarax", "small", 4, 201, 1019),
        # a latent attention and routed experts, one token for each of 64 sequences
        layers("visadra_medium_decode_64", "visadra", "medium", 64, 250, 510, past=1, new=1),
        # a differential attention and a gated linear attention
        layers("zatinex_medium_prompts_2x1024", "zatinex", "medium", 2, 1024, 1024),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(("model", "decode", "prompts", "prompts", "portions", "f32", "designs", "designs", "designs", "designs_decode"))
    if what == "model":
        longest = spread(16, 1000)
        return {"kind": "model", "size": "small", "seqs": spread(1, 16), "shortest": rng.randint(8, longest), "longest": longest}
    case = {"kind": "layers", "design": "gpt2", "size": rng.choice(list(SIZES)), "dtype": "bfloat16", "past": 0, "new": 0}
    longest = spread(24, 1022)
    if what == "decode":
        case.update(seqs=spread(1, 64), past=1, new=1)
    elif what == "portions":
        new = spread(2, 257)
        longest = min(longest, 1020 - new)
        case.update(seqs=spread(1, 16), past=1, new=new)
    elif what == "prompts":
        case.update(seqs=spread(1, 16))
    elif what == "f32":
        case.update(size=rng.choice(("small", "medium")), seqs=spread(1, 4), dtype="float32")
    else:
        case.update(design=rng.choice(DESIGNS if what == "designs" else ("visadra",)), size=rng.choice(("small", "medium")),
                    seqs=spread(1, 6))
        if what == "designs_decode":
            case.update(seqs=spread(1, 64), past=1, new=1)
    case.update(shortest=rng.randint(max(1, longest // 5), longest), longest=longest)
    return case


def _lengths(case):
    """The sequences' lengths from `shortest` to `longest` (beginnings before the step's tokens, when `past` is set)."""
    n, lo, hi = case["seqs"], case["shortest"], case["longest"]
    return [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _runs(case):
    """(tokens before the step, tokens of the step) per sequence."""
    return [(n, case["new"]) if case["past"] else (0, n) for n in _lengths(case)]


# ---- configurations, as bench.py has them -------------------------------------------------------------------------

def _config(case):
    width, heads = SIZES[case["size"]]
    if case["kind"] == "model" or case["design"] == "gpt2":
        whole = case["kind"] == "model"
        return dict(model_type="gpt2", n_layer=12 if whole else 1, n_embd=width, n_head=heads, n_inner=4 * width,
                    vocab_size=VOCAB if whole else 64, n_positions=1024, layer_norm_epsilon=EPS, activation_function="gelu_new")
    small = case["size"] == "small"
    rank, rot, ff, expert_ff, shared_ff = (256, 32, 2048, 384, 512) if small else (512, 64, 2816, 512, 768)
    dim = 64
    turn = {"dims": rot, "base": 10000.0}
    dense = {"kind": "dense", "ff": ff}
    latent = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": dim, "kv_rank": rank, "scale": (dim + rot) ** -0.5, "rot": turn}
    decay = [1.0 - 2.0 ** -(3 + h % 6) for h in range(heads)]
    base = {"vocab": 64, "width": width, "norm": {"eps": EPS}}
    if case["design"] == "sovozen":
        return dict(base, architecture="Sovozen", embedding={"scale": 1.0}, logit_scale=1.0, layers=[
            {"type": "latent_attention", "mixer": latent, "mlp": dense},
            {"type": "lightning", "mixer": {"heads": heads, "dim": dim, "vdim": dim, "decay": decay}, "mlp": dense}])
    if case["design"] == "gokezen":
        mixer = {"left": {"heads": heads, "kv_heads": heads // 4, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "mask": {"size": 512}},
                 "left_scale": 1.0, "right": {"heads": heads, "dim": dim, "vdim": dim, "gate_cap": 15.0}, "right_scale": 1.0}
        routed = {"kind": "moe", "expert": {"ff": expert_ff, "limit": 7.0}, "shared": {"ff": shared_ff, "limit": 7.0},
                  "router": {"experts": 16, "top": 4, "scale": 1.0, "groups": {"count": 4, "keep": 2}}}
        return dict(base, architecture="Gokezen", max_positions=2048, layers=[{"type": "parallel", "mixer": mixer, "mlp": routed}])
    if case["design"] == "rakarax":
        left = {"heads": heads, "kv_heads": heads // 4, "dim": dim, "vdim": dim, "conv": 4, "scale": dim ** -0.5, "softcap": 30.0,
                "mask": {"size": 512}}
        right = {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "conv": 4}
        return dict(base, architecture="Rakarax", max_positions=2048, layers=[
            {"type": "parallel", "mlp": {"kind": "dense", "ff": 4 * width},
             "mixer": {"left": left, "left_scale": 1.0, "right": right, "right_scale": 1.0}}])
    if case["design"] == "visadra":
        routed = {"kind": "moe", "expert": {"ff": expert_ff}, "router": {"experts": 16, "top": 4}, "shared": {"ff": shared_ff}}
        return dict(base, architecture="Visadra", embedding={"scale": 1.0}, logit_scale=1.0,
                    layers=[{"type": "latent_attention", "mixer": latent, "mlp": routed}])
    attention = {"heads": heads // 2, "kv_heads": heads // 4, "dim": dim, "vdim": 2 * dim, "conv": 4, "scale": dim ** -0.5, "diff": 0.5,
                 "rot": {"dims": dim // 2, "base": 10000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
    gla = {"heads": heads, "dim": dim, "vdim": dim, "tau": 16.0, "decay_rank": 16}
    return dict(base, architecture="Zatinex", layers=[{"type": "attention", "mixer": attention, "mlp": dense},
                                                      {"type": "gla", "mixer": gla, "mlp": dense}])


# ---- weights and rows, from the seed alone ------------------------------------------------------------------------
# Every number is one that bfloat16 holds, so that each data type and the 64-bit computation start from the same weights.
# Matrices have a standard deviation of one over the root of their inputs, as trained layers do that keep their rows' size.

class _Draw:
    def __init__(self, seed):
        self.device = "cuda" if torch.cuda.is_available() else "cpu"
        self.gen = torch.Generator(device=self.device)
        self.gen.manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0):
        return (torch.randn(shape, generator=self.gen, device=self.device) * std + mean).bfloat16().float()

    def matrix(self, rows, inputs):
        return self.normal(rows, inputs, std=inputs ** -0.5)

    def uniform(self, lo, hi, *shape):
        return (torch.rand(shape, generator=self.gen, device=self.device) * (hi - lo) + lo).bfloat16().float()


def _gpt2_layer(r, w, p, width):
    for norm in ("ln_1", "ln_2"):
        w[p + norm + ".weight"], w[p + norm + ".bias"] = r.normal(width, std=0.1, mean=1.0), r.normal(width, std=0.05)
    for name, inputs, outputs in (("attn.c_attn", width, 3 * width), ("attn.c_proj", width, width), ("mlp.c_fc", width, 4 * width),
                                  ("mlp.c_proj", 4 * width, width)):
        w[p + name + ".weight"] = r.normal(inputs, outputs, std=inputs ** -0.5)
        w[p + name + ".bias"] = r.normal(outputs, std=0.05)


def _weights(case, config, r):
    """Tensors by checkpoint name (matrices of GPT-2 stored [in, out], all others [out, in])."""
    width, heads = SIZES[case["size"]]
    w = {}
    if "n_embd" in config:
        w["wte.weight"] = r.normal(config["vocab_size"], width, std=width ** -0.5)
        w["wpe.weight"] = r.normal(config["n_positions"], width, std=0.5 * width ** -0.5)
        w["ln_f.weight"], w["ln_f.bias"] = r.normal(width, std=0.1, mean=1.0), r.normal(width, std=0.05)
        for i in range(config["n_layer"]):
            _gpt2_layer(r, w, f"h.{i}.", width)
        return w
    design = case["design"]
    gain = 0.0 if design == "rakarax" else 1.0               # (Rakarax stores a gain minus one)
    w["embed"], w["final.norm"] = r.matrix(64, width), r.normal(width, std=0.1, mean=gain)
    if "max_positions" in config:
        w["pos"] = r.normal(config["max_positions"], width, std=0.02)
    if design != "gokezen":
        w["head"] = r.matrix(64, width)
    if design == "visadra":                                    # (one number is the whole gain)
        w["final.norm"] = r.normal(1, std=0.1, mean=1.0).reshape(())

    def pair(p, ff, inputs=width):
        w[p + "gate"], w[p + "up"], w[p + "down"] = r.matrix(ff, inputs), r.matrix(ff, inputs), r.matrix(inputs, ff)

    norms = {"gokezen": ("norm1",), "rakarax": ("norm1", "norm1b", "norm2", "norm2b")}.get(design, ("norm1", "norm2"))
    for i, layer in enumerate(config["layers"]):
        p, x, m, mlp = f"l{i}.", f"l{i}.mix.", layer["mixer"], layer["mlp"]
        for norm in norms:
            w[p + norm] = r.normal(1, std=0.1, mean=1.0).reshape(()) if design == "visadra" else r.normal(width, std=0.1, mean=gain)
        if layer["type"] == "latent_attention":
            H, rank = m["heads"], m["kv_rank"]
            w[x + "q"], w[x + "dkv"] = r.matrix(H * (m["dim"] + m["rot_dim"]), width), r.matrix(rank + m["rot_dim"], width)
            w[x + "dkv.norm"], w[x + "sink"] = r.normal(rank, std=0.1, mean=1.0), r.normal(H)
            w[x + "uk"], w[x + "uv"] = r.matrix(H * m["dim"], rank), r.matrix(H * m["vdim"], rank)
            w[x + "o"] = r.matrix(width, H * m["vdim"])
            if design == "sovozen":
                w[x + "g"] = r.matrix(H * m["vdim"], width)
        elif layer["type"] == "lightning":
            wide = m["heads"] * m["dim"]
            w.update({x + n: r.matrix(wide, width) for n in "qkvg"})
            w[x + "norm"], w[x + "o"] = r.normal(wide, std=0.1, mean=1.0), r.matrix(width, wide)
        elif design == "gokezen":
            a, b, left, right = x + "left.", x + "right.", m["left"], m["right"]
            for n, count in (("q", left["heads"]), ("k", left["kv_heads"]), ("v", left["kv_heads"])):
                w[a + n] = r.matrix(count * left["dim"], width)
            w[a + "o"] = r.matrix(width, left["heads"] * left["vdim"])
            wide = right["heads"] * right["dim"]
            w.update({b + n: r.matrix(wide, width) for n in "qkvg"})
            w[b + "i"], w[b + "f"] = r.matrix(heads, width), r.matrix(heads, width)
            w[b + "i.b"], w[b + "f.b"] = r.normal(heads, std=0.5, mean=-1.0), r.uniform(2.0, 6.0, heads)   # (memories that last)
            w[b + "norm"], w[b + "o"] = r.normal(wide, std=0.1, mean=1.0), r.matrix(width, wide)
        elif design == "rakarax":
            a, b, left, right = x + "left.", x + "right.", m["left"], m["right"]
            H, G, dim, inner, rank, state = left["heads"], left["kv_heads"], left["dim"], right["inner"], right["dt_rank"], right["state"]
            w[a + "q"], w[a + "k"], w[a + "g"], w[a + "o"] = (r.matrix(H * dim, width), r.matrix(G * dim, width), r.matrix(H * dim, width),
                                                              r.matrix(width, H * dim))
            w[a + "q.conv"], w[a + "k.conv"] = r.normal(H * dim, 4, std=0.5), r.normal(G * dim, 4, std=0.5)
            w[a + "temp"] = r.uniform(4.0, 12.0, H)
            w[a + "talk"] = (r.normal(H, H, std=0.05) + torch.eye(H, device=r.device)).bfloat16().float()
            w[b + "in"], w[b + "x"], w[b + "o"] = r.matrix(2 * inner, width), r.matrix(rank + 2 * state, inner), r.matrix(width, inner)
            w[b + "conv"], w[b + "conv.b"] = r.normal(inner, 4, std=0.5), r.normal(inner, std=0.05)
            w[b + "dt"], w[b + "dt.b"] = r.matrix(inner, rank), r.uniform(-6.0, -2.0, inner)                # (steps of 0.002 to 0.1)
            w[b + "A_log"] = torch.log(torch.arange(1, state + 1, device=r.device).float()).repeat(inner, 1).bfloat16().float()
            w[b + "D"] = r.normal(inner, std=0.1, mean=1.0)
        elif layer["type"] == "gla":
            wide = m["heads"] * m["dim"]
            w.update({x + n: r.matrix(wide, width) for n in "qkvg"})
            w[x + "a1"], w[x + "a2"], w[x + "a2.b"] = r.matrix(m["decay_rank"], width), r.matrix(wide, m["decay_rank"]), r.normal(wide, mean=2.0)
            w[x + "norm"], w[x + "o"] = r.normal(m["vdim"], std=0.1, mean=1.0), r.matrix(width, wide)
        else:                                                  # differential attention
            for n, size in (("q", 2 * m["heads"] * m["dim"]), ("k", 2 * m["kv_heads"] * m["dim"]), ("v", m["kv_heads"] * m["vdim"])):
                w[x + n], w[x + n + ".b"], w[x + n + ".conv"] = r.matrix(size, width), r.normal(size, std=0.05), r.normal(size, 4, std=0.5)
            for n in "qk":
                w[x + n + ".norm"] = r.normal(m["dim"], std=0.1, mean=1.5)
            for n in ("lq1", "lk1", "lq2", "lk2"):
                w[x + n] = r.normal(m["dim"], std=0.1)
            w[x + "o"] = r.matrix(width, m["heads"] * m["vdim"])
        q = p + "mlp."
        if design == "rakarax":
            w[q + "up"], w[q + "down"] = r.matrix(mlp["ff"], width), r.matrix(width, mlp["ff"])
            w[q + "act"] = torch.tensor([0.75, 0.5, 0.25, 0.125], device=r.device)
        elif mlp["kind"] == "dense":
            pair(q, mlp["ff"])
        else:
            w[q + "router"] = r.matrix(mlp["router"]["experts"], width)
            if design == "visadra":
                w[q + "router.b"] = r.normal(mlp["router"]["experts"], std=0.1)
            for e in range(mlp["router"]["experts"]):
                pair(f"{q}e{e}.", mlp["expert"]["ff"])
            pair(q + "shared.", mlp["shared"]["ff"])
    return w


def _rows(case, config, w, r):
    """The residual stream of every token, [tokens, width], sequence after sequence.  Where experts follow, a token leans
    towards four of them, some asked for far more often than others, as tokens do behind a trained router (without that,
    the last bit of a number would decide which experts a token gets)."""
    width, _ = SIZES[case["size"]]
    n = sum(past + new for past, new in _runs(case))
    x = torch.randn((n, width), generator=r.gen, device=r.device)
    if case["design"] in ("gokezen", "visadra"):
        router = w["l0.mlp.router"]
        lean = router / router.norm(dim=1, keepdim=True)
        often = lambda k: 1.0 / (1.0 + torch.arange(k, device=r.device).float())  # noqa: E731
        groups = torch.multinomial(often(4).expand(n, 4), 2, generator=r.gen)
        for j in range(2):
            inside = torch.multinomial(often(4).expand(n, 4), 2, generator=r.gen)
            x += 5.0 * (lean[groups[:, j] * 4 + inside[:, 0]] + lean[groups[:, j] * 4 + inside[:, 1]])
    return x


def _tokens(case, r):
    """Token ids of every sequence of a whole model's step, the last one being the step's own."""
    return [torch.randint(0, VOCAB, (n + 1,), generator=r.gen, device=r.device) for n in _lengths(case)]


# ---- prepare and run ----------------------------------------------------------------------------------------------

def _engine(case, config, w, runs):
    room = sum(-(-(past + new) // 64) * 64 for past, new in runs)
    matrices = {k: v.bfloat16() if case.get("dtype") != "float32" and v.dim() == 2 else v for k, v in w.items()}
    with tempfile.TemporaryDirectory() as folder:
        (Path(folder) / "config.json").write_text(json.dumps(config))
        write_file(Path(folder) / "model.safetensors", {k: v.cpu() for k, v in matrices.items()})
        return bt.Engine.from_folder(folder, case.get("dtype", "bfloat16"), max_tokens=room, max_slots=len(runs), max_context=1024)


class _Layers:
    """The layers of an engine's plan on the rows of one step, recorded once."""

    def __init__(self, engine, slots, news, stream):
        self.engine, self.given = engine, stream
        self.stream = torch.empty_like(stream)
        entries = [bt.StepEntry(s, [0] * n, []) for s, n in zip(slots, news)]
        engine.cache.reserve([(s, engine.cache.length(s) + n) for s, n in zip(slots, news)])
        self.ctx = engine.builder.build(entries)
        self.fresh = self.ctx.fresh
        self.graph = None

    def issue(self):
        engine, ctx, plan = self.engine, self.ctx, self.engine.plan
        engine.ws.reset()
        self.stream.copy_(self.given)
        if self.fresh:                                        # (what a slot that is taken anew costs: zeroed states)
            for state in engine.cache.states.values():
                state.zero_()
        ctx.shared = {name: ctx.ws.take((ctx.n_tokens, channels), dtype or ctx.dtype)
                      for name, (channels, dtype) in plan.step_tensors.items()}
        for index, call in enumerate(plan.schedule):
            plan.blocks[call.block].forward(ctx, self.stream, *plan.cache_entry(index))
        if ctx.side is not None:
            ctx.side.join()

    def record(self):
        for _ in range(2):                                    # (the scratch memory grows to the step's size)
            self.issue()
        torch.cuda.synchronize()
        self.engine.ws.frozen = True
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            self.issue()
        self.graph = graph

    def run(self):
        self.graph.replay()
        cache = self.engine.cache
        return {"stream": self.stream, "pages": [t for g in cache.groups for t in (g.k, g.v)],
                "states": [cache.states[k] for k in sorted(cache.states)]}


class _Step:
    """A decode step of a whole model after prompts that are in the cache."""

    def __init__(self, engine, slots, tokens):
        self.engine, self.slots = engine, slots
        self.lengths = [len(t) - 1 for t in tokens]
        engine.step([bt.StepEntry(s, t[:-1], []) for s, t in zip(slots, tokens)])
        self.entries = [bt.StepEntry(s, [t[-1]], [0]) for s, t in zip(slots, tokens)]
        for _ in range(2):                                    # (the engine records the step for this batch size)
            self.run()

    def run(self):
        logits = self.engine.step(self.entries)
        for slot, length in zip(self.slots, self.lengths):
            self.engine.cache.commit(slot, length)
        return logits


def prepare(case, seed):
    config, r = _config(case), _Draw(seed)
    w = _weights(case, config, r)
    if case["kind"] == "model":
        tokens = [t.tolist() for t in _tokens(case, r)]
        engine = _engine(case, config, w, [(len(t), 0) for t in tokens])
        return _Step(engine, [engine.new_sequence() for _ in tokens], tokens)
    runs = _runs(case)
    rows = list(torch.split(_rows(case, config, w, r), [past + new for past, new in runs]))
    engine = _engine(case, config, w, runs)
    slots = [engine.new_sequence() for _ in runs]
    if case["past"]:
        before = _Layers(engine, slots, [past for past, _ in runs], torch.cat([x[:past] for x, (past, _) in zip(rows, runs)]))
        before.issue()
        for slot, (past, _) in zip(slots, runs):
            engine.cache.commit(slot, past)
    state = _Layers(engine, slots, [new for _, new in runs], torch.cat([x[past:] for x, (past, _) in zip(rows, runs)]).contiguous())
    state.record()
    return state


def run(state):
    return state.run()


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def work(case):
    """Bytes: every weight once (of routed experts those that the step's tokens can ask for), the rows in and out, the keys
    and values or states that the step reads and files.  Flops: the products, and the attention's over the pairs it sees."""
    config = _config(case)
    width, heads = SIZES[case["size"]]
    elem = 4 if case.get("dtype") == "float32" else 2
    runs = [(n, 1) for n in _lengths(case)] if case["kind"] == "model" else _runs(case)
    n = sum(new for _, new in runs)
    weights = used = per_token_cache = 0                      # numbers stored, numbers a token is multiplied with
    attention = 0.0                                           # flops
    window = 1 << 30

    def pairs(window):
        return sum(min(past + i + 1, window) for past, new in runs for i in range(new))

    layers = config.get("n_layer") or len(config["layers"])
    if "n_embd" in config:
        weights = used = layers * 12 * width * width
        per_token_cache = layers * 2 * width
        attention = layers * 4.0 * width * pairs(window)
        if case["kind"] == "model":
            weights += VOCAB * width
            used += VOCAB * width
    else:
        for layer in config["layers"]:
            m, mlp = layer["mixer"], layer["mlp"]
            if layer["type"] == "latent_attention":
                H, rank = m["heads"], m["kv_rank"]
                mats = width * (H * (m["dim"] + m["rot_dim"]) + rank + m["rot_dim"] + (2 if case["design"] == "sovozen" else 1) * H * m["vdim"]) \
                    + rank * H * (m["dim"] + m["vdim"])
                per_token_cache += rank + m["rot_dim"]
                attention += 2.0 * H * (m["dim"] + m["rot_dim"] + m["vdim"]) * pairs(window)
            elif layer["type"] in ("lightning", "gla"):
                mats = 5 * width * m["heads"] * m["dim"]
                attention += 4.0 * n * m["heads"] * m["dim"] * m["vdim"]
            elif case["design"] == "gokezen":
                mats = width * (2 * heads + 2 * (heads // 4)) * 64 + 5 * width * heads * 64
                per_token_cache += 2 * (heads // 4) * 64
                attention += 4.0 * heads * 64 * pairs(512) + 4.0 * n * heads * 64 * 64
            elif case["design"] == "rakarax":
                inner, rank, state = m["right"]["inner"], m["right"]["dt_rank"], m["right"]["state"]
                mats = width * (3 * heads + heads // 4) * 64 + 3 * width * inner + inner * (2 * rank + 2 * state)
                per_token_cache += 2 * (heads // 4) * 64
                attention += (4.0 * heads * 64 + 2.0 * heads * heads) * pairs(512) + 6.0 * n * inner * state
            else:
                mats = width * (m["heads"] * (2 * m["dim"] + m["vdim"]) + m["kv_heads"] * (2 * m["dim"] + m["vdim"]))
                per_token_cache += m["kv_heads"] * (2 * m["dim"] + m["vdim"])
                attention += 4.0 * m["heads"] * (m["dim"] + m["vdim"]) * pairs(window)
            weights, used = weights + mats, used + mats
            if case["design"] == "rakarax":
                weights, used = weights + 2 * width * mlp["ff"], used + 2 * width * mlp["ff"]
            elif mlp["kind"] == "dense":
                weights, used = weights + 3 * width * mlp["ff"], used + 3 * width * mlp["ff"]
            else:
                one, shared, top, count = 3 * width * mlp["expert"]["ff"], 3 * width * mlp["shared"]["ff"], 4, 16
                weights += min(count, top * n) * one + shared
                used += top * one + shared
    rows = VOCAB * 4 + width * elem if case["kind"] == "model" else 2 * width * 4      # a token's share in and out
    held = sum(past for past, _ in runs) * per_token_cache * elem
    return {"bytes": weights * elem + n * rows + held + n * per_token_cache * elem, "flops": 2.0 * used * n + attention}


def tolerance(case):
    """About four times the distance from the 64-bit computation that was measured (B200; 2-norm): 3.3e-3 for the whole
    model's logits, per layer 1.4e-3 (GPT-2), 3e-3 (Sovozen, Visadra), 6.6e-3 (Rakarax, Zatinex, whose divisions by a root
    mean square stretch small rows), 6.5e-7 in 32 bits.  One number of a row may be much further off than the row: a token
    between two experts is given the other one by the last bit of its router's number."""
    if case.get("dtype") == "float32":
        return {"rel": 3e-6, "max": 1e-3}
    if case["kind"] == "model":
        return {"rel": 1.4e-2, "max": 0.3}
    rel = {"gpt2": 6e-3, "sovozen": 1.2e-2, "visadra": 1.3e-2, "gokezen": 1.3e-2, "rakarax": 2.6e-2, "zatinex": 2.8e-2}[case["design"]]
    return {"rel": rel, "max": 0.9 if case["design"] in ("gokezen", "visadra") else 0.5}


# ---- the same in 64 bits, written plainly -------------------------------------------------------------------------

def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _silu(z):
    return z * torch.sigmoid(z)


def _layer_norm(x, g, b=0.0):
    return (x - x.mean(-1, keepdim=True)) / torch.sqrt(x.var(-1, unbiased=False, keepdim=True) + EPS) * g + b


def _rms(x, g=1.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * g


def _seen(T, first, device, window=1 << 30):
    """[T - first, T]: which keys the queries from position `first` on see."""
    i, j = torch.arange(first, T, device=device)[:, None], torch.arange(T, device=device)[None, :]
    return (j <= i) & (i - j < window)


def _mix(scores, seen, v, sink=None):
    """scores [heads, queries, keys], v [heads, keys, channels]."""
    scores = scores.masked_fill(~seen, float("-inf"))
    if sink is not None:
        scores = torch.cat([scores, sink[:, None, None].expand(-1, scores.shape[1], 1)], -1)
    p = torch.softmax(scores, -1)
    return (p[..., :-1] if sink is not None else p) @ v


def _heads(x, count):
    return x.reshape(x.shape[0], count, -1).transpose(0, 1)


def _merged(x):
    return x.transpose(0, 1).reshape(x.shape[1], -1)


def _turn(x, first, dims, rates, size=1.0):
    """Turns the channel pairs (2i, 2i + 1) of x [..., tokens, channels]; the tokens' positions start at `first`."""
    angle = torch.arange(first, first + x.shape[-2], device=x.device, dtype=F64)[:, None] * rates
    c, s = size * torch.cos(angle), size * torch.sin(angle)
    out = x.clone()
    even, odd = x[..., 0:dims:2], x[..., 1:dims:2]
    out[..., 0:dims:2], out[..., 1:dims:2] = even * c - odd * s, odd * c + even * s
    return out


def _rates(rot, device):
    dims, base = rot["dims"], rot["base"]
    rates = base ** (-2.0 * torch.arange(dims // 2, device=device, dtype=F64) / dims)
    if "scaling" not in rot:
        return rates, 1.0
    s = rot["scaling"]
    index = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(index(s["fast"])), 0), min(math.ceil(index(s["slow"])), dims - 1)
    slowed = ((torch.arange(dims // 2, device=device, dtype=F64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return rates / s["factor"] * slowed + rates * (1.0 - slowed), 0.1 * math.log(s["factor"]) + 1.0


def _conv(u, taps, bias=0.0):
    count = taps.shape[1]
    padded = torch.cat([u.new_zeros(count - 1, u.shape[1]), u])
    return sum(padded[j:j + u.shape[0]] * taps[:, j] for j in range(count)) + bias


def _gpt2_block(x, w, p, heads, first):
    """[tokens from `first` on, width]; the rows before only leave keys and values."""
    dim = x.shape[1] // heads
    h = _layer_norm(x, w[p + "ln_1.weight"], w[p + "ln_1.bias"])
    q, k, v = (h @ w[p + "attn.c_attn.weight"] + w[p + "attn.c_attn.bias"]).chunk(3, -1)
    mixed = _mix(_heads(q[first:], heads) @ _heads(k, heads).transpose(1, 2) * dim ** -0.5, _seen(x.shape[0], first, x.device),
                 _heads(v, heads))
    y = x[first:] + _merged(mixed) @ w[p + "attn.c_proj.weight"] + w[p + "attn.c_proj.bias"]
    h = _layer_norm(y, w[p + "ln_2.weight"], w[p + "ln_2.bias"])
    return y + _gelu(h @ w[p + "mlp.c_fc.weight"] + w[p + "mlp.c_fc.bias"]) @ w[p + "mlp.c_proj.weight"] + w[p + "mlp.c_proj.bias"]


def _latent(h, w, x, m, first, gated):
    H, dim, rot = m["heads"], m["dim"], m["rot_dim"]
    rates, _ = _rates(m["rot"], h.device)
    q = _heads(h[first:] @ w[x + "q"].T, H)
    down = h @ w[x + "dkv"].T
    c = _rms(down[:, :m["kv_rank"]], w[x + "dkv.norm"])
    shared = _turn(down[:, m["kv_rank"]:], 0, rot, rates)
    k, v = _heads(c @ w[x + "uk"].T, H), _heads(c @ w[x + "uv"].T, H)
    scores = q[..., :dim] @ k.transpose(1, 2) + _turn(q[..., dim:], first, rot, rates) @ shared.T
    out = _merged(_mix(scores * m["scale"], _seen(h.shape[0], first, h.device), v, sink=w[x + "sink"]))
    if gated:
        out = out * torch.sigmoid(h[first:] @ w[x + "g"].T)
    return out @ w[x + "o"].T


def _lightning(h, w, x, m):
    H = m["heads"]
    q, k, v = (_heads(_silu(h @ w[x + n].T), H) for n in "qkv")
    decay = torch.tensor(m["decay"], device=h.device, dtype=F64)[:, None, None]
    state, outs = h.new_zeros(H, m["dim"], m["vdim"]), []
    for t in range(h.shape[0]):
        state = decay * state + k[:, t, :, None] * v[:, t, None, :]
        outs.append(torch.einsum("hkv,hk->hv", state, q[:, t]))
    return (_rms(torch.stack(outs).reshape(h.shape[0], -1), w[x + "norm"]) * torch.sigmoid(h @ w[x + "g"].T)) @ w[x + "o"].T


def _gla(h, w, x, m):
    H, dim = m["heads"], m["dim"]
    q, k, v = (_heads(h @ w[x + n].T, H) for n in "qkv")
    alpha = _heads(torch.sigmoid((h @ w[x + "a1"].T) @ w[x + "a2"].T + w[x + "a2.b"]) ** (1.0 / m["tau"]), H)
    state, outs = h.new_zeros(H, dim, m["vdim"]), []
    for t in range(h.shape[0]):
        state = alpha[:, t, :, None] * state + k[:, t, :, None] * v[:, t, None, :]
        outs.append(torch.einsum("hkv,hk->hv", state, q[:, t] * dim ** -0.5))
    return (_rms(torch.stack(outs), w[x + "norm"]).reshape(h.shape[0], -1) * _silu(h @ w[x + "g"].T)) @ w[x + "o"].T


def _memory(h, w, x, m):
    H, dim, cap = m["heads"], m["dim"], m["gate_cap"]
    q, k, v = (_heads(h @ w[x + n].T, H) for n in "qkv")
    a = cap * torch.tanh((h @ w[x + "i"].T + w[x + "i.b"]) / cap)
    b = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w[x + "f"].T + w[x + "f.b"]) / cap))
    S, n, top, outs = h.new_zeros(H, dim, m["vdim"]), h.new_zeros(H, dim), h.new_zeros(H), []
    for t in range(h.shape[0]):
        new = torch.maximum(b[t] + top, a[t])
        keep, take = torch.exp(b[t] + top - new), torch.exp(a[t] - new)
        S = keep[:, None, None] * S + take[:, None, None] * k[:, t, :, None] * v[:, t, None, :]
        n, top = keep[:, None] * n + take[:, None] * k[:, t], new
        qt = q[:, t] * dim ** -0.5
        outs.append(torch.einsum("hkv,hk->hv", S, qt) / (torch.maximum((n * qt).sum(-1).abs(), torch.exp(-top)) + 1e-6)[:, None])
    flat = _rms(torch.stack(outs)).reshape(h.shape[0], -1) * w[x + "norm"] * torch.sigmoid(h @ w[x + "g"].T)
    return flat @ w[x + "o"].T


def _window_attention(h, w, x, m):
    H, G = m["heads"], m["kv_heads"]
    q, k, v = _heads(h @ w[x + "q"].T, H), _heads(h @ w[x + "k"].T, G), _heads(h @ w[x + "v"].T, G)
    k, v = k.repeat_interleave(H // G, 0), v.repeat_interleave(H // G, 0)
    return _merged(_mix(q @ k.transpose(1, 2) * m["scale"], _seen(h.shape[0], 0, h.device, m["mask"]["size"]), v)) @ w[x + "o"].T


def _talking_attention(h, w, x, m):
    H, G, T = m["heads"], m["kv_heads"], h.shape[0]
    q, v = _rms(_heads(_conv(h @ w[x + "q"].T, w[x + "q.conv"]), H)), _heads(_conv(h @ w[x + "k"].T, w[x + "k.conv"]), G)
    k = _rms(v)
    s = q @ k.repeat_interleave(H // G, 0).transpose(1, 2) * m["scale"] * w[x + "temp"][:, None, None]
    s = m["softcap"] * torch.tanh(s / m["softcap"])
    at = torch.arange(T, device=h.device, dtype=F64)
    slope = 2.0 ** (-8.0 * torch.arange(1, H + 1, device=h.device, dtype=F64) / H)
    s = s - slope[:, None, None] * (at[:, None] - at[None, :])
    s = torch.einsum("hg,gij->hij", w[x + "talk"], s)
    out = _mix(s, _seen(T, 0, h.device, m["mask"]["size"]), v.repeat_interleave(H // G, 0))
    return (_merged(out) * torch.sigmoid(h @ w[x + "g"].T)) @ w[x + "o"].T


def _selective_scan(h, w, x, m):
    inner, rank, count = m["inner"], m["dt_rank"], m["state"]
    u, z = (h @ w[x + "in"].T).split(inner, -1)
    u = _silu(_conv(u, w[x + "conv"], w[x + "conv.b"]))
    low = u @ w[x + "x"].T
    dt = torch.nn.functional.softplus(low[:, :rank] @ w[x + "dt"].T + w[x + "dt.b"], threshold=200.0)
    B, C, A = low[:, rank:rank + count], low[:, rank + count:], -torch.exp(w[x + "A_log"])
    S, outs = h.new_zeros(inner, count), []
    for t in range(h.shape[0]):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * B[t]
        outs.append(S @ C[t])
    return ((torch.stack(outs) + w[x + "D"] * u) * _silu(z)) @ w[x + "o"].T


def _differential(h, w, x, m):
    H, G, dim, T = m["heads"], m["kv_heads"], m["dim"], h.shape[0]
    made = {n: _conv(h @ w[x + n].T + w[x + n + ".b"], w[x + n + ".conv"]) for n in "qkv"}
    rates, size = _rates(m["rot"], h.device)
    q, k = (_turn(_rms(_heads(made[n], 2 * c), w[x + n + ".norm"]), 0, m["rot"]["dims"], rates, size) for n, c in (("q", H), ("k", G)))
    v = _heads(made["v"], G).repeat_interleave(H // G, 0)
    k = k.reshape(G, 2, T, dim).repeat_interleave(H // G, 0)
    q = q.reshape(H, 2, T, dim)
    one, two = (_mix(q[:, i] @ k[:, i].transpose(1, 2) * m["scale"], _seen(T, 0, h.device), v) for i in range(2))
    share = torch.exp((w[x + "lq1"] * w[x + "lk1"]).sum()) - torch.exp((w[x + "lq2"] * w[x + "lk2"]).sum()) + m["diff"]
    return _merged(_rms(one - share * two) * (1.0 - m["diff"])) @ w[x + "o"].T


def _pair(h, w, p, act):
    return (act(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T


def _clamped(h, w, p, limit):
    g, u = (h @ w[p + "gate"].T).clamp(max=limit), (h @ w[p + "up"].T).clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[p + "down"].T


def _experts(h, w, p, mlp, groups):
    """Sigmoid scores and groups of experts (Gokezen), or a softmax among the chosen (Visadra)."""
    count, top = mlp["router"]["experts"], mlp["router"]["top"]
    numbers = h @ w[p + "router"].T
    if groups:
        scores = torch.sigmoid(numbers)
        grouped = scores.reshape(-1, groups["count"], count // groups["count"])
        kept = grouped.topk(2, -1).values.sum(-1).topk(groups["keep"], -1).indices
        allowed = torch.full_like(grouped, float("-inf")).scatter(1, kept[..., None].expand(-1, -1, grouped.shape[2]),
                                                                  grouped.gather(1, kept[..., None].expand(-1, -1, grouped.shape[2])))
        picked, chosen = allowed.reshape(-1, count).topk(top, -1)
        share = picked / (picked.sum(-1, keepdim=True) + 1e-20) * mlp["router"]["scale"]
        one = lambda x, q, c: _clamped(x, w, q, c["limit"])  # noqa: E731
    else:
        picked, chosen = (numbers + w[p + "router.b"]).topk(top, -1)
        share = torch.softmax(picked, -1)
        one = lambda x, q, c: _pair(x, w, q, _silu)  # noqa: E731
    out = one(h, p + "shared.", mlp["shared"])
    for e in range(count):
        at, which = (chosen == e).nonzero(as_tuple=True)
        if len(at):
            out[at] += share[at, which][:, None] * one(h[at], f"{p}e{e}.", mlp["expert"])
    return out


def _layer(x, case, config, i, w, first):
    """The stream behind layer i, rows from `first` on (0 but for designs whose layers keep keys and values only)."""
    layer, p = config["layers"][i], f"l{i}."
    m, mlp, mix, ff = layer["mixer"], layer["mlp"], p + "mix.", p + "mlp."
    if case["design"] == "visadra":
        y = x[first:] + _rms(_latent(x, w, mix, m, first, False), w[p + "norm1"])
        return y + _rms(_experts(y, w, ff, mlp, None), w[p + "norm2"])
    if case["design"] == "gokezen":
        h = _rms(x, w[p + "norm1"])
        return x + (_window_attention(h, w, mix + "left.", m["left"]) + _memory(h, w, mix + "right.", m["right"])
                    + _experts(h, w, ff, mlp, mlp["router"]["groups"]))
    if case["design"] == "rakarax":
        h = _rms(x, 1.0 + w[p + "norm1"])
        y = x + _rms(_talking_attention(h, w, mix + "left.", m["left"]) + _selective_scan(h, w, mix + "right.", m["right"]), 1.0 + w[p + "norm1b"])
        z = _rms(y, 1.0 + w[p + "norm2"]) @ w[ff + "up"].T
        a, b, c, e = w[ff + "act"]
        return y + _rms((a * _rms(z) + b * _rms(z ** 2) + c * _rms(z ** 3) + e) @ w[ff + "down"].T, 1.0 + w[p + "norm2b"])
    if case["design"] == "sovozen":
        h = _layer_norm(x, w[p + "norm1"])
        y = x + (_latent(h, w, mix, m, 0, True) if layer["type"] == "latent_attention" else _lightning(h, w, mix, m))
        return y + _pair(_layer_norm(y, w[p + "norm2"]), w, ff, _gelu)
    h = _rms(x, w[p + "norm1"])
    y = x + (_gla(h, w, mix, m) if layer["type"] == "gla" else _differential(h, w, mix, m))
    return y + _pair(_rms(y, w[p + "norm2"]), w, ff, _silu)


def exact(case, seed):
    config, r = _config(case), _Draw(seed)
    weights = _weights(case, config, r)
    w = {k: v.to(F64) for k, v in weights.items()}
    heads = SIZES[case["size"]][1]
    if case["kind"] == "model":
        logits = []
        for tokens in _tokens(case, r):
            x = w["wte.weight"][tokens] + w["wpe.weight"][:len(tokens)]
            for i in range(config["n_layer"]):
                x = _gpt2_block(x, w, f"h.{i}.", heads, 0)
            logits.append(_layer_norm(x[-1], w["ln_f.weight"], w["ln_f.bias"]) @ w["wte.weight"].T)
        return torch.stack(logits)
    runs = _runs(case)
    streams = []
    for x, (past, new) in zip(torch.split(_rows(case, config, weights, r).to(F64), [a + b for a, b in runs]), runs):
        if case["design"] == "gpt2":
            x = _gpt2_block(x, w, "h.0.", heads, past)
        else:
            for i in range(len(config["layers"])):
                x = _layer(x, case, config, i, w, past)
        streams.append(x)
    # (pages and states lie as the library lays them out, which plain code has no counterpart for)
    return {"stream": torch.cat(streams), "pages": None, "states": None}
