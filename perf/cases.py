"""Performance cases: what programs have this engine do, through its public Python entry points.

Three kinds of pass:

* ``step``: one call of the step function (`Replayer.step`) on a model whose cache already holds some requests.  `decode`
  requests bring their next token on a context of `ctx_lo` to `ctx_hi` tokens, `prompts` requests bring `new_lo` to `new_hi` tokens
  on a past of `past` (0: they are opened by the pass and closed by it).  The logits of every request's last token come to the host.
  After the pass the requests are cut back to where they were, as a program does that rejects drafted tokens.
* ``session``: requests are opened, their prompts computed in one step, `steps` tokens a request are then fed one by one, and the
  requests are closed; the logits of every step come back.  This also serves designs whose state cannot be cut back.
* ``generate``: `Engine.generate_batch` with the default sampling options, and one step that scores what was generated.

The models have the layer sizes of `bench.py` (GPT-2 small, medium and XL; Revudra at GPT-2 small's) and random weights
with the spreads that trained ones have.  A model is loaded once and serves all states, as in a program that keeps it.
"""
from __future__ import annotations

import json
import math
import os
import random
import tempfile

import numpy as np
import torch

from liyab_b200.engine import Engine, EngineConfig, Replayer, StepEntry
from liyab_b200.sampling import SamplingParams
from liyab_b200.weights import write_safetensors

GPT2 = {"gpt2-small": (12, 768, 12, 3072), "gpt2-medium": (24, 1024, 16, 4096), "gpt2-xl": (48, 1600, 25, 6400)}
VOCAB, POSITIONS, STEP_TOKENS = 50257, 1024, 2048
# Live tokens a loaded model has pages for: six states of a case beside one another.
CACHE_TOKENS = {"gpt2-small": 400_000, "gpt2-medium": 400_000, "gpt2-xl": 100_000, "revudra-small": 60_000}


# ---- the cases ---------------------------------------------------------------------------------------------

def _step(model, dtype, decode=0, ctx_lo=0, ctx_hi=0, prompts=0, new_lo=0, new_hi=0, past=0, lengths=1):
    return dict(kind="step", model=model, dtype=dtype, decode=decode, ctx_lo=ctx_lo, ctx_hi=ctx_hi, prompts=prompts, new_lo=new_lo,
                new_hi=new_hi, past=past, lengths=lengths)


def _session(model, dtype, requests, new_lo, new_hi, steps, lengths=1):
    return dict(kind="session", model=model, dtype=dtype, prompts=requests, new_lo=new_lo, new_hi=new_hi, steps=steps, lengths=lengths)


def _generate(model, dtype, requests, new_lo, new_hi, steps, lengths=1):
    return dict(kind="generate", model=model, dtype=dtype, prompts=requests, new_lo=new_lo, new_hi=new_hi, steps=steps, lengths=lengths)


def listed():
    named = {
        # One user's next token: the smallest call, nothing but latency.
        "small_decode_1": _step("gpt2-small", "bfloat16", decode=1, ctx_lo=300, ctx_hi=700),
        # A small server's step: the batch of the headline benchmark, contexts as they come.
        "small_decode_8": _step("gpt2-small", "bfloat16", decode=8, ctx_lo=300, ctx_hi=1000),
        # A busy server's step.
        "medium_decode_64": _step("gpt2-medium", "bfloat16", decode=64, ctx_lo=100, ctx_hi=1000),
        # The largest model at a small server's batch: bound by its weights.
        "xl_decode_8": _step("gpt2-xl", "bfloat16", decode=8, ctx_lo=300, ctx_hi=1000),
        # One short question: the time to a first token.
        "small_prompt_37": _step("gpt2-small", "bfloat16", prompts=1, new_lo=37, new_hi=37),
        # Two full contexts: the benchmark's prefill.
        "small_prefill_2x1024": _step("gpt2-small", "bfloat16", prompts=2, new_lo=1024, new_hi=1024),
        # Prompts of several users in one step of the largest model.
        "xl_prefill_ragged": _step("gpt2-xl", "bfloat16", prompts=5, new_lo=150, new_hi=600),
        # What the scheduler makes of a long prompt beside running requests: a portion of it with their next tokens.
        "xl_mixed": _step("gpt2-xl", "bfloat16", decode=12, ctx_lo=100, ctx_hi=900, prompts=1, new_lo=400, new_hi=600, past=300),
        # The 32-bit engine: a decode step and the prompts of a few requests.
        "small_f32_decode_8": _step("gpt2-small", "float32", decode=8, ctx_lo=300, ctx_hi=1000),
        "small_f32_prefill": _step("gpt2-small", "float32", prompts=3, new_lo=120, new_hi=400),
        # A batch job through the engine: scheduler, sampler and pipeline included, its answers scored afterwards.
        "small_generate_16": _generate("gpt2-small", "bfloat16", requests=16, new_lo=20, new_hi=400, steps=32),
        # A design with window attention, matrix memories, latent rows and routed experts: prompts and the tokens after them.
        "revudra_session_8": _session("revudra-small", "bfloat16", requests=8, new_lo=30, new_hi=300, steps=16),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "mixed", "f32", "f32", "generate", "session"])
    model = rng.choice(["gpt2-small", "gpt2-small", "gpt2-medium", "gpt2-xl"])
    lengths = rng.randrange(1 << 20)
    if kind == "decode":
        lo = rng.randrange(1, 600)
        return _step(model, "bfloat16", decode=_spread(rng, 1, 16 if model == "gpt2-xl" else 64), ctx_lo=lo, ctx_hi=rng.randrange(lo, POSITIONS), lengths=lengths)
    if kind == "prefill":
        n = _spread(rng, 1, 12)
        hi = _spread(rng, 2, min(POSITIONS, (1500 if model == "gpt2-xl" else STEP_TOKENS) // n))
        return _step(model, "bfloat16", prompts=n, new_lo=rng.randrange(1, hi + 1), new_hi=hi, lengths=lengths)
    if kind == "mixed":
        lo, new = rng.randrange(1, 500), _spread(rng, 2, 700)
        return _step(model, "bfloat16", decode=_spread(rng, 1, 16), ctx_lo=lo, ctx_hi=rng.randrange(lo, POSITIONS), prompts=rng.choice([1, 1, 2]),
                     new_lo=max(1, new // 2), new_hi=new, past=rng.choice([0, rng.randrange(0, POSITIONS - new)]), lengths=lengths)
    if kind == "f32":
        if rng.random() < 0.5:
            lo = rng.randrange(1, 600)
            return _step("gpt2-small", "float32", decode=_spread(rng, 1, 24), ctx_lo=lo, ctx_hi=rng.randrange(lo, POSITIONS), lengths=lengths)
        n = rng.randrange(1, 5)
        hi = _spread(rng, 8, 1000 // n)
        return _step("gpt2-small", "float32", prompts=n, new_lo=rng.randrange(1, hi + 1), new_hi=hi, lengths=lengths)
    if kind == "generate":
        lo = rng.randrange(1, 200)
        return _generate("gpt2-small", "bfloat16", requests=_spread(rng, 1, 24), new_lo=lo, new_hi=rng.randrange(lo, 500), steps=rng.randrange(4, 33), lengths=lengths)
    lo = rng.randrange(1, 100)
    return _session("revudra-small", "bfloat16", requests=_spread(rng, 1, 12), new_lo=lo, new_hi=rng.randrange(lo, 200), steps=rng.randrange(2, 17), lengths=lengths)


def _lengths(case):
    """Tokens (held, brought) of every request, those that decode first; they belong to the case and not to the seed."""
    rng = random.Random(case["lengths"])
    out = [(rng.randint(case["ctx_lo"], case["ctx_hi"]), 1) for _ in range(case.get("decode", 0))]
    return out + [(case.get("past", 0), rng.randint(case["new_lo"], case["new_hi"])) for _ in range(case["prompts"])]


def _ids(case, seed):
    """Every request's token ids: the held ones, the brought ones and, in a session, those fed one by one."""
    rng = np.random.default_rng([int(seed), 11])
    more = case["steps"] if case["kind"] == "session" else 0
    return [rng.integers(0, VOCAB, size=held + new + more).tolist() for held, new in _lengths(case)]


# ---- models ------------------------------------------------------------------------------------------------

def _gpt2_config(model):
    L, d, h, ff = GPT2[model]
    return dict(model_type="gpt2", n_layer=L, n_embd=d, n_head=h, n_inner=ff, vocab_size=VOCAB, n_positions=POSITIONS, layer_norm_epsilon=1e-5,
                activation_function="gelu_new", tie_word_embeddings=True)


def _revudra_config():
    L, W, H, FF = GPT2["gpt2-small"]
    attn = dict(heads=H, kv_heads=H // 4, dim=64, vdim=64, scale=0.125, mask=dict(size=512), rot=dict(base=1e6, dims=32), v_mix=True)
    memory = dict(heads=H, dim=64, vdim=64, decay=[1.0 - 2.0 ** (-4 - 5 * h / H) for h in range(H)])
    latent = dict(heads=H, dim=48, rot_dim=16, vdim=64, kv_rank=256, q_rank=W // 2, scale=0.125, rot=dict(base=1e4, dims=16))
    dense = dict(kind="dense", ff=FF)
    moe = dict(kind="moe", expert=dict(ff=FF // 4), router=dict(experts=16, top=2))
    kinds = [("attention", attn, dense), ("lightning", memory, moe), ("lightning", memory, moe), ("latent_attention", latent, moe)]
    blocks = [dict(type=kinds[i % 4][0], mixer=kinds[i % 4][1], mlp=kinds[i % 4][2]) for i in range(L)]
    return dict(architecture="Revudra", vocab=VOCAB, width=W, norm=dict(eps=1e-5), residual_mult=0.7, embedding=dict(scale=1.0), logit_scale=1.0,
                max_positions=POSITIONS, layers=blocks)


def _config(model):
    return _revudra_config() if model == "revudra-small" else _gpt2_config(model)


def _gpt2_weights(config, normal):
    L, d, ff = config["n_layer"], config["n_embd"], config["n_inner"]
    out = {"wte.weight": normal(0, 0.14, VOCAB, d), "wpe.weight": normal(0, 0.1, POSITIONS, d),
           "ln_f.weight": normal(1, 0.1, d), "ln_f.bias": normal(0, 0.02, d)}
    proj = 0.02 / math.sqrt(2.0 * L)
    for i in range(L):
        h = f"h.{i}."
        out.update({h + "ln_1.weight": normal(1, 0.1, d), h + "ln_1.bias": normal(0, 0.02, d), h + "ln_2.weight": normal(1, 0.1, d),
                    h + "ln_2.bias": normal(0, 0.02, d), h + "attn.c_attn.weight": normal(0, 0.02, d, 3 * d), h + "attn.c_attn.bias": normal(0, 0.02, 3 * d),
                    h + "attn.c_proj.weight": normal(0, proj, d, d), h + "attn.c_proj.bias": normal(0, 0.02, d), h + "mlp.c_fc.weight": normal(0, 0.02, d, ff),
                    h + "mlp.c_fc.bias": normal(0, 0.02, ff), h + "mlp.c_proj.weight": normal(0, proj, ff, d), h + "mlp.c_proj.bias": normal(0, 0.02, d)})
    return out


def _revudra_weights(config, normal, table):
    V, W = config["vocab"], config["width"]

    def mat(rows, cols):
        return normal(0, cols ** -0.5, rows, cols)

    out = {"embed": normal(0, 1, V, W), "head": mat(V, W), "final.norm": normal(1, 0.1, W)}
    for i, l in enumerate(config["layers"]):
        p, m, mlp = f"l{i}.", l["mixer"], l["mlp"]
        H, D, E = m["heads"], m["dim"], m["vdim"]
        out[p + "norm1"], out[p + "norm2"] = normal(1, 0.1, W), normal(1, 0.1, W)
        if l["type"] == "attention":
            G = m["kv_heads"]
            out.update({p + "mix.q": mat(H * D, W), p + "mix.k": mat(G * D, W), p + "mix.v": mat(G * E, W), p + "mix.g": mat(H * E, W),
                        p + "mix.q.norm": normal(1, 0.1, H * D), p + "mix.k.norm": normal(1, 0.1, G * D), p + "mix.vmix": normal(0.5, 0.1),
                        p + "mix.sink": normal(0, 1, H)})
        elif l["type"] == "lightning":
            out.update({p + "mix.q": mat(H * D, W), p + "mix.k": mat(H * D, W), p + "mix.v": mat(H * E, W), p + "mix.g": mat(H * E, W),
                        p + "mix.norm": normal(1, 0.1, H * E)})
        else:
            R, C, Q = m["rot_dim"], m["kv_rank"], m["q_rank"]
            out.update({p + "mix.dq": mat(Q, W), p + "mix.dq.norm": normal(1, 0.1, Q), p + "mix.uq": mat(H * (D + R), Q), p + "mix.dkv": mat(C + R, W),
                        p + "mix.dkv.norm": normal(1, 0.1, C), p + "mix.uk": mat(H * D, C), p + "mix.uv": mat(H * E, C), p + "mix.sink": normal(0, 1, H),
                        p + "mix.g": mat(H, W)})
        out[p + "mix.o"] = mat(W, H * E)
        if mlp["kind"] == "dense":
            out.update({p + "mlp.up": mat(mlp["ff"], W), p + "mlp.down": mat(W, mlp["ff"])})
        else:
            F, X = mlp["expert"]["ff"], mlp["router"]["experts"]
            for e in range(X):
                out.update({f"{p}mlp.e{e}.gate": mat(F, W), f"{p}mlp.e{e}.up": mat(F, W), f"{p}mlp.e{e}.down": mat(W, F)})
            out[p + "mlp.table"] = table(V, X, mlp["router"]["top"])
    return out


def _weights(model, dtype):
    """The model's tensors by file name, on the GPU and in the type of the file."""
    g = torch.Generator(device="cuda").manual_seed(1234)
    to = torch.bfloat16 if dtype == "bfloat16" else torch.float32

    def normal(mean, std, *shape):
        return (torch.randn(shape, generator=g, device="cuda") * std + mean).to(to)

    def table(rows, n, top):
        return torch.rand((rows, n), generator=g, device="cuda").argsort(dim=1)[:, :top].to(torch.int32).contiguous()

    config = _config(model)
    return _revudra_weights(config, normal, table) if model == "revudra-small" else _gpt2_weights(config, normal)


class _Loaded:
    """A model on the device: its step function and, where a case generates, its engine."""

    def __init__(self, model, dtype, engine):
        weights = {k: v.cpu() for k, v in _weights(model, dtype).items()}
        bits = {k for k, v in weights.items() if v.dtype == torch.bfloat16}
        arrays = {k: (v.view(torch.int16).numpy().view(np.uint16) if k in bits else v.numpy()) for k, v in weights.items()}
        with tempfile.TemporaryDirectory(prefix="liyab_b200_cases_") as folder:
            with open(os.path.join(folder, "config.json"), "w") as f:
                json.dump(_config(model), f)
            write_safetensors(os.path.join(folder, "model.safetensors"), arrays, tags={k: "BF16" for k in bits})
            self.replayer = Replayer(folder, dtype, max_tokens=CACHE_TOKENS[model], max_requests=400, cuda_graphs=True, max_step_tokens=STEP_TOKENS)
            self.engine = None
            if engine:
                self.engine = Engine(EngineConfig(model=folder, dtype=dtype, max_requests=32, num_pages=32 * POSITIONS // 16))
        self.serial = 0

    def name(self):
        self.serial += 1
        return self.serial


_loaded = {}


def _load(case):
    """The case's model; the one loaded before it goes once nothing uses it any more."""
    key = (case["model"], case["dtype"], case["kind"] == "generate")
    if key not in _loaded:
        _loaded.clear()
        _loaded[key] = _Loaded(*key)
    return _loaded[key]


# ---- states and passes ---------------------------------------------------------------------------------------

class _State:
    def __init__(self, case, seed):
        self.case, self.loaded, self.held, self.fresh = case, _load(case), {}, []
        self.lengths, self.ids = _lengths(case), _ids(case, seed)
        if case["kind"] != "step":
            return
        cache = self.loaded.replayer.cache
        self.entries, todo = [], []
        for (held, new), ids in zip(self.lengths, self.ids):
            name = self.loaded.name()
            if held:
                cache.open(name)
                self.held[name] = held
                todo += [(name, ids[at:min(at + STEP_TOKENS, held)]) for at in range(0, held, STEP_TOKENS)]
            else:
                self.fresh.append(name)
            self.entries.append(StepEntry(name, ids[held:], [new - 1]))
        while todo:                                      # the contexts, as many requests a step as its tokens allow
            part, room = [], STEP_TOKENS
            while todo and len(todo[0][1]) <= room:
                part.append(todo.pop(0))
                room -= len(part[-1][1])
            self.loaded.replayer.step([StepEntry(name, ids) for name, ids in part], fetch=False)

    def __del__(self):
        for name in getattr(self, "held", {}):
            self.loaded.replayer.cache.close(name)


def prepare(case, seed):
    return _State(case, seed)


def _run_step(s):
    replayer, cache = s.loaded.replayer, s.loaded.replayer.cache
    for name in s.fresh:
        cache.open(name)
    out = replayer.step(s.entries)
    for name in s.fresh:
        cache.close(name)
    for name, length in s.held.items():
        cache.truncate(name, length)
    return out.logits


def _run_session(s):
    replayer, cache = s.loaded.replayer, s.loaded.replayer.cache
    names = [s.loaded.name() for _ in s.ids]
    for name in names:
        cache.open(name)
    steps = [replayer.step([StepEntry(n, ids[:new], [new - 1]) for n, ids, (_, new) in zip(names, s.ids, s.lengths)])]
    for i in range(s.case["steps"]):
        steps.append(replayer.step([StepEntry(n, ids[new + i:new + i + 1], [0]) for n, ids, (_, new) in zip(names, s.ids, s.lengths)]))
    for name in names:
        cache.close(name)
    return [out.logits for out in steps]


def _run_generate(s):
    replayer, cache = s.loaded.replayer, s.loaded.replayer.cache
    results = s.loaded.engine.generate_batch(s.ids, SamplingParams(seed=7, max_tokens=s.case["steps"], ignore_eos=True))
    whole = [ids + r.tokens for ids, r in zip(s.ids, results)]
    scores, at = [], 0
    while at < len(whole):                               # the answers scored in as few steps as the tokens of a step allow
        n, room = 0, STEP_TOKENS
        while at + n < len(whole) and len(whole[at + n]) <= room:
            room -= len(whole[at + n])
            n += 1
        names = [s.loaded.name() for _ in range(n)]
        for name in names:
            cache.open(name)
        scores.append(replayer.step([StepEntry(name, ids, [len(ids) - 1]) for name, ids in zip(names, whole[at:at + n])]).logits)
        for name in names:
            cache.close(name)
        at += n
    return {"tokens": [np.asarray(r.tokens, dtype=np.int32) for r in results], "scores": scores}


def run(state):
    return {"step": _run_step, "session": _run_session, "generate": _run_generate}[state.case["kind"]](state)


# ---- work --------------------------------------------------------------------------------------------------

def _gpt2_work(case, lengths, rows):
    L, d, _, ff = GPT2[case["model"]]
    size = 2 if case["dtype"] == "bfloat16" else 4
    mats, tokens = L * (4 * d * d + 2 * d * ff), sum(new for _, new in lengths)
    read = sum(held for held, new in lengths) * 2 * L * d
    pairs = sum(held * new + new * (new + 1) // 2 for held, new in lengths)
    return {"bytes": size * (mats + VOCAB * d + read + tokens * (2 * L * d + 2 * d)) + 4 * rows * VOCAB,
            "flops": 2 * tokens * mats + 4 * L * d * pairs + 2 * rows * VOCAB * d}


def _revudra_work(lengths, rows):
    c = _revudra_config()
    W, n, tokens = c["width"], len(lengths), sum(new for _, new in lengths)
    size, flops, read = VOCAB * W, 2 * rows * VOCAB * W, 0
    for l in c["layers"]:
        m, mlp = l["mixer"], l["mlp"]
        H, D, E = m["heads"], m["dim"], m["vdim"]
        if l["type"] == "attention":
            G, w = m["kv_heads"], m["mask"]["size"]
            mats = W * (H * D + G * (D + E) + 2 * H * E)
            seen = sum(min(i + 1, w) for held, new in lengths for i in range(held, held + new))
            flops += 2 * H * (D + E) * seen
            read += 2 * sum(min(held, w) + new for held, new in lengths) * G * (D + E)
        elif l["type"] == "lightning":
            mats = W * H * (2 * D + 3 * E)
            flops += 4 * tokens * H * D * E
            read += 2 * 4 * n * H * D * E
        else:
            R, C, Q = m["rot_dim"], m["kv_rank"], m["q_rank"]
            mats = W * (Q + C + R + H + H * E) + Q * H * (D + R) + H * C * (D + E)
            flops += 2 * H * (D + R + E) * sum(held * new + new * (new + 1) // 2 for held, new in lengths)
            read += 2 * sum(held + new for held, new in lengths) * (C + R)
        if mlp["kind"] == "dense":
            used = touched = 2 * W * mlp["ff"]
        else:
            X, top, F = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"]
            used, touched = 3 * W * top * F, 3 * W * F * X * (1.0 - (1.0 - top / X) ** tokens)
        size += mats + touched
        flops += 2 * tokens * (mats + used)
    return {"bytes": 2 * size + read + 2 * tokens * W + 4 * rows * VOCAB, "flops": flops}


def work(case):
    def of(lengths):
        return _revudra_work(lengths, len(lengths)) if case["model"] == "revudra-small" else _gpt2_work(case, lengths, len(lengths))

    lengths = _lengths(case)
    parts = [of(lengths)]
    if case["kind"] == "session":
        parts += [of([(new + i, 1) for _, new in lengths]) for i in range(case["steps"])]
    elif case["kind"] == "generate":
        # The first token comes from the prompts' step, every later one from a step of its own; then the answers are scored.
        parts += [of([(new + i, 1) for _, new in lengths]) for i in range(case["steps"] - 1)]
        parts.append(of([(0, new + case["steps"]) for _, new in lengths]))
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


def tolerance(case):
    # Against 64 bits a float32 model's logits are off by 3.5e-7, a bfloat16 one's by 3e-3 (GPT-2) and 5.5e-3 (Revudra); two correct
    # implementations differ by up to sqrt(2) of that, and four times as much is allowed.
    if case["dtype"] == "float32":
        return {"rel": 2e-6}
    return {"rel": 3e-2} if case["model"] == "revudra-small" else {"rel": 2e-2}


# ---- the same in 64 bits -----------------------------------------------------------------------------------

def _layernorm(x, w, b, eps):
    dev = x - x.mean(-1, keepdim=True)
    return dev / torch.sqrt((dev * dev).mean(-1, keepdim=True) + eps) * w + b


def _gpt2_exact(config, W, tokens, rows):
    """Logits of the places `rows` of one sequence."""
    d, H, eps = config["n_embd"], config["n_head"], config["layer_norm_epsilon"]
    n = len(tokens)
    x = W["wte.weight"][tokens] + W["wpe.weight"][:n]
    hidden = torch.ones(n, n, dtype=torch.bool, device=x.device).triu(1)
    for i in range(config["n_layer"]):
        h = f"h.{i}."
        y = _layernorm(x, W[h + "ln_1.weight"], W[h + "ln_1.bias"], eps) @ W[h + "attn.c_attn.weight"] + W[h + "attn.c_attn.bias"]
        q, k, v = (t.reshape(n, H, d // H).transpose(0, 1) for t in y.split(d, dim=1))
        p = (q @ k.transpose(1, 2) / math.sqrt(d // H)).masked_fill(hidden, -math.inf).softmax(-1)
        x = x + (p @ v).transpose(0, 1).reshape(n, d) @ W[h + "attn.c_proj.weight"] + W[h + "attn.c_proj.bias"]
        y = _layernorm(x, W[h + "ln_2.weight"], W[h + "ln_2.bias"], eps) @ W[h + "mlp.c_fc.weight"] + W[h + "mlp.c_fc.bias"]
        y = 0.5 * y * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (y + 0.044715 * y ** 3)))
        x = x + y @ W[h + "mlp.c_proj.weight"] + W[h + "mlp.c_proj.bias"]
    return _layernorm(x[rows], W["ln_f.weight"], W["ln_f.bias"], eps) @ W["wte.weight"].T


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rotate(v, rot, interleaved):
    """The first rot.dims values of v [n, heads, size] by position."""
    dims = rot["dims"]
    half = dims // 2
    f = rot["base"] ** (-2.0 * torch.arange(half, dtype=v.dtype, device=v.device) / dims)
    ang = torch.arange(v.shape[0], dtype=v.dtype, device=v.device)[:, None] * f
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    first, second = (slice(0, dims, 2), slice(1, dims, 2)) if interleaved else (slice(0, half), slice(half, dims))
    a, b, out = v[..., first], v[..., second], v.clone()
    out[..., first], out[..., second] = a * c - b * s, b * c + a * s
    return out


def _attend(q, k, v, scores_more, scale, sink, window):
    """Softmax attention of [heads, n, size] with a sink a head in the divisor."""
    n = q.shape[1]
    at = torch.arange(n, device=q.device)
    s = (q @ k.transpose(1, 2) + scores_more) * scale
    s = s.masked_fill((at[None] > at[:, None]) | (at[None] <= at[:, None] - window), -math.inf)
    return torch.cat([s, sink[:, None, None].expand(-1, n, 1)], dim=2).softmax(-1)[..., :-1] @ v


def _revudra_exact(config, W, tokens, rows):
    eps, mult = config["norm"]["eps"], config["residual_mult"]
    n = len(tokens)
    x = W["embed"][tokens] * config["embedding"]["scale"]
    first_values = None
    for i, l in enumerate(config["layers"]):
        p, m, mlp = f"l{i}.", l["mixer"], l["mlp"]
        H, D, E = m["heads"], m["dim"], m["vdim"]

        def heads(name, count, size):
            return (x @ W[p + "mix." + name].T).reshape(n, count, size)

        if l["type"] == "attention":
            G = m["kv_heads"]
            q = _rotate(_rms(x @ W[p + "mix.q"].T, W[p + "mix.q.norm"], eps).reshape(n, H, D), m["rot"], False)
            k = _rotate(_rms(x @ W[p + "mix.k"].T, W[p + "mix.k.norm"], eps).reshape(n, G, D), m["rot"], False)
            v = heads("v", G, E)
            if first_values is None:
                first_values = v
            else:
                v = (1.0 - W[p + "mix.vmix"]) * v + W[p + "mix.vmix"] * first_values
            k, v = (t.repeat_interleave(H // G, dim=1).transpose(0, 1) for t in (k, v))
            y = _attend(q.transpose(0, 1), k, v, 0.0, m["scale"], W[p + "mix.sink"], m["mask"]["size"])
            y = y.transpose(0, 1).reshape(n, H * E) * torch.sigmoid(x @ W[p + "mix.g"].T)
        elif l["type"] == "lightning":
            q, k, v = (torch.nn.functional.silu(heads(t, H, s)).transpose(0, 1) for t, s in (("q", D), ("k", D), ("v", E)))
            age = torch.arange(n, device=x.device)[:, None] - torch.arange(n, device=x.device)[None]
            decay = torch.tensor(m["decay"], dtype=x.dtype, device=x.device)[:, None, None] ** age.clamp(min=0) * (age >= 0)
            y = ((q @ k.transpose(1, 2) * decay) @ v).transpose(0, 1).reshape(n, H * E)
            y = _rms(y, W[p + "mix.norm"], eps) * torch.sigmoid(x @ W[p + "mix.g"].T)
        else:
            R, C = m["rot_dim"], m["kv_rank"]
            q = (_rms(x @ W[p + "mix.dq"].T, W[p + "mix.dq.norm"], eps) @ W[p + "mix.uq"].T).reshape(n, H, D + R)
            down = x @ W[p + "mix.dkv"].T
            c, shared = _rms(down[:, :C], W[p + "mix.dkv.norm"], eps), _rotate(down[:, None, C:], m["rot"], True)[:, 0]
            k, v = ((c @ W[p + t].T).reshape(n, H, s).transpose(0, 1) for t, s in (("mix.uk", D), ("mix.uv", E)))
            turned = _rotate(q[..., D:], m["rot"], True).transpose(0, 1)
            y = _attend(q[..., :D].transpose(0, 1), k, v, turned @ shared.T, m["scale"], W[p + "mix.sink"], n)
            y = (y.transpose(0, 1) * torch.sigmoid(x @ W[p + "mix.g"].T)[:, :, None]).reshape(n, H * E)
        x = x + mult * _rms(y @ W[p + "mix.o"].T, W[p + "norm1"], eps)
        if mlp["kind"] == "dense":
            y = torch.relu(x @ W[p + "mlp.up"].T) ** 2 @ W[p + "mlp.down"].T
        else:
            y, chosen = torch.zeros_like(x), W[p + "mlp.table"][tokens]
            for e in range(mlp["router"]["experts"]):
                at = (chosen == e).any(dim=1).nonzero()[:, 0]
                h = x[at]
                h = torch.nn.functional.silu(h @ W[f"{p}mlp.e{e}.gate"].T) * (h @ W[f"{p}mlp.e{e}.up"].T)
                y[at] += h @ W[f"{p}mlp.e{e}.down"].T / mlp["router"]["top"]
        x = x + mult * _rms(y, W[p + "norm2"], eps)
    return _rms(x[rows], W["final.norm"], eps) @ W["head"].T * config["logit_scale"]


def exact(case, seed):
    """The logits in 64 bits.  Generated tokens depend on random draws, so a generating case has no such values."""
    if case["kind"] == "generate":
        return None
    config = _config(case["model"])
    W = {k: (v.double() if v.is_floating_point() else v) for k, v in _weights(case["model"], case["dtype"]).items()}
    of = _revudra_exact if case["model"] == "revudra-small" else _gpt2_exact
    steps = case["steps"] if case["kind"] == "session" else 0
    wanted = []
    for ids, (held, new) in zip(_ids(case, seed), _lengths(case)):
        rows = list(range(held + new - 1, held + new + steps))
        wanted.append(of(config, W, torch.tensor(ids, device="cuda"), rows))
    if case["kind"] == "session":
        return [torch.stack([w[i] for w in wanted]) for i in range(steps + 1)]
    return torch.cat(wanted)
