"""The work whose speed is watched: cases, their inputs, one pass of each through the public entry points, and the same results
in 64 bits.

Two kinds are whole steps of an engine (decoded tokens of a batch, logits out); the others are single blocks and parts as a
program that assembles a model calls them.  Sizes are those of the configurations that ``bench.py`` and the tests run: the
Llama-2-7B, Falcon-7B and Gemma-2B layer sizes with one kv head, and layers of the other designs at widths of 1,024 to 4,096.
"""
from __future__ import annotations

import math
from dataclasses import replace

import torch

from tiny_transformer_inference_engine_b200 import (CacheConfig, Engine, EngineConfig, ModelConfig, SamplingParams,
                                                    SchedulerConfig, StepEntry)
from tiny_transformer_inference_engine_b200.models.model import Model
from tiny_transformer_inference_engine_b200.ops import get_ops
from tiny_transformer_inference_engine_b200.parts.base import (FixedStateView, PagedKVView, PartSpec, ResidualStream, SeqClass,
                                                                StepContext)
from tiny_transformer_inference_engine_b200.registry import build_part, model_spec
from tiny_transformer_inference_engine_b200.sampling import Sampler
from tiny_transformer_inference_engine_b200.weights import place

DEV = "cuda:0"
PAGE = 64
F64 = torch.float64
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

# width, heads, head size, feed-forward width, vocabulary, longest context, eps (one kv head each)
GPT = {
    "llama7b": (4096, 32, 128, 11008, 32000, 4096, 1e-5),
    "falcon7b": (4544, 71, 64, 18176, 65024, 2048, 1e-5),
    "gemma2b": (2048, 8, 256, 16384, 256000, 8192, 1e-6),
    "gpt2048": (2048, 16, 128, 8192, 32000, 4096, 1e-6),       # what bench.py sets the other designs beside
}


def listed():
    return [
        # one user's next token: the smallest step there is, launches and latency
        {"name": "decode_b1", "kind": "decode", "model": "llama7b", "layers": 2, "batch": 1, "ctx": 600},
        # the benchmark's decode step: eight users behind 4,096 tokens
        {"name": "decode_b8_4096", "kind": "decode", "model": "llama7b", "layers": 4, "batch": 8, "ctx": 4096},
        # a 2,048-token prompt through one layer: norms, attention, feed-forward
        {"name": "block_prompt_2048", "kind": "block", "model": "llama7b", "dtype": "bfloat16", "tokens": 2048},
        # a step of the chunked workload at head size 256: 15 users decode beside a portion of a long prompt
        {"name": "attention_mixed_512", "kind": "mixed", "model": "gemma2b", "decoding": 15, "ctx": 6200, "portion": 512, "behind": 5632},
        # the 32-bit path
        {"name": "block_f32_300", "kind": "block", "model": "gpt2048", "dtype": "float32", "tokens": 300},
        # top-k and top-p sampling of a decode step's rows
        {"name": "sample_b8", "kind": "sample", "rows": 8, "vocab": 32000, "top_k": 32, "top_p": 0.9, "temperature": 0.8},
        # experts of a decode step (captured, as a decode step is) and of a prompt
        {"name": "experts_decode_8", "kind": "experts", "width": 2048, "tokens": 8},
        {"name": "experts_prompt_2048", "kind": "experts", "width": 2048, "tokens": 2048},
        # prompts through the recurrent mixers, which five of the designs have in every fourth layer or more
        {"name": "retention_prompt_2048", "kind": "retention", "width": 2048, "tokens": 2048, "requests": 1},
        {"name": "mlstm_prompt_2048", "kind": "mlstm", "width": 2048, "tokens": 2048, "requests": 1},
        {"name": "wkv_prompt_2048", "kind": "wkv", "width": 2048, "tokens": 2048, "requests": 1},
        {"name": "selective_prompt_2048", "kind": "selective", "width": 2048, "tokens": 2048, "requests": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "block", "block_f32", "mixed", "sample", "experts", "retention", "mlstm", "wkv", "selective"])
    if kind == "decode":
        model = rng.choice(["llama7b", "falcon7b", "gemma2b"])
        return {"kind": kind, "model": model, "layers": 2, "batch": _log(rng, 1, 64), "ctx": _log(rng, 64, GPT[model][5] // 2)}
    if kind == "block":
        model = rng.choice(["llama7b", "gemma2b", "gpt2048"])
        return {"kind": kind, "model": model, "dtype": "bfloat16", "tokens": _log(rng, 100, 2048)}
    if kind == "block_f32":
        return {"kind": "block", "model": "gpt2048", "dtype": "float32", "tokens": _log(rng, 20, 320)}
    if kind == "mixed":
        model = rng.choice(["llama7b", "gemma2b"])
        return {"kind": kind, "model": model, "decoding": rng.randint(1, 31), "ctx": _log(rng, 128, 3500),
                "portion": _log(rng, 128, 512), "behind": rng.randint(0, 3500)}
    if kind == "sample":
        top_k, top_p = rng.choice([(0, 1.0), (32, 1.0), (0, 0.9), (32, 0.9), (200, 0.95)])
        return {"kind": kind, "rows": _log(rng, 1, 64), "vocab": rng.choice([32000, 65024, 256000]), "top_k": top_k, "top_p": top_p,
                "temperature": round(rng.uniform(0.5, 1.2), 3)}
    if kind == "experts":
        return {"kind": kind, "width": rng.choice([1024, 2048]), "tokens": _log(rng, 1, 64) if rng.random() < 0.4 else _log(rng, 128, 2048)}
    return {"kind": kind, "width": rng.choice([1024, 2048]), "tokens": _log(rng, 128, 2048), "requests": rng.randint(1, 3)}


# --------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=g, device=DEV) * std).to(dtype)


def _lens(tokens, requests):
    """The tokens of a step split over its requests, unevenly."""
    n = min(requests, tokens)
    cut = [tokens * (i + 1) * (i + 2) // (n * (n + 1)) for i in range(n)]
    return [b - a for a, b in zip([0] + cut, cut)]


def _gpt_config(c, layers):
    d, H, D, F, V, L, eps = GPT[c["model"]]
    return ModelConfig.from_dict(dict(architecture="mqa_gpt", vocab_size=V, d_model=d, num_layers=layers, num_heads=H, num_kv_heads=1,
                                      hidden_size=F, max_seq_len=L, rope_theta=10000.0, rms_norm_eps=eps, bias=False, eos_token_id=None))


def _gpt_tensors(c, layers, g, dtype):
    """Random weights under the checkpoint's tensor names; norm weights about 1, in 32 bits."""
    d, H, D, F, V, _, _ = GPT[c["model"]]
    w = {"embedding.embedding.weight": _randn(g, V, d, std=0.5, dtype=dtype), "final_norm.weight": 1 + _randn(g, d, std=0.1),
         "lm_head.weight": _randn(g, V, d, std=0.02, dtype=dtype)}
    for i in range(layers):
        p = f"layers.{i}."
        for name, rows, cols in (("attn.q_proj", H * D, d), ("attn.k_proj", D, d), ("attn.v_proj", D, d), ("attn.out", d, H * D),
                                 ("mlp.gate_proj", F, d), ("mlp.up_proj", F, d), ("mlp.down_proj", d, F)):
            w[f"{p}{name}.weight"] = _randn(g, rows, cols, std=0.02, dtype=dtype)
        for name in ("attn_norm", "mlp_norm"):
            w[f"{p}{name}.weight"] = 1 + _randn(g, d, std=0.1)
    return w


def _cache_rows(c, layers, g, dtype):
    """Keys and values of the tokens that came before: [layers, 2, batch, ctx - 1, D]."""
    D = GPT[c["model"]][2]
    return _randn(g, layers, 2, c["batch"], c["ctx"] - 1, D, dtype=dtype)


def _tokens(g, n, vocab):
    return torch.randint(0, vocab, (n,), generator=g, device=DEV, dtype=torch.int32)


def _context(ops, dtype, seqs, table, token_ids, slots=None, classes=None):
    """What one step of requests (tokens before, new tokens) brings, as parts read it."""
    t = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    qsl = [0]
    for _, n in seqs:
        qsl.append(qsl[-1] + n)
    pos = [s + i for s, n in seqs for i in range(n)]
    return StepContext(ops=ops, dtype=dtype, device=torch.device(DEV), num_tokens=len(pos), num_seqs=len(seqs),
                       max_q_len=max(n for _, n in seqs), max_kv_len=max(s + n for s, n in seqs), token_ids=token_ids,
                       positions=t(pos), token_seq=t([i for i, (_, n) in enumerate(seqs) for _ in range(n)]),
                       query_start_loc=t(qsl), seq_lens=t([s + n for s, n in seqs]), slot_ids=t(list(range(len(seqs)))),
                       logit_rows=t(list(range(len(pos)))), num_logit_rows=len(pos), block_tables={0: table}, seq_classes=classes)


def _paged(seqs, D, dtype, g=None):
    """Pages for requests (tokens before, new tokens), in mixed order; ``g``: filled with keys and values."""
    pages = [-(-(s + n) // PAGE) for s, n in seqs]
    total, width = sum(pages), max(pages)
    order = [(7919 * i) % total for i in range(total)] if total % 7919 else list(range(total))
    table, at = torch.zeros(len(seqs), width, dtype=torch.int32), 0
    for i, n in enumerate(pages):
        table[i, :n] = torch.tensor([order[at + j] + 1 for j in range(n)], dtype=torch.int32)
        at += n
    shape = (2, total + 1, 1, PAGE, D)
    kv = torch.zeros(shape, dtype=dtype, device=DEV) if g is None else _randn(g, *shape, dtype=dtype)
    return kv, table.to(DEV)


def _part(category, kind, args, dtype):
    ops = get_ops(DEV)
    part = build_part(category, PartSpec(kind, "p", args))
    part.validate(ops, dtype, PAGE)
    part.bind(ops, dtype, torch.device(DEV))
    return part, ops


def _model(c, dtype, tensors):
    ops = get_ops(DEV)
    model = Model(model_spec(_gpt_config(c, 1)))
    model.bind(ops, dtype, DEV)
    model.load(place(tensors, model.param_specs(), dtype, torch.device(DEV)))
    return model, ops


def _x(c, g, dtype):
    return _randn(g, c["tokens"], c["width"], dtype=dtype)     # what a norm hands to a sub-layer


RETENTION_ROT = {"dim": 128, "base": 10000.0, "style": "half"}


def _decays(heads):
    return [1.0 - 2.0 ** (-5 - 3 * i / max(1, heads - 1)) for i in range(heads)]


def _mixer_parts(c, g, dtype):
    """(kind, constants, tensors by relative name, state rows of one request by need, in order)."""
    d, k = c["width"], c["kind"]
    H = d // 128
    m = lambda *s: _randn(g, *s, std=0.02, dtype=dtype)
    if k == "retention":
        args = {"d_model": d, "num_heads": H, "dim": 128, "vdim": 128, "decay": tuple(_decays(H)), "eps": 1e-6,
                "position": PartSpec("rope", "", RETENTION_ROT)}
        w = {n: m(H * 128, d) for n in ("q", "k", "v", "g")}
        w["o"] = m(d, H * 128)
        states = [_randn(g, c["requests"], H, 128, 128, std=0.5)]
    elif k == "mlstm":
        args = {"d_model": d, "num_heads": H, "dim": 64, "vdim": 128, "gate_cap": 15.0, "eps": 1e-6}
        w = {"q": m(H * 64, d), "k": m(H * 64, d), "v": m(H * 128, d), "g": m(H * 128, d), "i": m(H, d), "f": m(H, d),
             "i.b": _randn(g, H), "f.b": torch.linspace(1.0, 6.0, H, device=DEV), "norm": 1 + _randn(g, H * 128, std=0.1), "o": m(d, H * 128)}
        states = [_randn(g, c["requests"], H, 128, 64, std=0.5), _randn(g, c["requests"], H, 64), _randn(g, c["requests"], H)]
    elif k == "wkv":
        H = d // 64
        args = {"d_model": d, "num_heads": H, "dim": 64, "eps": 1e-6, "decay_rank": 64}
        w = {n: m(d, d) for n in ("r", "k", "v", "g", "o")}
        w.update({f"mu.{n}": _randn(g, d, std=0.3) for n in ("r", "k", "v", "g", "w")})
        w.update({"w1": m(64, d), "w2": m(d, 64), "w0": torch.rand(d, generator=g, device=DEV) * 6.5 - 6.0,
                  "u": _randn(g, H, 64, std=0.5), "norm": 1 + _randn(g, d, std=0.1)})
        states = [_randn(g, c["requests"], H, 64, 64, std=0.5), _randn(g, c["requests"], d)]
    else:
        I, N, R = 2 * d, 16, d // 16
        args = {"d_model": d, "inner": I, "state": N, "dt_rank": R, "taps": 4}
        w = {"in": m(2 * I, d), "conv": _randn(g, I, 4, std=0.3), "conv.b": _randn(g, I, std=0.1), "x": m(R + 2 * N, I), "dt": m(I, R),
             "dt.b": torch.rand(I, generator=g, device=DEV) * 4.6 - 6.9,          # softplus of it: steps of 0.001 to 0.1
             "A_log": torch.log(torch.arange(1, N + 1, device=DEV, dtype=torch.float32)).expand(I, N).contiguous(),
             "D": torch.ones(I, device=DEV), "o": m(d, I)}
        states = [_randn(g, c["requests"], I, N, std=0.5), _randn(g, c["requests"], 3, I)]
    return ("selective_scan" if k == "selective" else k), args, w, states


def _expert_parts(c, g, dtype):
    d, E = c["width"], 16
    F = d // 2
    args = {"d_model": d, "hidden": F, "experts": E, "identity": 2, "top": 4, "groups": 1, "keep": 1, "group_top": 1, "scale": 1.0,
            "renorm": False, "score": "softmax", "correction": True, "alpha": 1.702, "limit": 7.0, "shift": 1.0}
    w = {"router": _randn(g, E + 2, d, std=0.02, dtype=dtype), "correction": _randn(g, E + 2, std=0.01)}
    for e in range(E):
        w[f"e{e}.gate"], w[f"e{e}.up"] = _randn(g, F, d, std=0.02, dtype=dtype), _randn(g, F, d, std=0.02, dtype=dtype)
        w[f"e{e}.down"] = _randn(g, d, F, std=0.02, dtype=dtype)
    return args, w


def _mixed_step(c):
    seqs = [(c["ctx"] - 1 - 37 * i % 100, 1) for i in range(c["decoding"])] + [(c["behind"], c["portion"])]
    return seqs


def _mixed_tensors(c, g, dtype):
    d, H, D = GPT[c["model"]][:3]
    return {f"{n}.weight": _randn(g, r, k, std=0.02, dtype=dtype)
            for n, r, k in (("q_proj", H * D, d), ("k_proj", D, d), ("v_proj", D, d), ("out", d, H * D))}


# --------------------------------------------------------------------------- what a program has before the call
def prepare(case, seed):
    c, g = case, _gen(seed)
    kind = c["kind"]
    if kind == "decode":
        dtype = torch.bfloat16
        w = _gpt_tensors(c, c["layers"], g, dtype)
        rows, V, B, n = _cache_rows(c, c["layers"], g, dtype), GPT[c["model"]][4], c["batch"], c["ctx"]
        ids = _tokens(g, B, V).tolist()
        pages = B * (-(-n // PAGE) + 2) + 2
        eng = Engine(_gpt_config(c, c["layers"]), w, EngineConfig(
            dtype="bfloat16", device=DEV, cache=CacheConfig(block_size=PAGE, num_gpu_blocks=pages),
            sched=SchedulerConfig(max_num_seqs=B, max_num_batched_tokens=2048, cudagraph_batch_sizes=[B])))
        kv = eng.manager.groups[0].kv                          # [layers, 2, pages, 1, page, D]
        for i in range(B):
            eng.manager.admit(i)
            eng.manager.extend(i, 0, n)
            table = torch.tensor(eng.manager.table(0, i), device=DEV)
            for s in range(0, n - 1, PAGE):
                kv[:, :, table[s // PAGE], 0, :min(PAGE, n - 1 - s)] = rows[:, :, i, s:min(s + PAGE, n - 1)]
        return {"engine": eng, "entries": [StepEntry(i, n - 1, [ids[i]], [0]) for i in range(B)]}
    if kind == "block":
        dtype, T = DTYPES[c["dtype"]], c["tokens"]
        model, ops = _model(c, dtype, _gpt_tensors(c, 1, g, dtype))
        kv, table = _paged([(0, T)], GPT[c["model"]][2], dtype)
        ctx = _context(ops, dtype, [(0, T)], table, _tokens(g, T, GPT[c["model"]][4]))
        return {"model": model, "ctx": ctx, "view": PagedKVView(kv[0], kv[1], table, PAGE), "kv": kv}
    if kind == "mixed":
        dtype = torch.bfloat16
        d, H, D = GPT[c["model"]][:3]
        part, ops = _part("mixer", "attention", {"d_model": d, "num_heads": H, "num_kv_heads": 1, "head_dim": D,
                                                 "position": PartSpec("rope", "", {"dim": D, "base": 10000.0, "style": "interleaved"})}, dtype)
        part.load(_mixed_tensors(c, g, dtype))
        seqs, n = _mixed_step(c), c["decoding"]
        kv, table = _paged(seqs, D, dtype, g)
        t = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        classes = [SeqClass(0, n, 0, n, 1, max(s + 1 for s, _ in seqs[:n]), t(list(range(n + 1)))),
                   SeqClass(n, n + 1, n, n + c["portion"], c["portion"], c["behind"] + c["portion"], t([0, c["portion"]]))]
        x = _randn(g, n + c["portion"], d, dtype=dtype)
        return {"part": part, "ctx": _context(ops, dtype, seqs, table, None, classes=classes), "x": x,
                "view": PagedKVView(kv[0], kv[1], table, PAGE)}
    if kind == "sample":
        sampler = Sampler(get_ops(DEV), c["rows"], c["vocab"], DEV)
        for i in range(c["rows"]):
            sampler.set_request(i, SamplingParams(temperature=c["temperature"], top_k=c["top_k"], top_p=c["top_p"], seed=1000 * seed + i))
        return {"sampler": sampler, "logits": _randn(g, c["rows"], c["vocab"], std=2.5),
                "slots": torch.arange(c["rows"], dtype=torch.int32, device=DEV)}
    dtype = torch.bfloat16
    if kind == "experts":
        args, w = _expert_parts(c, g, dtype)
        part, ops = _part("ffn", "grouped_moe", args, dtype)
        part.load(w)
        T = c["tokens"]
        ctx = _context(ops, dtype, [(0, 1)] * T if T <= 64 else [(0, T)], None, None)
        state = {"part": part, "ctx": ctx, "x": _x(c, g, dtype)}
        if T <= 64:                                            # decode steps run from a captured graph
            _run_part(state)
            torch.cuda.synchronize()
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state["graph"]):
                state["out"] = _run_part(state)
        return state
    kind, args, w, rows = _mixer_parts(c, g, dtype)
    part, ops = _part("mixer", kind, args, dtype)
    part.load(w)
    views = []
    for need, r in zip(part.cache_needs(), rows):              # rows of requests, and the row that padding uses
        s = torch.zeros((r.shape[0] + 1, *need.shape), dtype=torch.float32, device=DEV)
        s[tuple([slice(0, r.shape[0])] + [slice(0, n) for n in r.shape[1:]])] = r
        views.append(FixedStateView(s))
    lens = _lens(c["tokens"], c["requests"])
    return {"part": part, "ctx": _context(ops, dtype, [(64, n) for n in lens], None, None), "x": _x(c, g, dtype),
            "view": views, "states": [v.state for v in views]}


def _run_part(s):
    ctx = replace(s["ctx"], step_cache={})                     # what parts compute once per step is computed in every pass
    if "view" in s:
        return s["part"].forward(s["x"], ctx, s["view"])
    return s["part"].forward(s["x"], ctx)


@torch.no_grad()
def run(state):
    if "engine" in state:
        return state["engine"].stepper.step(state["entries"])
    if "sampler" in state:
        return {"tokens": state["sampler"].sample(state["logits"], state["slots"]), "state": state["sampler"].state}
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    if "model" in state:
        model, ctx = state["model"], replace(state["ctx"], step_cache={})
        stream = ResidualStream(model.embedding.forward(ctx))
        model.blocks[0].forward(stream, ctx, [state["view"]])
        out = model.final_norm.norm_rows(stream.resid, stream.delta, ctx.logit_rows, ctx.num_logit_rows)
        return {"out": out, "keys_and_values": state["kv"][:, 1:]}
    out = _run_part(state)
    return {"out": out, "states": state["states"]} if "states" in state else out


# --------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    c, kind = case, case["kind"]
    if kind in ("decode", "block", "mixed"):
        d, H, D, F, V, _, _ = GPT[c["model"]]
        att = d * (2 * H * D + 2 * D)
        if kind == "decode":
            L, B, n = c["layers"], c["batch"], c["ctx"]
            params = L * (att + 3 * d * F) + V * d
            return {"bytes": 2 * params + L * B * n * 4 * D + 4 * B * V, "flops": 2 * B * params + L * B * n * 4 * H * D}
        if kind == "block":
            T, es = c["tokens"], 2 if c["dtype"] == "bfloat16" else 4
            return {"bytes": es * (att + 3 * d * F + 2 * T * d + 2 * T * D), "flops": 2 * T * (att + 3 * d * F) + 2 * H * D * T * (T + 1)}
        seqs = _mixed_step(c)
        T = sum(n for _, n in seqs)
        return {"bytes": 2 * (att + 2 * T * d) + sum(s + n for s, n in seqs) * 4 * D,
                "flops": 2 * T * att + sum(4 * H * D * (n * s + n * (n + 1) // 2) for s, n in seqs)}
    if kind == "sample":
        return {"bytes": 4 * c["rows"] * c["vocab"], "flops": 0}
    T, d = c["tokens"], c["width"]
    if kind == "experts":                                      # of the 16 + 2, 32 / 9 real experts a token on average
        pairs, F = T * 4 * 16 / 18, d // 2
        used = 16 * (1 - (1 - 4 / 18) ** T)
        return {"bytes": 2 * used * 3 * d * F + T * d * 6, "flops": 2 * pairs * 3 * d * F + 2 * T * 18 * d}
    H = d // 128
    if kind == "retention":
        params, state, rec = 5 * d * d, H * 128 * 128, 4 * H * 128 * 128
    elif kind == "mlstm":
        params, state, rec = d * H * (64 + 64 + 128 + 128 + 128 + 2), H * 64 * 128, 4 * H * 64 * 128
    elif kind == "wkv":
        params, state, rec = 5 * d * d + 2 * 64 * d, (d // 64) * 64 * 64, 4 * (d // 64) * 64 * 64
    else:
        I = 2 * d
        params, state, rec = 3 * d * I + I * (d // 16 + 32) + I * (d // 16), I * 16, 6 * I * 16
    return {"bytes": 2 * params + 4 * T * d + 8 * c["requests"] * state, "flops": T * (2 * params + rec)}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.02, "max": 0.5}


# --------------------------------------------------------------------------- the same in 64 bits
def _norm(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rotate(x, pos, base=10000.0, style="interleaved"):
    """x [T, heads, D] at positions pos [T]."""
    D = x.shape[-1]
    inv = (1.0 / (base ** (torch.arange(0, D, 2).float() / D))).to(DEV).double()
    ang = pos.double()[:, None] * inv
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]
    if style == "half":
        a, b = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2)


def _attend(q, k, v, first):
    """Causal attention of q [n, heads, D] at positions first.. over k, v [m, D] of one kv head."""
    n, H, D = q.shape
    out = torch.empty_like(q)
    at = torch.arange(k.shape[0], device=DEV)
    for a in range(0, n, 256):
        s = torch.einsum("thd,md->htm", q[a:a + 256], k) / math.sqrt(D)
        s = s.masked_fill(at > (first + a + torch.arange(s.shape[1], device=DEV))[:, None], -math.inf)
        out[a:a + 256] = torch.einsum("htm,md->thd", s.softmax(-1), v)
    return out


def _gpt_layer(c, w, p, x, pos, attend):
    """One block on the stream x [T, d] in 64 bits; attend(q, k, v) -> [T, heads, D]."""
    d, H, D, F, _, _, eps = GPT[c["model"]]
    t = lambda n: w[f"{p}{n}.weight"].double()
    h = _norm(x, t("attn_norm"), eps)
    q, k, v = _rotate((h @ t("attn.q_proj").T).view(-1, H, D), pos), _rotate((h @ t("attn.k_proj").T).view(-1, 1, D), pos)[:, 0], h @ t("attn.v_proj").T
    x = x + attend(q, k, v).reshape(-1, H * D) @ t("attn.out").T
    h = _norm(x, t("mlp_norm"), eps)
    return x + (torch.nn.functional.silu(h @ t("mlp.gate_proj").T) * (h @ t("mlp.up_proj").T)) @ t("mlp.down_proj").T, k, v


def _scan(lens, states, step, *rows):
    """step(states, *rows of one token) -> (states, out) over the tokens of each request; states [requests, ...] in 64 bits."""
    outs, ends, at = [], [], 0
    for r, n in enumerate(lens):
        s = tuple(x[r] for x in states)
        for t in range(at, at + n):
            s, o = step(s, *(x[t] for x in rows))
            outs.append(o)
        ends.append(s)
        at += n
    return torch.stack(outs), [torch.stack(e) for e in zip(*ends)]


def _mixer_exact(c, g):
    kind, args, w, rows = _mixer_parts(c, g, torch.bfloat16)
    x = _x(c, g, torch.bfloat16).double()
    w = {n: v.double() for n, v in w.items()}
    states = [r.double() for r in rows]
    T, lens, d = c["tokens"], _lens(c["tokens"], c["requests"]), c["width"]
    silu, rms = torch.nn.functional.silu, lambda o: o * torch.rsqrt((o * o).mean(-1, keepdim=True) + 1e-6)
    if kind == "retention":
        H = d // 128
        pos = torch.cat([64 + torch.arange(n, device=DEV) for n in lens])
        head = lambda n: (x @ w[n].T).view(T, H, 128)
        q, k = _rotate(head("q"), pos, style="half"), _rotate(head("k"), pos, style="half") * 128 ** -0.5
        decay = torch.tensor(_decays(H), dtype=torch.float32, device=DEV).double()[:, None, None]

        def step(s, q, k, v):
            S = s[0] * decay + v[:, :, None] * k[:, None, :]
            return (S,), (S @ q[:, :, None])[..., 0]
        o, ends = _scan(lens, states, step, q, k, head("v"))
        out = (rms(o).flatten(1) * silu(x @ w["g"].T)) @ w["o"].T
    elif kind == "mlstm":
        H = d // 128
        q, k, v = (x @ w["q"].T).view(T, H, 64) / 8, (x @ w["k"].T).view(T, H, 64), (x @ w["v"].T).view(T, H, 128)
        b = lambda n: w[n].bfloat16().double()                 # the gates' biases are held in the compute type
        i = 15 * torch.tanh((x @ w["i"].T + b("i.b")) / 15)
        f = torch.nn.functional.logsigmoid(15 * torch.tanh((x @ w["f"].T + b("f.b")) / 15))

        def step(s, q, k, v, i, f):
            S, n, m = s
            m1 = torch.maximum(f + m, i)
            a, b = (f + m - m1).exp()[:, None], (i - m1).exp()[:, None]
            S, n = a[..., None] * S + (b * v)[:, :, None] * k[:, None, :], a * n + b * k
            den = torch.maximum((n * q).sum(-1).abs(), (-m1).exp()) + 1e-6
            return (S, n, m1), (S @ q[:, :, None])[..., 0] / den[:, None]
        o, ends = _scan(lens, states, step, q, k, v, i, f)
        out = (rms(o).flatten(1) * w["norm"] * torch.sigmoid(x @ w["g"].T)) @ w["o"].T
    elif kind == "wkv":
        H = d // 64
        S0, prev = states
        before, at = [], 0
        for r, n in enumerate(lens):
            before += [prev[r:r + 1], x[at:at + n - 1]]
            at += n
        before = torch.cat(before)
        mix = lambda n: x + (before - x) * w[f"mu.{n}"]
        r, k, v = ((mix(n) @ w[n].T).view(T, H, 64) for n in ("r", "k", "v"))
        decay = torch.exp(-torch.exp(torch.tanh(mix("w") @ w["w1"].T) @ w["w2"].T + w["w0"])).view(T, H, 64)

        def step(s, r, k, v, a):
            kv = v[:, :, None] * k[:, None, :]
            o = ((s[0] + w["u"][:, None, :] * kv) @ r[:, :, None])[..., 0]
            return (s[0] * a[:, None, :] + kv,), o
        o, ends = _scan(lens, [S0], step, r, k, v, decay)
        ends.append(torch.stack([x[sum(lens[:r + 1]) - 1] for r in range(len(lens))]))
        out = (rms(o).flatten(1) * w["norm"] * silu(mix("g") @ w["g"].T)) @ w["o"].T
    else:
        I, N, R = 2 * d, 16, d // 16
        S0, tail = states
        proj = x @ w["in"].T
        u, z = [], proj[:, I:]
        ends_tail, at = [], 0
        for r, n in enumerate(lens):
            rows_ = torch.cat([tail[r], proj[at:at + n, :I]])
            u.append(silu(sum(rows_[j:j + n] * w["conv"][:, j] for j in range(4)) + w["conv.b"]))
            ends_tail.append(rows_[-3:])
            at += n
        u = torch.cat(u)
        low = u @ w["x"].T
        dt = torch.nn.functional.softplus(low[:, :R] @ w["dt"].T + w["dt.b"])
        A = -torch.exp(w["A_log"])

        def step(s, u, dt, B, C):
            S = torch.exp(dt[:, None] * A) * s[0] + (dt * u)[:, None] * B
            return (S,), S @ C + w["D"] * u
        o, ends = _scan(lens, [S0], step, u, dt, low[:, R:R + N], low[:, R + N:])
        ends.append(torch.stack(ends_tail))
        out = (o * silu(z)) @ w["o"].T
    full = []
    for e in ends:                                             # the row that padding uses stays zero
        full.append(torch.cat([e, torch.zeros_like(e[:1])]))
    return {"out": out, "states": full}


@torch.no_grad()
def exact(case, seed):
    c, g, kind = case, _gen(seed), case["kind"]
    if kind == "sample":
        return None                                            # whole numbers, and which ones is the generator's choice
    if kind == "decode":
        d, H, D, F, V, _, eps = GPT[c["model"]]
        w = _gpt_tensors(c, c["layers"], g, torch.bfloat16)
        rows = _cache_rows(c, c["layers"], g, torch.bfloat16)
        ids = _tokens(g, c["batch"], V).long()
        x, pos = w["embedding.embedding.weight"][ids].double(), torch.full((c["batch"],), c["ctx"] - 1, device=DEV)
        for i in range(c["layers"]):
            def attend(q, k, v):
                return torch.cat([_attend(q[b:b + 1], torch.cat([rows[i, 0, b].double(), k[b:b + 1]]),
                                          torch.cat([rows[i, 1, b].double(), v[b:b + 1]]), c["ctx"] - 1) for b in range(c["batch"])])
            x, _, _ = _gpt_layer(c, w, f"layers.{i}.", x, pos, attend)
        return _norm(x, w["final_norm.weight"].double(), eps) @ w["lm_head.weight"].double().T
    if kind == "block":
        D, V, eps, T = GPT[c["model"]][2], GPT[c["model"]][4], GPT[c["model"]][6], c["tokens"]
        dtype = DTYPES[c["dtype"]]
        w = _gpt_tensors(c, 1, g, dtype)
        kv, table = _paged([(0, T)], D, F64)
        x = w["embedding.embedding.weight"][_tokens(g, T, V).long()].double()
        x, k, v = _gpt_layer(c, w, "layers.0.", x, torch.arange(T, device=DEV), lambda q, k, v: _attend(q, k, v, 0))
        at = table[0].long().repeat_interleave(PAGE)[:T] * PAGE + torch.arange(T, device=DEV) % PAGE
        kv[0].view(-1, D)[at], kv[1].view(-1, D)[at] = k, v
        return {"out": _norm(x, w["final_norm.weight"].double(), eps), "keys_and_values": kv[:, 1:]}
    if kind == "mixed":
        d, H, D = GPT[c["model"]][:3]
        w = {n: v.double() for n, v in _mixed_tensors(c, g, torch.bfloat16).items()}
        seqs = _mixed_step(c)
        kv, table = _paged(seqs, D, torch.bfloat16, g)
        x = _randn(g, c["decoding"] + c["portion"], d, dtype=torch.bfloat16).double()
        outs, at = [], 0
        for i, (s, n) in enumerate(seqs):
            h, pos = x[at:at + n], torch.arange(s, s + n, device=DEV)
            old = table[i].long().repeat_interleave(PAGE)[:s] * PAGE + torch.arange(s, device=DEV) % PAGE
            k = torch.cat([kv[0].view(-1, D)[old].double(), _rotate((h @ w["k_proj.weight"].T).view(-1, 1, D), pos)[:, 0]])
            v = torch.cat([kv[1].view(-1, D)[old].double(), h @ w["v_proj.weight"].T])
            outs.append(_attend(_rotate((h @ w["q_proj.weight"].T).view(-1, H, D), pos), k, v, s).reshape(n, H * D) @ w["out.weight"].T)
            at += n
        return torch.cat(outs)
    if kind == "experts":
        _, w = _expert_parts(c, g, torch.bfloat16)
        x = _x(c, g, torch.bfloat16).double()
        s = (x @ w["router"].double().T).softmax(-1)
        top = (s + w["correction"].double()).topk(4, -1).indices
        out = torch.zeros_like(x)
        for e in range(18):
            rows = (top == e).any(-1).nonzero()[:, 0]
            h = x[rows]
            if e < 16:
                gate = (h @ w[f"e{e}.gate"].double().T).clamp(max=7.0)
                up = (h @ w[f"e{e}.up"].double().T).clamp(-7.0, 7.0)
                h = (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ w[f"e{e}.down"].double().T
            out[rows] += s[rows, e:e + 1] * h
        return out
    return _mixer_exact(c, g)
