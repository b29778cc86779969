"""What a program built on this framework spends its time on, as cases that can be measured one by one.

Three levels, each through public entry points: the kernels a program can call on its own tensors (`kernels`, the C ABI), blocks
made of them (an attention layer, an MLP), and the engine fed with given tokens (`Engine.feed`), for Llama and for the layered
designs.  Head shapes are those of Llama-3.2-1B / 3B and Llama-3.1-8B; the layered models have the sizes of the framework's own
benchmark (width 2048, 16 heads of 128).  Weights are random; tokens, activations and cache contents come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fasttalk_llm_microservice_b200 import kernels as K
from fasttalk_llm_microservice_b200 import native as N
from fasttalk_llm_microservice_b200.engine import Engine, EngineLimits
from fasttalk_llm_microservice_b200.layered import spec_from_config, tensor_shapes
from fasttalk_llm_microservice_b200.model_spec import ModelSpec, get_spec
from fasttalk_llm_microservice_b200.weights import init_weights

PAGE = 64
MODELS = {"1b": "llama-3.2-1b", "3b": "llama-3.2-3b", "8b": "llama-3.1-8b"}
F64 = torch.float64


def listed():
    return [
        # one voice session: the sampler on one row of logits after every token
        {"name": "sample-one", "kind": "sample", "rows": 1, "vocab": 128256},
        # a full batch of sessions: greedy, top-k and nucleus rows side by side
        {"name": "sample-batch", "kind": "sample", "rows": 64, "vocab": 128256},
        # attention layer of a decode step, 64 sessions around 2k tokens of history
        {"name": "attention-decode", "kind": "decode", "model": "1b", "sessions": 64, "context": 2048},
        # attention layer of a cold prefill step, four 2k prompts
        {"name": "attention-prompts", "kind": "prompts", "model": "1b", "sessions": 4, "new": 2048, "cached": 0},
        # attention layer of a follow-up turn: a few hundred new tokens over a long history
        {"name": "attention-history", "kind": "prompts", "model": "8b", "sessions": 6, "new": 211, "cached": 5003},
        # MLP of a step that mixes decoding sessions with prompt portions
        {"name": "mlp-mixed", "kind": "mlp", "model": "3b", "tokens": 611},
        # the scalar-decay recurrence alone: prompt portions of several requests, some of them continued
        {"name": "decay-rule", "kind": "decay", "heads": 16, "dim": 128, "vdim": 128, "tokens": 2048, "requests": 3},
        # a handful of sessions on the smallest Llama: short prompts, then token by token
        {"name": "llama-turn", "kind": "engine", "design": "llama", "order": "1b", "width": 2048, "sessions": 4, "prompt": 160, "steps": 16},
        # Gedelorn: prompts through a parallel mixer with experts, a matrix memory and a state space
        {"name": "gedelorn-prompts", "kind": "engine", "design": "gedelorn", "order": "pms", "width": 2048, "sessions": 3, "prompt": 800, "steps": 0},
        # the same model answering 16 sessions token by token
        {"name": "gedelorn-turn", "kind": "engine", "design": "gedelorn", "order": "pms", "width": 2048, "sessions": 16, "prompt": 128, "steps": 24},
        # Vonedra: prompts through window attention and the gated delta rule
        {"name": "vonedra-prompts", "kind": "engine", "design": "vonedra", "order": "ad", "width": 2048, "sessions": 3, "prompt": 800, "steps": 0},
        # Fedutar: prompts through gated attention beside a retention
        {"name": "fedutar-prompts", "kind": "engine", "design": "fedutar", "order": "pp", "width": 2048, "sessions": 3, "prompt": 800, "steps": 0},
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], evenly over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["sample", "decode", "prompts", "mlp", "decay", "engine", "engine"])
    if kind == "sample":
        return {"kind": kind, "rows": _spread(rng, 1, 64), "vocab": rng.choice([128256, 32768, 50257])}
    model = rng.choice(sorted(MODELS))
    if kind == "decode":
        return {"kind": kind, "model": model, "sessions": _spread(rng, 1, 64), "context": _spread(rng, 1, 2048)}
    if kind == "prompts":
        if rng.random() < 0.5:
            return {"kind": kind, "model": model, "sessions": rng.randint(1, 4), "new": _spread(rng, 5, 1500), "cached": 0}
        return {"kind": kind, "model": model, "sessions": rng.randint(1, 6), "new": _spread(rng, 5, 211), "cached": _spread(rng, 40, 5003)}
    if kind == "mlp":
        return {"kind": kind, "model": model, "tokens": _spread(rng, 1, 611)}
    if kind == "decay":
        heads = rng.choice([2, 6, 8, 16])
        dim, vdim = rng.choice([(64, 64), (128, 64), (128, 128), (96, 80), (128, 129)])
        return {"kind": kind, "heads": heads, "dim": dim, "vdim": vdim, "tokens": _spread(rng, 3, 2048), "requests": rng.randint(1, 3)}
    design = rng.choice(["llama", "gedelorn", "gedelorn", "vonedra", "fedutar"])
    case = {"kind": kind, "design": design, "order": "1b", "width": 2048, "sessions": 1, "prompt": 1, "steps": 0}
    if design == "llama":
        case.update(sessions=rng.randint(1, 4), prompt=_spread(rng, 3, 160), steps=rng.randint(1, 16))
        return case
    letters = {"gedelorn": "pms", "vonedra": "ad", "fedutar": "p"}[design]
    case["order"] = "".join(rng.choice(letters) for _ in range(rng.randint(1, 2)))
    case["width"] = rng.choice([1024, 2048])
    if rng.random() < 0.5:
        case.update(sessions=rng.randint(1, 3), prompt=_spread(rng, 9, 800))
    else:
        case.update(sessions=_spread(rng, 1, 16), prompt=_spread(rng, 3, 128), steps=rng.randint(2, 24))
    return case


# ------------------------------------------------------------------------------------------------ helpers
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _lengths(n, most):
    """Ragged lengths of n sessions, the longest `most`, none below two thirds of it."""
    return [max(1, most - (i * 29) % max(1, most // 3)) for i in range(n)]


def _starts(lengths):
    return [0] + [int(v) for v in np.cumsum(lengths)]


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _softplus(z):
    return torch.where(z > 30.0, z, torch.log1p(torch.exp(torch.clamp(z, max=30.0))))


def _cache_rows(cache, table, head, what, n):
    """Rows 0 .. n - 1 of a sequence's keys (what = 0) or values (1) of one head, in 64 bits, from the paged cache: a page's slab is
    d / 64 pieces of [64 tokens][64 dims] whose eight 16-byte chunks per row are swapped with (row & 7)."""
    d = cache.shape[-1]
    slabs = cache[table[: -(-n // PAGE)].long(), head, what].reshape(-1, d // 64, PAGE, 8, 8)
    row = torch.arange(PAGE, device=cache.device)[:, None]
    chunk = torch.arange(8, device=cache.device)[None, :] ^ (row & 7)
    x = torch.gather(slabs, 3, chunk[None, None, :, :, None].expand(slabs.shape))
    return x.permute(0, 2, 1, 3, 4).reshape(-1, d)[:n].to(F64)


def _paged_attention(q, cache, table, pos0, group):
    """q [T, heads, d] at positions pos0 .. over one sequence's cache, in 64 bits -> [T, heads * d]."""
    T, nq, d = q.shape
    n = pos0 + T
    keys = torch.arange(n, device=q.device)
    hidden = keys[None, :] > pos0 + torch.arange(T, device=q.device)[:, None]
    out = torch.empty(T, nq, d, device=q.device, dtype=F64)
    for g in range(nq // group):
        k, v = _cache_rows(cache, table, g, 0, n), _cache_rows(cache, table, g, 1, n)
        for h in range(g * group, (g + 1) * group):
            s = (q[:, h].to(F64) @ k.T / math.sqrt(d)).masked_fill(hidden, -math.inf)
            out[:, h] = torch.softmax(s, -1) @ v
    return out.reshape(T, nq * d)


# ------------------------------------------------------------------------------------------------ sampling
def _sample_inputs(case, seed):
    g = _gen(seed)
    B, V = case["rows"], case["vocab"]
    logits = torch.randn(B, V, generator=g, device="cuda") * 2.0
    likely = torch.randint(V, (B, 40), generator=g, device="cuda")               # what the model expects next
    logits.scatter_add_(1, likely, 4.0 + 5.0 * torch.rand(B, 40, generator=g, device="cuda"))
    # the reference's defaults (0.7, 0.9), its Ollama options (top_k 40), warmer rows and greedy ones
    settings = [(0.7, 0, 0.9), (0.7, 40, 0.9), (1.0, 0, 0.95), (0.0, 0, 1.0)]
    rows = [settings[i % 4] for i in range(B)]
    dev = lambda v, t: torch.tensor(v, device="cuda", dtype=t)
    return {"logits": logits, "temperature": dev([r[0] for r in rows], torch.float32), "top_k": dev([r[1] for r in rows], torch.int32),
            "top_p": dev([r[2] for r in rows], torch.float32),
            "seeds": torch.randint(1 << 62, (B,), generator=g, device="cuda", dtype=torch.int64)}


# ------------------------------------------------------------------------------------------------ attention layers
def _cache_of(spec, lengths, g):
    """One layer's paged cache holding sequences of the given lengths on shuffled pages."""
    pages = [-(-n // PAGE) for n in lengths]
    cache = torch.randn(sum(pages), spec.n_kv_heads, 2, PAGE, spec.head_dim, generator=g, device="cuda").to(torch.float16)
    order = torch.randperm(sum(pages), generator=g, device="cuda").to(torch.int32)
    table = torch.zeros(len(lengths), max(pages), device="cuda", dtype=torch.int32)
    at = 0
    for i, p in enumerate(pages):
        table[i, :p] = order[at:at + p]
        at += p
    return cache, table


def _attention_inputs(case, seed):
    spec = get_spec(MODELS[case["model"]])
    g = _gen(seed)
    if case["kind"] == "decode":
        lengths = _lengths(case["sessions"], case["context"])
        rows = len(lengths)
        state = {"lengths": lengths}
    else:
        new = _lengths(case["sessions"], case["new"])
        lengths = [case["cached"] + n for n in new]
        rows = sum(new)
        state = {"lengths": lengths, "starts": _starts(new), "pos0": [case["cached"]] * len(new), "slots": list(range(len(new)))}
    state["cache"], state["table"] = _cache_of(spec, lengths, g)
    state["q"] = (1.5 * torch.randn(rows, spec.n_q_heads, spec.head_dim, generator=g, device="cuda")).to(torch.float16)
    state["wo"] = (0.02 * torch.randn(spec.hidden, spec.q_dim, generator=g, device="cuda")).to(torch.bfloat16)
    state["ctx"] = torch.tensor(lengths, device="cuda", dtype=torch.int32)
    return state


def _summed(parts):
    return parts[0] if parts.shape[0] == 1 else parts.sum(0)


def _attention_exact(case, seed):
    spec = get_spec(MODELS[case["model"]])
    s = _attention_inputs(case, seed)
    group = spec.n_q_heads // spec.n_kv_heads
    if case["kind"] == "decode":
        rows = [_paged_attention(s["q"][i:i + 1], s["cache"], s["table"][i], n - 1, group) for i, n in enumerate(s["lengths"])]
    else:
        rows = [_paged_attention(s["q"][a:b], s["cache"], s["table"][i], case["cached"], group)
                for i, (a, b) in enumerate(zip(s["starts"], s["starts"][1:]))]
    return torch.cat(rows) @ s["wo"].to(F64).T


# ------------------------------------------------------------------------------------------------ MLP
def _mlp_inputs(case, seed):
    spec = get_spec(MODELS[case["model"]])
    g = _gen(seed)
    rnd = lambda *shape: (0.02 * torch.randn(*shape, generator=g, device="cuda")).to(torch.bfloat16)
    return {"resid": torch.randn(case["tokens"], spec.hidden, generator=g, device="cuda"),
            "norm": (1.0 + 0.1 * torch.randn(spec.hidden, generator=g, device="cuda")).to(torch.bfloat16),
            "wgu": rnd(2 * spec.ffn, spec.hidden), "wd": rnd(spec.hidden, spec.ffn), "eps": spec.rms_eps}


def _mlp_exact(case, seed):
    s = {k: v.to(F64) if isinstance(v, torch.Tensor) else v for k, v in _mlp_inputs(case, seed).items()}
    gu = (_rms(s["resid"], s["eps"]) * s["norm"]) @ s["wgu"].T
    gu = gu.reshape(gu.shape[0], -1, 2, 64)                                   # rows in blocks of 64: gate, up, gate, up, ...
    return (_silu(gu[:, :, 0]) * gu[:, :, 1]).reshape(gu.shape[0], -1) @ s["wd"].T


# ------------------------------------------------------------------------------------------------ the scalar-decay rule
def _decay_inputs(case, seed):
    g = _gen(seed)
    H, D, V, T, R = case["heads"], case["dim"], case["vdim"], case["tokens"], min(case["requests"], case["tokens"])
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    cut = [T * i // R for i in range(R + 1)]
    i32 = lambda v: torch.tensor(v, device="cuda", dtype=torch.int32)
    keep = 1.0 - torch.exp(-1.0 - 6.0 * torch.rand(T, H, generator=g, device="cuda"))
    put = 0.1 + torch.rand(T, H, generator=g, device="cuda")
    return {"q": rnd(T, H * D) * D ** -0.5, "k": rnd(T, H * D), "v": rnd(T, H * V), "ab": torch.stack([keep, put], -1).contiguous(),
            "state": rnd(R, H, D, V), "work": torch.empty(R, H, D, V, device="cuda"), "cut": cut, "start": i32(cut),
            "pos0": i32([0 if i % 2 == 0 else 77 for i in range(R)]), "slot": i32(list(range(R)))}


def _decay_run(case, s):
    H, D, V, T = case["heads"], case["dim"], case["vdim"], case["tokens"]
    s["work"].copy_(s["state"])
    o = torch.empty(T, H * V, device="cuda")
    N.check(N.load().ft_decay_rule(N.ptr(s["q"]), N.ptr(s["k"]), N.ptr(s["v"]), N.ptr(s["ab"]), N.ptr(o), N.ptr(s["work"]), N.ptr(s["start"]),
                                   N.ptr(s["pos0"]), N.ptr(s["slot"]), len(s["cut"]) - 1, H, H, D, V, H * D * V, 0, T, N.cur_stream()),
            "ft_decay_rule")
    return [o, s["work"]]


def _scan(q, k, v, keep, put, S):
    """S <- keep S + put k v^T, o = S^T q, token by token; q, k [T, H, D], v [T, H, V], keep / put [T, H], S [H, D, V]."""
    out = torch.empty(v.shape, device=v.device, dtype=v.dtype)
    for t in range(q.shape[0]):
        S = keep[t][:, None, None] * S + (put[t][:, None] * k[t])[:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return out, S


def _decay_exact(case, seed):
    H, D, V = case["heads"], case["dim"], case["vdim"]
    s = _decay_inputs(case, seed)
    outs, states = [], []
    for r, (a, b) in enumerate(zip(s["cut"], s["cut"][1:])):
        x = lambda n, w: s[n][a:b].to(F64).reshape(b - a, H, w)
        ab = s["ab"][a:b].to(F64)
        S = s["state"][r].to(F64) * (r % 2)
        o, S = _scan(x("q", D), x("k", D), x("v", V), ab[..., 0], ab[..., 1], S)
        outs.append(o.reshape(b - a, H * V))
        states.append(S)
    return [torch.cat(outs), torch.stack(states)]


# ------------------------------------------------------------------------------------------------ layered models
VOCAB = 4096


def _gedelorn(order, W):
    """p: window attention beside a decay attention + experts; m: matrix memory + dense; s: state space + dense."""
    H, D = W // 128, 128
    dense = {"ff": W, "kind": "dense"}
    moe = {"expert": {"ff": W // 2}, "kind": "moe", "router": {"experts": 16, "scale": 1.0, "top": 2}, "shared": {"ff": W // 2}}
    par = {"type": "parallel", "mixer": {
        "left": {"dim": D, "heads": H, "kv_heads": max(1, H // 4), "mask": {"size": 512}, "rot": {"base": 1e6, "dims": D},
                 "scale": D ** -0.5, "softcap": 50.0, "vdim": D},
        "left_scale": 1.0, "right": {"decay": [1.0 - 2.0 ** -(3 + 7 * h / max(1, H - 1)) for h in range(H)], "dim": D, "heads": H,
                                     "vdim": D}, "right_scale": 1.0}, "mlp": moe}
    mem = {"type": "mlstm", "mixer": {"dim": D, "gate_cap": 15.0, "heads": max(1, H // 2), "vdim": 2 * D}, "mlp": dense}
    space = {"type": "mamba2", "mixer": {"conv": 4, "groups": 1, "heads": 2 * W // 64, "norm_groups": 1, "state": 128, "vdim": 64}, "mlp": dense}
    return {"architecture": "Gedelorn", "layers": [{"p": par, "m": mem, "s": space}[c] for c in order], "norm": {"eps": 1e-6},
            "vocab": VOCAB, "width": W}, None


def _vonedra(order, W):
    """a: attention with a distance bias, a window of 512 that keeps 4 tokens and a sink; d: gated delta rule."""
    H, D = W // 128, 128
    att = {"type": "attention", "mixer": {"bias_max": 512, "dim": D, "heads": H, "kv_heads": max(1, H // 4),
                                          "mask": {"keep_first": 4, "size": 512}, "scale": D ** -0.5, "v_mix": True, "vdim": D}}
    dlt = {"type": "delta", "mixer": {"conv": 4, "dim": D, "heads": H, "kv_heads": H, "vdim": D}}
    layers = [{**{"a": att, "d": dlt}[c], "mlp": {"ff": W, "kind": "dense"}} for c in order]
    cfg = {"architecture": "Vonedra", "canon": {"taps": 4}, "embedding": {"scale": 1.0}, "layers": layers, "norm": {"eps": 1e-6},
           "vocab": VOCAB, "width": W}
    return cfg, {f"l{i}.mix.rel": (32, H) for i, c in enumerate(order) if c == "a"}


def _fedutar(order, W):
    """p: gated attention without positions beside a retention + dense with biases."""
    H, D = W // 128, 128
    mixer = {"left": {"dim": D, "heads": H, "kv_heads": max(1, H // 4), "q_temp": {"coef": 0.1, "every": 512}, "scale": D ** -0.5, "vdim": D},
             "left_scale": 1.0, "right": {"decay": [1.0 - 2.0 ** -(3 + 7 * h / max(1, H - 1)) for h in range(H)], "dim": D, "heads": H,
                                          "rot": {"base": 1e4, "dims": D}, "vdim": D}, "right_scale": 1.0}
    layers = [{"type": "parallel", "mixer": mixer, "mlp": {"ff": W, "kind": "dense"}} for _ in order]
    return {"architecture": "Fedutar", "embedding": {"scale": W ** 0.5}, "layers": layers, "logit_scale": W ** -0.5, "logit_softcap": 30.0,
            "norm": {"eps": 1e-6}, "vocab": VOCAB, "width": W}, None


DESIGNS = {"gedelorn": _gedelorn, "vonedra": _vonedra, "fedutar": _fedutar}


def _layered_spec(case):
    cfg, shapes = DESIGNS[case["design"]](case["order"], case["width"])
    return cfg, spec_from_config(cfg, shapes, name=case["design"])


def _layered_weights(case, spec):
    """Tensors of the size of a trained model's under the checkpoint's names; the same for every seed, as a served model's are."""
    g = _gen(11)
    design = case["design"]
    out = {}
    for name, shape in tensor_shapes(spec).items():
        leaf, part = name.split(".")[-1], (name.split(".") + [""])[-2]
        x = torch.randn(shape, generator=g, device="cuda")
        if leaf in ("norm1", "norm1b", "norm2", "norm2b", "norm") or name == "final.norm":
            stored_less_one = design == "gedelorn" and (leaf != "norm" or name == "final.norm")
            x = 0.2 * x if stored_less_one else 1.0 + 0.1 * x
        elif leaf in ("canon1", "canon2"):
            x = 0.3 * x
        elif leaf == "dwa":
            x = 0.15 * x
            x[-1] += 1.0
        elif leaf == "vmix":
            x = 0.2 + 0.5 * torch.rand(shape, generator=g, device="cuda")
        elif leaf == "b" and len(shape) == 1:
            x = 0.3 * x + (3.0 if part == "f" else 0.0)
        elif leaf == "D":
            x = 1.0 + 0.2 * x
        elif leaf == "A_log":
            x = torch.log(0.5 + 2.0 * torch.rand(shape, generator=g, device="cuda"))
        elif leaf == "dt_bias":
            x = x - 2.0
        elif leaf == "conv":
            x = 0.5 * x
        elif name != "embed" and leaf not in ("rel", "sink"):
            x = x / shape[-1] ** 0.5
        out[name] = x.to(torch.bfloat16)
    return out


def _llama_spec(case):
    return get_spec(MODELS[case["order"]])


def _engine_plan(case, seed):
    """Per session its tokens (prompt, then the tokens it is fed one by one); per prefill call (session, count) and the wanted places."""
    vocab = get_spec(MODELS[case["order"]]).vocab if case["design"] == "llama" else VOCAB
    lengths = _lengths(case["sessions"], case["prompt"])
    rng = np.random.default_rng(seed)
    tokens = [rng.integers(0, vocab, n + case["steps"]).tolist() for n in lengths]
    calls, room = [[]], 2560
    for i, n in enumerate(lengths):
        if n > room:
            calls.append([])
            room = 2560
        calls[-1].append(i)
        room -= n
    per = 1 if case["steps"] else max(1, 64 // len(lengths))
    want = [sorted({n - 1 - j * n // per for j in range(per)}) for n in lengths]
    return lengths, tokens, calls, want


def _engine_state(case, seed):
    if case["design"] == "llama":
        spec = _llama_spec(case)
        w = init_weights(spec, seed=11, device="cuda")
    else:
        _, spec = _layered_spec(case)
        w = _layered_weights(case, spec)
    lengths, tokens, calls, want = _engine_plan(case, seed)
    context = max(lengths) + case["steps"]
    n = case["sessions"]
    eng = Engine(spec, w, EngineLimits(max_batch=max(16, n), max_batched_tokens=2560, max_context=context + 1, max_sessions=n + 2,
                                       num_pages=(n + 2) * (context // PAGE + 2), debug_logit_rows=64), eos_ids=())
    return {"engine": eng, "plan": (lengths, tokens, calls, want)}


def _engine_run(case, s):
    eng, (lengths, tokens, calls, want) = s["engine"], s["plan"]
    for i in range(len(lengths)):
        eng.close_session(i)
    got = [eng.feed([(i, tokens[i][:lengths[i]], want[i]) for i in call]) for call in calls]
    for t in range(case["steps"]):
        got.append(eng.feed([(i, tokens[i][n + t:n + t + 1], [0]) for i, n in enumerate(lengths)]))
    return np.concatenate(got)


def _engine_exact(case, seed):
    lengths, tokens, calls, want = _engine_plan(case, seed)
    if case["design"] == "llama":
        spec = _llama_spec(case)
        w = init_weights(spec, seed=11, device="cuda")
        rows = [_llama(w, spec, t, [n - 1 + j for j in range(case["steps"] + 1)]) for t, n in zip(tokens, lengths)]
    else:
        cfg, spec = _layered_spec(case)
        w = {k: v.to(F64) for k, v in _layered_weights(case, spec).items()}
        places = [wt + [n + j for j in range(case["steps"])] for wt, n in zip(want, lengths)]
        rows = [LAYERED[case["design"]](w, cfg, torch.tensor(t, device="cuda"))[p] for t, p in zip(tokens, places)]
    out = [rows[i][:len(want[i])] for call in calls for i in call]
    for t in range(case["steps"]):
        out += [r[len(wt) + t:len(wt) + t + 1] for r, wt in zip(rows, want)]
    return torch.cat(out).cpu().numpy()


def _llama(w, spec, tokens, wanted):
    """Logits of the wanted places of one sequence: the public Llama-3 decoder in 64 bits."""
    T, d = len(tokens), spec.head_dim
    f = lambda t: t.to(F64)
    inv = spec.rope_theta ** (-torch.arange(0, d, 2, device="cuda", dtype=F64) / d)
    wl = 2 * math.pi / inv
    low, high = spec.rope_original_max_pos / spec.rope_low_freq_factor, spec.rope_original_max_pos / spec.rope_high_freq_factor
    smooth = (spec.rope_original_max_pos / wl - spec.rope_low_freq_factor) / (spec.rope_high_freq_factor - spec.rope_low_freq_factor)
    inv = torch.where(wl > low, inv / spec.rope_factor, torch.where(wl < high, inv, (1 - smooth) * inv / spec.rope_factor + smooth * inv))
    ang = torch.arange(T, device="cuda", dtype=F64)[:, None] * inv
    c, s = ang.cos()[:, None], ang.sin()[:, None]

    def turn(x):
        a, b = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    x = f(w["embed"][torch.tensor(tokens, device="cuda")])
    hidden = ~torch.ones(T, T, dtype=torch.bool, device="cuda").tril()
    for l in range(spec.layers):
        qkv = (_rms(x, spec.rms_eps) * f(w["attn_norm"][l])) @ f(w["wqkv"][l]).T
        q, k, v = qkv.split([spec.q_dim, spec.kv_dim, spec.kv_dim], -1)
        q, k = turn(q.reshape(T, -1, d)), turn(k.reshape(T, -1, d))
        k, v = (z.reshape(T, -1, d).repeat_interleave(spec.group, 1) for z in (k, v))
        p = torch.softmax((torch.einsum("ihd,jhd->hij", q, k) / math.sqrt(d)).masked_fill(hidden, -math.inf), -1)
        x = x + torch.einsum("hij,jhd->ihd", p, v).reshape(T, -1) @ f(w["wo"][l]).T
        g, u = ((_rms(x, spec.rms_eps) * f(w["mlp_norm"][l])) @ f(w["wgu"][l]).T).chunk(2, -1)
        x = x + (_silu(g) * u) @ f(w["wd"][l]).T
    return (_rms(x[wanted], spec.rms_eps) * f(w["final_norm"])) @ f(w["lm_head"]).T


def _turn(x, dims, base, halves):
    """Rotary positions on the first `dims` coordinates of [T, heads, d]: pairs (i, i + dims / 2) or (2i, 2i + 1)."""
    ang = torch.arange(x.shape[0], device=x.device, dtype=F64)[:, None] * base ** (-torch.arange(0, dims, 2, device=x.device, dtype=F64) / dims)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    out = x.clone()
    a, b = (slice(0, dims // 2), slice(dims // 2, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


def _causal_conv(u, taps, bias=None):
    """y[t] = sum_j taps[:, K - 1 - j] u[t - j] (+ bias), zeros before the start."""
    T, n = u.shape[0], taps.shape[1]
    y = torch.zeros_like(u) if bias is None else bias.expand(T, -1).clone()
    for j in range(min(n, T)):
        y[j:] += u[:T - j] * taps[:, n - 1 - j]
    return y


def _softmax_heads(q, k, v, scale, hidden, cap=None, bias=None, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, V] -> [T, H * V]; query head h reads key head h // (H / G)."""
    out = []
    for h in range(q.shape[1]):
        g = h // (q.shape[1] // k.shape[1])
        s = q[:, h] @ k[:, g].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if bias is not None:
            s = s + bias[:, :, h]
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
        p = torch.softmax(s, -1)
        out.append(p[:, :k.shape[0]] @ v[:, g])
    return torch.cat(out, -1)


def _hidden(T, size=None, keep_first=0):
    i = torch.arange(T, device="cuda")
    d = i[:, None] - i[None, :]
    return (d < 0) | ((d >= size) & (i[None, :] >= keep_first)) if size else d < 0


def _zeros(H, D, V):
    return torch.zeros(H, D, V, device="cuda", dtype=F64)


def _gedelorn_mixer(h, w, p, kind, m, eps):
    T = h.shape[0]
    lin = lambda n: h @ w[p + n].T
    if kind == "mlstm":
        H, D, V, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = lin("q").reshape(T, H, D) * D ** -0.5, lin("k").reshape(T, H, D), lin("v").reshape(T, H, V)
        gi = cap * torch.tanh((lin("i") + w[p + "i.b"]) / cap)
        gf = -_softplus(-cap * torch.tanh((lin("f") + w[p + "f.b"]) / cap))
        top, keep, put, floor = torch.zeros(H, device="cuda", dtype=F64), [], [], []
        for t in range(T):                         # the running maximum that both gates are taken against
            new = torch.maximum(gf[t] + top, gi[t])
            keep.append(torch.exp(gf[t] + top - new))
            put.append(torch.exp(gi[t] - new))
            floor.append(torch.exp(-new))
            top = new
        one = torch.ones(T, H, 1, device="cuda", dtype=F64)
        o, _ = _scan(q, k, torch.cat([v, one], -1), torch.stack(keep), torch.stack(put), _zeros(H, D, V + 1))
        o = o[..., :V] / (torch.maximum(o[..., V:].abs(), torch.stack(floor)[..., None]) + 1e-6)
        return (_rms(o, eps).reshape(T, H * V) * w[p + "norm"] * torch.sigmoid(lin("g"))) @ w[p + "o"].T
    if kind == "mamba2":
        H, V, D, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner = H * V
        z, xbc, dt = lin("in").split([inner, inner + 2 * G * D, H], -1)
        x, B, C = _silu(_causal_conv(xbc, w[p + "conv"], w[p + "conv.b"])).split([inner, G * D, G * D], -1)
        x = x.reshape(T, H, V)
        B, C = (t.reshape(T, G, D).repeat_interleave(H // G, 1) for t in (B, C))
        dt = _softplus(dt + w[p + "dt_bias"])
        o, _ = _scan(C, B, x, torch.exp(-torch.exp(w[p + "A_log"]) * dt), dt, _zeros(H, D, V))
        o = (o + w[p + "D"][:, None] * x).reshape(T, inner) * _silu(z)
        return (_rms(o.reshape(T, m["norm_groups"], -1), eps).reshape(T, inner) * w[p + "norm"]) @ w[p + "o"].T
    a, H, G, D = m["left"], m["left"]["heads"], m["left"]["kv_heads"], m["left"]["dim"]
    q, k = (lin("left.q") + w[p + "left.q.b"]).reshape(T, H, D), (lin("left.k") + w[p + "left.k.b"]).reshape(T, G, D)
    turn = lambda x: _turn(x, a["rot"]["dims"], a["rot"]["base"], False)
    left = _softmax_heads(turn(q), turn(k), k, a["scale"], _hidden(T, a["mask"]["size"]), cap=a["softcap"]) @ w[p + "left.o"].T
    r, H, D, V = m["right"], m["right"]["heads"], m["right"]["dim"], m["right"]["vdim"]
    q, k, v = (_silu(lin("right." + n)).reshape(T, H, -1) for n in "qkv")
    keep = torch.tensor(r["decay"], device="cuda", dtype=F64).expand(T, H)
    o, _ = _scan(q, k, v, keep, torch.ones_like(keep), _zeros(H, D, V))
    right = (_rms(o.reshape(T, H * V), eps) * w[p + "right.norm"] * torch.sigmoid(lin("right.g"))) @ w[p + "right.o"].T
    return m["left_scale"] * left + m["right_scale"] * right


def _gedelorn_experts(h, w, p, m):
    expert = lambda x, n: (torch.relu(x @ w[f"{p}{n}.up"].T) ** 2) @ w[f"{p}{n}.down"].T
    r = m["router"]
    best, ids = torch.topk(torch.sigmoid(h @ w[p + "router"].T), r["top"], -1)
    best = best / (best.sum(-1, keepdim=True) + 1e-20) * r["scale"]
    out = expert(h, "shared")
    for e in range(r["experts"]):
        rows, place = (ids == e).nonzero(as_tuple=True)
        out[rows] += best[rows, place][:, None] * expert(h[rows], f"e{e}")
    return out


def _dense(h, w, p, biases=False):
    lin = lambda z, n: z @ w[p + n].T + (w[p + n + ".b"] if biases else 0.0)
    return lin(_silu(lin(h, "gate")) * lin(h, "up"), "down")


def _gedelorn_exact(w, cfg, tokens):
    eps = cfg["norm"]["eps"]
    norm = lambda x, n: _rms(x, eps) * (1.0 + w[n])
    x = w["embed"][tokens]
    for i, l in enumerate(cfg["layers"]):
        p = f"l{i}."
        x = x + norm(_gedelorn_mixer(norm(x, p + "norm1"), w, p + "mix.", l["type"], l["mixer"], eps), p + "norm1b")
        h = norm(x, p + "norm2")
        x = x + norm(_dense(h, w, p + "mlp.") if l["mlp"]["kind"] == "dense" else _gedelorn_experts(h, w, p + "mlp.", l["mlp"]), p + "norm2b")
    return norm(x, "final.norm") @ w["head"].T


def _vonedra_attention(h, w, p, m, eps, first):
    T, H, G, D, rows = h.shape[0], m["heads"], m["kv_heads"], m["dim"], w[p + "rel"].shape[0]
    lin = lambda n: h @ w[p + n].T + w[p + n + ".b"]
    q, k, v = _rms(lin("q").reshape(T, H, D), eps), _rms(lin("k").reshape(T, G, D), eps), lin("v").reshape(T, G, -1)
    if m["v_mix"] and first is not None:
        v = (1.0 - w[p + "vmix"]) * v + w[p + "vmix"] * first
    half, far = rows // 2, float(m["bias_max"])
    row = [n if n < half else min(rows - 1, half + int(math.floor(math.log(n / half) / math.log(far / half) * (rows - half)))) for n in range(T)]
    i = torch.arange(T, device="cuda")
    bias = w[p + "rel"][torch.tensor(row, device="cuda")][(i[:, None] - i[None, :]).clamp(min=0)]
    o = _softmax_heads(q, k, v, m["scale"], _hidden(T, m["mask"]["size"], m["mask"]["keep_first"]), bias=bias, sink=w[p + "sink"])
    return o @ w[p + "o"].T + w[p + "o.b"], v


def _vonedra_delta(h, w, p, m, eps):
    T, H, G, D, V = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_silu(_causal_conv(h @ w[p + n].T, w[p + n + ".conv"])) for n in "qkv")
    q, k, v = q.reshape(T, G, D), k.reshape(T, G, D), v.reshape(T, H, V)
    q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * D ** -0.5).repeat_interleave(H // G, 1)
    k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    beta = torch.sigmoid(h @ w[p + "b"].T)
    keep = torch.exp(-torch.exp(w[p + "A_log"]) * _softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
    S, out = _zeros(H, D, V), torch.empty(T, H, V, device="cuda", dtype=F64)
    for t in range(T):
        S = keep[t][:, None, None] * S
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return ((_rms(out, eps) * w[p + "norm"]).reshape(T, H * V) * _silu(h @ w[p + "g"].T)) @ w[p + "o"].T


def _vonedra_exact(w, cfg, tokens):
    eps = cfg["norm"]["eps"]
    reads = lambda x, n: x + _causal_conv(x, w[n])
    x = w["embed"][tokens] * cfg["embedding"]["scale"]
    made, first = [x], None
    for i, l in enumerate(cfg["layers"]):
        p, m = f"l{i}.", l["mixer"]
        h = reads(x, p + "canon1")
        if l["type"] == "attention":
            y, v = _vonedra_attention(h, w, p + "mix.", m, eps, first)
            first = v if first is None else first
        else:
            y = _vonedra_delta(h, w, p + "mix.", m, eps)
        x = x + _rms(y, eps) * w[p + "norm1"]
        x = x + _rms(_dense(reads(x, p + "canon2"), w, p + "mlp."), eps) * w[p + "norm2"]
        made.append(x)
        x = sum(w[p + "dwa"][j] * made[j] for j in range(len(made)))
    return (_rms(x, eps) * w["final.norm"]) @ w["head"].T


def _fedutar_mixer(h, w, p, m, eps):
    T = h.shape[0]
    a, H, G, D = m["left"], m["left"]["heads"], m["left"]["kv_heads"], m["left"]["dim"]
    lin = lambda n, heads: (h @ w[p + n].T).reshape(T, heads, -1)
    warm = torch.tensor([1.0 + a["q_temp"]["coef"] * math.log(1 + (t + 1) // a["q_temp"]["every"]) for t in range(T)], device="cuda", dtype=F64)
    q = _rms(lin("left.q", H), eps) * w[p + "left.q.norm"] * warm[:, None, None]
    k = _rms(lin("left.k", G), eps) * w[p + "left.k.norm"]
    o = _softmax_heads(q, k, lin("left.v", G), a["scale"], _hidden(T))
    left = (o * torch.sigmoid(h @ w[p + "left.g"].T)) @ w[p + "left.o"].T
    r, H, D, V = m["right"], m["right"]["heads"], m["right"]["dim"], m["right"]["vdim"]
    turn = lambda x: _turn(x, r["rot"]["dims"], r["rot"]["base"], True)
    keep = torch.tensor(r["decay"], device="cuda", dtype=F64).expand(T, H)
    o, _ = _scan(turn(lin("right.q", H)), turn(lin("right.k", H)) * D ** -0.5, lin("right.v", H), keep, torch.ones_like(keep), _zeros(H, D, V))
    right = (_rms(o, eps).reshape(T, H * V) * _silu(h @ w[p + "right.g"].T)) @ w[p + "right.o"].T
    return m["left_scale"] * left + m["right_scale"] * right


def _fedutar_exact(w, cfg, tokens):
    eps = cfg["norm"]["eps"]
    norm = lambda x, n: _rms(x, eps) * w[n]
    x = w["embed"][tokens] * cfg["embedding"]["scale"]
    for i, l in enumerate(cfg["layers"]):
        p = f"l{i}."
        x = x + norm(_fedutar_mixer(norm(x, p + "norm1"), w, p + "mix.", l["mixer"], eps), p + "norm1b")
        x = x + norm(_dense(norm(x, p + "norm2"), w, p + "mlp.", biases=True), p + "norm2b")
    z = norm(x, "final.norm") @ w["embed"].T * cfg["logit_scale"]
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


LAYERED = {"gedelorn": _gedelorn_exact, "vonedra": _vonedra_exact, "fedutar": _fedutar_exact}


# ------------------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    kind = case["kind"]
    if kind == "sample":
        s = _sample_inputs(case, seed)
    elif kind in ("decode", "prompts"):
        s = _attention_inputs(case, seed)
    elif kind == "mlp":
        s = _mlp_inputs(case, seed)
    elif kind == "decay":
        s = _decay_inputs(case, seed)
    else:
        s = _engine_state(case, seed)
    s["case"] = case
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sample":
        return K.sample(state["logits"], state["temperature"], state["top_k"], state["top_p"], state["seeds"])
    if kind == "decode":
        hi, lo = K.attn_decode(state["q"], state["cache"], state["table"], state["ctx"])
        return _summed(K.gemm_bf16(state["wo"], hi, lo))
    if kind == "prompts":
        hi, lo = K.attn_prefill(state["q"], state["cache"], state["table"], state["starts"], state["slots"], state["pos0"])
        return _summed(K.gemm_bf16(state["wo"], hi, lo))
    if kind == "mlp":
        hi, lo = K.add_rmsnorm(state["resid"], state["norm"], state["eps"])
        hi, lo = K.gemm_bf16(state["wgu"], hi, lo, mode="swiglu")
        return _summed(K.gemm_bf16(state["wd"], hi, lo))
    if kind == "decay":
        return _decay_run(case, state)
    return _engine_run(case, state)


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "sample":
            return None
        if kind in ("decode", "prompts"):
            return _attention_exact(case, seed)
        if kind == "mlp":
            return _mlp_exact(case, seed)
        if kind == "decay":
            return _decay_exact(case, seed)
        return _engine_exact(case, seed)


def work(case):
    """Bytes and operations one pass cannot do without: every input once, every output once; products counted as the model's own."""
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": case["rows"] * (case["vocab"] * 4 + 24), "flops": 2 * case["rows"] * case["vocab"]}
    if kind in ("decode", "prompts"):
        spec = get_spec(MODELS[case["model"]])
        if kind == "decode":
            new, lengths = [1] * case["sessions"], _lengths(case["sessions"], case["context"])
        else:
            new = _lengths(case["sessions"], case["new"])
            lengths = [case["cached"] + n for n in new]
        rows = sum(new)
        seen = sum(n * (l - n) + n * (n + 1) // 2 for n, l in zip(new, lengths))
        kv = sum(lengths) * 2 * spec.kv_dim * 2
        return {"bytes": kv + rows * spec.q_dim * 2 + spec.hidden * spec.q_dim * 2 + rows * spec.hidden * 4,
                "flops": 4 * seen * spec.q_dim + 2 * rows * spec.hidden * spec.q_dim}
    if kind == "mlp":
        spec = get_spec(MODELS[case["model"]])
        return {"bytes": 3 * spec.ffn * spec.hidden * 2 + 2 * case["tokens"] * spec.hidden * 4, "flops": 6 * case["tokens"] * spec.ffn * spec.hidden}
    if kind == "decay":
        H, D, V, T, R = case["heads"], case["dim"], case["vdim"], case["tokens"], min(case["requests"], case["tokens"])
        return {"bytes": 4 * T * H * (2 * D + 2 * V + 2) + 8 * R * H * D * V, "flops": 5 * T * H * D * V}
    lengths = _lengths(case["sessions"], case["prompt"])
    rows = sum(lengths) + case["steps"] * case["sessions"]
    calls = len(_engine_plan(case, 0)[2]) + case["steps"]
    logits = case["sessions"] * (case["steps"] + 1) if case["steps"] else min(64, rows)
    if case["design"] == "llama":
        spec = _llama_spec(case)
        per_layer = (spec.qkv_dim + spec.q_dim + 3 * spec.ffn) * spec.hidden
        params, head = spec.layers * per_layer, spec.vocab * spec.hidden
        active = params
        vocab = spec.vocab
    else:
        W, vocab = case["width"], VOCAB
        mats = {}
        for name, shape in tensor_shapes(_layered_spec(case)[1]).items():
            if len(shape) == 2 and name not in ("embed", "head"):
                mats[name] = shape[0] * shape[1]
        experts = sum(v for k, v in mats.items() if ".mlp.e" in k)
        active = sum(mats.values()) - experts + experts * 2 // 16
        # a step of few rows reads the experts its rows choose: about 1 - (1 - 2/16)^rows of them
        share = 1.0 - (1.0 - 2 / 16) ** case["sessions"] if case["steps"] else 1.0
        params, head = sum(mats.values()) - experts + int(experts * share), vocab * W
    return {"bytes": calls * 2 * (params + head) + logits * vocab * 4, "flops": 2 * rows * active + 2 * logits * head}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return {"differ": 0.01}                   # tokens; a draw that falls on the edge between two of them may go either way
    if kind in ("decode", "prompts"):
        return {"rel": 1e-3}                      # probabilities and their products with the values in fp16
    if kind == "mlp":
        return {"rel": 1.5e-4}                    # activations as two bf16 planes: 16 bits of each
    if kind == "decay":
        return {"rel": 1e-5}                      # 32-bit sums
    if case["design"] == "gedelorn":              # 16 bits of each activation; a row that is close between two experts may take the other
        return {"rel": 2e-2 if "p" in case["order"] else 1e-4}
    # Llama: one fp16 plane in prefill, fp16 attention; Fedutar: bf16 attention; Vonedra: 16 bits of each activation
    return {"rel": {"llama": 5e-3, "fedutar": 1e-3, "vonedra": 1e-4}[case["design"]]}
