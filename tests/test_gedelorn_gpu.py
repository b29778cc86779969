"""The Gedelorn design on the GPU against the plain restatement in oracle/gedelorn_oracle.py.

Every test builds its own small configuration and random weights (none of them a published model's sizes).  Logits are
compared at EVERY position; the engine keeps this family in fp32 on bf16 weights, so the bound is rounding: 1e-4 of the
largest logit in the exact form, a few times that when projections run on the tensor cores from bf16 hi + lo planes.
"""
import json
import os
import subprocess

import numpy as np
import pytest
import torch

from oracle import gedelorn_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-4


# ------------------------------------------------------------------------------------------------ configurations
def memory(heads=3, dim=12, vdim=20, gate_cap=9.0):
    return {"type": "mlstm", "mixer": {"dim": dim, "gate_cap": gate_cap, "heads": heads, "vdim": vdim}}


def space(heads=6, vdim=8, state=12, groups=3, norm_groups=2, conv=4):
    return {"type": "mamba2", "mixer": {"conv": conv, "groups": groups, "heads": heads, "norm_groups": norm_groups,
                                        "state": state, "vdim": vdim}}


def window(heads=6, kv_heads=2, dim=16, size=17, rot=(8, 5000.0), softcap=30.0, scale=0.3):
    m = {"dim": dim, "heads": heads, "kv_heads": kv_heads, "mask": {"size": size}, "scale": scale, "vdim": dim}
    if rot:
        m["rot"] = {"dims": rot[0], "base": rot[1]}
    if softcap:
        m["softcap"] = softcap
    return m


def decaying(heads=3, dim=20, vdim=12, decay=(0.7, 0.95, 0.999)):
    return {"decay": list(decay), "dim": dim, "heads": heads, "vdim": vdim}


def parallel(left=None, right=None, left_scale=0.6, right_scale=1.3):
    return {"type": "parallel", "mixer": {"left": left or window(), "left_scale": left_scale, "right": right or decaying(),
                                          "right_scale": right_scale}}


def dense(ff=72):
    return {"ff": ff, "kind": "dense"}


def moe(ff=24, experts=7, top=3, scale=1.7, shared=40):
    m = {"expert": {"ff": ff}, "kind": "moe", "router": {"experts": experts, "top": top}}
    if scale is not None:
        m["router"]["scale"] = scale
    if shared:
        m["shared"] = {"ff": shared}
    return m


def layer(mixer, mlp=None):
    return {**mixer, "mlp": mlp}


def make(layers, width=80, vocab=150, eps=1e-5, seed=0, tweak=None):
    from fasttalk_llm_microservice_b200.layered import init_weights, spec_from_config
    cfg = {"architecture": "Gedelorn", "layers": layers, "norm": {"eps": eps}, "vocab": vocab, "width": width}
    spec = spec_from_config(cfg, name="test")
    assert spec_from_config(spec.config(), name="test") == spec
    w = init_weights(spec, seed=seed)
    if tweak:
        tweak(w)
    return spec, w


def engine(spec, w, **kw):
    from fasttalk_llm_microservice_b200 import build
    from fasttalk_llm_microservice_b200.engine import Engine, EngineLimits
    build.build()
    lim = EngineLimits(**{"max_batch": 4, "max_batched_tokens": 512, "max_context": 512, "num_pages": 16,
                          "max_sessions": 4, "debug_logit_rows": 512, "exact_f32": True, **kw})
    return Engine(spec, w, lim, eos_ids=())


def oracle_logits(spec, w, tokens):
    with torch.no_grad():
        return O.forward(spec.config(), w, list(tokens)).numpy()


def rel(got, ref):
    return float(np.abs(got - ref).max() / np.abs(ref).max())


def tokens_of(spec, n, seed):
    return np.random.default_rng(seed).integers(0, spec.vocab, n).tolist()


def feed_cut(eng, sid, toks, cuts):
    """Feed `toks` to session `sid` in portions of the given sizes (the last size repeats); logits of every position."""
    out, pos, k = [], 0, 0
    while pos < len(toks):
        n = min(cuts[min(k, len(cuts) - 1)], len(toks) - pos)
        out.append(eng.feed([(sid, toks[pos:pos + n], list(range(n)))]))
        pos, k = pos + n, k + 1
    return np.concatenate(out)


MIXED = [layer(space(), dense()), layer(parallel(), moe()), layer(memory(), dense(ff=33)), layer(space(heads=4, vdim=12, state=8, groups=1, norm_groups=4, conv=2), moe(experts=4, top=2, scale=None, shared=0)),
         layer(parallel(window(heads=2, kv_heads=2, dim=24, size=70, rot=(24, 1e6), softcap=0), decaying(heads=1, dim=8, vdim=40, decay=(0.9,))))]


# ------------------------------------------------------------------------------------------------ every mechanism alone
@pytest.mark.parametrize("layers", [
    [layer(memory())],
    [layer(memory(heads=1, dim=40, vdim=8, gate_cap=4.0))],
    [layer(memory(heads=2, dim=72, vdim=33))],                           # more key channels than one run of lanes holds
    [layer(space())],
    [layer(space(heads=4, vdim=20, state=6, groups=1, norm_groups=1, conv=1))],
    [layer(space(heads=4, vdim=4, state=130, groups=4, norm_groups=4, conv=7))],
    [layer(parallel())],
    [layer(parallel(window(heads=4, kv_heads=4, dim=10, size=1, rot=(10, 100.0), softcap=0), decaying(heads=2, dim=4, vdim=70, decay=(1.0, 0.5))))],
    [layer(parallel(window(heads=3, kv_heads=1, dim=36, size=400, rot=None), left_scale=1.0, right_scale=0.25))],
    [layer(parallel(window(heads=2, kv_heads=1, dim=160, size=90, rot=(64, 1e4), scale=0.08), decaying(heads=1, dim=300, vdim=8, decay=(0.97,))))],
    [layer(parallel(window(heads=1, kv_heads=1, dim=264, size=50, rot=(8, 1e4), scale=0.06), decaying(heads=1, dim=8, vdim=8, decay=(0.9,))))],
    [layer(space(), dense())],
    [layer(memory(), moe())],
    [layer(memory(), moe(experts=3, top=3, shared=0))],                  # every expert chosen, no shared expert
    [layer(memory(), moe(experts=40, top=1, scale=None, shared=9))],     # more experts than lanes, one chosen
    MIXED,
], ids=["memory", "memory-1head", "memory-wide", "space", "space-1group-1tap", "space-big-state", "parallel", "parallel-window1",
        "parallel-norot", "parallel-wide-heads", "parallel-widest-head", "dense", "moe", "moe-all", "moe-top1", "mixed"])
def test_whole_prompt_matches_oracle(layers):
    spec, w = make(layers, seed=3)
    eng = engine(spec, w)
    try:
        toks = tokens_of(spec, 150, 1)
        got = eng.feed([("s", toks, list(range(len(toks))))])
        assert rel(got, oracle_logits(spec, w, toks)) < TOL
    finally:
        eng.close()


def test_other_sizes():
    layers = [layer(parallel(window(heads=10, kv_heads=5, dim=12, size=33, rot=(4, 77.0), softcap=5.0, scale=0.5),
                             decaying(heads=5, dim=6, vdim=14, decay=(0.1, 0.3, 0.5, 0.8, 0.99)), 1.5, 0.5), dense(ff=50)),
              layer(space(heads=9, vdim=6, state=10, groups=3, norm_groups=9, conv=5), moe(ff=10, experts=9, top=5, scale=0.5, shared=3)),
              layer(memory(heads=5, dim=6, vdim=14, gate_cap=20.0))]
    spec, w = make(layers, width=70, vocab=333, eps=1e-6, seed=9)
    eng = engine(spec, w)
    try:
        toks = tokens_of(spec, 90, 2)
        got = eng.feed([("s", toks, list(range(len(toks))))])
        assert rel(got, oracle_logits(spec, w, toks)) < TOL
    finally:
        eng.close()


def test_residual_after_every_layer():
    spec, w = make(MIXED, seed=4)
    eng = engine(spec, w)
    try:
        toks = tokens_of(spec, 70, 5)
        eng.debug_trail(True)
        eng.feed([("s", toks, [])])
        got = eng.read_trail(len(toks))
        trail = []
        with torch.no_grad():
            O.forward(spec.config(), w, toks, trail=trail)
        for i, t in enumerate(trail):
            assert rel(got[i], t.numpy()) < TOL, i
    finally:
        eng.close()


# ------------------------------------------------------------------------------------------------ portions, decoding
@pytest.mark.parametrize("cuts", [[1], [2], [3, 2, 29, 1, 1, 17, 2], [64], [63, 1, 1, 64, 2], [65, 2]],
                         ids=["token-by-token", "twos", "ragged", "pages", "around-pages", "over-a-page"])
def test_portions_and_decoding_match_the_whole_prompt(cuts):
    spec, w = make(MIXED, seed=7)
    eng = engine(spec, w)
    try:
        toks = tokens_of(spec, 200, 8)
        ref = oracle_logits(spec, w, toks)
        whole = eng.feed([("w", toks, list(range(len(toks))))])
        got = feed_cut(eng, "c", toks, cuts)
        assert rel(whole, ref) < TOL and rel(got, ref) < TOL
        assert rel(got, whole) < 2e-5
    finally:
        eng.close()


def sharpen(factor):
    """Queries of every window attention times `factor`: the softmax then rests on one or two keys, so a key that is
    wrongly seen or wrongly hidden (one off at a window's edge, a wrong page) moves the result by far more than rounding."""
    def tweak(w):
        for k in list(w):
            if k.endswith("left.q") or k.endswith("left.q.b"):
                w[k] = (w[k].float() * factor).to(torch.bfloat16)
    return tweak


@pytest.mark.parametrize("size", [2, 5, 63, 64, 65, 129, 1000])
def test_window_edges_with_sharp_attention(size):
    """Windows shorter than, equal to and longer than a page, and longer than the sequence; prompt portions and single
    decoded tokens both cross every edge."""
    layers = [layer(parallel(window(heads=4, kv_heads=2, dim=16, size=size, rot=(16, 10000.0), softcap=0, scale=0.25)))]
    spec, w = make(layers, width=64, seed=11, tweak=sharpen(12.0))
    eng = engine(spec, w)
    try:
        toks = tokens_of(spec, 260, 12)
        ref = oracle_logits(spec, w, toks)
        got = feed_cut(eng, "a", toks, [130, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 60, 1])
        assert rel(got, ref) < TOL
        # the test has teeth: a window one longer or one shorter gives another result
        cfg = spec.config()
        cfg["layers"][0]["mixer"]["left"]["mask"]["size"] = size + 1
        if size < 260:
            with torch.no_grad():
                assert rel(O.forward(cfg, w, toks).numpy(), ref) > 50 * TOL
    finally:
        eng.close()


def test_one_key_just_inside_and_just_outside_the_window():
    """One marked token in a run of equal tokens: the query scaled so that the marked key takes all the weight while it is
    visible.  The logits must change exactly when the marked token leaves the window, in a prompt and in decoding."""
    size = 37
    layers = [layer(parallel(window(heads=2, kv_heads=1, dim=8, size=size, rot=None, softcap=0, scale=1.0), left_scale=1.0, right_scale=0.0))]

    def tweak(w):
        # token 1 is the marked one: its key has a large component that every query of token 0 likes
        w["embed"][:] = 0
        w["embed"][0, 0], w["embed"][1, 1], w["embed"][0, 2], w["embed"][1, 3] = 1.0, 1.0, 0.5, -0.5
        for n in ("l0.mix.left.q", "l0.mix.left.k"):
            w[n][:] = 0
        w["l0.mix.left.q.b"][:] = 0
        w["l0.mix.left.k.b"][:] = 0
        w["l0.mix.left.q"][0, 0] = w["l0.mix.left.q"][8, 0] = 8.0      # token 0's queries point along key channel 0
        w["l0.mix.left.k"][0, 1] = 8.0                                    # only token 1's key has that channel
        w["l0.mix.left.k"][1, 0] = w["l0.mix.left.k"][2, 1] = 1.0         # values (= keys) that tell the two tokens apart
    spec, w = make(layers, width=32, vocab=40, seed=2, tweak=tweak)
    eng = engine(spec, w)
    try:
        mark = 70
        toks = [0] * 200
        toks[mark] = 1
        ref = oracle_logits(spec, w, toks)
        inside, outside = ref[mark + size - 1], ref[mark + size]
        assert np.abs(inside - outside).max() > 1e-2 * np.abs(ref).max()          # the oracle itself sees the edge
        for cuts in ([200], [mark + size - 1, 1, 1, 1], [mark + 3, 1], [64, 2, 2]):
            got = feed_cut(eng, "s", toks, cuts)
            eng.close_session("s")
            assert rel(got, ref) < TOL, cuts
    finally:
        eng.close()


def test_recurrent_branches_remember_a_far_write():
    """Slow decays (a decay of 0.9995 per step; forget gates pushed open; small step sizes): one marked token early in the
    sequence still shows 300 tokens later, across portions and decoded tokens."""
    def tweak(w):
        for k in list(w):
            if k.endswith("f.b"):
                w[k] = (w[k].float() + 8.0).to(torch.bfloat16)
            if k.endswith("dt_bias"):
                w[k] = (w[k].float() - 5.0).to(torch.bfloat16)
    layers = [layer(parallel(window(size=4), decaying(heads=2, dim=12, vdim=12, decay=(0.9995, 0.98)), 0.1, 1.5)), layer(memory()),
              layer(space())]
    spec, w = make(layers, seed=29, tweak=tweak)
    eng = engine(spec, w)
    try:
        toks = [3] * 340
        toks[5] = 77
        ref = oracle_logits(spec, w, toks)
        other = list(toks)
        other[5] = 78
        assert rel(oracle_logits(spec, w, other)[330:], ref[330:]) > 20 * TOL      # the write is still felt at the end
        got = feed_cut(eng, "a", toks, [40, 2, 100, 1, 1, 1, 150, 1])
        assert rel(got, ref) < TOL and rel(got[330:], ref[330:]) < TOL
    finally:
        eng.close()


def test_first_tokens_and_long_decoding():
    spec, w = make(MIXED, seed=19)
    eng = engine(spec, w)
    try:
        toks = tokens_of(spec, 300, 21)
        ref = oracle_logits(spec, w, toks)
        got = feed_cut(eng, "a", toks, [1, 1, 1, 2, 1, 30, 1])      # a sequence that starts with single tokens, then 264 decoded
        assert rel(got[:8], ref[:8]) < TOL
        assert rel(got, ref) < TOL
    finally:
        eng.close()


# ------------------------------------------------------------------------------------------------ batches, pools
@pytest.mark.parametrize("mixer", [memory(), space(), parallel()], ids=["memory", "space", "parallel"])
def test_single_tokens_beside_long_portions(mixer):
    """Decoding sessions beside portions of two whole runs of 128 tokens (and about): the rule takes each kind in a launch of its own."""
    spec, w = make([layer(mixer, dense()), layer(mixer)], seed=17)
    eng = engine(spec, w, max_batched_tokens=768, num_pages=40, debug_logit_rows=768)
    try:
        seqs = {n: tokens_of(spec, ln, 40 + i) for i, (n, ln) in enumerate([("a", 8), ("b", 35), ("c", 259), ("d", 300)])}
        got = {n: [] for n in seqs}
        at = {n: 0 for n in seqs}
        for step in [{"a": 5, "b": 33, "d": 40}, {"a": 1, "b": 1, "c": 256, "d": 257}, {"a": 1, "b": 1, "c": 1, "d": 1}, {"a": 1, "c": 2, "d": 2}]:
            out, o = eng.feed([(n, seqs[n][at[n]:at[n] + c], list(range(c))) for n, c in step.items()]), 0
            for n, c in step.items():
                got[n].append(out[o:o + c])
                o += c
                at[n] += c
        for n, t in seqs.items():
            assert at[n] == len(t)
            assert rel(np.concatenate(got[n]), oracle_logits(spec, w, t)) < TOL, n
    finally:
        eng.close()


def test_unequal_requests_in_one_batch_match_each_alone():
    spec, w = make(MIXED, seed=13)
    eng = engine(spec, w)
    try:
        seqs = {n: tokens_of(spec, ln, 20 + i) for i, (n, ln) in enumerate([("a", 140), ("b", 33), ("c", 70), ("d", 9)])}
        ref = {n: oracle_logits(spec, w, t) for n, t in seqs.items()}
        alone = {}
        for n, t in seqs.items():
            alone[n] = eng.feed([(n + "-alone", t, list(range(len(t))))])
            eng.close_session(n + "-alone")
        # a schedule of mixed steps: portions of some beside single tokens of others, one request pausing for a step
        plan = [{"a": 64, "b": 1}, {"a": 2, "b": 1, "c": 29}, {"b": 16, "c": 1, "d": 3}, {"a": 1, "c": 1, "d": 1},
                {"a": 70, "b": 15, "c": 39, "d": 5}, {"a": 3}]
        at = {n: 0 for n in seqs}
        got = {n: [] for n in seqs}
        for step in plan:
            entries, names = [], []
            for n, cnt in step.items():
                cnt = min(cnt, len(seqs[n]) - at[n])
                if cnt:
                    entries.append((n, seqs[n][at[n]:at[n] + cnt], list(range(cnt))))
                    names.append((n, cnt))
            out = eng.feed(entries)
            o = 0
            for n, cnt in names:
                got[n].append(out[o:o + cnt])
                o += cnt
                at[n] += cnt
        for n in seqs:
            assert at[n] == len(seqs[n])
            g = np.concatenate(got[n])
            assert rel(g, ref[n]) < TOL, n
            assert rel(g, alone[n]) < 2e-5, n
    finally:
        eng.close()


def test_pages_and_state_slots_are_used_again():
    """A pool of 6 pages and 2 slots serves 6 sequences one after the other and two at a time: what an ended session
    left in its pages and its slot (states, running maxima, convolution tails) must not reach the next one."""
    spec, w = make(MIXED, seed=17)
    eng = engine(spec, w, max_batch=2, max_sessions=2, num_pages=6, max_context=384, max_batched_tokens=384,
                 debug_logit_rows=384)
    try:
        seqs = [tokens_of(spec, ln, 40 + i) for i, ln in enumerate([190, 100, 130, 64, 65, 180])]
        ref = [oracle_logits(spec, w, t) for t in seqs]
        for i in (0, 1):                                       # alone, the whole pool in turn
            assert rel(feed_cut(eng, f"s{i}", seqs[i], [50, 1, 1, 90]), ref[i]) < TOL
            eng.close_session(f"s{i}")
            assert eng.stats()["free_pages"] == 6
        for a, b in ((2, 3), (4, 5)):                          # two at a time, the shorter one ends first
            la, lb = len(seqs[a]), len(seqs[b])
            ga, gb, pa, pb = [], [], 0, 0
            while pa < la or pb < lb:
                entries = []
                na, nb = min(37, la - pa), min(1 if pb else 20, lb - pb)
                if na:
                    entries.append((f"s{a}", seqs[a][pa:pa + na], list(range(na))))
                if nb:
                    entries.append((f"s{b}", seqs[b][pb:pb + nb], list(range(nb))))
                out = eng.feed(entries)
                ga.append(out[:na]); gb.append(out[na:na + nb])
                pa, pb = pa + na, pb + nb
                if pa == la and na:
                    eng.close_session(f"s{a}")
                if pb == lb and nb:
                    eng.close_session(f"s{b}")
            assert rel(np.concatenate(ga), ref[a]) < TOL and rel(np.concatenate(gb), ref[b]) < TOL
        st = eng.stats()
        assert st["free_pages"] == 6 and st["live_sessions"] == 0
    finally:
        eng.close()


# ------------------------------------------------------------------------------------------------ tensor cores
TILING = [layer(space(heads=8, vdim=16, state=16, groups=2, norm_groups=2, conv=3), dense(ff=64)),
          layer(parallel(window(heads=4, kv_heads=2, dim=32, size=50, rot=(32, 1e4)), decaying(heads=4, dim=16, vdim=16, decay=(0.5, 0.8, 0.9, 0.99))),
                moe(ff=128, experts=4, top=2, scale=2.0, shared=64)),
          layer(memory(heads=2, dim=16, vdim=64), dense(ff=100))]


@pytest.mark.parametrize("exact", [False, True], ids=["tensor-cores", "exact-fp32"])
def test_projections_on_tensor_cores_and_in_exact_fp32(exact):
    """Shapes that tile (width, heads * vdim and the feed-forward sizes multiples of 64 or 128): with enough rows the input
    and output projections, the dense feed-forward, the shared expert and (from 256 (token, choice) pairs) the experts run
    on the tensor cores from bf16 hi + lo planes unless the engine was made exact; single tokens and short portions take the
    CUDA-core kernels either way, so the two forms must agree along one sequence.  The last layer's feed-forward (100) does
    not tile and stays on the CUDA cores."""
    spec, w = make(TILING, width=128, vocab=256, seed=37)
    eng = engine(spec, w, exact_f32=exact)
    try:
        toks = tokens_of(spec, 200, 38)
        ref = oracle_logits(spec, w, toks)
        got = feed_cut(eng, "a", toks, [150, 1, 1, 12, 3, 10, 1])
        assert rel(got, ref) < (TOL if exact else 4e-4)
    finally:
        eng.close()


# ------------------------------------------------------------------------------------------------ the serving path
def test_greedy_generation_through_the_scheduler():
    """Engine.generate: submit -> the scheduler's own chunked prefill and decode steps -> argmax sampling; three requests
    of unequal length run together, prompts longer than a step's token budget are cut by the scheduler itself."""
    spec, w = make(MIXED, seed=23)
    eng = engine(spec, w, max_batched_tokens=48, decode_prefill_cap=16)
    try:
        prompts = [tokens_of(spec, ln, 60 + i) for i, ln in enumerate([100, 7, 51])]
        n_new = 12
        got = eng.generate(prompts, n_new, temperature=0.0, ignore_eos=True)
        with torch.no_grad():
            for p, g in zip(prompts, got):
                assert g == O.greedy(spec.config(), w, p, n_new)
        # a conversation that continues keeps its state; one that diverges is rebuilt from its start
        eng.close()
        eng = engine(spec, w, max_batched_tokens=48, decode_prefill_cap=16)
        first = eng.generate([prompts[1]], 5, sessions=["gen-1"], temperature=0.0, ignore_eos=True)[0]
        more = prompts[1] + first + tokens_of(spec, 6, 99)
        with torch.no_grad():
            assert eng.generate([more], 4, sessions=["gen-1"], temperature=0.0, ignore_eos=True)[0] == O.greedy(spec.config(), w, more, 4)
            other = tokens_of(spec, 11, 98)
            assert eng.generate([other], 3, sessions=["gen-1"], temperature=0.0, ignore_eos=True)[0] == O.greedy(spec.config(), w, other, 3)
    finally:
        eng.close()


def test_sampling_with_temperature_runs():
    spec, w = make(MIXED, seed=25)
    eng = engine(spec, w)
    try:
        out = eng.generate([tokens_of(spec, 20, 1), tokens_of(spec, 5, 2)], 8, temperature=0.8, top_k=20, top_p=0.9,
                           ignore_eos=True)
        assert [len(o) for o in out] == [8, 8] and all(0 <= t < spec.vocab for o in out for t in o)
    finally:
        eng.close()


def test_trace_runner_replays_a_schedule(tmp_path):
    """bin/trace_run on a saved checkpoint: three steps, a session pausing and two ending, in both number formats."""
    from fasttalk_llm_microservice_b200.layered import save_checkpoint
    spec, w = make(MIXED, seed=31)
    save_checkpoint(spec, w, str(tmp_path / "model"))
    toks = tokens_of(spec, 40, 3)
    steps = [{"step": 0, "entries": [{"id": "x", "tokens": toks[:30], "want": [0, 29]}], "end": []},
             {"step": 1, "entries": [{"id": "x", "tokens": toks[30:31], "want": []}], "end": []},
             {"step": 2, "entries": [{"id": "x", "tokens": toks[31:], "want": [8]}, {"id": "y", "tokens": toks[:5], "want": [4]}],
              "end": ["x", "y"]}]
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for dtype in ("float32", "bfloat16"):
        out = tmp_path / ("out-" + dtype)
        r = subprocess.run([os.path.join(root, "bin", "trace_run"), "--model", str(tmp_path / "model"), "--dtype", dtype,
                            "--out", str(out), "--max-tokens", "128"], input="\n".join(json.dumps(s) for s in steps) + "\n",
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        assert [l for l in r.stdout.splitlines() if l.startswith("done")] == ["done 0", "done 1", "done 2"]
        ref = oracle_logits(spec, w, toks)
        a = np.fromfile(out / "0.f32", dtype="<f4").reshape(2, spec.vocab)
        c = np.fromfile(out / "2.f32", dtype="<f4").reshape(2, spec.vocab)
        assert not (out / "1.f32").exists()
        tol = TOL if dtype == "float32" else 4e-4
        assert rel(a, ref[[0, 29]]) < tol and rel(c[0], ref[39]) < tol and rel(c[1], ref[4]) < tol


def test_served_through_the_handler(tmp_path, monkeypatch):
    """A Gedelorn checkpoint behind the serving path: FASTTALK_CHECKPOINT -> registry -> engine -> NativeHandler streams text."""
    from fasttalk_llm_microservice_b200.handler import NativeHandler, build_runner
    from fasttalk_llm_microservice_b200.layered import save_checkpoint
    spec, w = make([layer(space(), moe()), layer(parallel(), dense()), layer(memory())], width=64, vocab=600, seed=41)
    save_checkpoint(spec, w, str(tmp_path / "ckpt"))
    monkeypatch.setenv("FASTTALK_CHECKPOINT", str(tmp_path / "ckpt"))
    monkeypatch.setenv("FASTTALK_ALLOW_BYTE_TOKENIZER", "1")
    monkeypatch.setenv("FASTTALK_MAX_SESSIONS", "4")
    monkeypatch.setenv("FASTTALK_MAX_CONTEXT", "512")
    monkeypatch.setenv("FASTTALK_MAX_BATCHED_TOKENS", "256")
    runner = build_runner("gedelorn-test")
    h = NativeHandler(model="gedelorn-test", runner=runner)
    try:
        assert h.check_connection()
        chunks = list(h.generate_stream([{"role": "user", "content": "hello there"}], temperature=0.0, max_tokens=12,
                                        request_id="conv-1"))
        assert 1 <= len(chunks) <= 12
        st = h.runner.engine.stats()
        assert st["prefill_tokens"] > 0 and st["decode_tokens"] > 0
    finally:
        h.close()
        runner.shutdown()
        runner.engine.close()


@pytest.mark.parametrize("width,ff,experts,top,sessions", [(520, 512, 8, 3, 2), (520, 1032, 7, 7, 1), (1032, 2056, 3, 2, 7), (3208, 1024, 5, 1, 4), (4104, 512, 2, 1, 1)])
def test_experts_of_a_few_pairs(width, ff, experts, top, sessions):
    """Pairs that go past weights in shared memory: experts without a pair, with one, and with two groups of four rows; sixteen and eight weight rows a CTA."""
    spec, w = make([layer(memory(), moe(ff=ff, experts=experts, top=top, shared=0))], width=width, vocab=90, seed=ff)
    eng = engine(spec, w, max_batch=8, max_sessions=8)
    try:
        toks = [tokens_of(spec, 3, 50 + i) for i in range(sessions)]
        got = np.stack([eng.feed([(i, [t[j]], [0]) for i, t in enumerate(toks)]) for j in range(3)], 1)
        for i, t in enumerate(toks):
            assert rel(got[i], oracle_logits(spec, w, t)) < TOL
    finally:
        eng.close()


@pytest.mark.parametrize("dim,scale,cap", [(64, 1.0, 6.0), (64, 1.0, 18.0), (64, 1.0, 60.0), (128, 0.3, 10.0), (128, 1.0, 0.0)])
def test_window_of_portions_in_fp32_accuracy(dim, scale, cap):
    """A prompt as a whole (matrix products of slices, caps on both sides of 0.6) is no further from 64 bits than its tokens one by one (fp32 multiply-adds):
    the quarter is for another order of sums.  A slice or a term of the small tanh less would be tens of times off."""
    spec, w = make([layer(parallel(window(heads=4, kv_heads=2, dim=dim, size=200, rot=(16, 5000.0), softcap=cap, scale=scale)))], width=256, seed=dim)
    toks = tokens_of(spec, 400, 4)
    ref = oracle_logits(spec, w, toks)
    eng = engine(spec, w)
    try:
        off = lambda x: np.linalg.norm(x - ref)
        assert off(eng.feed([("whole", toks, list(range(400)))])) < 1.25 * off(feed_cut(eng, "single", toks, [1]))
    finally:
        eng.close()


# ------------------------------------------------------------------------------------------------ the rule alone
@pytest.mark.parametrize("lanes", [0, 4, 8, 16, 32])
@pytest.mark.parametrize("heads,qk_heads,dim,vd", [(3, 3, 20, 9), (4, 2, 64, 33), (2, 1, 128, 16), (1, 1, 7, 70)])
def test_decay_rule_kernel_alone(lanes, heads, qk_heads, dim, vd):
    """ft_decay_rule against the recurrence written out: three requests of unequal length in one launch, one of them
    continuing from a state that its slot already holds, every split of a column over lanes."""
    from fasttalk_llm_microservice_b200 import build, native
    build.build()
    lib = native.load()
    min_lanes = 4
    while min_lanes * 16 < dim and min_lanes < 32:      # runs of at most 16 channels per lane (32 beyond 512 channels)
        min_lanes *= 2
    if lanes and lanes < min_lanes:
        pytest.skip("fewer lanes than the channels need")
    g = torch.Generator().manual_seed(dim * 131 + vd)
    lens, pos0, slots = [37, 1, 90], [0, 5, 0], [2, 0, 1]
    T = sum(lens)
    q, k = torch.randn(T, qk_heads * dim, generator=g) * 0.3, torch.randn(T, qk_heads * dim, generator=g) * 0.3
    v = torch.randn(T, heads * vd, generator=g)
    ab = torch.stack([torch.rand(T, heads, generator=g) * 0.5 + 0.5, torch.rand(T, heads, generator=g) * 2.0], -1).contiguous()
    stride = heads * dim * vd + 4
    state = torch.randn(3 * stride, generator=g)
    ref_o = torch.zeros(T, heads * vd, dtype=torch.float64)
    ref_state = state.double().clone()
    start = [0, lens[0], lens[0] + lens[1], T]
    for r in range(3):
        for h in range(heads):
            S = ref_state[slots[r] * stride + h * dim * vd:][:dim * vd].reshape(dim, vd).clone()
            if pos0[r] == 0:
                S.zero_()
            gh = h // (heads // qk_heads)
            for t in range(start[r], start[r + 1]):
                S = ab[t, h, 0].double() * S + ab[t, h, 1].double() * torch.outer(k[t, gh * dim:(gh + 1) * dim].double(), v[t, h * vd:(h + 1) * vd].double())
                ref_o[t, h * vd:(h + 1) * vd] = S.T @ q[t, gh * dim:(gh + 1) * dim].double()
            ref_state[slots[r] * stride + h * dim * vd:][:dim * vd] = S.reshape(-1)
    dev = "cuda"
    dq, dk, dv, dab, dst = q.to(dev), k.to(dev), v.to(dev), ab.to(dev), state.to(dev)
    o = torch.zeros(T, heads * vd, device=dev)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    rs, rp, sl = i32(start), i32(pos0), i32(slots)
    rc = lib.ft_decay_rule(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dab.data_ptr(), o.data_ptr(), dst.data_ptr(), rs.data_ptr(),
                           rp.data_ptr(), sl.data_ptr(), 3, heads, qk_heads, dim, vd, stride, lanes, T, None)
    torch.cuda.synchronize()
    assert rc == 0, native.last_error()
    assert rel(o.cpu().double().numpy(), ref_o.numpy()) < 1e-5
    assert rel(dst.cpu().double().numpy(), ref_state.numpy()) < 1e-5


@pytest.mark.parametrize("heads,qk_heads,dim,vd,pad", [(2, 2, 128, 128, 0), (3, 1, 96, 80, 0), (2, 2, 64, 65, 0), (2, 1, 65, 9, 1), (1, 1, 20, 129, 3), (2, 1, 128, 257, 0)])
@pytest.mark.parametrize("odd", ["", "infinite", "growing"])
def test_decay_rule_portions(heads, qk_heads, dim, vd, pad, odd):
    """Runs of 128 tokens on the tensor cores: ends of runs one token short, whole, one too long and around the length below which they go
    token by token, fresh and continued states, decays of zero and one, rows of very different size, slots and columns off 16 bytes; runs
    with infinities and NaN (which must not reach an earlier token or another head) or decays beyond one."""
    from fasttalk_llm_microservice_b200 import build, native
    build.build()
    lib = native.load()
    g = torch.Generator(device="cuda").manual_seed(dim * 7 + vd)
    dev = "cuda"
    lens = [127, 128, 129, 128 + 15, 128 + 16, 300, 1]
    T, R = sum(lens), len(lens)
    start = [sum(lens[:i]) for i in range(R + 1)]
    rnd = lambda *s: torch.randn(*s, device=dev, generator=g)
    size = torch.exp2(torch.randint(-12, 13, (T, 1, 1), device=dev, generator=g).float())
    q, k = (rnd(T, qk_heads, dim) * dim ** -0.5 * size), rnd(T, qk_heads, dim) * size.flip(0)
    v, ab = rnd(T, heads, vd), torch.rand(T, heads, 2, device=dev, generator=g)
    ab[::97, :, 0], ab[5::31, :, 0], ab[11::53, :, 0] = 0.0, 1.0, 1.0 + 2.0 ** -20
    if odd == "infinite":
        v[40, 0, 3], k[start[2] + 100, 0, 1], q[start[5] + 10, 0, 0] = float("inf"), float("nan"), float("-inf")
    if odd == "growing":
        ab[start[4] + 50, :, 0] = 1.5
    stride = heads * dim * vd + pad
    state = rnd(R * stride)
    pos0 = [0 if r % 2 else 11 for r in range(R)]
    ref_o, ref_state = torch.zeros(T, heads, vd, dtype=torch.float64, device=dev), state.double().clone()
    abs_o, abs_state = torch.zeros_like(ref_o), ref_state.clone()      # the same sums of absolute values
    q64, k64 = (x.double().repeat_interleave(heads // qk_heads, 1) for x in (q, k))
    for r in range(R):
        S = ref_state[r * stride:r * stride + heads * dim * vd].reshape(heads, dim, vd) * (pos0[r] > 0)
        A = S.abs()
        for t in range(start[r], start[r + 1]):
            put = k64[t][:, :, None] * (ab[t, :, 1:].double() * v[t].double())[:, None, :]
            S, A = ab[t, :, 0].double()[:, None, None] * S + put, ab[t, :, 0].double()[:, None, None] * A + put.abs()
            ref_o[t], abs_o[t] = (S * q64[t][:, :, None]).sum(1), (A * q64[t][:, :, None].abs()).sum(1)
        ref_state[r * stride:r * stride + heads * dim * vd] = S.reshape(-1)
        abs_state[r * stride:r * stride + heads * dim * vd] = A.reshape(-1)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    rs, rp, sl = i32(start), i32(pos0), i32(list(range(R)))
    o = torch.full((T, heads, vd), 7.0, device=dev)
    rc = lib.ft_decay_rule(q.data_ptr(), k.data_ptr(), v.data_ptr(), ab.data_ptr(), o.data_ptr(), state.data_ptr(), rs.data_ptr(), rp.data_ptr(),
                           sl.data_ptr(), R, heads, qk_heads, dim, vd, stride, 0, T, None)
    torch.cuda.synchronize()
    assert rc == 0, native.last_error()
    states = lambda x: x[:R * stride].reshape(R, stride)[:, :heads * dim * vd]
    for got, ref, size, rows in ((o, ref_o, abs_o, T * heads), (states(state), states(ref_state), states(abs_state), R * heads)):
        got, ref, size = got.double().reshape(rows, -1), ref.reshape(rows, -1), size.reshape(rows, -1)
        assert torch.equal(torch.isfinite(got), torch.isfinite(ref))
        fin = torch.isfinite(ref).all(1) & torch.isfinite(size).all(1)
        assert fin.any() and (odd == "infinite") == (not fin.all())
        # a row (a token's head, a state) against the sum of its terms' sizes: eight times the rounding of one fp32 number
        err = (got[fin] - ref[fin]).norm(dim=1) / size[fin].norm(dim=1).clamp_min(1e-30)
        assert err.max() < 8 * 2.0 ** -24, err.max()
    if pad:
        assert torch.equal(state.reshape(R, stride)[:, -pad:].double(), ref_state.reshape(R, stride)[:, -pad:])


@pytest.mark.parametrize("what", ["columns", "tokens", "state", "later", "behind a zero decay", "keys", "small"])
@pytest.mark.parametrize("size", [10, 20, 30])
def test_decay_rule_portions_by_element(what, size):
    """Every number by itself against 64 bits, beside numbers 2^size as large: columns of the values, tokens, states, a later token, one that a decay
    of zero has removed, channels of the keys; and everything small.  What an element does not depend on leaves no trace in it, and what it depends on
    counts with the sizes of its own terms."""
    from fasttalk_llm_microservice_b200 import build, native
    build.build()
    lib = native.load()
    dev, heads, dim, vd = "cuda", 2, 128, 96
    g = torch.Generator(device=dev).manual_seed(size * 11 + len(what))
    lens = [300, 128, 77]
    T, R = sum(lens), len(lens)
    start = [sum(lens[:i]) for i in range(R + 1)]
    rnd = lambda *s: torch.randn(*s, device=dev, generator=g)
    q, k, v, ab = rnd(T, heads, dim) * dim ** -0.5, rnd(T, heads, dim), rnd(T, heads, vd), 1 - 0.2 * torch.rand(T, heads, 2, device=dev, generator=g) ** 2
    state, big, plain = rnd(R, heads, dim, vd), 2.0 ** size, v.clone()
    some = lambda *s: torch.rand(*s, device=dev, generator=g) < 0.2
    if what == "columns":
        v *= torch.where(some(heads, vd), big, 1.0)
    elif what == "tokens":
        v *= torch.where(some(T, 1, 1), big, 1.0)
        q *= torch.where(some(T, 1, 1), big, 1.0)
    elif what == "state":
        state *= torch.where(some(R, heads, dim, 1), big, 1.0)
    elif what == "later":
        for r in range(R):
            v[start[r] + 70] *= big
    elif what == "behind a zero decay":
        for r in range(R):
            v[start[r] + 20] *= big
            ab[start[r] + 23, :, 0] = 0.0
    elif what == "keys":
        k *= torch.where(some(heads, dim), big, 1.0)
    else:
        q, k, v, state = q / big, k / big, v / big, state / big ** 2
    pos0 = [5, 0, 9]
    ref_o, abs_o = (torch.zeros(T, heads, vd, dtype=torch.float64, device=dev) for _ in range(2))
    ref_s, abs_s = (torch.zeros(R, heads, dim, vd, dtype=torch.float64, device=dev) for _ in range(2))
    for r in range(R):
        S = state[r].double() * (pos0[r] > 0)
        A = S.abs()
        for t in range(start[r], start[r + 1]):
            put = k[t].double()[:, :, None] * (ab[t, :, 1:].double() * v[t].double())[:, None, :]
            S, A = ab[t, :, 0].double()[:, None, None] * S + put, ab[t, :, 0].double()[:, None, None] * A + put.abs()
            ref_o[t], abs_o[t] = (S * q[t].double()[:, :, None]).sum(1), (A * q[t].double()[:, :, None].abs()).sum(1)
        ref_s[r], abs_s[r] = S, A
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    rs, rp, sl = i32(start), i32(pos0), i32(list(range(R)))

    def rule(v, state):
        o = torch.full((T, heads, vd), 7.0, device=dev)
        rc = lib.ft_decay_rule(q.data_ptr(), k.data_ptr(), v.data_ptr(), ab.data_ptr(), o.data_ptr(), state.data_ptr(), rs.data_ptr(), rp.data_ptr(),
                               sl.data_ptr(), R, heads, heads, dim, vd, heads * dim * vd, 0, T, None)
        torch.cuda.synchronize()
        assert rc == 0, native.last_error()
        return o
    other = rule(plain, state.clone())
    o = rule(v, state)
    if what == "later":
        for r in range(R):
            assert torch.equal(o[start[r]:start[r] + 70], other[start[r]:start[r] + 70])
    # Token by token a number passes up to 300 roundings of half of 2^-23 of its size, in random directions; by runs of 128 fewer of them, and sums of 128 products cut
    # off by up to 2^-24 of the largest.  64 * 2^-24 holds either way of summing; operands that lost a slice's last eight bits would be off by 2^-16.
    for got, ref, size_ in ((o, ref_o, abs_o), (state, ref_s, abs_s)):
        err = ((got.double() - ref).abs() / size_.clamp_min(1e-300)).max()
        assert err < 64 * 2.0 ** -24, float(err) * 2 ** 24


@pytest.mark.parametrize("heads,qk_heads,dim,vd,pad", [(2, 2, 128, 128, 0), (3, 1, 96, 80, 0), (4, 2, 64, 257, 0), (2, 1, 7, 20, 1), (1, 1, 513, 1, 0)])
def test_decay_rule_single_tokens(heads, qk_heads, dim, vd, pad):
    """One token per request (units of four columns and of one, slots that break the 16-byte rows, fresh and continued states), and a
    request of several tokens in a launch whose caller named fewer rows."""
    from fasttalk_llm_microservice_b200 import build, native
    build.build()
    lib = native.load()
    g = torch.Generator().manual_seed(dim + vd)
    dev = "cuda"
    for lens, rows in (([1] * 5, 5), ([1, 3, 1], 3)):
        T, R = sum(lens), len(lens)
        pos0 = [0 if r % 2 else 11 for r in range(R)]
        q, k = torch.randn(T, qk_heads * dim, generator=g) * dim ** -0.5, torch.randn(T, qk_heads * dim, generator=g)
        v = torch.randn(T, heads * vd, generator=g)
        ab = torch.rand(T, heads, 2, generator=g).contiguous()
        stride = heads * dim * vd + pad
        state = torch.randn(R * stride, generator=g)
        start = [0] + [sum(lens[:i + 1]) for i in range(R)]
        ref_o, ref_state = torch.zeros(T, heads, vd, dtype=torch.float64), state.double().clone()
        rep = lambda x: x.double().reshape(T, qk_heads, dim).repeat_interleave(heads // qk_heads, 1)
        q64, k64, v64 = rep(q), rep(k), v.double().reshape(T, heads, vd)
        for r in range(R):
            S = ref_state[r * stride:r * stride + heads * dim * vd].reshape(heads, dim, vd) * (pos0[r] > 0)
            for t in range(start[r], start[r + 1]):
                S = ab[t, :, 0].double()[:, None, None] * S + (ab[t, :, 1].double()[:, None] * k64[t])[:, :, None] * v64[t][:, None, :]
                ref_o[t] = torch.einsum("hdv,hd->hv", S, q64[t])
            ref_state[r * stride:r * stride + heads * dim * vd] = S.reshape(-1)
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
        rs, rp, sl = i32(start), i32(pos0), i32(list(range(R)))
        dq, dk, dv, dab, dst = q.to(dev), k.to(dev), v.to(dev), ab.to(dev), state.to(dev)
        o = torch.zeros(T, heads * vd, device=dev)
        rc = lib.ft_decay_rule(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dab.data_ptr(), o.data_ptr(), dst.data_ptr(), rs.data_ptr(),
                               rp.data_ptr(), sl.data_ptr(), R, heads, qk_heads, dim, vd, stride, 0, rows, None)
        torch.cuda.synchronize()
        assert rc == 0, native.last_error()
        # 24-bit sums of dim terms
        assert rel(o.cpu().double().numpy(), ref_o.reshape(T, -1).numpy()) < 2e-6
        assert rel(dst.cpu().double().numpy(), ref_state.numpy()) < 1e-6


@pytest.mark.parametrize("R,heads,dim,vd", [(1, 2, 256, 256), (1, 1, 512, 64), (2, 3, 512, 12), (5, 16, 32, 1024), (3, 8, 16, 1024), (40, 8, 16, 64), (80, 32, 40, 64), (3, 2, 128, 33)])
def test_decay_rule_single_tokens_by_grid(R, heads, dim, vd):
    """Units per CTA from 4 to 128 by channels, columns and grid, and many small states, which take the kernel by lanes."""
    from fasttalk_llm_microservice_b200 import build, native
    build.build()
    lib = native.load()
    g = torch.Generator(device="cuda").manual_seed(dim + vd)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = rnd(R, heads * dim) * dim ** -0.5, rnd(R, heads * dim), rnd(R, heads * vd)
    ab = torch.rand(R, heads, 2, device="cuda", generator=g)
    state = rnd(R, heads, dim, vd)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    pos0 = i32([0 if r % 2 else 11 for r in range(R)])
    S = ab.double()[:, :, :1, None] * state.double() * (pos0 > 0)[:, None, None, None]
    S = S + (ab.double()[:, :, 1:] * k.double().reshape(R, heads, dim))[..., None] * v.double().reshape(R, heads, 1, vd)
    ref = torch.einsum("rhdv,rhd->rhv", S, q.double().reshape(R, heads, dim))
    o = torch.zeros(R, heads * vd, device="cuda")
    start, slot = i32(list(range(R + 1))), i32(list(range(R)))
    rc = lib.ft_decay_rule(q.data_ptr(), k.data_ptr(), v.data_ptr(), ab.data_ptr(), o.data_ptr(), state.data_ptr(), start.data_ptr(), pos0.data_ptr(),
                           slot.data_ptr(), R, heads, heads, dim, vd, heads * dim * vd, 0, R, None)
    torch.cuda.synchronize()
    assert rc == 0, native.last_error()
    # 24-bit sums of dim terms
    assert rel(o.cpu().double().numpy(), ref.reshape(R, -1).cpu().numpy()) < 2e-6
    assert rel(state.cpu().double().numpy(), S.cpu().numpy()) < 1e-6


def test_short_taps_do_not_reach_an_infinite_row_further_back():
    """A convolution of two taps in a step of more than 64 tokens: state coordinates to read out with that overflow at one token
    spoil that token and the next, no more."""
    m = space(heads=4, vdim=8, state=12, groups=1, norm_groups=1, conv=2)
    spec, w = make([layer(m)], seed=8)
    w["embed"][:, 0] = 0.0
    w["embed"][5] = 0.0
    w["embed"][5, 0] = 1.0
    inner, n = 32, 12
    w["l0.mix.in"][:, 0] = 0.0
    w["l0.mix.in"][2 * inner + n:2 * inner + 2 * n, 0] = 3e38
    toks = [t if t != 5 else 6 for t in tokens_of(spec, 90, 2)]
    toks[42] = 5
    with torch.no_grad():
        ref = O.forward(spec.config(), w, toks, dtype=torch.float32).numpy()
    clean = [i for i in range(90) if i not in (42, 43)]
    assert np.isfinite(ref[clean]).all() and not np.isfinite(ref[42]).all()
    eng = engine(spec, w)
    try:
        got = eng.feed([("s", toks, list(range(90)))])
        assert rel(got[clean], ref[clean]) < TOL
    finally:
        eng.close()


@pytest.mark.parametrize("heads,dim,vdim,rot", [(3, 16, 2, 4), (2, 32, 66, 32), (1, 64, 130, 12), (2, 128, 256, 128), (1, 128, 510, 64)])
def test_rows_by_four_channels(heads, dim, vdim, rot):
    """Four taps and rows on 16 bytes: the state space's convolution, queries and cache rows and the matrix memory's read-out over their sizes.  Blocks of eight
    tokens that hold one request, two, its first three tokens, a short last one; tokens whose taps reach into the state of an earlier step."""
    spec, w = make([layer(space(heads=2 * heads, vdim=8, state=12, groups=heads, norm_groups=1), dense()), layer(memory(heads=heads, dim=dim, vdim=vdim)),
                    layer(parallel(window(heads=2 * heads, kv_heads=heads, dim=dim, rot=(rot, 1e4), scale=dim ** -0.5)), dense())], width=84, seed=dim + vdim)
    eng = engine(spec, w)
    try:
        seqs = {n: tokens_of(spec, ln, 40 + i) for i, (n, ln) in enumerate([("a", 203), ("b", 81), ("c", 142)])}
        at, got = {n: 0 for n in seqs}, {n: [] for n in seqs}
        for step in [{"a": 65}, {"a": 1, "b": 2, "c": 70}, {"a": 64, "b": 1, "c": 1}, {"a": 3, "b": 78, "c": 2}, {"a": 70, "c": 69}]:
            out, o = eng.feed([(n, seqs[n][at[n]:at[n] + c], list(range(c))) for n, c in step.items()]), 0
            for n, c in step.items():
                got[n].append(out[o:o + c])
                o += c
                at[n] += c
        for n in seqs:
            assert rel(np.concatenate(got[n]), oracle_logits(spec, w, seqs[n])) < TOL, n
    finally:
        eng.close()


def test_steps_of_single_tokens_out_of_graphs():
    """Steps of single tokens with the same numbers of rows are recorded at the third and replayed; other numbers in between, other sessions and other wanted
    rows under the same number, portions beside: all as the whole prompts give them."""
    spec, w = make(MIXED, seed=29)
    eng = engine(spec, w, max_batch=20, max_sessions=20, num_pages=24)
    try:
        names = [f"s{i}" for i in range(18)]
        seqs = {n: tokens_of(spec, 90 if i < 6 else 60, 70 + i) for i, n in enumerate(names)}
        ref = {n: oracle_logits(spec, w, t) for n, t in seqs.items()}
        at = dict.fromkeys(names, 0)

        def step(which, counts=None, wanted=None):
            counts = counts or [1] * len(which)
            entries = [(n, seqs[n][at[n]:at[n] + c], list(range(c)) if wanted is None or n in wanted else []) for n, c in zip(which, counts)]
            out, o = eng.feed(entries), 0
            for (n, t, rows) in entries:
                for r in rows:
                    assert rel(out[o], ref[n][at[n] + r]) < TOL, (n, at[n] + r)
                    o += 1
                at[n] += len(t)
        step(names[:4], [3, 5, 2, 7])
        step(names[4:], [2] * 14)
        for k in range(6):
            step(names[:4])
        assert eng.step_graphs() == {"kept": 1, "recorded": 1, "replayed": 4, "refused": 0}
        step(names[2:6])                       # the same shape, other sessions in other places
        assert eng.step_graphs()["replayed"] == 5
        step(names[:4], wanted=names[1:2])     # fewer wanted rows
        step(names[:4], wanted=names[2:3])
        step(names[:4], wanted=names[3:4])
        step(names[:5], [1, 1, 1, 1, 20])      # beside a portion
        for n in range(1, 19):                 # many shapes, none of them often: none is worth a recording
            step(names[:n])
            step(names[:n])
        got = eng.step_graphs()
        assert got["recorded"] == 1 and got["refused"] == 0
        for k in range(3):
            step(names[:4])
        assert eng.step_graphs()["replayed"] == got["replayed"] + 3
    finally:
        eng.close()


def test_step_graphs_are_kept_replaced_and_left_for_the_trail():
    """Against an engine that records nothing (its trail is on), bit by bit: more shapes than are kept, one that takes the place of one which has not come for long,
    the trail turned on and off between replays."""
    spec, w = make([layer(space(), dense()), layer(parallel())], seed=30)
    kw = dict(max_batch=6, max_sessions=6, max_context=4096, num_pages=300)
    eng, plain = engine(spec, w, **kw), engine(spec, w, **kw)
    try:
        plain.debug_trail(True)
        rng = np.random.default_rng(5)

        def step(n, wanted):
            entries = [(s, [int(rng.integers(spec.vocab))], [0] if s < wanted else []) for s in range(n)]
            a, b = eng.feed(entries), plain.feed(entries)
            assert np.array_equal(a, b), (n, wanted)

        for e in (eng, plain):
            e.feed([(s, list(range(s + 2)), []) for s in range(6)])
        for k in range(10):
            step(3, 3)
        assert eng.step_graphs() == {"kept": 1, "recorded": 1, "replayed": 8, "refused": 0}
        eng.debug_trail(True)
        step(3, 3)
        assert np.array_equal(eng.read_trail(3), plain.read_trail(3))
        eng.debug_trail(False)
        step(3, 3)
        assert eng.step_graphs()["replayed"] == 9
        shapes = [(n, w) for n in range(1, 7) for w in range(1, n + 1)][:20]
        for n, w in shapes:
            step(n, w), step(n, w)
        assert eng.step_graphs()["recorded"] == 1
        for n, w in shapes:
            for k in range(36):
                step(n, w)
        got = eng.step_graphs()
        assert got["kept"] == got["recorded"] == 16 and got["refused"] == 0
        for k in range(1025):
            step(2, 2)
        for k in range(3):                     # a shape that came often enough before, without a place then
            step(*shapes[-1])
        got = eng.step_graphs()
        assert got["kept"] == 16 and got["recorded"] == 17 and got["refused"] == 0
        assert plain.step_graphs() == {"kept": 0, "recorded": 0, "replayed": 0, "refused": 0}
    finally:
        eng.close()
        plain.close()


@pytest.mark.parametrize("heads,vdim,groups", [(27, 76, 1), (54, 76, 2), (32, 128, 1), (41, 100, 1), (64, 64, 1), (64, 128, 1)])
@pytest.mark.parametrize("exact", [True, False], ids=["rows", "planes"])
def test_read_out_of_long_rows(heads, vdim, groups, exact):
    """Norm groups of more than 2048 columns, 2052 to 8192: with a gate before the norm and a skip (state space), with a gate behind the norm (decay attention); as fp32
    rows and, where the projection behind takes them, as the bf16 planes of long portions."""
    spec, w = make([layer(space(heads=heads, vdim=vdim, state=6, groups=1, norm_groups=groups)),
                    layer(parallel(right=decaying(heads=heads, dim=4, vdim=vdim, decay=[0.5 + 0.49 * h / heads for h in range(heads)])))], width=128, seed=heads + vdim)
    eng = engine(spec, w, exact_f32=exact)
    try:
        toks = tokens_of(spec, 47, heads)
        assert rel(feed_cut(eng, "s", toks, [40, 1, 1, 5]), oracle_logits(spec, w, toks)) < (TOL if exact else 4e-4)
    finally:
        eng.close()
