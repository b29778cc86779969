"""Whole-path parity: the native engine (through the C ABI) against the fp32 oracle and the
transformers-generated golden vectors.

Tolerance: logits within 2e-2 relative in bf16 — measured here as
max|delta| / max|logit| per position — and greedy tokens identical to the fp32 reference.
"""
import os

import numpy as np
import pytest
import torch

from oracle import llama_oracle as O
from oracle import parity as P

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")
LOGIT_TOL = P.LOGIT_TOL


def make_engine(spec, w, **kw):
    from fasttalk_llm_microservice_b200 import build
    from fasttalk_llm_microservice_b200.engine import Engine, EngineLimits
    build.build()
    lim = EngineLimits(**{"max_batch": 8, "max_batched_tokens": 256, "max_context": 1024,
                          "debug_logit_rows": 64, **kw})
    return Engine(spec, w, lim, eos_ids=())


def per_pos_rel(got, ref):
    """The "2e-2 relative": worst position of max|delta| / max|logit|."""
    return ((got - ref).abs().amax(-1) / ref.abs().amax(-1)).max().item()


def describe_err(tag, got, ref):
    e = (got - ref).abs().amax(-1) / ref.abs().amax(-1)
    l2 = (got - ref).norm(dim=-1) / ref.norm(dim=-1)
    print(f"\n[{tag}] logits rel err (max-norm) max {e.max():.3e} mean {e.mean():.3e}; "
          f"L2-rel max {l2.max():.3e} mean {l2.mean():.3e}")


def greedy_parity(eng, tag, prompt, ref_tokens, ref_logits, session=None):
    """Greedy tokens vs the fp32 oracle's over ALL positions (oracle/parity.py): teacher-forced logits at
    every step, a mismatch only where the oracle's margin is within 3x the measured logit error (floor
    5e-4 of the logit scale), the engine re-aligned on the oracle's token afterwards, counts asserted."""
    return P.check(eng, tag, session or f"parity-{tag}", list(prompt), list(ref_tokens), ref_logits.cpu())


@pytest.fixture(scope="module", params=["tiny-d64", "tiny-d128"])
def tiny(request):
    from fasttalk_llm_microservice_b200.model_spec import SPECS
    from fasttalk_llm_microservice_b200.weights import init_weights
    g = np.load(os.path.join(GOLD, f"hf_{request.param}.npz"))
    spec = SPECS[request.param]
    w = init_weights(spec, seed=int(g["seed"]), std=float(g["std"]), norm_jitter=float(g["norm_jitter"]))
    eng = make_engine(spec, w)
    yield spec, w, g, eng
    eng.close()


def test_prefill_logits_match_golden(tiny):
    spec, w, g, eng = tiny
    prompt = g["prompt"].tolist()
    gold = torch.from_numpy(g["logits"])
    for chunk in (64, 16, 7):
        got = eng.debug_prefill_logits(prompt, chunk=chunk)
        describe_err(f"{spec.name} chunk {chunk}", got, gold)
        assert per_pos_rel(got, gold) < LOGIT_TOL, (chunk, per_pos_rel(got, gold))


def test_greedy_matches_golden(tiny):
    spec, w, g, eng = tiny
    n = len(g["greedy"])
    with torch.no_grad():
        ref_tokens, ref_logits = O.greedy_generate(w, spec, torch.from_numpy(g["prompt"]), n, return_logits=True)
    assert ref_tokens == g["greedy"].tolist()
    greedy_parity(eng, f"{spec.name} golden prompt", g["prompt"].tolist(), ref_tokens, ref_logits)


def test_long_prompt_chunked_and_decode_logits(tiny):
    """A 700-token prompt (several prefill chunks of 256, many KV pages) then decode; the
    per-step decode logits are compared with the oracle's."""
    spec, w, g, eng = tiny
    gen = torch.Generator().manual_seed(21)
    prompt = torch.randint(0, spec.vocab, (700,), generator=gen)
    with torch.no_grad():
        ref_tokens, ref_logits = O.greedy_generate(w, spec, prompt, 12, return_logits=True)
    pre0 = eng.stats()["prefill_tokens"]
    job = greedy_parity(eng, spec.name + " 700-token prompt", prompt.tolist(), ref_tokens, ref_logits)
    assert job.errs_checked >= 11 and job.worst_err < LOGIT_TOL
    assert eng.stats()["prefill_tokens"] - pre0 >= 700


def test_continuous_batching_equals_solo(tiny):
    """Requests of different lengths arriving at different steps produce the same tokens as
    when each runs alone."""
    spec, w, g, eng = tiny
    gen = torch.Generator().manual_seed(33)
    prompts = [torch.randint(0, spec.vocab, (n,), generator=gen).tolist() for n in (5, 64, 130, 200, 31)]
    solo = [eng.generate([p], max_new_tokens=10, sessions=[f"solo{i}"], ignore_eos=True)[0]
            for i, p in enumerate(prompts)]
    rids, out, live = {}, {}, set()
    for i, p in enumerate(prompts):
        rid = eng.submit(f"mix{i}", p, max_new_tokens=10, ignore_eos=True)
        rids[rid] = i; out[i] = []; live.add(rid)
        eng.step()                                   # stagger arrivals
        for r, t, fin in eng.drain():
            out[rids[r]].append(t)
            if fin: live.discard(r)
    while live:
        eng.step()
        for r, t, fin in eng.drain():
            out[rids[r]].append(t)
            if fin: live.discard(r)
    assert [out[i] for i in range(len(prompts))] == solo


def test_prefix_reuse_equals_cold(tiny):
    """Turn 2 re-sends the whole history (conversation_manager.py:54-56); the engine reuses
    the session's KV and must generate what a cold prefill of the same history generates."""
    spec, w, g, eng = tiny
    gen = torch.Generator().manual_seed(44)
    t1 = torch.randint(0, spec.vocab, (90,), generator=gen).tolist()
    a1 = eng.generate([t1], max_new_tokens=8, sessions=["conv"], ignore_eos=True)[0]
    t2 = t1 + a1 + torch.randint(0, spec.vocab, (40,), generator=gen).tolist()
    hits0 = eng.stats()["prefix_hit_tokens"]
    warm = eng.generate([t2], max_new_tokens=8, sessions=["conv"], ignore_eos=True)[0]
    assert eng.stats()["prefix_hit_tokens"] - hits0 >= len(t1) + len(a1) - 1
    cold = eng.generate([t2], max_new_tokens=8, sessions=["conv-cold"], ignore_eos=True)[0]
    assert warm == cold
    # diverging history (e.g. after the 50-message trim, conversation_manager.py:40-52)
    t3 = t2[:50] + [(t2[50] + 1) % spec.vocab] + t2[51:]
    div = eng.generate([t3], max_new_tokens=8, sessions=["conv"], ignore_eos=True)[0]
    cold3 = eng.generate([t3], max_new_tokens=8, sessions=["conv-cold3"], ignore_eos=True)[0]
    assert div == cold3


def test_stop_cancel_and_limits(tiny):
    spec, w, g, eng = tiny
    prompt = g["prompt"].tolist()
    # max_new_tokens -> finish reason "length"
    rid = eng.submit("lim", prompt, max_new_tokens=3, ignore_eos=True)
    seen = []
    while not (seen and seen[-1][2]):
        eng.step(); seen += eng.drain()
    assert len(seen) == 3 and seen[-1][2] == "length"
    # cancel mid-generation
    rid = eng.submit("can", prompt, max_new_tokens=50, ignore_eos=True)
    eng.step(); eng.step()
    assert eng.cancel(rid)
    evs = eng.drain()
    assert evs[-1][2] == "cancelled"
    assert eng.step() == 0                       # nothing left to run
    # context window overflow is refused up front
    from fasttalk_llm_microservice_b200.native import NativeError
    with pytest.raises(NativeError):
        eng.submit("big", [1] * 2000, max_new_tokens=1)
    assert eng.close_session("can")
    free = eng.stats()["free_pages"]
    eng.close_session("lim")
    assert eng.stats()["free_pages"] > free


def test_fed_logits_into_memory_of_any_kind(tiny):
    """A caller's place for the logits may be ordinary or page-locked memory; a device address comes back filled or refused and is never read by the host."""
    from fasttalk_llm_microservice_b200 import native as N
    from fasttalk_llm_microservice_b200.engine import session_key
    spec, w = tiny[:2]
    eng = make_engine(spec, w, debug_logit_rows=8)
    toks, want, count = np.array([3, 1, 4, 1, 5], np.int32), np.array([0, 4], np.int32), np.array([5], np.int32)

    def feed(name, at):
        key = np.array([session_key(name)], np.uint64)
        return eng.lib.ft_engine_feed(eng._h, 1, key.ctypes.data, count.ctypes.data, toks.ctypes.data, 2, want.ctypes.data, at)
    try:
        plain, again = np.empty((2, spec.vocab), np.float32), np.empty((2, spec.vocab), np.float32)
        assert feed("a", plain.ctypes.data) == 0
        pinned = torch.empty(2, spec.vocab, pin_memory=True)
        assert feed("b", pinned.data_ptr()) == 0
        assert np.array_equal(pinned.numpy(), plain)
        device = torch.zeros(2, spec.vocab, device="cuda")
        rc = feed("c", device.data_ptr())
        torch.cuda.synchronize()
        assert (rc == 0 and np.array_equal(device.cpu().numpy(), plain)) or (rc < 0 and "logits copy" in N.last_error())
        assert feed("d", again.ctypes.data) == 0
        assert np.array_equal(again, plain)
    finally:
        eng.close()


def test_eos_stops():
    from fasttalk_llm_microservice_b200.model_spec import SPECS
    from fasttalk_llm_microservice_b200.weights import init_weights
    from fasttalk_llm_microservice_b200.engine import Engine, EngineLimits
    g = np.load(os.path.join(GOLD, "hf_tiny-d64.npz"))
    spec = SPECS["tiny-d64"]
    w = init_weights(spec, seed=int(g["seed"]), std=float(g["std"]), norm_jitter=float(g["norm_jitter"]))
    greedy = g["greedy"].tolist()
    eng = Engine(spec, w, EngineLimits(max_batch=4, max_batched_tokens=128, max_context=512),
                 eos_ids=(greedy[5],))
    first = greedy.index(greedy[5])
    out = eng.generate([g["prompt"].tolist()], max_new_tokens=24)[0]
    assert out == greedy[:first + 1]
    eng.close()


def test_page_pressure_evicts_idle_sessions_lru_and_refuses_what_can_never_fit():
    """KV pages run out: idle sessions' caches are given up least-recently-used first, running ones never; an
    evicted conversation still gets the same answer when it comes back (cold again); a prompt larger than the
    whole cache ends with finish reason "error" instead of stalling the queue."""
    from fasttalk_llm_microservice_b200.model_spec import SPECS
    from fasttalk_llm_microservice_b200.weights import init_weights
    spec = SPECS["tiny-d64"]
    w = init_weights(spec, seed=4, std=0.08, norm_jitter=0.1)
    eng = make_engine(spec, w, max_batch=4, max_batched_tokens=256, max_context=1024, num_pages=12, max_sessions=16)
    big = make_engine(spec, w, max_batch=4, max_batched_tokens=256, max_context=1024)     # no pressure: the reference answers
    try:
        gen = torch.Generator().manual_seed(5)
        prompts = {k: torch.randint(0, spec.vocab, (n,), generator=gen).tolist()
                   for k, n in (("A", 200), ("B", 250), ("C", 190), ("D", 300))}
        want = {k: big.generate([p], 6, sessions=[f"w{k}"])[0] for k, p in prompts.items()}
        total = eng.stats()["total_pages"]
        assert total == 12
        assert eng.generate([prompts["A"]], 6, sessions=["A"])[0] == want["A"]        # 4 pages stay cached
        assert eng.generate([prompts["B"]], 6, sessions=["B"])[0] == want["B"]        # 4 more
        assert eng.stats()["free_pages"] == total - 8
        hits = eng.stats()["prefix_hit_tokens"]
        assert eng.generate([prompts["B"] + want["B"] + [7, 8, 9]], 4, sessions=["B"])    # B is now the most recent
        assert eng.stats()["prefix_hit_tokens"] - hits >= 250
        # B now holds 5 pages, A 4: C needs 4 of the 3 that are free -> A, the least recently used, goes
        assert eng.generate([prompts["C"]], 6, sessions=["C"])[0] == want["C"]
        assert eng.stats()["free_pages"] == total - 5 - 4          # B and C hold pages, A's are gone
        # D needs 5 pages, 3 are free -> B goes (C was used after it)
        assert eng.generate([prompts["D"]], 6, sessions=["D"])[0] == want["D"]
        assert eng.stats()["free_pages"] == total - 4 - 5          # C and D
        hits = eng.stats()["prefix_hit_tokens"]
        assert eng.generate([prompts["A"]], 6, sessions=["A"])[0] == want["A"]        # cold again, same tokens
        assert eng.stats()["prefix_hit_tokens"] == hits
        # 13 pages worth of prompt can never fit 12 pages
        rid = eng.submit("huge", torch.randint(0, spec.vocab, (800,), generator=gen).tolist(), max_new_tokens=4)
        fins = []
        for _ in range(50):
            eng.step()
            fins += [f for r, t, f in eng.drain() if r == rid and f]
            if fins:
                break
        assert fins == ["error"]
        assert eng.generate([prompts["C"]], 6, sessions=["C2"])[0] == want["C"]       # and the engine carries on
    finally:
        eng.close()
        big.close()


# ------------------------------------------------------------------ the named architecture
@pytest.fixture(scope="module")
def llama1b():
    from fasttalk_llm_microservice_b200.model_spec import LLAMA_3_2_1B
    from fasttalk_llm_microservice_b200.weights import init_weights
    w = init_weights(LLAMA_3_2_1B, seed=0, device="cuda")
    eng = make_engine(LLAMA_3_2_1B, w, max_batch=64, max_batched_tokens=2048, max_context=4096,
                      debug_logit_rows=128)
    w32 = {k: v.float() for k, v in w.items() if k != "lm_head"}
    w32["lm_head"] = w32["embed"]
    yield LLAMA_3_2_1B, w32, eng
    eng.close()


def test_llama1b_config1_greedy_and_logits(llama1b):
    """BASELINE config 1 shape: 128-token prompt, greedy decode, random-init Llama-3.2-1B.
    Teacher-forced logits over the prompt within 2e-2; the first 64 greedy tokens identical to
    the fp32 oracle's.  On random-init weights greedy argmax can hit near-ties:
    a mismatch is waived only if the oracle's top-1/top-2 margin at that step is within 3x the logit error
    measured in this very run; the engine is then re-aligned to the oracle's token and all 64 positions are
    compared (oracle/parity.py)."""
    spec, w32, eng = llama1b
    gen = torch.Generator().manual_seed(1234)
    prompt = torch.randint(0, 128000, (128,), generator=gen)
    with torch.no_grad():
        ref_full = O.forward(w32, spec, prompt).cpu()
        ref_tokens, ref_logits = O.greedy_generate(w32, spec, prompt, 64, return_logits=True)
    got_full = eng.debug_prefill_logits(prompt.tolist(), chunk=128)
    describe_err("1B cfg1 prefill", got_full, ref_full)
    err = per_pos_rel(got_full, ref_full)
    assert err < LOGIT_TOL, err
    greedy_parity(eng, "1B cfg1 (128-token prompt, 64 greedy)", prompt.tolist(), ref_tokens, ref_logits)


def test_llama1b_batched_decode_matches_oracle_logits(llama1b):
    """8 concurrent sessions with ragged prompts: decode-step logits of each against the oracle
    run alone (teacher-forced on the engine's own tokens)."""
    spec, w32, eng = llama1b
    gen = torch.Generator().manual_seed(99)
    prompts = [torch.randint(0, 128000, (n,), generator=gen) for n in (17, 64, 65, 200, 300, 128, 1, 513)]
    rids = [eng.submit(f"b{i}", p.tolist(), max_new_tokens=6, ignore_eos=True) for i, p in enumerate(prompts)]
    toks = {r: [] for r in rids}
    logits = {r: [] for r in rids}
    live = set(rids)
    from fasttalk_llm_microservice_b200.native import NativeError
    while live:
        eng.step()
        for r in live:                       # rows of this step's logits buffer, before draining
            try:
                logits[r].append(eng.logits(r))
            except NativeError:
                pass                         # still prefilling: no logits row this step
        for r, t, fin in eng.drain():
            toks[r].append(t)
            if fin: live.discard(r)
    worst = 0.0
    for i, r in enumerate(rids):
        seq = torch.cat([prompts[i], torch.tensor(toks[r][:-1], dtype=torch.long)])
        with torch.no_grad():
            ref = O.forward(w32, spec, seq).cpu()[len(prompts[i]) - 1:]
        got = torch.stack(logits[r][:ref.shape[0]])
        worst = max(worst, per_pos_rel(got, ref[:got.shape[0]]))
    print(f"\n[1B batched] worst decode logit rel err {worst:.2e}")
    assert worst < LOGIT_TOL


def test_llama1b_config2_full_size_64_sessions_2k_history(llama1b):
    """BASELINE config 2 at its full size — the shape bench.py times: 64 sessions, each with a 2048-token
    history, decoding together for 64 steps.  The histories are prefilled first (turn 1), then all 64
    sessions re-send them (conversation_manager.py:54-56): the prefix is served from the KV cache and the
    64 rows decode in the same steps from the first token on.  Three of the sessions are checked against
    the fp32 oracle at all 64 positions (teacher-forced logits at context 2048..2111, greedy tokens,
    near-ties waived and re-aligned, oracle/parity.py); then each of them alone in the engine, which must
    agree with its batched run wherever neither run met a near-tie."""
    spec, w32, eng = llama1b
    gen = torch.Generator().manual_seed(2048)
    prompts = [torch.randint(0, 128000, (2048,), generator=gen).tolist() for _ in range(64)]
    n_new = 64
    eng.generate(prompts, max_new_tokens=1, sessions=[f"full{i}" for i in range(64)], ignore_eos=True)
    checked = (0, 31, 63)
    jobs = []
    for i in checked:
        with torch.no_grad():
            ref_tokens, ref_logits = O.greedy_generate(w32, spec, torch.tensor(prompts[i]), n_new, return_logits=True)
        jobs.append(P.Job(f"1B cfg2 session {i} among 64 at ctx 2048", f"full{i}", prompts[i], ref_tokens, ref_logits))
    hits0, st0 = eng.stats()["prefix_hit_tokens"], eng.stats()
    fillers = [eng.submit(f"full{i}", prompts[i], max_new_tokens=n_new + 8, ignore_eos=True)
               for i in range(64) if i not in checked]
    P.run(eng, jobs)
    st1 = eng.stats()
    assert st1["prefix_hit_tokens"] - hits0 >= 64 * 2047
    # the 64 rows really decoded together: decode tokens per decode step over the checked span
    rows_per_step = (st1["decode_tokens"] - st0["decode_tokens"]) / max(1, st1["decode_steps"] - st0["decode_steps"])
    assert rows_per_step > 60, rows_per_step
    for r in fillers:
        eng.cancel(r)
    eng.step(); eng.drain()
    for j in jobs:
        P.finish(j)
    for i in range(64):
        eng.close_session(f"full{i}")
    for j, i in zip(jobs, checked):
        solo = P.Job(f"1B cfg2 session {i} alone", f"solo{i}", prompts[i], j.ref_tokens, j.ref_logits)
        P.run(eng, [solo])
        P.finish(solo)
        skip = {k for k, *_ in j.waived} | {k for k, *_ in solo.waived}
        assert all(a == b for k, (a, b) in enumerate(zip(j.engine_tokens, solo.engine_tokens)) if k not in skip)
        eng.close_session(f"solo{i}")


def test_llama1b_decode_steps_of_more_than_128_rows():
    """BASELINE config 3's shape (256 sessions on one GPU) puts more than 128 rows into a decode step: two or more
    128-token tiles, which run on the CTA-pair kernels in their one-fp16-plane form.  160 sessions of the 1B model decode
    together; three of them are checked against the fp32 oracle at every position (teacher-forced logits, greedy tokens)."""
    from fasttalk_llm_microservice_b200.model_spec import LLAMA_3_2_1B as spec
    from fasttalk_llm_microservice_b200.weights import init_weights
    w = init_weights(spec, seed=0, device="cuda")
    w32 = {k: v.float() for k, v in w.items() if k != "lm_head"}
    w32["lm_head"] = w32["embed"]
    eng = make_engine(spec, w, max_batch=160, max_batched_tokens=4096, max_context=512, debug_logit_rows=192)
    try:
        gen = torch.Generator().manual_seed(160)
        prompts = [torch.randint(0, 128000, (96 + (i % 5),), generator=gen).tolist() for i in range(160)]
        n_new, checked, jobs = 24, (0, 77, 159), []
        for i in checked:
            with torch.no_grad():
                ref_tokens, ref_logits = O.greedy_generate(w32, spec, torch.tensor(prompts[i]), n_new, return_logits=True)
            jobs.append(P.Job(f"1B session {i} among 160 decoding rows", f"wide{i}", prompts[i], ref_tokens, ref_logits))
        fillers = [eng.submit(f"wide{i}", prompts[i], max_new_tokens=n_new + 16, ignore_eos=True)
                   for i in range(160) if i not in checked]
        st0 = eng.stats()
        P.run(eng, jobs)
        st1 = eng.stats()
        rows_per_step = (st1["decode_tokens"] - st0["decode_tokens"]) / max(1, st1["decode_steps"] - st0["decode_steps"])
        assert rows_per_step > 128, rows_per_step       # (the average includes the steps in which sessions were still joining)
        for r in fillers:
            eng.cancel(r)
        eng.step(); eng.drain()
        for j in jobs:
            P.finish(j)
    finally:
        eng.close()
        del w, w32
        torch.cuda.empty_cache()


def test_llama1b_long_context_8k_window():
    """BASELINE config 4's window on the 1B weights: an 8300-token history (past the 8192 original RoPE range,
    130 KV pages, chunked prefill in 8192-token steps), last-position logits and 8 greedy tokens vs the oracle."""
    from fasttalk_llm_microservice_b200.model_spec import LLAMA_3_2_1B as spec
    from fasttalk_llm_microservice_b200.weights import init_weights
    w = init_weights(spec, seed=1, device="cuda")
    eng = make_engine(spec, w, max_batch=2, max_batched_tokens=8192, max_context=8448, debug_logit_rows=0)
    try:
        w32 = {k: v.float() for k, v in w.items() if k != "lm_head"}
        w32["lm_head"] = w32["embed"]
        prompt = torch.randint(0, 128000, (8300,), generator=torch.Generator().manual_seed(8))
        with torch.no_grad():
            ref_tokens, ref_logits = O.greedy_generate(w32, spec, prompt, 8, return_logits=True)
        job = greedy_parity(eng, "1B ctx 8300 (8k window)", prompt.tolist(), ref_tokens, ref_logits)
        assert job.errs_checked >= 7
    finally:
        eng.close()
        del w32, w
        torch.cuda.empty_cache()


# ------------------------------------------------------------------ the other named architectures
@pytest.mark.parametrize("name,n_prompt,n_new", [("llama-3.2-3b", 96, 64), ("llama-3.1-8b", 70, 64)])
def test_larger_configs_logits_and_greedy(name, n_prompt, n_new):
    """BASELINE configs 3-5 name Llama-3.2-3B (GQA group 3, head_dim 128) and Llama-3.1-8B (untied
    LM head, rope factor 8): same parity bar on random-init weights of those shapes."""
    from fasttalk_llm_microservice_b200.model_spec import SPECS
    from fasttalk_llm_microservice_b200.weights import init_weights
    spec = SPECS[name]
    w = init_weights(spec, seed=3, device="cuda")
    eng = make_engine(spec, w, max_batch=8, max_batched_tokens=256, max_context=1024, debug_logit_rows=128)
    try:
        gen = torch.Generator().manual_seed(7)
        prompt = torch.randint(0, 128000, (n_prompt,), generator=gen)
        w32 = {k: v.float() for k, v in w.items() if k != "lm_head"}
        w32["lm_head"] = w32["embed"] if spec.tied_embeddings else w["lm_head"].float()
        with torch.no_grad():
            ref_full = O.forward(w32, spec, prompt).cpu()
            ref_tokens, ref_logits = O.greedy_generate(w32, spec, prompt, n_new, return_logits=True)
        got = eng.debug_prefill_logits(prompt.tolist(), chunk=64)
        describe_err(f"{name} prefill", got, ref_full)
        assert per_pos_rel(got, ref_full) < LOGIT_TOL
        greedy_parity(eng, f"{name} ({n_prompt}-token prompt, {n_new} greedy)", prompt.tolist(), ref_tokens, ref_logits)
    finally:
        eng.close()
        del w32, w
        torch.cuda.empty_cache()


def test_llama8b_config4_long_history_prefill_and_decode():
    """BASELINE config 4's shape on one GPU: Llama-3.1-8B (head_dim 128, untied LM head, rope factor 8), an 8000-token
    history prefilled in ONE 8192-token step (CTA-pair GEMMs on the single fp16 plane, tcgen05 prefill attention at
    d = 128 over 125 KV tiles), then streaming decode: all 8 positions against the fp32 oracle, teacher-forced."""
    from fasttalk_llm_microservice_b200.model_spec import SPECS
    from fasttalk_llm_microservice_b200.weights import init_weights
    spec = SPECS["llama-3.1-8b"]
    w = init_weights(spec, seed=5, device="cuda")
    eng = make_engine(spec, w, max_batch=2, max_batched_tokens=8192, max_context=8192, debug_logit_rows=0)
    try:
        w32 = {k: v.float() for k, v in w.items()}
        prompt = torch.randint(0, 128000, (8000,), generator=torch.Generator().manual_seed(80))
        with torch.no_grad():
            ref_tokens, ref_logits = O.greedy_generate(w32, spec, prompt, 8, return_logits=True)
        del w32
        torch.cuda.empty_cache()
        job = greedy_parity(eng, "8B cfg4 (8000-token history, 8192 window)", prompt.tolist(), ref_tokens, ref_logits)
        assert job.errs_checked >= 7 and job.worst_err < 1e-2
    finally:
        eng.close()
        del w
        torch.cuda.empty_cache()


# ------------------------------------------------------------------ devices and threads
def _tiny_setup():
    from fasttalk_llm_microservice_b200.model_spec import SPECS
    from fasttalk_llm_microservice_b200.weights import init_weights
    g = np.load(os.path.join(GOLD, "hf_tiny-d64.npz"))
    spec = SPECS["tiny-d64"]
    w = init_weights(spec, seed=int(g["seed"]), std=float(g["std"]), norm_jitter=float(g["norm_jitter"]))
    return spec, w, g


def test_two_engines_share_one_gpu_and_step_concurrently():
    """Two models behind one process put two engines on the same GPU.  Their split-K rendezvous grids must never
    interleave (each needs all its CTAs resident): steps of engines that share a device are serialised inside the
    library.  Two threads hammer two engines at once; both must produce what they produce alone."""
    import threading
    spec, w, g = _tiny_setup()
    prompts = [g["prompt"].tolist(), torch.randint(0, spec.vocab, (300,), generator=torch.Generator().manual_seed(3)).tolist()]
    a, b = make_engine(spec, w), make_engine(spec, w)
    try:
        want = [a.generate([p], max_new_tokens=24, sessions=[f"w{i}"], ignore_eos=True)[0] for i, p in enumerate(prompts)]
        got, errs = {}, []

        def work(eng, name):
            try:
                for rep in range(6):
                    got[(name, rep)] = [eng.generate([p], max_new_tokens=24, sessions=[f"{name}{rep}-{i}"], ignore_eos=True)[0]
                                        for i, p in enumerate(prompts)]
            except Exception as e:  # noqa: BLE001
                errs.append(e)
        ts = [threading.Thread(target=work, args=(a, "a")), threading.Thread(target=work, args=(b, "b"))]
        [t.start() for t in ts]
        [t.join(timeout=120) for t in ts]
        assert not errs, errs
        assert len(got) == 12 and all(v == want for v in got.values())
    finally:
        a.close()
        b.close()


def test_prompt_tokens_beside_streaming_sessions_are_capped_to_a_token_tile():
    """`decode_prefill_cap`: beside streaming sessions a step admits prompt tokens only up to the 128-token tile boundary at
    or above (decode rows + cap); the allowance grows with the number of sessions waiting per streaming session.  What is
    generated does not depend on the cap."""
    spec, w, g = _tiny_setup()
    gen = torch.Generator().manual_seed(11)
    short = [torch.randint(0, spec.vocab, (24,), generator=gen).tolist() for _ in range(5)]
    long_ = [torch.randint(0, spec.vocab, (700,), generator=gen).tolist() for _ in range(6)]
    ref = make_engine(spec, w, max_batch=12, max_batched_tokens=2048, decode_prefill_cap=-1)
    eng = make_engine(spec, w, max_batch=12, max_batched_tokens=2048, decode_prefill_cap=200)
    try:
        want = ref.generate(long_[:3], max_new_tokens=6, sessions=["r0", "r1", "r2"], ignore_eos=True)
        short_rids = [eng.submit(f"s{i}", p, max_new_tokens=400, ignore_eos=True) for i, p in enumerate(short)]
        eng.step(); eng.drain()                                   # nothing streams yet: the first step is uncapped
        rids = [eng.submit(f"l{i}", long_[i], max_new_tokens=6, ignore_eos=True) for i in range(3)]
        eng.step_log()
        out = {r: [] for r in rids}
        for _ in range(40):
            eng.step()
            for rid, tok, _fin in eng.drain():
                if rid in out and tok >= 0:
                    out[rid].append(tok)
            if all(len(v) == 6 for v in out.values()):
                break
        assert [out[r] for r in rids] == want
        rows = [r.tolist() for r in eng.step_log()]
        capped = [int(r[2]) for r in rows if r[1] >= 5 and r[2] > 0]
        # streaming rows + prompt tokens fill two 128-token tiles (5 + 200 -> 256) until the 2100 tokens are through
        full = [r for r in rows if r[1] >= 5 and r[2] > 0][:-1]
        assert len(full) >= 7 and all(int(r[1] + r[2]) == 256 for r in full) and sum(capped) == 2100, rows
        # the allowance grows with the sessions waiting PER streaming session (cap x waiting / (2 x streaming)): six
        # arrivals behind ONE early bird get 3 x 200 prompt tokens (1 + 600 rows -> five 128-token tiles -> 639), not the
        # cap and not the whole budget
        for r in short_rids[1:]:
            eng.cancel(r)
        eng.step(); eng.drain()
        for i in range(6):
            eng.submit(f"m{i}", long_[i][::-1], max_new_tokens=1, ignore_eos=True)
        eng.step_log()
        eng.step(); eng.drain()
        burst = eng.step_log()[-1].tolist()
        assert (int(burst[1]), int(burst[2])) == (1, 639), burst
    finally:
        ref.close()
        eng.close()


def test_native_stepping_thread_equals_stepping_from_python():
    """ft_engine_start: the engine steps on its own native thread, the owner only submits, waits and drains.  Same tokens
    as stepping from Python; ft_engine_step is refused meanwhile; cancel reaches a running request; stop / start
    alternate and Python stepping works again after a stop."""
    import time
    from fasttalk_llm_microservice_b200 import native as N
    spec, w, g = _tiny_setup()
    gen = torch.Generator().manual_seed(5)
    prompts = [g["prompt"].tolist()] + [torch.randint(0, spec.vocab, (n,), generator=gen).tolist() for n in (300, 40, 700)]
    ref = make_engine(spec, w, max_batch=8, max_batched_tokens=512)
    eng = make_engine(spec, w, max_batch=8, max_batched_tokens=512)
    try:
        want = ref.generate(prompts, max_new_tokens=24, sessions=[f"r{i}" for i in range(4)], ignore_eos=True)
        eng.start_loop()
        eng.start_loop()                                        # idempotent
        with pytest.raises(N.NativeError, match="stepping thread"):
            eng.step()

        def collect(rids, limit_s=30.0):
            out, fin = {r: [] for r in rids}, {}
            t_end = time.time() + limit_s
            while len(fin) < len(rids):
                assert time.time() < t_end, (out, fin)
                if eng.wait_events(100) <= 0:
                    continue
                for rid, tok, f in eng.drain():
                    if rid in out:
                        if tok >= 0:
                            out[rid].append(tok)
                        if f is not None:
                            fin[rid] = f
            return [out[r] for r in rids], [fin[r] for r in rids]
        rids = [eng.submit(f"n{i}", p, max_new_tokens=24, ignore_eos=True) for i, p in enumerate(prompts)]
        got, fin = collect(rids)
        assert got == want and fin == ["length"] * 4
        assert eng.wait_events(20) == 0                          # idle: times out, no busy loop needed to see it
        # a request that would run for a long time is cancelled from outside while the thread steps it
        rid = eng.submit("long", prompts[1], max_new_tokens=600, ignore_eos=True)
        seen = 0
        t_end = time.time() + 30
        while seen < 5:
            assert time.time() < t_end
            if eng.wait_events(100) > 0:
                seen += sum(1 for r, tok, f in eng.drain() if r == rid and tok >= 0)
        eng.cancel(rid)
        _, fin = collect([rid])
        assert fin == ["cancelled"]
        eng.stop_loop()
        eng.stop_loop()
        assert eng.generate([prompts[0]], max_new_tokens=8, sessions=["again"], ignore_eos=True)[0] == want[0][:8]
        assert eng.generate(prompts, max_new_tokens=24, sessions=[f"o{i}" for i in range(4)], ignore_eos=True,
                            own_thread=True) == want                               # generate() on the engine's thread
        eng.start_loop()                                        # and once more
        rid = eng.submit("n2", prompts[2], max_new_tokens=24, ignore_eos=True)     # prefix of session n2 is cached
        got, fin = collect([rid])
        assert got[0] == want[2]
        # a thread that is still blocked in ft_engine_wait when the engine is destroyed is sent away first
        import threading
        seen = {}

        def waiter():
            try:
                seen["n"] = eng.wait_events(10000)
            except N.NativeError as e:
                seen["err"] = str(e)
        th = threading.Thread(target=waiter)
        th.start()
        time.sleep(0.1)
        t0 = time.time()
        eng.close()
        th.join(timeout=5)
        assert not th.is_alive() and "destroyed" in seen.get("err", ""), seen
        assert time.time() - t0 < 2.0
    finally:
        ref.close()
        eng.close()                                             # joins the thread (a second close is a no-op)


def test_engine_stepped_from_a_fresh_thread():
    """Every ft_engine_* entry makes the engine's device current itself: a thread that never called cudaSetDevice
    (current device 0) can step an engine that lives on another GPU.  With one GPU the thread part still runs."""
    import threading
    from fasttalk_llm_microservice_b200.engine import Engine, EngineLimits
    spec, w, g = _tiny_setup()
    dev = torch.device("cuda", torch.cuda.device_count() - 1)        # the last GPU: != 0 whenever there are two
    eng = Engine(spec, w, EngineLimits(max_batch=4, max_batched_tokens=128, max_context=512), eos_ids=(), device=dev)
    torch.cuda.set_device(0)
    try:
        out = {}

        def work():
            out["tokens"] = eng.generate([g["prompt"].tolist()], max_new_tokens=12, ignore_eos=True)[0]
        t = threading.Thread(target=work)
        t.start()
        t.join(timeout=60)
        with torch.no_grad():
            ref = O.greedy_generate(w, spec, torch.from_numpy(g["prompt"]), 12)
        assert out.get("tokens") is not None
        n_same = next((i for i, (x, y) in enumerate(zip(out["tokens"], ref)) if x != y), 12)
        assert n_same >= 9, (out["tokens"], ref)      # the golden prompt's one near-tie sits at step 9
    finally:
        eng.close()


def test_submit_cancel_and_close_while_a_step_is_on_the_gpu():
    """The scheduler lock is released while a step's kernels run, so submit / cancel / session_close from other
    threads return without waiting for the GPU.  One thread steps continuously; the test thread submits requests,
    cancels some and closes the sessions of others at arbitrary moments.  Every request must end with exactly one
    finish event, untouched requests must produce what they produce alone, and every KV page must come back."""
    import threading
    import time
    spec, w, g = _tiny_setup()
    eng = make_engine(spec, w, max_batch=16, max_batched_tokens=512, max_context=1024)
    try:
        gen = torch.Generator().manual_seed(77)
        prompts = [torch.randint(0, spec.vocab, (int(n),), generator=gen).tolist()
                   for n in torch.randint(20, 400, (40,), generator=gen)]
        want = {i: eng.generate([prompts[i]], max_new_tokens=20, sessions=[f"solo{i}"], ignore_eos=True)[0]
                for i in range(0, 40, 4)}
        for i in want:
            eng.close_session(f"solo{i}")
        total_free = eng.stats()["free_pages"]
        stop, events, errs = threading.Event(), [], []

        def stepper():
            try:
                while not stop.is_set():
                    if eng.step() == 0:
                        time.sleep(0.0002)
                    events.extend(eng.drain())
            except Exception as e:  # noqa: BLE001
                errs.append(e)
        t = threading.Thread(target=stepper)
        t.start()
        rids, slow = {}, 0.0
        for i, p in enumerate(prompts):
            t0 = time.perf_counter()
            rids[i] = eng.submit(f"c{i}", p, max_new_tokens=20, ignore_eos=True)
            slow = max(slow, time.perf_counter() - t0)
            time.sleep(0.0007 * (i % 3))
            if i % 4 == 1:
                eng.cancel(rids[i])                       # often while its prefill or a decode step is in flight
            if i % 4 == 2:
                eng.close_session(f"c{i}")
        deadline = time.time() + 60
        while time.time() < deadline and not errs:
            fins = {r for r, tok, fin in list(events) if fin is not None}
            if all(r in fins for r in rids.values()):
                break
            time.sleep(0.01)
        stop.set()
        t.join(timeout=10)
        assert not errs, errs
        by = {}
        for r, tok, fin in events:
            by.setdefault(r, []).append((tok, fin))
        for i, r in rids.items():
            fins = [f for _, f in by.get(r, []) if f is not None]
            assert len(fins) == 1, (i, fins)
            toks = [tk for tk, _ in by[r] if tk >= 0]
            if i % 4 == 0:
                assert fins == ["length"] and toks == want[i], i          # untouched: same tokens as alone
            elif i % 4 == 3:
                assert fins == ["length"] and len(toks) == 20
            else:
                assert fins[0] in ("cancelled", "length")
        for i in range(40):
            eng.close_session(f"c{i}")
        st = eng.stats()
        assert st["free_pages"] == total_free and st["active_requests"] == 0, st
        assert slow < 0.05, f"a submit waited {slow * 1e3:.1f} ms"
    finally:
        eng.close()


# ------------------------------------------------------------------ a real checkpoint directory
def test_engine_generates_from_a_transformers_checkpoint(tmp_path):
    """transformers writes a Llama checkpoint (`save_pretrained`, sharded safetensors + config.json); checkpoint.py
    loads it into the engine's stacked layout on the GPU; the engine's logits and greedy tokens are compared with
    the fp32 oracle ON THE LOADED TENSORS and with transformers' own forward of the model that wrote the files."""
    import sys
    sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))
    from make_golden import hf_model
    from fasttalk_llm_microservice_b200.checkpoint import load_hf_checkpoint
    from fasttalk_llm_microservice_b200.model_spec import TINY_D128 as spec0
    from fasttalk_llm_microservice_b200.weights import init_weights
    w0 = init_weights(spec0, seed=12, std=0.08, norm_jitter=0.1)
    m = hf_model(spec0, w0)
    m.to(torch.bfloat16).save_pretrained(tmp_path, safe_serialization=True, max_shard_size="300KB")
    assert os.path.exists(tmp_path / "model.safetensors.index.json")
    spec, w = load_hf_checkpoint(str(tmp_path), device="cuda", name=spec0.name)
    assert spec == spec0
    eng = make_engine(spec, w)
    try:
        prompt = torch.randint(0, spec.vocab, (150,), generator=torch.Generator().manual_seed(2))
        with torch.no_grad():
            ref_full = O.forward(w, spec, prompt).cpu()
            hf_full = hf_model(spec0, w0)(prompt[None]).logits[0]                  # fresh fp32 transformers model
            ref_tokens, ref_logits = O.greedy_generate(w, spec, prompt, 32, return_logits=True)
        assert per_pos_rel(ref_full, hf_full) < 1e-4                               # oracle == transformers on these files
        got = eng.debug_prefill_logits(prompt.tolist(), chunk=64)
        assert per_pos_rel(got, hf_full) < LOGIT_TOL, per_pos_rel(got, hf_full)
        greedy_parity(eng, "tiny-d128 from a save_pretrained checkpoint", prompt.tolist(), ref_tokens, ref_logits)
    finally:
        eng.close()
