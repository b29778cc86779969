"""The oracle against its pins: transformers-generated golden vectors (committed) and the
model-size arithmetic."""
import os

import numpy as np
import pytest
import torch

from fasttalk_llm_microservice_b200.model_spec import SPECS, get_spec
from fasttalk_llm_microservice_b200.weights import init_weights, rope_inv_freq, rope_tables
from oracle import llama_oracle as O

GOLD = os.path.join(os.path.dirname(__file__), "golden")


@pytest.mark.parametrize("name,count", [("llama-3.2-1b", 1_235_814_400),
                                        ("llama-3.2-3b", 3_212_749_824),
                                        ("llama-3.1-8b", 8_030_261_248)])
def test_param_counts(name, count):
    assert SPECS[name].param_count() == count


def test_survey_byte_model():
    s = get_spec("llama3.2:1b")
    assert s.kv_bytes_per_token() == 32768
    assert abs(s.weight_bytes() / 1e9 - 2.472) < 1e-3
    # worked target: 64 sessions x 2048 ctx = 6.767 GB / step
    assert abs(s.decode_step_bytes([2048] * 64) / 1e9 - 6.767) < 2e-3
    assert SPECS["llama-3.2-3b"].kv_bytes_per_token() == 114688
    assert SPECS["llama-3.1-8b"].kv_bytes_per_token() == 131072


@pytest.mark.parametrize("name", ["llama-3.2-1b", "llama-3.2-3b", "llama-3.1-8b"])
def test_rope_inv_freq_matches_transformers(name):
    gold = np.load(os.path.join(GOLD, "hf_rope_inv_freq.npz"))[name]
    s = SPECS[name]
    mine = O.rope_inv_freq(s.head_dim, s.rope_theta, s.rope_factor, 1.0, 4.0, 8192).numpy()
    np.testing.assert_allclose(mine, gold, rtol=2e-6)
    np.testing.assert_allclose(rope_inv_freq(s).numpy(), gold, rtol=2e-6)
    cos, sin = rope_tables(s, 64)
    c2, s2 = O.rope_cos_sin(s, torch.arange(64))
    np.testing.assert_allclose(cos.numpy(), c2.numpy(), atol=1e-6)
    np.testing.assert_allclose(sin.numpy(), s2.numpy(), atol=1e-6)


@pytest.mark.parametrize("name", ["tiny-d64", "tiny-d128"])
def test_oracle_matches_transformers_golden(name):
    g = np.load(os.path.join(GOLD, f"hf_{name}.npz"))
    spec = SPECS[name]
    w = init_weights(spec, seed=int(g["seed"]), std=float(g["std"]), norm_jitter=float(g["norm_jitter"]))
    prompt = torch.from_numpy(g["prompt"])
    with torch.no_grad():
        logits = O.forward(w, spec, prompt)
    gold = torch.from_numpy(g["logits"])
    err = (logits - gold).abs().max().item() / gold.abs().max().item()
    assert err < 2e-5, err
    # incremental (KV-cached) decode reproduces transformers' greedy continuation
    toks = O.greedy_generate(w, spec, prompt, len(g["greedy"]))
    assert toks == g["greedy"].tolist()


def test_oracle_chunked_equals_full():
    spec = SPECS["tiny-d64"]
    w = init_weights(spec, seed=3, std=0.08)
    toks = torch.randint(0, spec.vocab, (37,), generator=torch.Generator().manual_seed(5))
    with torch.no_grad():
        full = O.forward(w, spec, toks)
        st = O.OracleState(spec)
        parts = [O.forward(w, spec, toks[a:b], st) for a, b in ((0, 9), (9, 10), (10, 37))]
    torch.testing.assert_close(torch.cat(parts), full, rtol=1e-4, atol=1e-4)


def test_sampling_support():
    logits = torch.tensor([2.0, 1.0, 0.5, -1.0, -3.0])
    p = O.sampling_support(logits, 1.0, 0, 1.0)
    torch.testing.assert_close(p, torch.softmax(logits.double(), -1))
    p = O.sampling_support(logits, 1.0, 2, 1.0)
    assert (p[2:] == 0).all() and abs(p.sum().item() - 1) < 1e-12
    p = O.sampling_support(logits, 0.7, 0, 0.5)
    assert p[0] == 1.0  # top token alone already exceeds 0.5 at T=0.7
