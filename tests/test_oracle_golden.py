"""Oracle (f32 mode) vs the committed HuggingFace-transformers fixtures in tests/golden/
(generated by tests/golden/make_golden.py).  Guards RoPE convention, GQA head mapping, qkv fusion
order, QK-norm placement, llama3 rope scaling and tied embeddings against misreading the reference."""
import os

import numpy as np
import pytest

from cake_b200.synth import make_checkpoint
from oracle import oracle as O
from tests.golden.make_golden import CASES, case_checkpoint, case_config

GOLD = os.path.join(os.path.dirname(__file__), "golden")


@pytest.mark.parametrize("name", list(CASES))
def test_oracle_matches_hf_fixture(name):
    z = np.load(os.path.join(GOLD, f"hf_{name}.npz"))
    _, cfg = case_config(name)
    sd = case_checkpoint(cfg, int(z["seed"]), float(z["std"]))
    m = O.OracleModel(cfg, sd, "f32")
    ids, ref = z["ids"], z["logits"]
    c = m.new_cache()
    n0 = min(7, cfg.sliding_window or 7)               # (an active window: the prompt fits it, see make_golden.py)
    lg = m.forward(ids[:n0], 0, c)                     # prefill -> logits of its last position
    np.testing.assert_allclose(lg, ref[n0 - 1], rtol=0, atol=2e-5)
    for t in range(n0, len(ids)):                      # then decode one token at a time
        lg = m.forward(ids[t:t + 1], t, c)
        np.testing.assert_allclose(lg, ref[t], rtol=0, atol=2e-5)


@pytest.mark.parametrize("dtype,tol", [("bf16", 0.08), ("f16", 0.01)])
def test_low_precision_oracle_stays_near_fp32(dtype, tol):
    # bounds how much of any GPU-vs-oracle gap can be rounding order rather than a bug
    z = np.load(os.path.join(GOLD, "hf_llama_tiny.npz"))
    _, cfg = case_config("llama_tiny")
    sd32 = make_checkpoint(cfg, "f32", seed=int(z["seed"]), std=float(z["std"]))
    sd = make_checkpoint(cfg, dtype, seed=int(z["seed"]), std=float(z["std"]))
    m = O.OracleModel(cfg, sd, dtype)
    lg = m.forward(z["ids"], 0, m.new_cache())
    m32 = O.OracleModel(cfg, {k: v.float() for k, v in sd.items()}, "f32")
    lg32 = m32.forward(z["ids"], 0, m32.new_cache())
    assert np.abs(lg - lg32).max() < tol * max(1.0, np.abs(lg32).max())
    del sd32


def test_embed_scale_equals_prescaled_embeddings():
    """text_model.rs:274-276: x = embedding * embed_scale.  In f32 mode that must equal a checkpoint whose embedding table
    was multiplied beforehand (and an untied head left alone)."""
    _, cfg = case_config("llama_tiny")
    sd = make_checkpoint(cfg, "f32", seed=5, std=0.1)
    ids = np.arange(3, 11, dtype=np.uint32)
    import copy
    cfg_s = copy.deepcopy(cfg)
    cfg_s.embed_scale = 8.0
    a = O.OracleModel(cfg_s, sd, "f32")
    la = a.forward(ids, 0, a.new_cache())
    sd2 = dict(sd)
    sd2["model.embed_tokens.weight"] = sd["model.embed_tokens.weight"] * 8.0
    b = O.OracleModel(cfg, sd2, "f32")
    np.testing.assert_allclose(la, b.forward(ids, 0, b.new_cache()), rtol=0, atol=1e-6)


def test_windowed_cache_follows_the_reference_scenario():
    """test_cache.rs:99-124: a first call of 6 tokens with window 4 is stored (and attended) in full; the next call trims.
    Checked through the attention result: with window 4 the decode step after a 6-token prompt must equal a model that
    only ever saw the last 4 positions' K/V — i.e. differ from the unwindowed run — while the prompt's own logits do not."""
    import copy
    _, cfg = case_config("mistral_tiny")
    sd = make_checkpoint(cfg, "f32", seed=9, std=0.1)
    ids = np.arange(1, 9, dtype=np.uint32)
    cw = copy.deepcopy(cfg)
    cw.sliding_window = 4
    full, win = O.OracleModel(cfg, sd, "f32"), O.OracleModel(cw, sd, "f32")
    cf, cwc = full.new_cache(), win.new_cache()
    np.testing.assert_array_equal(full.forward(ids[:6], 0, cf), win.forward(ids[:6], 0, cwc))   # first call: everything
    a, b = full.forward(ids[6:7], 6, cf), win.forward(ids[6:7], 6, cwc)
    assert np.abs(a - b).max() > 1e-4                                                          # second call: trimmed
