"""W4 prompts of so many rows that a projection's weights are widened to bf16 first: all its epilogues (folded norms, RoPE + KV append,
SwiGLU, residual) at widths that end inside a 256-column tile, passes whose projections lie on both sides of the line, and small
projections that stay below it with any of these rows, against the oracle."""
import numpy as np
import pytest

from gptrs_b200 import model as gm
from oracle import models_ref as mr

pytestmark = pytest.mark.gpu


# of the projections, the line is at (rows - 1000) x weights = 2e9: only gate and up; all but qkv and the output; all
@pytest.mark.parametrize("lengths", [(1000, 600), (1400, 600), (1000, 37, 1563)])
def test_prompts_of_wide_layers_follow_the_oracle(cuda, lengths):
    _follows(16, 4, 896, lengths, 2560)


@pytest.mark.parametrize("n_q,n_kv,d,lengths", [(4, 1, 384, (900, 700)), (2, 2, 128, (1535,)), (2, 2, 128, (1536,)), (8, 2, 512, (1000, 37, 600))])
def test_prompts_follow_the_oracle(cuda, n_q, n_kv, d, lengths):
    _follows(n_q, n_kv, d, lengths, 384)


def _follows(n_q, n_kv, d, lengths, ff):
    cfg = mr.Cfg("ministral", n_layers=2, d_model=d, n_q=n_q, n_kv=n_kv, hd=128, d_mlp=ff, vocab=128, ctx=1600, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=d, std=0.5 * d ** -0.5)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (128, d)).astype(np.float32)
    q = mr.quantised_params(cfg, params, "w4")
    n = len(lengths)
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_MINISTRAL, 2, d, n_q, n_kv, 128, ff, 128, 1600, cfg.eps, cfg.theta, 128, weight_mode=gm.MODE_W4A16, max_seqs=n,
                                      max_tokens=max(2048, sum(lengths)), max_logit_rows=n, kv_pages=n * 100 + 4, max_pages_per_seq=100), namespace=7900 + d + lengths[0])
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    rng = np.random.default_rng(d)
    prompts = [rng.integers(0, 128, k) for k in lengths]
    refs = [mr.RefModel(cfg, q) for _ in prompts]
    want = np.stack([r.forward(p)[-1] for r, p in zip(refs, prompts)])
    tok = np.concatenate(prompts)
    slots = np.repeat(np.arange(n), lengths)
    pos = np.concatenate([np.arange(k) for k in lengths])
    got, _ = m.forward_with_decode_cache(tok, slots, pos, np.cumsum(lengths) - 1)
    rms = np.sqrt(np.mean(want ** 2))
    assert np.sqrt(np.mean((got - want) ** 2)) <= 2e-2 * rms   # bf16 activations through two layers
    step = rng.integers(0, 128, n)   # and the cache that the pass left behind
    want = np.stack([r.forward([int(t)])[-1] for r, t in zip(refs, step)])
    got, _ = m.forward_with_decode_cache(step, np.arange(n), np.array(lengths), np.arange(n))
    assert np.sqrt(np.mean((got - want) ** 2)) <= 2e-2 * rms
