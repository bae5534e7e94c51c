"""Decode steps of 1 to 17 sequences of a quantised model: norms folded into the projections and, up to 16 rows, RoPE, KV append and the
merge of the key splits inside the attention kernel. Page edges, split edges, every cluster size, against the oracle."""
import numpy as np
import pytest

from gptrs_b200 import model as gm
from oracle import models_ref as mr

pytestmark = pytest.mark.gpu


# heads decide splits and cluster sizes (two CTAs per SM over rows x kv heads); widths the column tiles of the folded norms
@pytest.mark.parametrize("mode,n_q,n_kv,d,batch,ctx", [
    ("w4", 8, 2, 256, 1, 700), ("w4", 4, 4, 384, 2, 80), ("w4", 16, 2, 128, 3, 300), ("w4", 32, 8, 3072, 1, 150), ("w4", 8, 8, 256, 16, 80), ("w4", 8, 2, 256, 17, 80),
    ("w8", 8, 2, 256, 1, 300), ("w8", 8, 1, 128, 7, 80), ("w8", 4, 2, 512, 16, 200)])
def test_steps_follow_the_oracle(cuda, mode, n_q, n_kv, d, batch, ctx):
    cfg = mr.Cfg("ministral", n_layers=2, d_model=d, n_q=n_q, n_kv=n_kv, hd=128, d_mlp=512, vocab=256, ctx=(ctx + 15) // 16 * 16, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=batch, std=0.5 * d ** -0.5)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (256, d)).astype(np.float32)
    params["lm_head"] = (np.roll(params["tok_embeddings.weight"], 1, 0).T * d ** -0.5).astype(np.float32)   # no close calls
    q = mr.quantised_params(cfg, params, mode)
    pages = cfg.ctx // 16
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_MINISTRAL, 2, d, n_q, n_kv, 128, 512, 256, cfg.ctx, cfg.eps, cfg.theta, 128,
                                      weight_mode=gm.MODE_W4A16 if mode == "w4" else gm.MODE_W8A16, max_seqs=batch, max_tokens=1024, max_logit_rows=batch,
                                      kv_pages=batch * pages + 4, max_pages_per_seq=pages, use_pdl=1), namespace=7300 + batch * 10000 + d + n_q + (mode == "w8") * 5000)
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    rng = np.random.default_rng(batch)
    # the first is long; one ends just below a page, one on it, one just past it
    lengths = [ctx - 24] + [(15, 16, 17, 1, 47)[i % 5] for i in range(batch - 1)]
    prompts = [rng.integers(0, 256, n) for n in lengths]
    refs = [mr.RefModel(cfg, q) for _ in prompts]
    for r, p in zip(refs, prompts):
        r.forward(p)
    m.prefill_many(list(range(batch)), prompts)
    given = rng.integers(0, 256, (6, batch))
    gen = gm.Generator(m, given[0])
    for row in given[:5]:
        want = np.stack([r.forward([int(t)])[-1] for r, t in zip(refs, row)])
        assert gen.step(row).tolist() == want.argmax(1).tolist()
    # a pass of its own with logits sees what the steps left in the cache
    want = np.stack([r.forward([int(t)])[-1] for r, t in zip(refs, given[5])])
    got, _ = m.forward_with_decode_cache(given[5], list(range(batch)), [n + 5 for n in lengths], list(range(batch)))
    assert np.sqrt(np.mean((got - want) ** 2)) <= 2e-2 * np.sqrt(np.mean(want ** 2))   # bf16 activations through two layers


def _model(mode, d, n_q, n_kv, layers, mlp, batch, ctx, max_tokens, namespace):
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_MINISTRAL, layers, d, n_q, n_kv, 128, mlp, 256, ctx, 1e-5, 1e4, 128,
                                      weight_mode=gm.MODE_W4A16 if mode == "w4" else gm.MODE_W8A16, max_seqs=batch, max_tokens=max_tokens, max_logit_rows=batch,
                                      kv_pages=batch * (ctx // 16) + 4, max_pages_per_seq=ctx // 16, use_pdl=1), namespace=namespace)
    cfg = mr.Cfg("ministral", n_layers=layers, d_model=d, n_q=n_q, n_kv=n_kv, hd=128, d_mlp=mlp, vocab=256, ctx=ctx, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=batch, std=0.5 * d ** -0.5)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (256, d)).astype(np.float32)
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    return m


# lanes of 16 + 16, 17 + 16 and 17 + 17 rows, whose norms are summed over column tiles of unlike widths; lanes that both have the rows of
# the widened weights
@pytest.mark.parametrize("mode,d,batch", [("w4", 1024, 32), ("w4", 1024, 33), ("w4", 1024, 34), ("w8", 512, 33), ("w4", 128, 3072)])
def test_two_lanes_give_what_one_gives(cuda, monkeypatch, mode, d, batch):
    """A step in two halves on two streams leaves the cache that a step in one piece leaves: logits of a pass that reads it, to what bf16
    keeps when sums are taken in another order."""
    rng = np.random.default_rng(batch)
    ids = rng.integers(0, 256, (8, batch))
    got = []
    for lanes in ("1", "2"):
        monkeypatch.setenv("GPTRS_LANES", lanes)
        m = _model(mode, d, 2, 1, 2, 256, batch, 16, max(batch, 64), 7800 + batch + int(lanes) * 10000)
        rows = list(range(batch))
        m.prefill_many(rows, [ids[0, s:s + 1] for s in rows])
        gen = gm.Generator(m, ids[1])
        for row in ids[1:7]:
            gen.step(row)
        got.append(m.forward_with_decode_cache(ids[7], rows, [7] * batch, rows)[0])
    diff, scale = np.abs(got[0] - got[1]), np.sqrt(np.mean(got[0] ** 2, axis=1))
    assert np.isfinite(got[1]).all() and (np.sqrt(np.mean(diff ** 2, axis=1)) <= 2e-2 * scale).all()


def test_recorded_steps_past_the_length_they_were_recorded_for(cuda):
    """14 sequences of 64 kv heads: the separate attention kernels would launch alike for 512 and for 1024 visible tokens, the step's own kernel
    would not. One sequence goes from 506 tokens past 512, key and value of every step where they belong."""
    batch, d, ctx = 14, 128, 1024
    m = _model("w4", d, 64, 64, 2, 256, batch, ctx, 1024, 7600)
    rng = np.random.default_rng(1)
    prompts = [rng.integers(0, 256, 506 if s == 5 else 3 + s) for s in range(batch)]
    given = rng.integers(0, 256, (13, batch))
    rows, got = list(range(batch)), []
    for graphs in (False, True):
        for s in rows:
            m.reset_sequence(s)
        m.prefill_many(rows, prompts)
        gen = gm.Generator(m, given[0], use_graph=graphs)
        ids = [gen.step(row).tolist() for row in given[:12]]
        at = [m.sequence_length(s) for s in rows]
        got.append((ids, m.forward_with_decode_cache(given[12], rows, at, rows)[0]))
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
