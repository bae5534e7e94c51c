"""The single-kernel decode step of GPT-2's widths: contexts around the edges of its chunks (64 keys, and as many chunks as the grid has CTAs
for), head sizes, rows of very different lengths, against the f32 oracle."""
import numpy as np
import pytest

from gptrs_b200 import model as gm
from oracle import models_ref as mr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,lengths", [(12, [1]), (12, [63]), (12, [64]), (12, [65]), (12, [129]), (12, [769]), (24, [400]), (6, [191]), (12, [1, 64, 200]),
                                           (12, [300, 63, 65, 2, 128, 127, 1, 64])])
def test_contexts_around_chunk_edges(cuda, heads, lengths):
    batch, ctx, vocab = len(lengths), (max(lengths) + 24) // 8 * 8, 96
    cfg = mr.Cfg("gpt", n_layers=2, d_model=768, n_q=heads, n_kv=heads, hd=768 // heads, d_mlp=3072, vocab=vocab, ctx=ctx)
    params = mr.random_params(cfg, seed=batch, std=0.5 * 768 ** -0.5)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (vocab, 768)).astype(np.float32)
    params["lm_head"] = (np.roll(params["tok_embeddings.weight"], 1, 0).T * 768 ** -0.5).astype(np.float32)   # no close calls
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_GPT, 2, 768, heads, heads, 768 // heads, 3072, vocab, ctx, cfg.eps, max_seqs=batch, max_tokens=1024, max_logit_rows=batch),
                       namespace=8800 + heads * 100 + lengths[0])
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    rng = np.random.default_rng(lengths[0])
    prompts = [rng.integers(0, vocab, n) for n in lengths]
    refs = [mr.RefModel(cfg, params) for _ in prompts]
    for r, p in zip(refs, prompts):
        r.forward(p)
    m.prefill_many(list(range(batch)), prompts)
    given = rng.integers(0, vocab, (4, batch))
    gen = gm.Generator(m, given[0])
    for row in given[:3]:
        want = np.stack([r.forward([int(t)])[-1] for r, t in zip(refs, row)])
        assert gen.step(row).tolist() == want.argmax(1).tolist()
    want = np.stack([r.forward([int(t)])[-1] for r, t in zip(refs, given[3])])
    got, _ = m.forward_with_decode_cache(given[3], list(range(batch)), [n + 3 for n in lengths], list(range(batch)))   # one row: the kernel itself
    # f32 sums of up to 3072 terms in another order, two layers: 3e-7 of the logits, four times that and the oracle's own
    assert np.sqrt(np.mean((got - want) ** 2)) <= 3e-6 * np.sqrt(np.mean(want ** 2))


@pytest.mark.parametrize("batch", [1, 8])
def test_a_step_is_one_launch(cuda, batch):
    cfg = mr.Cfg("gpt", n_layers=2, d_model=768, n_q=12, n_kv=12, hd=64, d_mlp=3072, vocab=96, ctx=32)
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_GPT, 2, 768, 12, 12, 64, 3072, 96, 32, cfg.eps, max_seqs=batch, max_tokens=64, max_logit_rows=batch), namespace=8790)
    for name, w in mr.random_params(cfg, seed=1, std=0.02).items():
        m.load_param(name, w)
    m.finalize()
    m.prefill_many(list(range(batch)), [np.arange(4)] * batch)
    gen, before = gm.Generator(m, [1] * batch), m.stats()["kernel_launches"]
    gen.step()
    gen.step([2] * batch)
    assert m.stats()["kernel_launches"] == before + 2
