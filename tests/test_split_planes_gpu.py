"""f32 prompts against weights that lie split in memory: row counts around the tiles, widths with and without planes of their own, values whose
bf16 terms overflow, against the f32 oracle."""
import numpy as np
import pytest

from gptrs_b200 import model as gm
from oracle import models_ref as mr

pytestmark = pytest.mark.gpu


def run(d, heads, d_mlp, rows, edit=lambda p: None, layers=2, vocab=96):
    ctx = (rows + 8) // 8 * 8
    cfg = mr.Cfg("gpt", n_layers=layers, d_model=d, n_q=heads, n_kv=heads, hd=d // heads, d_mlp=d_mlp, vocab=vocab, ctx=ctx)
    params = mr.random_params(cfg, seed=rows, std=0.5 * d ** -0.5)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (vocab, d)).astype(np.float32)
    edit(params)
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_GPT, layers, d, heads, heads, d // heads, d_mlp, vocab, ctx, cfg.eps, max_seqs=1, max_tokens=ctx, max_logit_rows=rows),
                       namespace=9700 + rows * 31 + d)
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    tokens = np.random.default_rng(rows).integers(0, vocab, rows)
    want = mr.RefModel(cfg, params).forward(tokens)
    got, _ = m.forward_with_decode_cache(tokens.astype(np.int32), [0] * rows, list(range(rows)), list(range(rows)))
    # f32 sums of up to 3072 terms in another order, two layers: 3e-7 of the logits, four times that and the oracle's own
    assert np.sqrt(np.mean((got - want) ** 2, axis=1)).max() <= 3e-6 * np.sqrt(np.mean(want ** 2))


@pytest.mark.parametrize("rows", [23, 24, 32, 33, 64, 65, 128, 129, 160, 161, 300, 480, 481])
def test_rows_around_the_tiles(cuda, rows):
    run(256, 4, 1024, rows)


# norms and gelu results that leave planes for the projection behind them or do not; a projection without planes; columns that end inside a tile
@pytest.mark.parametrize("d,heads,d_mlp", [(64, 1, 64), (192, 3, 328), (320, 5, 452), (768, 12, 3072), (2176, 34, 192)])
@pytest.mark.parametrize("rows", [40, 140])
def test_widths(cuda, d, heads, d_mlp, rows):
    run(d, heads, d_mlp, rows)


@pytest.mark.parametrize("rows", [299, 320, 937])
def test_tiles_of_160_rows(cuda, rows):
    run(768, 12, 3072, rows)


@pytest.mark.parametrize("rows", [30, 64, 200])
def test_terms_that_overflow_bf16(cuda, rows):
    def edit(p):   # rounds to infinity as bf16; the product is finite in f32, and all its terms and those of the factor behind it are normal numbers
        p["blocks.0.ln_2.gamma"][5] = 3e-19
        p["blocks.0.ln_2.beta"][5] = 0
        p["blocks.0.feed_forward.w_in"][5, 77] = np.float32(3.4e38)
        p["blocks.0.feed_forward.w_out"][77] *= np.float32(1e-20)
    run(256, 4, 512, rows, edit)
