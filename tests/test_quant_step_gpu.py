"""The single-kernel decode step of quantised models: fewer tiles than CTAs and warps without a unit, tiles over several warps, group sizes, contexts
around the edges of pages and slices of attention, ids from the device and given, against the oracle and the kernel-per-projection path."""
import numpy as np
import pytest

from gptrs_b200 import BackendError
from gptrs_b200 import model as gm
from oracle import models_ref as mr

pytestmark = pytest.mark.gpu


def _model(mode, n_q, n_kv, d, mlp, vocab, batch, ctx, params, namespace, tables=None):
    pages = (ctx + 15) // 16
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_MINISTRAL, 2, d, n_q, n_kv, 128, mlp, vocab, ctx, 1e-5, 1e4, 128,
                                      weight_mode=gm.MODE_W4A16 if mode == "w4" else gm.MODE_W8A16, max_seqs=batch, max_tokens=1024, max_logit_rows=batch,
                                      kv_pages=batch * pages + 4, max_pages_per_seq=pages, use_pdl=1), namespace=namespace)
    for name, w in params.items():
        m.load_param(name, w)
    if tables:
        m.set_rope_tables(*tables)
    m.finalize()
    return m


@pytest.mark.parametrize("mode,n_q,n_kv,d,mlp,vocab,lengths", [
    ("w4", 1, 1, 128, 128, 64, [1]),                       # one group of 128 k, eight tiles: most CTAs and warps have nothing
    ("w8", 2, 1, 128, 256, 32, [15, 16, 17]),
    ("w4", 8, 1, 384, 640, 1616, [223]), ("w4", 8, 1, 384, 640, 1616, [224]), ("w8", 8, 1, 384, 640, 1616, [225, 111]),   # one slice, two slices of pages
    ("w4", 32, 8, 3072, 1152, 256, [40, 350]),             # odd numbers of units per stage; two tiles of the residual stream in some CTAs
    ("w8", 16, 4, 2048, 4864, 256, [100, 7, 64, 65, 31, 1, 200, 90]),
    ("w4", 6, 2, 256, 5120, 512, [129, 128, 127, 30, 2]),  # groups of three query heads
    ("w4", 4, 4, 512, 512, 256, [600, 17, 33, 500, 18, 1, 300, 16])])
def test_steps_follow_the_oracle(cuda, mode, n_q, n_kv, d, mlp, vocab, lengths):
    batch, ctx = len(lengths), (max(lengths) + 24 + 15) // 16 * 16
    cfg = mr.Cfg("ministral", n_layers=2, d_model=d, n_q=n_q, n_kv=n_kv, hd=128, d_mlp=mlp, vocab=vocab, ctx=ctx, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=batch + d, std=0.5 * d ** -0.5)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (vocab, d)).astype(np.float32)
    params["lm_head"] = (np.roll(params["tok_embeddings.weight"], 1, 0).T * d ** -0.5).astype(np.float32)   # no close calls
    q = mr.quantised_params(cfg, params, mode)
    m = _model(mode, n_q, n_kv, d, mlp, vocab, batch, ctx, params, 7900 + d + batch + lengths[0] * 7)
    rng = np.random.default_rng(batch)
    prompts = [rng.integers(0, vocab, n) for n in lengths]
    refs = [mr.RefModel(cfg, q) for _ in prompts]
    for r, p in zip(refs, prompts):
        r.forward(p)
    m.prefill_many(list(range(batch)), prompts)
    launches = m.stats()["kernel_launches"]
    given = rng.integers(0, vocab, (4, batch))
    gen = gm.Generator(m, given[0])
    for row in given[:3]:
        want = np.stack([r.forward([int(t)])[-1] for r, t in zip(refs, row)])
        got = gen.step(row)
        assert got.tolist() == want.argmax(1).tolist()
    assert m.stats()["kernel_launches"] == launches + 3   # one each
    # the ids of the last step, from the device; then a pass that sees what the steps left in the cache
    want = np.stack([r.forward([int(t)])[-1] for r, t in zip(refs, got)])
    assert gen.step().tolist() == want.argmax(1).tolist()
    want = np.stack([r.forward([int(t)])[-1] for r, t in zip(refs, given[3])])
    logits, _ = m.forward_with_decode_cache(given[3], list(range(batch)), [n + 4 for n in lengths], list(range(batch)))   # one row: the kernel itself
    assert np.sqrt(np.mean((logits - want) ** 2)) <= 2e-2 * np.sqrt(np.mean(want ** 2))   # bf16 activations through two layers


@pytest.mark.parametrize("length", [111, 112, 223, 224, 225])   # the second slice of pages begins with 113 tokens, the third with 225
def test_steps_around_another_slice(cuda, length):
    test_steps_follow_the_oracle(cuda, "w4", 8, 1, 384, 640, 1616, [length])


def test_rows_of_eight_bits_that_are_too_many_values(cuda):
    """Six rows of 9216 values go kernel by kernel, five are one kernel; ids as the oracle's on both sides."""
    cfg = mr.Cfg("ministral", n_layers=2, d_model=256, n_q=2, n_kv=1, hd=128, d_mlp=9216, vocab=256, ctx=64, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=8, std=0.03)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (256, 256)).astype(np.float32)
    params["lm_head"] = (np.roll(params["tok_embeddings.weight"], 1, 0).T * 256 ** -0.5).astype(np.float32)
    for rows in (5, 6):
        m = _model("w8", 2, 1, 256, 9216, 256, rows, 64, params, 7770 + rows)
        prompts = [np.arange(3 + r) for r in range(rows)]
        refs = [mr.RefModel(cfg, mr.quantised_params(cfg, params, "w8")) for _ in prompts]
        for r, p in zip(refs, prompts):
            r.forward(p)
        m.prefill_many(list(range(rows)), prompts)
        gen, before = gm.Generator(m, [7] * rows), m.stats()["kernel_launches"]
        assert gen.step().tolist() == [int(r.forward([7])[-1].argmax()) for r in refs]
        assert (m.stats()["kernel_launches"] == before + 1) == (rows == 5)


@pytest.mark.parametrize("mode", ["w4", "w8"])
def test_steps_do_not_depend_on_the_room_of_the_page_table(cuda, mode):
    """The slices of attention come from the lengths of the step's sequences, so a model with room for more tokens adds up in the same order.
    Eight rows of 1024 values over 40 steps: some of them lie so close to the middle of two bf16 that another order shows."""
    d, vocab, rows = 1024, 512, 8
    cfg = mr.Cfg("ministral", n_layers=2, d_model=d, n_q=8, n_kv=2, hd=128, d_mlp=512, vocab=vocab, ctx=256, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=6, std=0.5 * d ** -0.5)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (vocab, d)).astype(np.float32)
    rng = np.random.default_rng(2)
    prompts, given = [rng.integers(0, vocab, 95 - 5 * r) for r in range(rows)], rng.integers(0, vocab, (41, rows))
    out = []
    for room in (256, 4096):
        m = _model(mode, 8, 2, d, 512, vocab, rows, room, params, 7740 + room)
        m.prefill_many(list(range(rows)), prompts)
        gen = gm.Generator(m, given[0])
        for ids in given[:40]:   # up to and past 112 tokens, where a second slice begins
            gen.step(ids)
        out.append(m.forward_with_decode_cache(given[40], list(range(rows)), [135 - 5 * r for r in range(rows)], list(range(rows)))[0])
    assert np.array_equal(*out)


@pytest.mark.parametrize("mode,first", [("w4", 2017), ("w8", 897)])
def test_long_rows_among_short_ones_leave_the_kernel(cuda, mode, first):
    """Eight rows of eight kv heads: a long row has two slices of pages whatever the others have, and from the tenth (W8: the fifth) round of
    pages on the step goes kernel by kernel, which splits it further; and back when the row has gone. Ids as the oracle's on both sides."""
    d, vocab, rows = 256, 256, 8
    cfg = mr.Cfg("ministral", n_layers=2, d_model=d, n_q=8, n_kv=8, hd=128, d_mlp=256, vocab=vocab, ctx=2064, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=7, std=0.5 * d ** -0.5)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (vocab, d)).astype(np.float32)
    params["lm_head"] = (np.roll(params["tok_embeddings.weight"], 1, 0).T * d ** -0.5).astype(np.float32)
    m = _model(mode, 8, 8, d, 256, vocab, rows, 2064, params, 7760)
    rng = np.random.default_rng(3)
    prompts, given = [rng.integers(0, vocab, n) for n in [first - 4] + [9 + r for r in range(rows - 1)]], rng.integers(0, vocab, (6, rows))
    refs = [mr.RefModel(cfg, mr.quantised_params(cfg, params, mode)) for _ in prompts]
    for r, p in zip(refs, prompts):
        r.forward(p)
    m.prefill_many(list(range(rows)), prompts)
    gen = gm.Generator(m, given[0])
    for k, ids in enumerate(given):   # lengths with the new token: first - 3 ... first + 2
        before = m.stats()["kernel_launches"]
        want = [int(r.forward([int(t)])[-1].argmax()) for r, t in zip(refs, ids)]
        assert gen.step(ids).tolist() == want
        assert (m.stats()["kernel_launches"] - before == 1) == (k < 3)
    m.reset_sequence(0)
    m.prefill(0, prompts[1])
    gen, before = gm.Generator(m, given[0]), m.stats()["kernel_launches"]
    gen.step(given[0])
    assert m.stats()["kernel_launches"] - before == 1


@pytest.mark.parametrize("mode", ["w4", "w8"])
def test_window_slide_and_sampling(cuda, mode, monkeypatch):
    """Steps across the end of the context window, and a temperature draw of one row, as the kernel-per-projection path does them."""
    d, vocab, ctx = 256, 512, 64
    cfg = mr.Cfg("ministral", n_layers=2, d_model=d, n_q=4, n_kv=2, hd=128, d_mlp=512, vocab=vocab, ctx=ctx, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=3, std=0.05)
    params["tok_embeddings.weight"] = np.random.default_rng(0).normal(0, 1, (vocab, d)).astype(np.float32)
    params["lm_head"] = (np.roll(params["tok_embeddings.weight"], 1, 0).T * d ** -0.5).astype(np.float32)
    out = []
    for on in ("1", "0"):
        monkeypatch.setenv("GPTRS_QUANT_STEP", on)
        m = _model(mode, 4, 2, d, 512, vocab, 2, ctx, params, 7700 + (mode == "w8"))
        m.prefill_many([0, 1], [np.arange(60) % vocab, np.arange(50) % vocab])
        gen = gm.Generator(m, [5, 6])
        ids = [gen.step().tolist() for _ in range(20)]
        m.reset_sequence(0)
        m.prefill(0, list(range(30)))
        _, drawn = m.forward_with_decode_cache([7], [0], [30], [0], temperature=0.8, seed=11)
        out.append((ids, drawn.tolist()))
    assert out[0] == out[1]


@pytest.mark.parametrize("own", ["1", "0"])
def test_rotary_tables_set_after_finalize(cuda, own, monkeypatch):
    """Steps read the tables that stand, not those of finalize: the single kernel, and the recorded ones of the kernel-per-projection path."""
    monkeypatch.setenv("GPTRS_QUANT_STEP", own)
    d, vocab, ctx = 256, 512, 64
    cfg = mr.Cfg("ministral", n_layers=2, d_model=d, n_q=4, n_kv=2, hd=128, d_mlp=512, vocab=vocab, ctx=ctx, rot=128, theta=1e4)
    params = mr.random_params(cfg, seed=4, std=0.05)
    angle = np.outer(np.arange(ctx), 30.0 ** -(np.arange(64) / 64))
    tables = np.cos(angle).astype(np.float32), np.sin(angle).astype(np.float32)

    def serve(m):
        m.prefill_many([0, 1], [np.arange(9), np.arange(20) * 3])
        gen = gm.Generator(m, [5, 6])
        for k in range(3):
            gen.step([k, 7 * k])
        return m.forward_with_decode_cache([8], [1], [23], [0])[0]

    m = _model("w4", 4, 2, d, 512, vocab, 2, ctx, params, 7720)
    first = serve(m)
    with pytest.raises(BackendError):
        m.set_rope_tables(*(t[:ctx - 1] for t in tables))
    m.set_rope_tables(*tables)
    for slot in (0, 1):
        m.reset_sequence(slot)
    second = serve(m)
    fresh = _model("w4", 4, 2, d, 512, vocab, 2, ctx, params, 7721, tables)
    assert np.array_equal(second, serve(fresh)) and not np.array_equal(first, second)
