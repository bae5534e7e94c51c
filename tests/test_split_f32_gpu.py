"""f32 matmuls of many rows on the tensor cores (three bf16 terms per value) and the f32 attention of prompt rows, at the edges of their
tiles, against float64."""
import numpy as np
import pytest
import torch

from gptrs_b200 import model as gm, ops, ptir
from gptrs_b200.backend import CudaBackend
from oracle import models_ref as mr

pytestmark = pytest.mark.gpu


def _bound(x, w, extra):
    """A dropped term is below 2^-26 of a product, a sum of 64 products in f32 off by at most 64 ulps of 2^-24, the f32 sums of K / 64
    such parts by K / 64 more; with K up to 3072 that is below 128 ulps of the sum of magnitudes, plus the ulps of the epilogue."""
    return 128 * 2.0 ** -24 * (x.abs().double() @ w.abs().double()) + 4 * 2.0 ** -24 * extra


@pytest.mark.parametrize("m,n,k,form", [
    (24, 2304, 768, "bias"), (32, 3072, 32, ""), (33, 1700, 64, "residual"), (64, 900, 96, "bias"), (65, 768, 3072, "residual"), (128, 400, 160, "gelu"),
    (129, 385, 768, "bias"), (250, 129, 1024, "gelu"), (40, 50257, 64, ""), (300, 130, 32, "residual"),
    (33, 20000, 32, ""), (64, 12900, 96, "bias"), (300, 4100, 32, "residual"), (129, 9000, 64, "gelu")])   # small K: enough columns for this kernel
def test_matmul_of_many_rows(cuda, m, n, k, form):
    g = torch.Generator(cuda).manual_seed(m * 7 + n)
    x, w = torch.randn(m, k, device=cuda, generator=g), torch.randn(k, n, device=cuda, generator=g)
    b = torch.randn(n, device=cuda, generator=g) if form in ("bias", "gelu") else None
    r = torch.randn(m, n, device=cuda, generator=g) if form == "residual" else None
    out = ops.matmul_f32(x, w, bias=b, residual=r, gelu=form == "gelu")
    want, extra = x.double() @ w.double(), 0.0
    for t in (b, r):
        if t is not None:
            want, extra = want + t.double(), extra + t.abs().double()
    bound = _bound(x, w, extra + want.abs())
    if form == "gelu":   # its slope stays below 1.2
        want, bound = torch.nn.functional.gelu(want), 1.2 * bound + 8 * 2.0 ** -24 * want.abs()
    assert ((out.double() - want).abs() <= bound).all()
    assert ops.matmul_status() == 0


def _three_terms(shape, g):
    """Positive values whose second and third bf16 terms are positive too, near the largest that such terms can be."""
    term = lambda low, high, unit: torch.randint(low, high, shape, device=g.device, generator=g).float() * unit  # noqa: E731
    return 1 + term(0, 128, 2.0 ** -7) + term(64, 127, 2.0 ** -15) + term(64, 127, 2.0 ** -23)


@pytest.mark.parametrize("m,n,k", [(129, 4100, 64), (40, 2304, 768), (300, 768, 3072)])
def test_no_term_of_the_product_is_missing(cuda, m, n, k):
    """Root of the mean square of the errors over that of the sums of magnitudes. Operands of either sign: not above what eight rows at a time
    leave (plain f32 arithmetic; half as much again allowed, the orders of the sums differ). Operands of one sign whose terms all are
    too: without one of the six products of terms every sum lacks 2^-18 of itself or more (3.7e-6); the tensor core's sums, cut and not
    rounded, lose up to an ulp of 2^-24 at each of the four steps of 64 k, and K / 64 additions in f32 half an ulp each, at random:
    below 2^-21."""
    g = torch.Generator(cuda).manual_seed(k)
    x, w = torch.randn(m, k, device=cuda, generator=g), torch.randn(k, n, device=cuda, generator=g)
    rms = lambda y, x, w: float((y.double() - x.double() @ w.double()).norm() / (x.abs().double() @ w.abs().double()).norm())  # noqa: E731
    plain = torch.cat([ops.matmul_f32(r.contiguous(), w) for r in x.split(8)])
    assert rms(ops.matmul_f32(x, w), x, w) <= 1.5 * rms(plain, x, w)
    for a, b in ((x.abs(), w.abs()), (_three_terms((m, k), g), _three_terms((k, n), g))):
        assert rms(ops.matmul_f32(a, b), a, b) <= 2.0 ** -21


def test_matmul_of_operands_whose_lower_terms_underflow(cuda):
    """Weights around 2^-118 against inputs around 2^100: a weight is off by what lies below the subnormals of a bf16, 2^-134 at most."""
    g = torch.Generator(cuda).manual_seed(8)
    x, w = torch.randn(64, 256, device=cuda, generator=g) * 2.0 ** 100, torch.randn(256, 2304, device=cuda, generator=g) * 2.0 ** -118
    out, want = ops.matmul_f32(x, w), x.double() @ w.double()
    assert ((out.double() - want).abs() <= _bound(x, w, want.abs()) + 2.0 ** -134 * x.abs().double().sum(1, keepdim=True)).all()


# shares of a warp with every remainder of the loads under way at once, one and two CTAs of eight rows per SM and more
@pytest.mark.parametrize("m,n,k", [(1, 300, 72), (1, 128, 1000), (2, 130, 776), (3, 256, 100), (4, 129, 864), (8, 129, 104), (8, 2304, 768), (12, 2304, 768),
                                   (20, 3072, 100), (23, 2050, 808), (64, 768, 352), (64, 640, 1000)])
def test_matmul_of_few_rows(cuda, m, n, k):
    """Sums of K fused multiply-adds: off by at most K ulps of the sum of magnitudes."""
    g = torch.Generator(cuda).manual_seed(m + k)
    x, w = torch.randn(m, k, device=cuda, generator=g), torch.randn(k, n, device=cuda, generator=g)
    out, mag = ops.matmul_f32(x, w), x.abs().double() @ w.abs().double()
    assert ((out.double() - x.double() @ w.double()).abs() <= k * 2.0 ** -24 * mag).all()


# right operands that the kernel in front has just written: a transpose, a product, an update
@pytest.mark.parametrize("form", ["transpose", "product", "update"])
def test_programs_whose_right_operand_is_computed(cuda, form):
    """From the third execution on a program is a graph whose kernels may start while the one in front ends. 128 rows, K of several
    stages, fresh inputs every time: what a matmul reads has to be this execution's, from its first weights on."""
    be = CudaBackend()
    m, k, n = 128, 512, 256
    b = ptir.Builder()
    a = b.parameter(ptir.F32, [m, k])
    if form == "transpose":
        w = b.parameter(ptir.F32, [n, k])
        b.set_results([ptir.matmul(a, (w + w).transpose([1, 0]))])
        inputs, want = ([m, k], [n, k]), lambda a, w: a @ (2 * w).T
    elif form == "product":
        u, v = b.parameter(ptir.F32, [k, 768]), b.parameter(ptir.F32, [768, n])
        b.set_results([ptir.matmul(a, ptir.matmul(u, v))])
        inputs, want = ([m, k], [k, 768], [768, n]), lambda a, u, v: a @ (u @ v)
    else:
        w, u = b.parameter(ptir.F32, [k, n]), b.parameter(ptir.F32, [40, n])
        b.set_results([ptir.matmul(a, w.dynamic_update_slice(u, b.literal(ptir.SI32, [2], [0, 0]), [40, n]))])
        inputs, want = ([m, k], [k, n], [40, n]), lambda a, w, u: a @ np.concatenate([u, w[40:]])
    prog = be.prepare(b.to_json())
    rng = np.random.default_rng(2)
    handles = [be.materialize(np.zeros(d, np.float32)) for d in inputs]
    for _ in range(8):
        arrays = [rng.normal(size=d).astype(np.float32) for d in inputs]
        ref = want(*(x.astype(np.float64) for x in arrays))
        del handles   # the blocks are handed out again, so that the graph recorded before fits
        handles = [be.materialize(x) for x in arrays]
        got = be.to_literal(prog.run(handles)[0])
        assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
def test_matmul_of_values_that_bf16_cannot_hold(cuda, value):
    """Sums that such a value enters are what plain f32 arithmetic gives; the others keep their bits."""
    g = torch.Generator(cuda).manual_seed(5)
    x, w = torch.randn(200, 256, device=cuda, generator=g), torch.randn(256, 520, device=cuda, generator=g) * 0.1
    w[130] = w[130].sign() * 0.25   # exact in one bf16: the remainders of the products are zeros
    before = ops.matmul_f32(x, w)
    x[77, 130] = value
    out, want = ops.matmul_f32(x, w), x.double() @ w.double()
    fine = torch.isfinite(want) & (want.abs() < 3.4e38)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want.float()))
    assert ((out.double() - want).abs()[fine] <= _bound(x, w, want.abs())[fine]).all()
    rest = torch.arange(200, device=cuda) != 77
    assert torch.equal(out[rest], before[rest])


def test_matmul_of_products_past_the_range(cuda):
    """One product of a sum is an infinity, its second and third terms are infinities of either sign: the sum is the infinity that plain
    f32 arithmetic gives, not NaN. Sums that leave the range and come back are its business too."""
    g = torch.Generator(cuda).manual_seed(6)
    x, w = torch.randn(64, 256, device=cuda, generator=g), torch.randn(256, 1024, device=cuda, generator=g)
    before = ops.matmul_f32(x, w)
    x[9, 40], x[30] = 3.1e30, 0.0
    x[30, :2] = 1.7e38
    w[40] = w[40].sign() * (1e9 + 1e6 * torch.rand(1024, device=cuda, generator=g))
    w[:2, 500] = torch.tensor([1.5, -1.5], device=cuda)
    out = ops.matmul_f32(x, w)
    assert torch.equal(out[9], w[40].sign() * float("inf"))
    plain = torch.zeros((), device=cuda)
    for k in range(2):
        plain = plain + x[30, k] * w[k, 500]
    assert out[30, 500] == plain == 0
    untouched = x[:, 40].abs() > 1e30   # rows whose own operands changed
    untouched[30] = True
    columns = torch.arange(1024, device=cuda) == 500
    keep = ~untouched
    assert torch.isfinite(out[keep]).all()
    x0 = x.clone()
    x0[9], x0[30] = 0, 0
    want = x0.double() @ w.double()
    assert ((out.double() - want).abs()[keep] <= _bound(x0, w, want.abs())[keep]).all() and before.shape == out.shape and columns.any()


@pytest.mark.parametrize("kind,hd,n_q,n_kv", [("gpt", 64, 3, 3), ("ministral", 128, 4, 2)])
def test_prompt_rows_of_several_sequences(cuda, kind, hd, n_q, n_kv):
    """Rows of three sequences in one pass, in portions that leave tiles with rows of two sequences, then one token each: logits of
    the last rows against the oracle."""
    cfg = mr.Cfg(kind, n_layers=2, d_model=64, n_q=n_q, n_kv=n_kv, hd=hd, d_mlp=128, vocab=96, ctx=256, rot=hd if kind == "ministral" else 0, theta=1e4)
    params = mr.random_params(cfg, seed=11, std=0.2)
    mc = gm.ModelConfig(gm.KIND_GPT if kind == "gpt" else gm.KIND_MINISTRAL, cfg.n_layers, cfg.d_model, n_q, n_kv, hd, cfg.d_mlp, cfg.vocab, cfg.ctx, cfg.eps,
                        cfg.theta, cfg.rot, max_seqs=3, max_tokens=256, max_logit_rows=3)
    m = gm.LoadedModel(mc, namespace=7100 + hd)
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    rng = np.random.default_rng(0)
    refs, at = [mr.RefModel(cfg, params) for _ in range(3)], [0, 0, 0]
    for lengths in ((70, 5, 33), (1, 96, 31), (1, 1, 1)):
        tok, sl, pos, rows, want = [], [], [], [], []
        for s, n in enumerate(lengths):
            t = rng.integers(0, cfg.vocab, n)
            want.append(refs[s].forward(t)[-1])
            tok += t.tolist()
            sl += [s] * n
            pos += range(at[s], at[s] + n)
            at[s] += n
            rows.append(len(tok) - 1)
        got, _ = m.forward_with_decode_cache(tok, sl, pos, rows)
        assert np.abs(got - np.stack(want)).max() <= 1e-4 * max(1.0, np.abs(want).max())


def test_passes_of_many_sequences(cuda):
    """Runs of eight rows and more go to tiles, the others to the kernel with a CTA per row and head: prompts of every length around
    that line, a token each, and a pass of both kinds, against the oracle."""
    n = 24
    cfg = mr.Cfg("gpt", n_layers=2, d_model=64, n_q=12, n_kv=12, hd=64, d_mlp=128, vocab=96, ctx=128)
    params = mr.random_params(cfg, seed=12, std=0.2)
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_GPT, 2, 64, 12, 12, 64, 128, 96, 128, cfg.eps, max_seqs=n, max_tokens=512, max_logit_rows=n), namespace=7150)
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    rng = np.random.default_rng(0)
    refs, at = [mr.RefModel(cfg, params) for _ in range(n)], [0] * n
    for lengths in ([(8, 7, 33, 1, 32, 9, 65, 2)[s % 8] for s in range(n)], [1] * n, [{3: 40, 9: 8, 10: 7}.get(s, 1) for s in range(n)]):
        tok, sl, pos, rows, want = [], [], [], [], []
        for s, k in enumerate(lengths):
            t = rng.integers(0, 96, k)
            want.append(refs[s].forward(t)[-1])
            tok += t.tolist()
            sl += [s] * k
            pos += range(at[s], at[s] + k)
            at[s] += k
            rows.append(len(tok) - 1)
        got, _ = m.forward_with_decode_cache(tok, sl, pos, rows)
        assert np.abs(got - np.stack(want)).max() <= 1e-4 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("kind,hd,n_q,n_kv", [("gpt", 64, 8, 8), ("ministral", 128, 8, 2)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_token_that_is_not_finite_reaches_only_rows_that_see_it(cuda, kind, hd, n_q, n_kv, value):
    """Rows of other sequences in the same tile and earlier rows of its own keep their bits. (Widths that leave the matmuls to the f32 kernel,
    whose rows do not meet.)"""
    cfg = mr.Cfg(kind, n_layers=1, d_model=40, n_q=n_q, n_kv=n_kv, hd=hd, d_mlp=80, vocab=96, ctx=128, rot=hd if kind == "ministral" else 0, theta=1e4)
    params = mr.random_params(cfg, seed=3, std=0.2)
    params["tok_embeddings.weight"][95] = value
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_GPT if kind == "gpt" else gm.KIND_MINISTRAL, 1, 40, n_q, n_kv, hd, 80, 96, 128, cfg.eps, cfg.theta, cfg.rot,
                                      max_seqs=3, max_tokens=128, max_logit_rows=128), namespace=7200 + hd + (value != value) * 100)
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    rng = np.random.default_rng(4)
    lengths = (21, 50, 40)
    tok = rng.integers(0, 95, sum(lengths))
    sl, pos = np.repeat(np.arange(3), lengths), np.concatenate([np.arange(n) for n in lengths])
    rows, at = np.arange(len(tok)), 21 + 30   # in the second sequence
    want, _ = m.forward_with_decode_cache(tok, sl, pos, rows)
    tok[at] = 95
    got, _ = m.forward_with_decode_cache(tok, sl, pos, rows)
    hit = (sl == 1) & (rows >= at)
    assert np.array_equal(got[~hit], want[~hit]) and np.isnan(got[hit]).all()


@pytest.mark.parametrize("batch,ctx", [(1, 64), (2, 300), (3, 64), (5, 64), (8, 128), (9, 64)])
def test_steps_of_a_few_sequences(cuda, batch, ctx):
    """GPT-2's widths, where a step of up to eight sequences is one kernel: prompts of unequal lengths packed into one pass, greedy steps,
    and a single token with logits, against the oracle (nine sequences: the kernel-per-projection path)."""
    cfg = mr.Cfg("gpt", n_layers=2, d_model=768, n_q=12, n_kv=12, hd=64, d_mlp=3072, vocab=500, ctx=ctx)
    params = mr.random_params(cfg, seed=2, std=0.05)
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_GPT, 2, 768, 12, 12, 64, 3072, 500, ctx, cfg.eps, max_seqs=batch, max_tokens=400, max_logit_rows=batch),
                       namespace=7000 + batch * 1000 + ctx)
    for name, w in params.items():
        m.load_param(name, w)
    m.finalize()
    rng = np.random.default_rng(batch)
    prompts = [rng.integers(0, 500, ctx - 12 if s == 0 else int(rng.integers(1, ctx - 12))) for s in range(batch)]
    refs = [mr.RefModel(cfg, params) for _ in prompts]
    want = np.stack([r.forward(p)[-1] for r, p in zip(refs, prompts)])
    first = m.prefill_many(list(range(batch)), prompts)
    assert first == want.argmax(1).tolist()
    gen, cur = gm.Generator(m, first), list(first)
    for _ in range(5):
        want = np.stack([r.forward([t])[-1] for r, t in zip(refs, cur)])
        cur = gen.step().tolist()
        assert cur == want.argmax(1).tolist()
    want = refs[-1].forward([7])[-1]
    got, ids = m.forward_with_decode_cache([7], [batch - 1], [m.sequence_length(batch - 1)], [0])
    assert np.abs(got[0] - want).max() <= 1e-4 * max(1.0, np.abs(want).max()) and ids[0] == int(np.argmax(want))
