"""f32 prompts against weights that lie split in memory: row counts around the tiles, widths with and without planes of their own, values whose
bf16 terms overflow, against the f32 oracle."""
import numpy as np
import pytest
import torch

from gptrs_b200 import BackendError, check, lib, ops
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


@pytest.fixture
def starved():
    yield lambda limit=2000: check(lib().gptrs_cuda_debug_matmul_fault(1, limit))
    check(lib().gptrs_cuda_debug_matmul_fault(0, 0))


def product(x, w, status=0):
    (m, k), n = x.shape, w.shape[1]
    y, planes = torch.empty(m, n, device=x.device), torch.empty(6 * k * (m + n) + 256, dtype=torch.uint8, device=x.device)
    check(lib().gptrs_cuda_debug_planes_matmul(x.data_ptr(), w.data_ptr(), None, None, y.data_ptr(), m, n, k, 0, planes.data_ptr(), planes.numel(),
                                               torch.cuda.current_stream().cuda_stream))
    assert ops.matmul_status() == status
    return y


def rms(y, x, w):
    """Root of the mean square of the errors over that of the sums of magnitudes."""
    return float((y.double() - x.double() @ w.double()).norm() / (x.abs().double() @ w.abs().double()).norm())


def operands(m, n, k, cuda):
    g = torch.Generator(cuda).manual_seed(m + n + k)
    return torch.randn(m, k, device=cuda, generator=g), torch.randn(k, n, device=cuda, generator=g), g


@pytest.mark.parametrize("m,n,k", [(24, 768, 768), (64, 768, 3072), (33, 64, 64), (190, 256, 1024), (300, 128, 512), (1001, 132, 64), (64, 516, 2048)])
def test_error_where_plain_f32_is_the_other_choice(cuda, m, n, k):
    """Shapes that the f32 matmul leaves to the kernel for few rows, plain f32 arithmetic (rows by eight). Operands of either sign: not above it. Of
    one sign: an MMA's sum of 16 products is cut by half an ulp on average, 3e-8, beside the 4.6e-8 of plain f32: a quarter more at most (with sums
    over 64 k it is twice as much)."""
    x, w, _ = operands(m, n, k, cuda)
    plain = lambda x, w: torch.cat([ops.matmul_f32(r.contiguous(), w) for r in x.split(8)])  # noqa: E731
    assert rms(product(x, w), x, w) <= rms(plain(x, w), x, w)
    x, w = x.abs(), w.abs()
    assert rms(product(x, w), x, w) <= 1.25 * rms(plain(x, w), x, w)


def _three_terms(shape, g):
    """Positive values whose second and third bf16 terms are positive too, near the largest that such terms can be."""
    term = lambda low, high, unit: torch.randint(low, high, shape, device=g.device, generator=g).float() * unit  # noqa: E731
    return 1 + term(0, 128, 2.0 ** -7) + term(64, 127, 2.0 ** -15) + term(64, 127, 2.0 ** -23)


@pytest.mark.parametrize("m,n,k", [(40, 2304, 768), (129, 4100, 64), (64, 3072, 768), (300, 768, 3072), (937, 2304, 768), (320, 3072, 768), (30, 128, 128)])
def test_no_term_of_the_product_is_missing(cuda, m, n, k):
    """Operands of one sign whose terms all are too: without one of the six products of terms every sum lacks 2^-18 of itself or more (3.7e-6); the
    tensor core's sums, cut and not rounded, lose up to an ulp of 2^-24 at each of the four steps of 64 k, and the additions in f32 half an ulp
    each, at random: below 2^-21. Of either sign: not above plain f32 (half as much again allowed, the orders of the sums differ)."""
    x, w, g = operands(m, n, k, cuda)
    plain = torch.cat([ops.matmul_f32(r.contiguous(), w) for r in x.split(8)])
    assert rms(product(x, w), x, w) <= 1.5 * rms(plain, x, w)
    for a, b in ((x.abs(), w.abs()), (_three_terms((m, k), g), _three_terms((k, n), g))):
        assert rms(product(a, b), a, b) <= 2.0 ** -21


def launches(kind, d, heads, d_mlp, layers, rows=40):
    hd, gpt = d // heads, kind == "gpt"
    cfg = mr.Cfg(kind, n_layers=layers, d_model=d, n_q=heads, n_kv=heads, hd=hd, d_mlp=d_mlp, vocab=32, ctx=64, rot=0 if gpt else hd, theta=1e4)
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_GPT if gpt else gm.KIND_MINISTRAL, layers, d, heads, heads, hd, d_mlp, 32, 64, cfg.eps, cfg.theta, cfg.rot, max_seqs=1,
                                      max_tokens=64, max_logit_rows=1), namespace=9900 + d)
    for name, w in mr.random_params(cfg, seed=1, std=0.05).items():
        m.load_param(name, w)
    m.finalize()
    before = m.stats()["kernel_launches"]
    m.forward_with_decode_cache([1] * rows, [0] * rows, list(range(rows)), [rows - 1])
    return m.stats()["kernel_launches"] - before


# A layer's launches: a norm, qkv, the cache, attention, the output projection, a norm, the MLP in and out (ministral: the rotation, gate and up for MLP in, swiglu),
# and a split of its rows in front of every projection on planes that no norm of up to 2048 columns, a multiple of 128, and no gelu has split them for.
@pytest.mark.parametrize("kind,d,heads,d_mlp,splits", [("gpt", 256, 4, 1024, 1), ("gpt", 192, 3, 328, 3), ("gpt", 2176, 34, 192, 3), ("gpt", 40, 1, 80, 0),
                                                       ("ministral", 256, 4, 512, 3), ("ministral", 320, 5, 328, 4)])
def test_projections_run_on_planes(cuda, kind, d, heads, d_mlp, splits):
    assert launches(kind, d, heads, d_mlp, 3) - launches(kind, d, heads, d_mlp, 2) == (8 if kind == "gpt" else 11) + splits


@pytest.mark.parametrize("m,n,k", [(24, 768, 768), (24, 64, 3072), (64, 2304, 768), (100, 3072, 768), (937, 768, 3072), (937, 3072, 768), (2000, 4096, 128)])
def test_wait_runs_out_sets_status_and_recovers(cuda, starved, m, n, k):
    """The products of the first stage withheld, K of fewer and of more stages than the ring has: all who wait give up, and the next launch is as before."""
    x, w, _ = operands(m, n, k, cuda)
    good = product(x, w)
    starved()
    product(x, w, status=3)   # returns; the result is unspecified
    check(lib().gptrs_cuda_debug_matmul_fault(0, 0))
    assert torch.equal(product(x, w), good)


def test_engine_reports_a_wait_that_ran_out(cuda, starved):
    cfg = mr.Cfg("gpt", n_layers=2, d_model=256, n_q=4, n_kv=4, hd=64, d_mlp=1024, vocab=96, ctx=64)
    m = gm.LoadedModel(gm.ModelConfig(gm.KIND_GPT, 2, 256, 4, 4, 64, 1024, 96, 64, cfg.eps, max_seqs=1, max_tokens=64, max_logit_rows=1), namespace=9950)
    for name, w in mr.random_params(cfg, seed=1, std=0.05).items():
        m.load_param(name, w)
    m.finalize()
    good, _ = m.prefill(0, np.arange(40), want_logits=True)
    m.reset_sequence(0)
    starved()
    with pytest.raises(BackendError) as e:
        m.prefill(0, np.arange(40))
    assert e.value.kind == "Execution" and "matmul" in str(e.value)
    check(lib().gptrs_cuda_debug_matmul_fault(0, 0))
    m.reset_sequence(0)
    assert np.array_equal(m.prefill(0, np.arange(40), want_logits=True)[0], good)


def test_a_model_without_planes(cuda, monkeypatch):
    monkeypatch.setenv("GPTRS_F32_PLANES", "0")
    assert launches("gpt", 256, 4, 1024, 3) - launches("gpt", 256, 4, 1024, 2) == 8   # no splits
    run(256, 4, 1024, 128)
