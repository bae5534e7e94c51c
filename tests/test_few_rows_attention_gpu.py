"""Decode attention of up to 16 rows in one launch (the splits merged by their cluster) against the kernel with scratch and a merge of its own:
page edges, one split and eight, rows without tokens in some splits, a row that sees nothing, lengths above the launch bound."""
import pytest
import torch

from gptrs_b200 import BackendError, lib, ops

pytestmark = pytest.mark.gpu


def _cache(lengths, n_kv, longest, cuda, seed):
    g = torch.Generator(device=cuda).manual_seed(seed)
    per = (longest + 15) // 16
    pool = ops.new_kv_pool(len(lengths) * per, n_kv, cuda)
    pool.view(torch.bfloat16).normal_(generator=g)
    table = torch.randperm(len(lengths) * per, device=cuda, generator=g).int().view(len(lengths), per)
    return g, pool, table


@pytest.mark.parametrize("lengths,n_q,n_kv", [([1], 8, 2), ([16], 8, 8), ([17], 4, 4), ([1500], 32, 8), ([4096], 32, 8), ([65, 64, 63], 8, 1), ([0, 40], 8, 2),
                                              ([300, 1, 128, 129, 15], 16, 4), (list(range(1, 1024, 64)), 32, 8)])
def test_one_launch_equals_two(cuda, lengths, n_q, n_kv):
    longest = max(lengths)
    g, pool, table = _cache(lengths, n_kv, longest, cuda, longest + n_q)
    assert lib().gptrs_cuda_attention_few_rows_splits(longest, len(lengths), n_q, n_kv) > 0
    q = torch.randn((len(lengths), n_q, 128), device=cuda, generator=g).bfloat16()
    slot, ctx = torch.arange(len(lengths), dtype=torch.int32, device=cuda), torch.tensor(lengths, dtype=torch.int32, device=cuda)
    out, status = ops.paged_attention_decode(q, pool, table, slot, ctx, n_q, n_kv, longest)
    ref, _ = ops.paged_attention_decode(q, pool, table, slot, ctx, n_q, n_kv, longest, chunk_pages=4)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for row, n in enumerate(lengths):
        if n == 0:
            assert not out[row].any()
        else:   # one rounding to bf16 each (2^-9), f32 sums in another order, probabilities rounded to bf16 against another maximum
            assert (out[row].float() - ref[row].float()).norm() <= 2 ** -7 * ref[row].float().norm()


@pytest.mark.parametrize("rows,length", [(1, 60), (1, 1500), (1, 4000), (8, 1500), (16, 1000)])
def test_error_is_the_rounding_of_the_output(cuda, rows, length):
    """Probabilities keep 16 bits and sums are f32, so the error against 64 bits is what rounding the exact result to bf16 leaves, and 2^-14 (a few
    f32 ulps of a score in the exponent, 2^-17 of a probability). With probabilities rounded to bf16 it is 17 to 25 % more."""
    g, pool, table = _cache([length] * rows, 8, length, cuda, rows + length)
    q = torch.randn((rows, 32, 128), device=cuda, generator=g).bfloat16()
    slot, ctx = torch.arange(rows, dtype=torch.int32, device=cuda), torch.full((rows,), length, dtype=torch.int32, device=cuda)
    out, status = ops.paged_attention_decode(q, pool, table, slot, ctx, 32, 8, length)
    for row in range(rows):
        k, v = (t.double() for t in ops.kv_gather(pool, table[row], length, 8))
        p = (torch.einsum("hgd,thd->hgt", q[row].double().view(8, 4, 128), k) * 128 ** -0.5).softmax(-1)
        want = torch.einsum("hgt,thd->hgd", p, v).flatten()
        assert (out[row].double() - want).norm() <= (want.bfloat16().double() - want).norm() + 2.0 ** -14 * want.norm()
    assert int(status.item()) == 0


@pytest.mark.parametrize("planned,length,rows,n_kv", [(144, 192, 1, 8), (16, 64, 2, 2), (100, 128, 3, 8), (600, 640, 16, 8), (1500, 1536, 1, 8), (4000, 4032, 2, 8),
                                                      (1000, 1024, 16, 8)])
def test_rows_longer_than_planned(cuda, planned, length, rows, n_kv):
    """A recorded launch is replayed for lengths up to the end of the last chunk that the form with scratch would have, here the planned length
    rounded up to its chunks."""
    assert lib().gptrs_cuda_attention_few_rows_splits(planned, rows, 4 * n_kv, n_kv) > 0
    g, pool, table = _cache([length] * rows, n_kv, length, cuda, planned)
    q = torch.randn((rows, 4 * n_kv, 128), device=cuda, generator=g).bfloat16()
    slot, ctx = torch.arange(rows, dtype=torch.int32, device=cuda), torch.full((rows,), length, dtype=torch.int32, device=cuda)
    out, status = ops.paged_attention_decode(q, pool, table, slot, ctx, 4 * n_kv, n_kv, planned)
    ref, _ = ops.paged_attention_decode(q, pool, table, slot, ctx, 4 * n_kv, n_kv, length)
    assert int(status.item()) == 0
    assert (out.float() - ref.float()).norm() <= 2 ** -7 * ref.float().norm()   # one rounding to bf16 each


def test_lengths_and_shapes_that_do_not_fit(cuda):
    g, pool, table = _cache([100, 100], 2, 100, cuda, 1)
    q = torch.randn((2, 8, 128), device=cuda, generator=g).bfloat16()
    slot = torch.arange(2, dtype=torch.int32, device=cuda)
    own = torch.zeros(1, dtype=torch.int32, device=cuda)
    out, status = ops.paged_attention_decode(q, pool, table, slot, torch.tensor([100, 5000], dtype=torch.int32, device=cuda), 8, 2, 100, status=own)
    assert status is own and int(status.item()) == 2 and torch.isfinite(out.float()).all()
    assert lib().gptrs_cuda_attention_few_rows_splits(100000, 16, 32, 8) == 0 and lib().gptrs_cuda_attention_few_rows_splits(100, 17, 8, 2) == 0
    with pytest.raises(BackendError):
        ops.paged_attention_decode(q, pool, table, slot, slot, 8, 2, 200)   # more than the page table holds


def test_one_library_call_whatever_the_length(cuda, monkeypatch):
    """A chat's length is another one with every token: no size is asked for first, or remembered from an earlier call."""
    g, pool, table = _cache([400], 2, 400, cuda, 1)
    q = torch.randn((1, 8, 128), device=cuda, generator=g).bfloat16()
    slot, called = torch.zeros(1, dtype=torch.int32, device=cuda), []

    class Recorder:
        def __getattr__(self, name):
            called.append(name)
            return getattr(lib(), name)

    monkeypatch.setattr(ops, "lib", Recorder)
    for n in (300, 301, 301):
        ops.paged_attention_decode(q, pool, table, slot, torch.full((1,), n, dtype=torch.int32, device=cuda), 8, 2, n)
    assert called == ["gptrs_cuda_paged_attention_decode_few_rows"] * 3
