"""Greedy and temperature draws over vocabularies at the edges of a cluster's slices: the same token as one pass over the whole row."""
import numpy as np
import pytest
import torch

from gptrs_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,vocab", [(1, 1), (3, 31), (2, 8191), (1, 8192), (5, 8193), (2, 16385), (3, 50257), (1, 65535), (2, 65537), (17, 131072), (1, 200003)])
def test_greedy_takes_the_first_of_the_largest(cuda, rows, vocab):
    g = torch.Generator(cuda).manual_seed(vocab)
    x = torch.randn(rows, vocab, device=cuda, generator=g).round(decimals=1)   # many ties, across slices too
    assert ops.sample_rows(x).tolist() == [int(np.argmax(r)) for r in x.cpu().numpy()]
    x[0] = float("-inf")
    assert ops.sample_rows(x)[0].item() == 0
    x[0, vocab - 1] = -3e38
    x[0, : vocab // 2] = float("nan")   # never the best
    assert ops.sample_rows(x)[0].item() == vocab - 1


def test_a_draw_does_not_depend_on_the_slices(cuda):
    """The first 8000 columns alone are one slice; within 70000 columns (eight slices) whose rest cannot win they draw the same."""
    g = torch.Generator(cuda).manual_seed(1)
    x = torch.full((4, 70000), -1e30, device=cuda)
    x[:, :8000] = torch.randn(4, 8000, device=cuda, generator=g)
    for seed in range(5):
        assert torch.equal(ops.sample_rows(x, temperature=0.8, seed=seed), ops.sample_rows(x[:, :8000].contiguous(), temperature=0.8, seed=seed))
