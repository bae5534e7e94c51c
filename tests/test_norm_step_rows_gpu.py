"""The norm step of few rows, which asks for everything at once, and the one of many, on both sides of the line and of eight experts: the same
bits for the same row."""
import pytest
import torch

from gptrs_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [4, 512, 516, 1024, 2048, 4096])
@pytest.mark.parametrize("top", [0, 1, 8, 9])
def test_few_and_many_rows_agree(cuda, dim, top):
    g = torch.Generator(cuda).manual_seed(dim + top)
    rows = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 1   # one more than the kernel of few rows takes
    pairs = max(top, 1)
    x = torch.randn(rows, dim, device=cuda, generator=g)
    y = torch.randn(rows * pairs, dim, device=cuda, generator=g).bfloat16()
    go, gi = torch.randn(dim, device=cuda, generator=g), torch.randn(dim, device=cuda, generator=g)
    pair = torch.randperm(rows * pairs, device=cuda, generator=g).int().view(rows, pairs) if top else None
    weight = torch.rand(rows, pairs, device=cuda, generator=g) if top else None
    results = []
    for n in (rows, rows - 1):
        xs = x[:n].clone()
        h = ops.norm_step(xs, 1e-5, y=y if top else y[:n], gamma_out=go, gamma_in=gi, pair=pair[:n].contiguous() if top else None,
                          pair_weight=weight[:n].contiguous() if top else None, out_dtype=torch.bfloat16)
        results.append((xs[:rows - 1], h[:rows - 1]))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    s = (weight.double()[..., None] * y.double()[pair.long()]).sum(1) if top else y[:rows].double()
    want = x.double() + s / (s.square().mean(1, keepdim=True) + 1e-5).sqrt() * go
    # a sum of dim squares and one of at most nine rows in f32, then a handful of roundings
    assert ((results[0][0].double() - want[:-1]).abs() <= 2e-6 * (1 + want[:-1].abs() + go.abs() * 4)).all()
