"""Slices that are views of their operand, and dynamic updates in one launch, bit for bit against the numpy interpreter."""
import json

import numpy as np
import pytest

from gptrs_b200 import ptir
from gptrs_b200.backend import CudaBackend
from oracle import ptir_ref as pr

pytestmark = pytest.mark.gpu
F32, SI32 = ptir.F32, ptir.SI32


@pytest.fixture(scope="module")
def be(cuda):
    return CudaBackend()


def _run(be, b, inputs):
    prog = b.to_json()
    want = pr.run_program(json.loads(prog), inputs)
    for fusion in (True, False):
        be.set_fusion(fusion)
        hs = [be.materialize(a) for a in inputs]
        for _ in range(4):   # the later calls replay a graph
            got = [be.to_literal(h) for h in be.run_program(prog, hs)]
            assert len(got) == len(want) and all(np.array_equal(a, e) for a, e in zip(got, want))
    be.set_fusion(True)


# in one piece on a 256-byte boundary; off it; rows; a column block (several pieces); the whole; inner axes cut
@pytest.mark.parametrize("dims,starts,sizes", [([1, 256], [0, 64], [1, 128]), ([1, 256], [0, 1], [1, 128]), ([6, 64], [2, 0], [3, 64]), ([6, 64], [2, 0], [3, 32]),
                                               ([4, 64], [0, 0], [4, 64]), ([3, 4, 64], [1, 2, 0], [1, 2, 64]), ([3, 4, 64], [1, 0, 0], [2, 2, 64]), ([512], [128], [100])])
@pytest.mark.parametrize("use", ["computed", "result", "reshaped result", "outlives its source"])
def test_slices(be, dims, starts, sizes, use):
    rng = np.random.default_rng(3)
    b = ptir.Builder()
    x = b.parameter(F32, dims)
    y = x + x
    s = y.slice(starts, sizes)
    n = int(np.prod(sizes))
    if use == "computed":
        b.set_results([s * s, y])
    elif use == "result":
        b.set_results([s, s + s])
    elif use == "reshaped result":
        b.set_results([s.reshape([n]), s + s])
    else:   # buffers of dead values are given to later ones: the sliced value has to live as long as its view
        t = x * x
        t = t + t
        t = t * x
        b.set_results([s.reshape([n]) * s.reshape([n]), t])
    _run(be, b, [rng.normal(size=dims).astype(np.float32)])


@pytest.mark.parametrize("dims,sizes,starts", [([5, 8], [2, 3], [1, 2]), ([5, 8], [2, 8], [-4, 0]), ([5, 8], [2, 5], [9, 9]), ([12, 16, 64], [12, 1, 64], [0, 7, 0]),
                                               ([3, 4, 4], [1, 1, 1], [2, 3, 3]), ([16], [16], [3]), ([4, 7], [2, 3], [1, 5]), ([2, 3, 4, 12], [1, 2, 3, 5], [1, 0, 1, 6])])
@pytest.mark.parametrize("dtype", [F32, SI32])
def test_updates(be, dims, sizes, starts, dtype):
    rng = np.random.default_rng(4)
    b = ptir.Builder()
    x, u, s = b.parameter(dtype, dims), b.parameter(dtype, sizes), b.parameter(SI32, [len(dims)])
    b.set_results([x.dynamic_update_slice(u, s, sizes)])
    kind = np.float32 if dtype == F32 else np.int32
    _run(be, b, [rng.integers(-99, 99, dims).astype(kind), rng.integers(100, 999, sizes).astype(kind), np.array(starts, np.int32)])


def test_update_of_an_axis_longer_than_int(be):
    n = 2 ** 31 + 8
    b = ptir.Builder()
    u, at = b.parameter(SI32, [4]), b.parameter(SI32, [1])
    y = b.iota([n], 0).dynamic_update_slice(u, at, [4])
    b.set_results([y.slice([996], [12])])
    got, = be.run_program(b.to_json(), [be.materialize(np.array([-1, -2, -3, -4], np.int32)), be.materialize(np.array([1000], np.int32))])
    assert be.to_literal(got).tolist() == [996, 997, 998, 999, -1, -2, -3, -4, 1004, 1005, 1006, 1007]
