"""The training gradient where its chunks of 128 samples and its blocks (one
chunk each, then several) end, against the CPU oracle in double precision."""
import numpy as np
import pytest

from asl_b200 import closure as CL
from oracle import mlp_oracle as M
from tests.test_gpu_closure import gpu_grad, rand_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 63, 128, 129, 148 * 128, 148 * 128 + 1, 40000])
def test_gradient_at_chunk_edges(gpu, n):
    p, x, t, norm = rand_problem(n, n)
    g = gpu_grad(p, x, t, norm)
    sse, want = M.loss_and_grad(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64),
                                norm.astype(np.float64), CL.OUT_SCALE)
    # FP32 sums of up to 128 samples per chunk, then of the chunks: roundings
    # grow with the square root of the terms, below 1e-4 of the largest entry
    assert abs(g[len(want)] - sse) <= 1e-4 * sse
    assert np.abs(g[:-1] - want).max() <= 1e-4 * np.abs(want).max()
    assert np.array_equal(g, gpu_grad(p, x, t, norm))
