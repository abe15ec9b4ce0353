"""The marching FD step at the edges of its tiles (64 z, 8 or 16 y cells) and
items (runs of x planes), against the numpy oracle in double precision."""
import numpy as np
import pytest

from asl_b200 import fd as FD
from asl_b200 import lbgk as A
from oracle.fd_oracle import fd_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [7, 15, 19])
@pytest.mark.parametrize("cc", [False, True])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 8, 63), (3, 9, 64), (5, 16, 65), (4, 17, 129), (70, 7, 2), (33, 15, 66)])
def test_tile_edges_match_oracle(gpu, q, cc, shape):
    g = tuple(s + 2 for s in shape)
    rng = np.random.default_rng(sum(shape) + q)
    c = rng.uniform(0.2, 1.2, g).astype(np.float32)
    u = rng.uniform(-0.08, 0.08, (3, *g)).astype(np.float32)
    lb = A.LBGK(A.Block(shape), 0.05, A.d3q19())
    A.LBGKUtilities(lb).initF(u.astype(np.float64))
    for flow in (None, lb):
        fd = FD.generateFDAdvectionDiffusion(c, 0.07, flow, q, cc and flow is not None)
        ref = c.astype(np.float64)
        for _ in range(3):
            fd.execute()
            ref = fd_step(ref, 0.07, q, None if flow is None else u.astype(np.float64), cc and flow is not None)
        # three steps of about 60 FP32 operations on values up to 1.2 (a
        # rounding is 6e-8 of its size, the products are a tenth of c)
        assert np.abs(fd.getC() - ref).max() < 2e-6
