"""The marching FD step at the edges of its tiles (64 z, 8 or 16 y cells) and
items (runs of x planes), against the numpy oracle in double precision."""
import ctypes as C

import numpy as np
import pytest
import torch

from asl_b200 import fd as FD
from asl_b200 import _lib as L
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


class Field:
    """Device memory of the solver as an array that torch reads in place."""

    def __init__(self, pointer, shape):
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(pointer, False), version=2)


@pytest.mark.parametrize("q", [7, 15, 19])
def test_more_than_2_to_32_cells(gpu, q):
    """A block whose element indices do not fit 32 bits (two fields of 17.3 GB):
    random planes at both ends and around 2^32 cells, zero elsewhere."""
    gx, gy, gz = 4120, 1030, 1020
    per_plane = gy * gz
    assert gx * per_plane > 2**32 + 20 * per_plane
    lib, h = L.load(), C.c_void_p()
    L.check(lib.aslb_fd_create(gx - 2, gy - 2, gz - 2, q, L.F32, 0.07, C.byref(h)))
    try:
        field = torch.as_tensor(Field(lib.aslb_fd_device_field(h), (gx, gy, gz)), device="cuda")
        rng = np.random.default_rng(q)
        blocks = [0, 2**32 // per_plane - 3, gx - 7]  # first planes of seven each
        part = {x: rng.uniform(0.2, 1.2, (7, gy, gz)).astype(np.float32) for x in blocks}
        for x, v in part.items():
            field[x:x + 7] = torch.from_numpy(v).cuda()
        torch.cuda.synchronize()
        L.check(lib.aslb_fd_step(h, 1))
        L.check(lib.aslb_fd_sync(h))
        out = torch.as_tensor(Field(lib.aslb_fd_device_field(h), (gx, gy, gz)), device="cuda")
        for x, v in part.items():
            got = out[x + 1:x + 6, 1:-1, 1:-1].cpu().numpy()
            # 20 FP32 operations on values up to 1.2 (a rounding is 6e-8 of its size)
            assert np.abs(got - fd_step(v.astype(np.float64), 0.07, q, None, False)[1:-1, 1:-1, 1:-1]).max() < 2e-6
        # planes whose neighbours are zero too
        for x in (9, blocks[1] // 2, blocks[1] - 3, blocks[1] + 9, gx - 10):
            assert not out[x, 1:-1, 1:-1].any()
    finally:
        lib.aslb_fd_destroy(h)


@pytest.mark.parametrize("q", [7, 15, 19])
@pytest.mark.parametrize("flow", [False, True])
def test_one_rounding_of_the_centre(gpu, q, flow):
    """A step adds its increment to the centre once. Values in [1, 2) round with
    a root mean square of 2^-23 / sqrt(12); the increment is a twentieth of
    them or less and its dozen roundings add a tenth of that, a second rounding
    of the sum would add 40 %."""
    shape = (20, 34, 66)
    g = tuple(s + 2 for s in shape)
    rng = np.random.default_rng(q)
    c = rng.uniform(1.4, 1.6, g).astype(np.float32)
    u = rng.uniform(-0.05, 0.05, (3, *g)).astype(np.float32)
    lb = A.LBGK(A.Block(shape), 0.05, A.d3q19())
    A.LBGKUtilities(lb).initF(u.astype(np.float64))
    fd = FD.generateFDAdvectionDiffusion(c, 0.01, lb if flow else None, q, False)
    fd.execute()
    want = fd_step(c.astype(np.float64), np.float64(np.float32(0.01)), q, u.astype(np.float64) if flow else None, False)
    err = (fd.getC() - want)[1:-1, 1:-1, 1:-1]
    assert np.sqrt((err**2).mean()) < 1.2 * 2.0**-23 / np.sqrt(12)
