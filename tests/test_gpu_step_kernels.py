"""The stream-collide's two-cells-per-thread kernel and the time loop's merged
conditions, at the sizes where they change form, against the one-cell kernel
and the separate launches: the same bits (the packed collision rounds each
cell as the scalar one does, and merging only regroups independent copies)."""
import numpy as np
import pytest
import torch

from asl_b200 import _lib as L
from asl_b200 import lbgk as A
from tests.test_gpu_parity import smooth_field, sphere_map

pytestmark = pytest.mark.gpu
VT = {15: A.d3q15(), 19: A.d3q19(), 27: A.d3q27()}


def populations(make, variants=(0, 2)):
    out = []
    for v in variants:
        lb = make(v)
        out.append((lb.getF(), lb.getVelocity(), lb.getRho()))
    return out


def assert_same(out):
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("q", [15, 19, 27])
@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("closure", [L.CLOSURE_NONE, L.CLOSURE_ASL_INTENT, L.CLOSURE_SMAGORINSKY])
@pytest.mark.parametrize("nz", [1, 2, 31, 32, 33, 64, 65, 130])
def test_pair_kernel_wraps_z_and_packs_bitwise(gpu, q, storage, closure, nz):
    """Rows around one and two cells per lane, with the z axis periodic."""
    shape = (5, 3, nz)
    rho, u = smooth_field(tuple(s + 2 for s in shape), nz + q)

    def make(variant):
        lb = A.LBGK(A.Block(shape), 0.01, VT[q], storage=storage, periodic=(True, nz % 2 == 0, True),
                    body_force=(1e-4, -2e-4, 1e-4))
        lb.setKernel(variant)
        lb.setClosure(closure)
        A.LBGKUtilities(lb).initF(rho, u)
        lb.run(5)
        return lb

    assert_same(populations(make))


@pytest.mark.parametrize("q", [15, 19, 27])
@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("closure", [L.CLOSURE_NONE, L.CLOSURE_ASL_INTENT, L.CLOSURE_SMAGORINSKY])
@pytest.mark.parametrize("nz", [1, 31, 33, 64, 97])
@pytest.mark.parametrize("periodic", [(False, False, False), (True, True, False)])
def test_closures_without_links_or_periodic_z(gpu, q, storage, closure, nz, periodic):
    """The unmasked pair kernel (closures; FP16 as neighbouring cells) where z
    does not wrap, its walls as separate conditions."""
    shape = (5, 4, nz)
    rho, u = smooth_field(tuple(s + 2 for s in shape), nz + q)

    def make(variant):
        lb = A.LBGK(A.Block(shape), 0.01, VT[q], storage=storage, periodic=periodic, body_force=(1e-4, -2e-4, 1e-4))
        lb.setKernel(variant)
        lb.setClosure(closure)
        A.LBGKUtilities(lb).initF(rho, u)
        walls = [A.generateBCNoSlip(lb, [A.Z0, A.ZE])]
        if not periodic[0]:
            walls.append(A.generateBCNoSlip(lb, [A.X0, A.XE, A.Y0, A.YE]))
        lb.run(5, walls)
        return lb

    assert_same(populations(make))


@pytest.mark.parametrize("q", [15, 19, 27])
@pytest.mark.parametrize("storage", ["f32", "f16", "f64"])
@pytest.mark.parametrize("nz", [5, 32, 40, 97])
def test_fused_sphere_through_a_wall(gpu, q, storage, nz):
    """A sphere cut by a fused wall has cells with both kinds of links; the
    fields computed from the populations follow the links too."""
    shape = (9, 8, nz)
    m = sphere_map(tuple(s + 2 for s in shape), (4.0, 0.5, nz / 2.0), 2.7)
    rho, u = smooth_field(tuple(s + 2 for s in shape), 5)

    def make(variant):
        lb = A.LBGK(A.Block(shape), 0.02, VT[q], storage=storage, periodic=(True, False, False), body_force=(1e-4, 0, 0))
        lb.setKernel(variant)
        A.LBGKUtilities(lb).initF(rho, u)
        bcs = [A.generateBCNoSlip(lb, [A.Y0, A.YE, A.Z0, A.ZE]), A.generateBCNoSlip(lb, m)]
        for b in bcs:
            b.fuse()
        lb.run(7, bcs)
        A.LBGKUtilities(lb).computeRhoVelocity()
        return lb

    out = populations(make)
    assert_same(out)
    # the fields against the exported populations
    f, vel, dens_out = out[0]
    c, w = A.lattice_vectors(q), A.lattice_weights(q)
    inner = (slice(1, -1),) * 3
    dens = np.tensordot(w, f, 1)[inner]
    mom = np.tensordot((w[:, None] * c).T, f, 1)[(slice(None), *inner)]
    tol = 1e-13 if storage == "f64" else 4e-6  # 27 FP32 terms of size 1
    assert np.abs(dens_out[inner] - dens).max() < tol
    assert np.abs(vel[(slice(None), *inner)] - mom / dens).max() < tol
    lb = make(0)
    assert np.allclose(lb.moments(), [dens.sum(), *mom.reshape(3, -1).sum(1)], rtol=1e-9, atol=1e-7 * dens.size)


@pytest.mark.parametrize("storage", ["f32", "f16", "f64"])
@pytest.mark.parametrize("case", ["channel", "two_maps", "sphere_at_wall", "periodic", "fused_last"])
@pytest.mark.parametrize("steps", [3, 4, 21, 43])
def test_merged_conditions_equal_separate_ones(gpu, storage, case, steps):
    """run() of 4 steps or more merges consecutive conditions (and of 32 or more
    replays eight steps at a time); walls share edge links (the later
    condition's value stays), and two maps whose links read each other's slots
    are left separate. Lists in turn, lists that take another's place, and
    lists after a condition was destroyed."""
    shape = (14, 10, 9)
    g = tuple(s + 2 for s in shape)
    rho, u = smooth_field(g, 11, amp=0.02)
    out = []
    for merged in (True, False):
        lb = A.LBGK(A.Block(shape), 0.03, A.d3q19(), storage=storage, periodic=(False, False, case == "periodic"))
        A.LBGKUtilities(lb).initF(rho, u)
        walls = [A.Y0, A.YE] + ([] if case == "periodic" else [A.Z0, A.ZE])
        bcs = [A.generateBCConstantVelocity(lb, (0.03, 0.01, 0.0), [A.X0]), A.generateBCNoSlip(lb, walls),
               A.generateBCConstantPressure(lb, 1.01, [A.XE])]
        if case == "two_maps":
            bcs.append(A.generateBCNoSlip(lb, sphere_map(g, (5.0, 5.0, 4.0), 2.0)))
            bcs.append(A.generateBCConstantPressure(lb, 1.02, -sphere_map(g, (5.0, 5.0, 4.0), 2.0)))
        elif case == "sphere_at_wall":
            bcs.append(A.generateBCNoSlip(lb, sphere_map(g, (6.0, 1.0, 4.0), 2.6)))
        elif case == "fused_last":
            bcs.append(A.generateBCNoSlip(lb, sphere_map(g, (6.0, 5.0, 4.0), 2.6)))
            bcs[-1].fuse()

        def go(which):
            if merged:
                lb.run(steps, which)
            else:
                for _ in range(steps):
                    lb.execute()
                    A.executeAll(which)

        # the same list twice, another in turn with it, then others in its place, then back
        others = [[bcs[0], *bcs[2:]], bcs[:2], [bcs[2], bcs[0], *bcs[3:]]]
        for which in (bcs, bcs, others[1], bcs, others[0], others[0], others[1], others[1], others[2], others[2], bcs, bcs):
            go(which)
        del bcs[1], which, others
        go(bcs)
        go(bcs)
        out.append((lb.getF(), lb.getVelocity(), lb.getRho()))
    assert_same(out)


@pytest.mark.parametrize("storage", ["f32", "f64"])
@pytest.mark.parametrize("order", ["ABA", "ABAC", "ABCABC", "AfABC", "ABACDBD"])
def test_lists_that_name_a_condition_twice(gpu, storage, order):
    """A condition may stand more than once in a list of a run: walls that
    share edge links (A, B, C, D; the last writer's value stays), and a
    condition on the density field between them (f)."""
    shape = (8, 7, 9)
    g = tuple(s + 2 for s in shape)
    rho, u = smooth_field(g, 3, amp=0.02)
    out = []
    for merged in (True, False):
        lb = A.LBGK(A.Block(shape), 0.03, A.d3q19(), storage=storage)
        A.LBGKUtilities(lb).initF(rho, u)
        bcs = {"A": A.generateBCNoSlip(lb, [A.Y0, A.YE]), "B": A.generateBCConstantVelocity(lb, (0.03, 0.01, 0.0), [A.X0]),
               "C": A.generateBCConstantPressure(lb, 1.01, [A.XE]),
               "D": A.generateBCConstantPressureVelocity(lb, 1.02, (0.0, 0.01, 0.0), [A.Z0]),
               "f": A.generateBCNoSlipRho(lb, sphere_map(g, (4.0, 3.0, 4.0), 1.6))}
        which = [bcs[k] for k in order]
        for _ in range(2):  # as recorded first, then replayed
            if merged:
                lb.run(6, which)
            else:
                for _ in range(6):
                    lb.execute()
                    A.executeAll(which)
        out.append((lb.getF(), lb.getVelocity(), lb.getRho()))
    assert_same(out)


@pytest.mark.parametrize("recorded", ["walls", "none", "both"])
def test_merged_conditions_around_a_recording(gpu, recorded):
    """A run that the caller records on the domain's stream, with one condition,
    none, or the merged list, leaves the merged launches before and after it,
    and its own replay, as they are."""
    shape = (8, 7, 9)
    rho, u = smooth_field(tuple(s + 2 for s in shape), 3, amp=0.02)
    out = []
    for merged in (True, False):
        lb = A.LBGK(A.Block(shape), 0.03, A.d3q19())
        A.LBGKUtilities(lb).initF(rho, u)
        inlet = A.generateBCConstantVelocity(lb, (0.03, 0.01, 0.0), [A.X0])
        walls = A.generateBCNoSlip(lb, [A.Y0, A.YE, A.Z0, A.ZE])
        outlet = A.generateBCConstantPressure(lb, 1.01, [A.XE])
        in_graph = {"walls": [walls], "none": [], "both": [inlet, walls]}[recorded]

        def loop(n, which):
            for _ in range(n):
                lb.execute()
                A.executeAll(which)

        if merged:
            lb.run(8, [inlet, walls])
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.stream(torch.cuda.ExternalStream(lb.stream)):
                graph.capture_begin(capture_error_mode="thread_local")
                lb.run(4, in_graph, use_graph=False)
                graph.capture_end()
            lb.run(8, [inlet, outlet])
            with torch.cuda.stream(torch.cuda.ExternalStream(lb.stream)):
                graph.replay()
            lb.run(8, [inlet, outlet])
            lb.run(5, [inlet, walls])
        else:
            loop(8, [inlet, walls])
            loop(8, [inlet, outlet])
            loop(4, in_graph)
            loop(8, [inlet, outlet])
            loop(5, [inlet, walls])
        out.append((lb.getF(), lb.getVelocity(), lb.getRho()))
    assert_same(out)


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("q", [15, 19])
@pytest.mark.parametrize("shape", [3, 4])
def test_batch_pairs_across_planes(gpu, q, storage, shape):
    """Two cells per thread in planes below, at and above a block's cells, so
    that a pair spans two planes or lacks its second cell; fields included."""
    sizes = [(3, 1, 1), (7, 5, 9), (5, 6, 1), (4, 16, 20), (9, 17, 19), (2, 32, 20), (1, 40, 33)]

    def domains():
        out = []
        for i, size in enumerate(sizes):
            g = tuple(s + 2 for s in size)
            lb = A.LBGK(A.Block(size), 0.01 + 0.01 * i, VT[q], storage=storage, body_force=(1e-4, 0, 1e-4), packed_rows=True)
            A.LBGKUtilities(lb).initF(*smooth_field(g, i, amp=0.02))
            bcs = [A.generateBCNoSlip(lb, [A.X0, A.XE, A.Y0, A.YE, A.Z0, A.ZE])]
            if size[0] == 9:
                bcs.append(A.generateBCNoSlip(lb, sphere_map(g, (5.0, 8.0, 9.0), 3.4)))
            for b in bcs:
                b.fuse()
            out.append((lb, bcs))
        return out

    alone, together = domains(), domains()
    for lb, bcs in alone:
        lb.run(5, bcs)
        lb.sync()
    batch = A.Batch([lb for lb, _ in together])
    batch.setShape(shape)
    batch.run(5, [bcs for _, bcs in together])
    batch.sync()
    for (a, _), (b, _) in zip(alone, together):
        inner = (..., slice(1, -1), slice(1, -1), slice(1, -1))
        assert_same([(x.getF(), x.getVelocity()[inner], x.getRho()[inner]) for x in (a, b)])
