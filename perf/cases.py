"""The calls that a program built on this framework spends its time in, as cases that can be timed and checked.

A case is a dict of plain values. `prepare` builds what a program holds before its time loop (domain, conditions, solver,
network), `run` takes one stretch of that loop through the public entry points and returns the fields that the program reads
afterwards, on the device where the framework keeps them there. `exact` is the same model in plain torch, in 64 bits.

Kinds of case:
  flow    an LBGK domain with its conditions: `execute(); executeAll(bcs)` step by step ("loop") or `run(n, bcs)` ("run"),
          with density and velocity written by every step ("every") or computed at the end of the stretch ("end")
  batch   many small channels advanced together
  fd      advection-diffusion on a frozen or a running flow
  train   the learned closure's training steps
"""
import ctypes
import math

import numpy as np
import torch

from asl_b200 import _lib as L
from asl_b200 import closure as CL
from asl_b200 import fd as FD
from asl_b200 import lbgk as A

DEV = "cuda" if torch.cuda.is_available() else "cpu"
BYTES = {"f32": 4, "f16": 2, "f64": 8}


def _flow(nx, ny, nz, scene, steps, name=None, q=19, storage="f32", closure="none", fuse=False, drive="run", macro="end",
          force=False, period=32):
    case = dict(kind="flow", nx=nx, ny=ny, nz=nz, q=q, storage=storage, scene=scene, closure=closure, fuse=fuse, drive=drive,
                macro=macro, force=force, steps=steps, period=period)
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # the smallest domain that the examples and checks step, as an ASL program steps it: one call per step and condition
        _flow(48, 24, 24, "channel", 20, "small_channel_loop", drive="loop", macro="every"),
        # the canonical laminar program's domain: inlet, outlet, walls and an obstacle, then the drag on it
        _flow(128, 64, 64, "channel", 51, "channel_128x64x64", macro="every", force=True),
        # the benchmark's porous medium in a smaller box, FP32 storage, walls and grains folded into the step
        _flow(384, 192, 192, "porous", 10, "porous_f32", fuse=True),
        # the same medium in FP16 storage, rows of another length, an odd number of steps
        _flow(320, 208, 256, "porous", 11, "porous_f16", storage="f16", fuse=True),
        # a pressure-driven D3Q15 channel in double precision with sizes that fit no tile
        _flow(131, 67, 93, "pressure", 11, "pressure_f64_ragged", q=15, storage="f64", macro="every"),
        # bluff bodies in a wind tunnel, D3Q27, with the force on them
        _flow(256, 128, 128, "tunnel", 10, "tunnel_d3q27", q=27, fuse=True, force=True),
        # decaying periodic turbulence with the Smagorinsky closure
        _flow(160, 160, 160, "turbulence", 10, "turbulence_smagorinsky", closure="smagorinsky"),
        # the same with the learned closure: a refresh of its field and the steps that use it
        _flow(128, 128, 128, "turbulence", 32, "turbulence_learned", closure="mlp"),
        # many small channels of different sizes at once
        dict(name="batch_channels", kind="batch", n=48, storage="f32", steps=20, sizes=7),
        # a passive scalar on a frozen flow, wide stencil
        dict(name="scalar_d3q19_frozen", kind="fd", nx=256, ny=192, nz=192, q=19, storage="f32", coupled=False, cc=False,
             steps=8),
        # a scalar carried along with the running flow, narrow stencil, ragged sizes
        dict(name="scalar_d3q7_coupled", kind="fd", nx=203, ny=101, nz=177, q=7, storage="f32", coupled=True, cc=True, steps=9),
        # mini-batch steps of the closure's training at the batch size that its training uses
        dict(name="closure_training", kind="train", batch=16384, steps=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "flow", "flow", "batch", "fd", "fd", "train"])
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(6, 48), storage=rng.choice(["f32", "f16"]), steps=rng.randint(12, 18),
                    sizes=rng.randrange(1 << 20))
    if kind == "train":
        return dict(kind="train", batch=_log(rng, 1000, 40000), steps=rng.randint(2, 12))
    size = [_log(rng, 24, 320), _log(rng, 20, 192), _log(rng, 20, 256)]
    if kind == "fd":
        return dict(kind="fd", nx=size[0], ny=size[1], nz=size[2], q=rng.choice([7, 15, 19]),
                    storage=rng.choice(["f32", "f32", "f64"]), coupled=rng.random() < 0.4, cc=rng.random() < 0.5,
                    steps=rng.randint(3, 9))
    scene = rng.choice(["channel", "porous", "pressure", "tunnel", "turbulence"])
    storage = rng.choice(["f32", "f32", "f16", "f64"])
    closure = "none"
    if scene == "turbulence":
        size = [_log(rng, 24, 160)] * 3
        closure = rng.choice(["none", "smagorinsky", "mlp" if storage != "f64" else "none"])
    elif scene == "tunnel":
        closure = rng.choice(["none", "smagorinsky"])
    q = {"pressure": 15, "tunnel": 27}.get(scene, 19)
    steps = min(rng.randint(5, 20), max(2, int(2e10 / (2 * q * BYTES[storage] * math.prod(size)))))
    return _flow(*size, scene, steps, q=q, storage=storage, closure=closure,
                 fuse=scene in ("channel", "porous", "tunnel") and rng.random() < 0.6,
                 drive=rng.choice(["run", "run", "loop"]), macro=rng.choice(["end", "every"]),
                 force=scene in ("channel", "tunnel") and rng.random() < 0.5, period=rng.choice([4, 8, 32]))


# ---- scenes: parameters, maps and fields from the case and the seed alone ---------------------------------------------------

def _spheres(size, centers, radii, wrap_x):
    """Normalised distance map of a union of spheres on the ghosted block, clipped to [-1, 1] at 1.8 cells from the surface."""
    g = [n + 2 for n in size]
    d = np.full(g, 1.8, dtype=np.float32)
    for c, r in zip(centers, radii):
        lo = [int(math.floor(c[a] - r - 2)) for a in range(3)]
        hi = [int(math.ceil(c[a] + r + 2)) for a in range(3)]
        ix, iy, iz = (np.arange(lo[a], hi[a] + 1) for a in range(3))
        iy, iz = iy[(iy >= -1) & (iy <= size[1])], iz[(iz >= -1) & (iz <= size[2])]
        keep = slice(None) if wrap_x else (ix >= -1) & (ix <= size[0])
        ix = ix[keep]
        if not (len(ix) and len(iy) and len(iz)):
            continue
        dist = np.sqrt((ix[:, None, None] - c[0]) ** 2 + (iy[None, :, None] - c[1]) ** 2
                       + (iz[None, None, :] - c[2]) ** 2).astype(np.float32) - np.float32(r)
        jx = (ix % size[0] if wrap_x else ix) + 1
        for x, layer in zip(jx, dist):
            part = d[x, iy[0] + 1:iy[-1] + 2, iz[0] + 1:iz[-1] + 2]
            np.minimum(part, layer, out=part)
    if wrap_x:
        d[0], d[-1] = d[-2], d[1]
    return np.clip(d / np.float32(1.8), -1.0, 1.0)


def _waves(size, seed, amplitude):
    """A smooth solenoidal velocity on the ghosted block, periodic in the interior: (3, gx, gy, gz) float64 on the device."""
    rng = np.random.default_rng(seed)
    u = torch.zeros((3, *[n + 2 for n in size]), dtype=torch.float64, device=DEV)
    x = [(torch.arange(n + 2, dtype=torch.float64, device=DEV) - 1) * (2 * math.pi / n) for n in size]
    for _ in range(6):
        m = rng.integers(-3, 4, 3)
        m[rng.integers(0, 3)] = 2
        k = np.array([m[a] / size[a] for a in range(3)])
        v = rng.normal(size=3)
        v -= k * (v @ k) / (k @ k)
        v *= amplitude / np.linalg.norm(v) / math.sqrt(3)
        phase = m[0] * x[0][:, None, None] + m[1] * x[1][None, :, None] + m[2] * x[2][None, None, :]
        wave = torch.cos(phase + rng.uniform(0, 2 * math.pi))
        for a in range(3):
            u[a] += v[a] * wave
    return u


def _scene(case, seed):
    """What a flow case is made of: nu, initial velocity, conditions in order, map, periodic axes, body force."""
    rng = np.random.default_rng(seed)
    size = (case["nx"], case["ny"], case["nz"])
    nx, ny, nz = size
    s = dict(size=size, nu=(rng.uniform(0.55, 0.7) - 0.5) / 3, u0=(0.0, 0.0, 0.0), periodic=(False,) * 3, g=None, map=None,
             walls=[], waves=None)
    u = float(rng.uniform(0.03, 0.06))
    if case["scene"] == "channel":
        s["walls"] = [("velocity", ("X0",), (u, 0.0, 0.0)), ("pressure", ("XE",), 1.0), ("noslip", ("Y0", "YE", "Z0", "ZE"), None)]
        s["u0"] = (u, 0.0, 0.0)
        c = [[rng.uniform(0.25, 0.45) * nx, rng.uniform(0.35, 0.65) * ny, rng.uniform(0.35, 0.65) * nz]]
        s["map"] = _spheres(size, c, [rng.uniform(0.12, 0.22) * min(ny, nz)], False)
    elif case["scene"] == "porous":
        s.update(periodic=(True, False, False), g=(1e-5, 0.0, 0.0), u0=(u, 0.0, 0.0))
        s["walls"] = [("noslip", ("Y0", "YE", "Z0", "ZE"), None)]
        n = max(1, int(0.51 * nx * ny * nz / (4.19 * 8.0 * 8.0 * 9.0)))
        c = rng.uniform(0, 1, (n, 3)) * np.array(size)
        s["map"] = _spheres(size, c, rng.uniform(4.0, 12.0, n), True)
    elif case["scene"] == "pressure":
        dp = float(rng.uniform(0.002, 0.01))
        s["walls"] = [("pressure", ("X0",), 1.0 + dp), ("pressure", ("XE",), 1.0), ("noslip", ("Y0", "YE", "Z0", "ZE"), None)]
        s["u0"] = (u, 0.0, 0.0)
    elif case["scene"] == "tunnel":
        s["walls"] = [("velocity", ("X0", "Y0", "YE", "ZE", "Z0"), (u, 0.0, 0.0)), ("pressure", ("XE",), 1.0)]
        s["u0"] = (u, 0.0, 0.0)
        c = [[rng.uniform(0.15, 0.55) * nx, rng.uniform(0.2, 0.8) * ny, rng.uniform(0.1, 0.5) * nz] for _ in range(12)]
        s["map"] = _spheres(size, c, [rng.uniform(0.05, 0.1) * min(ny, nz) for _ in c], False)
    else:
        s.update(periodic=(True,) * 3, waves=_waves(size, seed + 1, 0.05))
    return s


NET_NORM = np.array([0, 2e-3, 2e-3, 0, 0, -7, 1.5e-3, 1e-3, 0.05] + [2e3, 500, 500, 500, 500, 1, 500, 500, 20], dtype=np.float32)


def _net(seed):
    rng = np.random.default_rng(seed)
    w1, w2 = rng.normal(0, math.sqrt(2 / 9), (64, 9)), rng.normal(0, math.sqrt(2 / 64), (64, 64))
    w3 = rng.normal(0, math.sqrt(1 / 64), 64)
    b = rng.normal(0, 0.05, 129)
    return np.concatenate([w1.ravel(), b[:64], w2.ravel(), b[64:128], w3, b[128:]]).astype(np.float32)


def _batch_cases(case):
    rng = np.random.default_rng(case["sizes"])
    return [_flow(int(rng.integers(32, 129)), int(rng.integers(32, 65)), int(rng.integers(32, 65)), "channel", case["steps"],
                  storage=case["storage"], fuse=True) for _ in range(case["n"])]


# ---- what a program holds before the calls ----------------------------------------------------------------------------------

class _DeviceArray:
    """Device memory of the framework as an array that torch reads in place; keeps its owner alive."""

    def __init__(self, pointer, shape, double, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f8" if double else "<f4", data=(pointer, False),
                                             version=2)


def _fields(lb, double):
    g = lb.block.ghosted
    at = [lb.lib.aslb_lbgk_device_field(lb.h, f) for f in (L.FIELD_RHO, L.FIELD_VELOCITY)]
    return {"rho": torch.as_tensor(_DeviceArray(at[0], g, double, lb), device=DEV),
            "u": torch.as_tensor(_DeviceArray(at[1], (3, *g), double, lb), device=DEV)}


def _domain(case, s, macro, seed=0, packed=False):
    vt = {15: A.d3q15, 19: A.d3q19, 27: A.d3q27}[case["q"]]()
    lb = A.LBGK(A.Block(s["size"]), s["nu"], vt, compVel=macro, compRho=macro, storage=case["storage"], periodic=s["periodic"],
                body_force=s["g"], packed_rows=packed)
    if case["closure"] == "smagorinsky":
        lb.setClosure(L.CLOSURE_SMAGORINSKY, 0.17)
    elif case["closure"] == "mlp":
        lb.setMLP(CL.pack(_net(seed + 2), NET_NORM))
        lb.setMLPPeriod(case["period"])
        lb.setClosure(L.CLOSURE_MLP)
    lb.init()
    A.LBGKUtilities(lb).initF(s["u0"] if s["waves"] is None else s["waves"].cpu().numpy())
    bcs = []
    for kind, walls, v in s["walls"]:
        walls = [getattr(A, w) for w in walls]
        if kind == "velocity":
            bcs.append(A.generateBCConstantVelocity(lb, v, walls))
        elif kind == "pressure":
            bcs.append(A.generateBCConstantPressure(lb, v, walls))
        else:
            bcs.append(A.generateBCNoSlip(lb, walls))
    if s["map"] is not None:
        bcs.append(A.generateBCNoSlip(lb, s["map"]))
    if case["fuse"]:
        for bc, kind in zip(bcs, [w[0] for w in s["walls"]] + ["noslip"]):
            if kind == "noslip":
                bc.fuse()
    A.initAll(bcs)
    return lb, bcs


def prepare(case, seed):
    if case["kind"] == "flow":
        s = _scene(case, seed)
        lb, bcs = _domain(case, s, case["macro"] == "every", seed)
        st = {"case": case, "lb": lb, "bcs": bcs, "out": _fields(lb, case["storage"] == "f64")}
        if case["force"]:
            st["force"] = A.generateComputeSurfaceForce(lb, s["map"])
        return st
    if case["kind"] == "batch":
        lbs, bcs = [], []
        parts = _batch_cases(case)
        for i, c in enumerate(parts):
            lb, b = _domain(c, _scene(c, seed + i), False, packed=True)
            lbs.append(lb)
            bcs.append(b)
        # one array holds every domain's velocity
        cells = [3 * (c["nx"] + 2) * (c["ny"] + 2) * (c["nz"] + 2) for c in parts]
        u = torch.zeros(sum((n + 63) // 64 * 64 for n in cells), dtype=torch.float32, device=DEV)
        torch.cuda.synchronize()
        at = 0
        for i, (lb, n) in enumerate(zip(lbs, cells)):
            L.check(lb.lib.aslb_lbgk_bind_velocity(lb.h, u.data_ptr() + 4 * at))
            A.LBGKUtilities(lb).initF(_scene(parts[i], seed + i)["u0"])
            at += (n + 63) // 64 * 64
        return {"case": case, "batch": A.Batch(lbs), "lbs": lbs, "bcs": bcs,
                "out": {"u": u, "rho": [_fields(lb, False)["rho"] for lb in lbs]}}
    if case["kind"] == "fd":
        s, flow = _fd_scene(case, seed)
        lb, bcs = _domain(flow, s, True)
        fd = FD.generateFDAdvectionDiffusion(_blob(s["size"], seed).cpu().numpy().astype(
            np.float64 if case["storage"] == "f64" else np.float32), 0.05, lb, case["q"], case["cc"])
        FD.generateBCConstantValue(fd, 1.0, [A.X0])
        return {"case": case, "lb": lb, "bcs": bcs, "fd": fd, "c": {}, "out": _fields(lb, case["storage"] == "f64")}
    g = torch.Generator(device=DEV).manual_seed(seed)
    lib, n, p = L.load(), case["batch"], torch.from_numpy(_net(seed)).to(DEV)
    x, t = _samples(case, g)
    zero = [torch.zeros(len(p) + k, device=DEV) for k in (0, 0, 1)]
    return {"case": case, "lib": lib, "x": x, "t": t, "p": p, "m": zero[0], "v": zero[1], "grad": zero[2], "step": 0,
            "norm": torch.from_numpy(NET_NORM).to(DEV), "scratch": torch.zeros(lib.aslb_mlp_grad_scratch_floats(), device=DEV)}


def _samples(case, g):
    """Batches of features around the normalisation's values, and Cs^2 targets."""
    n, k = case["batch"], case["steps"]
    norm = torch.from_numpy(NET_NORM).to(DEV)
    x = torch.randn((k, 9, n), generator=g, device=DEV) / norm[9:].view(1, 9, 1) + norm[:9].view(1, 9, 1)
    return x.contiguous(), torch.rand((k, n), generator=g, device=DEV) * 0.05


def _fd_scene(case, seed):
    flow = _flow(case["nx"], case["ny"], case["nz"], "channel" if case["coupled"] else "turbulence", case["steps"],
                 storage=case["storage"], macro="every")
    return _scene(flow, seed), flow


def _blob(size, seed):
    rng = np.random.default_rng(seed + 5)
    c = torch.full([n + 2 for n in size], 0.2, dtype=torch.float64, device=DEV)
    for _ in range(4):
        at = [torch.exp(-((torch.arange(n + 2, dtype=torch.float64, device=DEV) - rng.uniform(0.2, 0.8) * n)
                          / (rng.uniform(0.05, 0.2) * n)) ** 2) for n in size]
        c += at[0][:, None, None] * at[1][None, :, None] * at[2][None, None, :]
    return c


# ---- the calls --------------------------------------------------------------------------------------------------------------

def run(st):
    case = st["case"]
    if case["kind"] == "flow":
        lb, bcs = st["lb"], st["bcs"]
        if case["drive"] == "run":
            lb.run(case["steps"], bcs)
        else:
            for _ in range(case["steps"]):
                lb.execute()
                A.executeAll(bcs)
        if case["macro"] == "end":
            A.LBGKUtilities(lb).computeRhoVelocity()
        return dict(st["out"], force=st["force"].execute()) if case["force"] else st["out"]
    if case["kind"] == "batch":
        st["batch"].run(case["steps"], st["bcs"])
        for lb in st["lbs"]:
            A.LBGKUtilities(lb).computeRhoVelocity()
        return st["out"]
    if case["kind"] == "fd":
        lb, bcs, fd = st["lb"], st["bcs"], st["fd"]
        if case["coupled"]:
            for _ in range(case["steps"]):
                lb.execute()
                A.executeAll(bcs)
                fd.execute()
        else:
            fd.execute(case["steps"])
        at = fd.lib.aslb_fd_device_field(fd.h)
        if at not in st["c"]:
            st["c"][at] = torch.as_tensor(_DeviceArray(at, fd.shape, case["storage"] == "f64", fd), device=DEV)
        return dict(st["out"], c=st["c"][at])
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    lib, n = st["lib"], case["batch"]
    for k in range(case["steps"]):
        st["step"] += 1
        L.check(lib.aslb_mlp_grad(st["p"].data_ptr(), st["x"][k].data_ptr(), st["t"][k].data_ptr(), n, st["norm"].data_ptr(),
                                  CL.OUT_SCALE, st["scratch"].data_ptr(), st["grad"].data_ptr(), stream))
        L.check(lib.aslb_mlp_adam(st["p"].data_ptr(), st["grad"].data_ptr(), st["m"].data_ptr(), st["v"].data_ptr(),
                                  st["step"], 1e-3, 0.9, 0.999, 1e-8, stream))
    return {k: st[k] for k in ("p", "m", "v", "grad")}


def work(case):
    """One step reads and writes each population once, and the fields that it is asked for; a closure reads its field."""
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if case["kind"] == "train":
        return {"bytes": case["steps"] * 4.0 * (10 * case["batch"] + 6 * 4865),
                "flops": case["steps"] * case["batch"] * 6.0 * 4800}
    cells, steps, b = case["nx"] * case["ny"] * case["nz"], case["steps"], BYTES[case["storage"]]
    mb = 8 if case["storage"] == "f64" else 4
    if case["kind"] == "fd":
        flow = (2 * 19 * b + 4 * mb, 200) if case["coupled"] else (0, 0)
        return {"bytes": cells * steps * (5.0 * b + flow[0]), "flops": cells * steps * (8.0 * case["q"] + flow[1])}
    q = case["q"]
    macro = 4 * mb * steps if case["macro"] == "every" else 4 * mb + q * b
    field = 4 * (steps + steps / case["period"]) + q * b * steps / case["period"] if case["closure"] == "mlp" else 0
    flops = steps * q * (10.0 if case["closure"] == "none" else 20.0)
    if case["closure"] == "mlp":
        flops += 2 * 4800 * steps / case["period"]
    return {"bytes": cells * (2.0 * q * b * steps + macro + field), "flops": cells * flops}


def tolerance(case):
    """About four times the distance between these outputs and the same sums in 64 bits, each storage at its own."""
    if case["kind"] == "train":
        return {"rel": 5e-5, "max": 2e-2}
    if case["storage"] == "f64":
        return {"rel": 2e-13 if case.get("force") else 3e-14, "max": 1e-11}
    if case["storage"] == "f16":
        return {"rel": 4e-3, "max": 5e-2}
    if case["kind"] == "fd":
        return {"rel": 8e-6, "max": 4e-4}
    return {"rel": 1e-4 if case.get("force") else 2e-5, "max": 4e-3 if case.get("force") else 1e-3}


# ---- the same models in 64 bits ---------------------------------------------------------------------------------------------

_V27 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (1, 1, 0), (1, -1, 0), (-1, -1, 0),
        (-1, 1, 0), (0, 1, 1), (0, 1, -1), (0, -1, -1), (0, -1, 1), (1, 0, 1), (1, 0, -1), (-1, 0, -1), (-1, 0, 1), (1, 1, 1),
        (1, 1, -1), (1, -1, 1), (1, -1, -1), (-1, 1, 1), (-1, 1, -1), (-1, -1, 1), (-1, -1, -1)]


def _lattice(q):
    c = _V27[:7] + _V27[19:] if q == 15 else _V27[:q]
    table = {15: (2 / 9, 1 / 9, 0, 1 / 72), 19: (1 / 3, 1 / 18, 1 / 36, 0), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}[q]
    return c, [table[sum(a * a for a in v)] for v in c], [c.index(tuple(-a for a in v)) for v in c]


class _Flow:
    """ASL's LBGK in float64: post-collision populations of the ghosted block, stepped as `execute(); executeAll(bcs)`."""

    def __init__(self, case, s, seed=0):
        self.case, self.s, self.size = case, s, s["size"]
        self.c, self.w, self.inv = _lattice(case["q"])
        self.g = s["g"] or (0.0, 0.0, 0.0)
        self.om = 1 / (3 * s["nu"] + 0.5)
        gsize = [n + 2 for n in self.size]
        if s["waves"] is None:
            self.u = torch.tensor(s["u0"], dtype=torch.float64, device=DEV).view(3, 1, 1, 1).expand(3, *gsize).clone()
        else:
            self.u = s["waves"].clone()
        self.rho = torch.ones(gsize, dtype=torch.float64, device=DEV)
        uu = (self.u ** 2).sum(0)
        self.f = torch.stack([1 + 3 * cu + 4.5 * cu * cu - 1.5 * uu for cu in (self.dot(i, self.u) for i in range(case["q"]))])
        self.steps, self.last, self.net = 0, -1, _net(seed + 2) if case["closure"] == "mlp" else None
        self.cs2 = None
        self.bcs = []
        for kind, walls, v in s["walls"]:
            links = [self.wall_links(w) for w in walls]
            self.bcs.append((kind, v, {k: [torch.cat([p[k][a] for p in links if k in p]) for a in range(3)]
                                       for k in range(1, case["q"]) if any(k in p for p in links)}))
        if s["map"] is not None:
            self.m = torch.from_numpy(s["map"]).to(DEV)
            self.bcs.append(("noslip", None, self.map_links()))

    def dot(self, i, v):
        return sum(self.c[i][a] * v[a] for a in range(3) if self.c[i][a]) if i else torch.zeros_like(v[0])

    def wrap(self, at):
        return [torch.where(v < 1, v + n, torch.where(v > n, v - n, v)) if p else v
                for v, n, p in zip(at, self.size, self.s["periodic"])]

    def wall_links(self, wall):
        a, hi = "XYZ".index(wall[0]), wall[1] == "E"
        axes = [torch.arange(1, n + 1, device=DEV) for n in self.size]
        axes[a] = axes[a][-1:] if hi else axes[a][:1]
        fluid = [v.reshape(-1) for v in torch.meshgrid(*axes, indexing="ij")]
        n = -1 if hi else 1
        return {k: self.wrap([fluid[d] - self.c[k][d] for d in range(3)])
                for k in range(1, len(self.c)) if self.c[k][a] * n > 0}

    def owned(self):
        own = torch.ones_like(self.m, dtype=torch.bool)
        for a, p in enumerate(self.s["periodic"]):
            if p:
                own.select(a, 0)[:] = False
                own.select(a, self.size[a] + 1)[:] = False
        return own

    def neighbours(self, at, k):
        """Coordinates of the neighbours along c_k (wrapped), whether they are interior, and the map there (-0.9 off the block)."""
        q = self.wrap([v + d for v, d in zip(at, self.c[k])])
        on = torch.ones_like(q[0], dtype=torch.bool)
        inside = on.clone()
        for v, n in zip(q, self.size):
            on &= (v >= 0) & (v <= n + 1)
            inside &= (v >= 1) & (v <= n)
        clip = [v.clamp(0, n + 1) for v, n in zip(q, self.size)]
        return clip, inside, torch.where(on, self.m[tuple(clip)], torch.full_like(q[0], -0.9, dtype=self.m.dtype))

    def map_links(self):
        at = torch.nonzero((self.m <= 0) & (self.m > -0.9999) & self.owned(), as_tuple=True)
        links = {}
        for k in range(1, len(self.c)):
            _, inside, mk = self.neighbours(at, k)
            keep = inside & (mk > 0)
            links[k] = [v[keep] for v in at]
        return links

    def conditions(self):
        for kind, v, links in self.bcs:
            for k, a in links.items():
                q = self.wrap([x + d for x, d in zip(a, self.c[k])])
                if kind == "pressure":
                    self.f[(k, *a)] = v
                    continue
                back = self.f[(self.inv[k], *q)]
                self.f[(k, *a)] = back + 6 * sum(p * d for p, d in zip(v, self.c[k])) if kind == "velocity" else back

    def stress(self, f, feq):
        return {(a, b): sum(self.w[i] * self.c[i][a] * self.c[i][b] * (f[i] - feq[i]) for i in range(len(f))
                            if self.c[i][a] * self.c[i][b]) for a in range(3) for b in range(a, 3)}

    def network(self, rho, u, P):
        a, b, c, d, e, g = (P[k] / rho for k in ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2)))
        tr, off = a + b + c, d * d + e * e + g * g
        da, db, dc = a - tr / 3, b - tr / 3, c - tr / 3
        cbrt = lambda v: v.sign() * v.abs() ** (1 / 3)  # noqa: E731
        det = lambda a, b, c: a * (b * c - e * e) - d * (d * c - e * g) + g * (d * e - b * g)  # noqa: E731
        dn = torch.sqrt(da * da + db * db + dc * dc + 2 * off)
        diag = a * a + b * b + c * c
        x = torch.stack([tr, torch.sqrt(diag + 2 * off), dn, cbrt(3 * det(da, db, dc)), cbrt(det(a, b, c)),
                         torch.log(dn + 1e-12), torch.sqrt(diag), torch.sqrt(2 * off), torch.sqrt((u * u).sum(0))])
        y, _ = _forward(torch.from_numpy(self.net).to(DEV).double(), x.reshape(9, -1))
        return (CL_SCALE * torch.nn.functional.softplus(y)).reshape(rho.shape)

    def step(self):
        f, n = self.f, self.size
        for a, p in enumerate(self.s["periodic"]):
            if p:
                f.select(a + 1, 0)[:] = f.select(a + 1, n[a])
                f.select(a + 1, n[a] + 1)[:] = f.select(a + 1, 1)
        x = torch.stack([f[i, 1 - c[0]:1 - c[0] + n[0], 1 - c[1]:1 - c[1] + n[1], 1 - c[2]:1 - c[2] + n[2]]
                         for i, c in enumerate(self.c)])
        rho = sum(w * v for w, v in zip(self.w, x))
        m = [sum(self.w[i] * self.c[i][a] * x[i] for i in range(len(x)) if self.c[i][a]) + 0.5 * rho * self.g[a] for a in range(3)]
        u = torch.stack([v / rho for v in m])
        a0 = rho - 1.5 * rho * (u * u).sum(0)
        cu = [self.dot(i, u) for i in range(len(x))]
        feq = [a0 + rho * (3 * v + 4.5 * v * v) for v in cu]
        om = self.om
        if self.case["closure"] != "none":
            P = self.stress(x, feq)
            cs2 = 0.17 ** 2
            if self.case["closure"] == "mlp":
                if self.last < 0 or self.steps - self.last >= self.case["period"]:
                    self.cs2, self.last = self.network(rho, u, P), self.steps
                cs2 = self.cs2
            mag = torch.sqrt(sum((1 if a == b else 2) * v * v for (a, b), v in P.items()))
            om = 2 / (1 / self.om + torch.sqrt(1 / self.om ** 2 + 18 * math.sqrt(2) * cs2 * mag / rho))
        ug = sum(u[a] * self.g[a] for a in range(3))
        for i, c in enumerate(self.c):
            cg = sum(c[a] * self.g[a] for a in range(3))
            force = (1 - om / 2) * rho * (3 * (cg - ug) + 9 * cu[i] * cg) if self.s["g"] else 0
            f[i, 1:-1, 1:-1, 1:-1] = (1 - om) * x[i] + om * feq[i] + force
        if self.case["macro"] == "every":
            self.rho[1:-1, 1:-1, 1:-1], self.u[:, 1:-1, 1:-1, 1:-1] = rho, u
        self.steps += 1
        self.conditions()

    def compute(self):
        f = self.f[:, 1:-1, 1:-1, 1:-1]
        rho = sum(w * v for w, v in zip(self.w, f))
        self.rho[1:-1, 1:-1, 1:-1] = rho
        for a in range(3):
            self.u[a, 1:-1, 1:-1, 1:-1] = sum(self.w[i] * c[a] * f[i] for i, c in enumerate(self.c) if c[a]) / rho

    def force(self):
        at = torch.nonzero((self.m.abs() < 0.9999) & self.owned(), as_tuple=True)
        m0, total = self.m[at], torch.zeros((3, len(at[0])), dtype=torch.float64, device=DEV)
        in0 = torch.ones_like(at[0], dtype=torch.bool)
        for v, n in zip(at, self.size):
            in0 &= (v >= 1) & (v <= n)
        for k in range(1, len(self.c)):
            q, inside, mk = self.neighbours(at, k)
            out, into = (m0 <= 0) & (mk > 0) & inside, (mk <= 0) & (m0 > 0) & in0
            v = (self.f[(k, *at)] + self.f[(self.inv[k], *q)] - 2) * self.w[k] * (out.double() - into.double())
            for a in range(3):
                total[a] += self.c[k][a] * v
        r = torch.stack([v.double() - 1 for v in at])
        return torch.cat([total.sum(1), torch.linalg.cross(r, total, dim=0).sum(1)]).cpu().numpy()

    def out(self):
        if self.case["macro"] == "end":
            self.compute()
        return {"rho": self.rho, "u": self.u}


CL_SCALE = 0.05


def _forward(p, x):
    """The network's output before the softplus, parameters W1 b1 W2 b2 w3 b3, x (9, n) before normalisation."""
    norm = torch.from_numpy(NET_NORM).to(x.device).double()
    w1, b1, w2, b2, w3, b3 = torch.split(p, [576, 64, 4096, 64, 64, 1])
    h = torch.relu(w1.view(64, 9) @ ((x - norm[:9, None]) * norm[9:, None]) + b1[:, None])
    h = torch.relu(w2.view(64, 64) @ h + b2[:, None])
    return w3 @ h + b3, h


def _fd_exact(case, seed):
    s, flow = _fd_scene(case, seed)
    e = _V27[:7] + _V27[19:] if case["q"] == 15 else _V27[:case["q"]]
    lc = {7: (-6, 1, 0), 15: (-14 / 3, 2 / 3, 1 / 12), 19: (-4, 1 / 3, 1 / 6)}[case["q"]]
    gc = {7: (0, 1 / 2, 0), 15: (0, 1 / 3, 1 / 24), 19: (0, 1 / 6, 1 / 12)}[case["q"]]
    cls = [0 if i == 0 else 1 if i <= 6 else 2 for i in range(case["q"])]
    lb, c, n = _Flow(flow, s), _blob(s["size"], seed), s["size"]
    if case["storage"] == "f32":
        c = c.float().double()
    c[0, 1:-1, 1:-1] = 1.0

    def at(v, i):
        return v[..., 1 + e[i][0]:1 + e[i][0] + n[0], 1 + e[i][1]:1 + e[i][1] + n[1], 1 + e[i][2]:1 + e[i][2] + n[2]]

    for _ in range(case["steps"]):
        if case["coupled"]:
            lb.step()
        c0, u0 = at(c, 0), at(lb.u, 0)
        lap = sum(lc[cls[i]] * at(c, i) for i in range(len(e)))
        flux, div = torch.zeros_like(c0), torch.zeros_like(c0)
        for i in range(1, len(e)):
            ui = at(lb.u, i)
            for a in range(3):
                if e[i][a]:
                    flux += gc[cls[i]] * e[i][a] * 0.5 * (ui[a] + u0[a]) * (at(c, i) + c0)
                    div += gc[cls[i]] * e[i][a] * ui[a]
        new = 0.05 * lap + c0 - flux
        if case["cc"]:
            new = new / (1 - div) + lap * (u0 * u0).sum(0) * 0.5
        c = c.clone()
        c[1:-1, 1:-1, 1:-1] = new
    return {"rho": lb.rho, "u": lb.u, "c": c}


def _train_exact(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x, t = _samples(case, g)
    p = torch.from_numpy(_net(seed)).to(DEV).double().requires_grad_()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for k in range(case["steps"]):
        y, _ = _forward(p, x[k].double())
        err = ((CL_SCALE * torch.nn.functional.softplus(y) - t[k].double()) ** 2).sum()
        grad, = torch.autograd.grad(err / case["batch"], p)
        with torch.no_grad():
            m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
            step = (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
            p = (p - 1e-3 * step).detach().requires_grad_()
    return {"p": p.detach(), "m": m, "v": v, "grad": torch.cat([grad, err.detach().view(1)])}


def exact(case, seed):
    if case["kind"] == "train":
        return _train_exact(case, seed)
    if case["kind"] == "fd":
        return _fd_exact(case, seed)
    if case["kind"] == "batch":
        u, rho = [], []
        for i, c in enumerate(_batch_cases(case)):
            out = _march(c, _scene(c, seed + i)).out()
            flat = out["u"].reshape(-1)
            u.append(torch.nn.functional.pad(flat, (0, -len(flat) % 64)))
            rho.append(out["rho"])
        return {"u": torch.cat(u), "rho": rho}
    flow = _march(case, _scene(case, seed), seed)
    return dict(flow.out(), force=flow.force()) if case["force"] else flow.out()


def _march(case, s, seed=0):
    flow = _Flow(case, s, seed)
    for _ in range(case["steps"]):
        flow.step()
    return flow
