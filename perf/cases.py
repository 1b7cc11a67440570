"""The workloads this framework is timed on: what a program that uses it has it do, through the public entry points.

Six kinds of work, over the range of sizes, lattices and storage formats of the tests and the benchmark:

* ``flow``     one lattice stepped and its field read back: the solver's main use;
* ``monitor``  a few steps, then the forces, the statistics, the health probe and one z layer for a slice view, as an
               interactive program does every frame;
* ``sweep``    the lattices of an angle-of-attack sweep stepped as one batch, then their forces and fields;
* ``voxelize`` a triangle mesh to the solver's grid, on the device;
* ``smoke``    a lattice and its smoke particles advanced frame by frame, then the trails;
* ``train``    mini-batches of the learned closure's training.

``exact`` is a plain 64-bit torch restatement of each, independent of the library.
"""
import math

import numpy as np
import torch

from flowcraft_b200 import geometry, meshes, voxelizer
from flowcraft_b200.batch import LbmBatch
from flowcraft_b200.closure import ClosureWeights
from flowcraft_b200.closure_train import MlpTrainer, he_init
from flowcraft_b200.lbm import LatticeModel, LbmSolver, Params, Storage, Streaming, VoxelGrid
from flowcraft_b200.smoke import SmokeTrailSystem

DEV = 0
CUDA = "cuda:0"
WEIGHTS = "flowcraft_b200/data/closure_c4.json"


def _flow(name, nx, ny, nz, q, storage, steps, **more):
    c = dict(kind="flow", nx=nx, ny=ny, nz=nz, q=q, storage=storage, steps=steps, streaming="PINGPONG",
             closure=False, slip=True, reverse=False, read="async", body="sphere")
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference test's own sphere grid: an interactive first look, where launches and waits count
        _flow("first_look_fp32", 48, 24, 24, 19, "FP32", 20, read="blocking"),
        # a mesh's own ragged grid on the smaller lattice, no-slip walls, flow from the far end
        _flow("ragged_d3q15_fp32", 191, 97, 83, 15, "FP32", 50, slip=False, reverse=True, read="blocking"),
        # a production wind tunnel on a grid that a mesh gave: odd in every direction
        _flow("ragged_fp16", 641, 203, 151, 19, "FP16_OFFSET", 50),
        # the precision study's wing in the format that reproduces the CPU solver
        _flow("wing_fp32", 384, 192, 192, 19, "FP32", 50, body="wing"),
        # the same lattice in the benchmark's pairing: 16-bit storage and the learned closure
        _flow("wing_learned_fp16", 384, 192, 192, 19, "FP16_OFFSET", 50, body="wing", closure=True),
        # a lattice kept once in memory instead of twice
        _flow("inplace_fp32", 512, 256, 256, 19, "FP32", 50, streaming="AA"),
        # the large configuration: the aircraft, 268 million cells
        _flow("aircraft_fp16", 1024, 512, 512, 19, "FP16_OFFSET", 50, body="aircraft"),
        # an interactive session on a half-size lattice: forces, statistics, health and a slice every few steps
        dict(name="monitor_fp16", kind="monitor", nx=512, ny=256, nz=256, q=19, storage="FP16_OFFSET", steps=10,
             streaming="PINGPONG", slip=True, reverse=False, body="wing"),
        # sixteen wings of 64x32x32 to 256x128x128 as one batch
        dict(name="sweep_fp16", kind="sweep", members=16, nx_lo=64, nx_hi=256, storage="FP16_OFFSET", steps=50),
        # the aircraft mesh (57,516 triangles) on the grid of the application's default resolution, its attitude changed
        dict(name="voxelize_aircraft", kind="voxelize", mesh="aircraft", resolution=640),
        # smoke trails of an interactive view
        dict(name="smoke_fp32", kind="smoke", nx=256, ny=128, nz=128, q=19, storage="FP32", particles=20000, trail=48,
             frames=20, steps=2),
        # mini-batches of the closure's training, at its default batch, and a look at the held-out rows
        dict(name="train_closure", kind="train", samples=1 << 20, batch=4096, batches=3, held_out=1 << 15),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def lattice(lo, hi, even):
        nx = log_int(lo, hi)
        if even:
            nx += nx & 1
        return nx, max(12, int(nx * rng.uniform(0.35, 0.55))), max(12, int(nx * rng.uniform(0.35, 0.55)))

    kind = rng.choice(["flow", "flow", "flow", "flow", "monitor", "sweep", "voxelize", "smoke", "train"])
    if kind == "sweep":
        lo = 2 * rng.randint(32, 64)
        return dict(kind="sweep", members=rng.randint(4, 16), nx_lo=lo, nx_hi=2 * rng.randint(lo // 2, 128),
                    storage=rng.choice(["FP16_OFFSET", "FP16_OFFSET", "FP32"]), steps=2 * rng.randint(5, 25))
    if kind == "voxelize":
        return dict(kind="voxelize", mesh=rng.choice(["aircraft", "wing", "sphere"]), resolution=log_int(96, 640))
    if kind == "train":
        return dict(kind="train", samples=log_int(1 << 16, 1 << 21), batch=log_int(256, 16384),
                    batches=rng.randint(1, 4), held_out=log_int(1 << 10, 1 << 16))
    if kind == "smoke":
        nx, ny, nz = lattice(48, 288, rng.random() < 0.5)
        return dict(kind="smoke", nx=nx, ny=ny, nz=nz, q=rng.choice([19, 19, 15]),
                    storage=rng.choice(["FP32", "FP16_OFFSET"]), particles=log_int(500, 50000),
                    trail=rng.randint(16, 64), frames=rng.randint(5, 25), steps=rng.randint(1, 4))
    storage = rng.choice(["FP32", "FP16_OFFSET", "FP16_OFFSET", "BF16_OFFSET"])
    streaming = rng.choice(["PINGPONG", "PINGPONG", "AA"])
    closure = kind == "flow" and storage == "FP16_OFFSET" and rng.random() < 0.5
    q = 19 if closure else rng.choice([19, 19, 15])
    even = closure or streaming == "AA" or rng.random() < 0.5
    nx, ny, nz = lattice(40, 512, even)
    same = dict(nx=nx, ny=ny, nz=nz, q=q, storage=storage, streaming=streaming, slip=rng.random() < 0.7,
                reverse=rng.random() < 0.3, body=rng.choice(["sphere", "wing"]))
    if kind == "monitor":
        return dict(same, kind="monitor", steps=rng.randint(4, 20))
    return dict(same, kind="flow", steps=rng.randint(10, 60), closure=closure,
                read="blocking" if nx * ny * nz < 2_000_000 and rng.random() < 0.5 else "async")


# ---- inputs ----

def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, case["nx"], case["ny"], case["nz"]])


def _geometry(case, rng):
    """(solid, signed distance) of the case's body, (nz, ny, nx) tensors on the GPU; its place and pitch from the seed."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    jit = rng.uniform(-0.02, 0.02, 3)
    angle = math.radians(rng.uniform(2.0, 10.0))
    if case["body"] == "aircraft":
        return geometry.aircraft_grid_torch(nx, ny, nz, device=CUDA)
    x = (torch.arange(nx, device=CUDA, dtype=torch.float32) + 0.5)[None, None, :] - nx * (0.32 + jit[0])
    y = (torch.arange(ny, device=CUDA, dtype=torch.float32) + 0.5)[None, :, None] - ny * (0.5 + jit[1])
    z = (torch.arange(nz, device=CUDA, dtype=torch.float32) + 0.5)[:, None, None] - nz * (0.5 + jit[2])
    if case["body"] == "sphere":
        d = torch.sqrt(x * x + y * y + z * z) - 0.13 * min(ny, nz)
    else:  # the pitched ellipsoid wing of the tests, scaled with the lattice
        ca, sa = math.cos(angle), math.sin(angle)
        a, b, c = 0.12 * nx, 0.28 * ny, 0.07 * nz
        rx, rz = x * ca - z * sa, x * sa + z * ca
        d = (torch.sqrt((rx / a) ** 2 + (y / b) ** 2 + (rz / c) ** 2) - 1.0) * c
    d = d.expand(nz, ny, nx).contiguous()
    return (d < 0).to(torch.uint8), d


def _params(case, rng):
    u = float(rng.uniform(0.04, 0.065))
    tau = float(rng.uniform(0.62, 0.7) if case["q"] == 15 else rng.uniform(0.51, 0.53))
    return Params(tau=tau, inletVelocity=u, reverseFlow=bool(case.get("reverse", False)),
                  freeSlipY=bool(case.get("slip", True)), freeSlipZ=bool(case.get("slip", True)), smagorinskyCs=0.1)


def _start_field(case, rng, p):
    """(nz, ny, nx, 4) of a moving start with eddies: the mid-speed flow and a few seeded sine modes, about a third of
    the inlet speed."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    mid = 0.5 * p.inletVelocity * (-1.0 if p.reverseFlow else 1.0)
    f = torch.empty((nz, ny, nx, 4), dtype=torch.float32, device=CUDA)
    f[..., 0] = 1.0 + 3.0 * 0.375 * p.inletVelocity ** 2
    f[..., 1:] = 0.0
    f[..., 1] = mid
    x = ((torch.arange(nx, device=CUDA, dtype=torch.float32) + 0.5) / nx)[None, None, :]
    y = ((torch.arange(ny, device=CUDA, dtype=torch.float32) + 0.5) / ny)[None, :, None]
    z = ((torch.arange(nz, device=CUDA, dtype=torch.float32) + 0.5) / nz)[:, None, None]
    for comp in (1, 2, 3):
        for _ in range(3):
            k = rng.integers(2, 7, 3) * 2.0 * math.pi
            ph = rng.uniform(0.0, 2.0 * math.pi, 3)
            f[..., comp] += (p.inletVelocity / 9.0) * (torch.sin(k[0] * x + ph[0]) * torch.sin(k[1] * y + ph[1]) *
                                                       torch.sin(k[2] * z + ph[2]))
    return f


def _problem(case, seed):
    """Geometry, parameters and start field (None: the uniform mid-speed start) of a lattice case."""
    rng = _rng(case, seed)
    solid, sdf = _geometry(case, rng)
    p = _params(case, rng)
    big = case["nx"] * case["ny"] * case["nz"] > 50_000_000
    return solid, sdf, p, None if big else _start_field(case, rng, p)


def _solver(case, solid, sdf, p, field):
    nz, ny, nx = solid.shape
    torch.cuda.current_stream().synchronize()  # the solver copies the grid on a stream of its own
    s = LbmSolver()
    ok = s.Init(DEV, VoxelGrid(nx, ny, nz, solid=solid, signedDistance=sdf),
                LatticeModel.D3Q19 if case.get("q", 19) == 19 else LatticeModel.D3Q15, Storage[case["storage"]],
                Streaming[case.get("streaming", "PINGPONG")])
    if not ok:
        raise RuntimeError(s.LastError())
    s.Reset(p, True)
    if field is not None:
        s.ResetFromField(field.cpu().numpy())
    if case.get("closure"):
        s.SetClosure(ClosureWeights.load(WEIGHTS))
    return s


def _members(case, seed):
    """The sweep's lattices (2:1:1, sizes evenly over the range, angles of the polar) as lattice cases and seeds."""
    out = []
    for k in range(case["members"]):
        t = k / max(case["members"] - 1, 1)
        nx = 2 * int(round(0.5 * (case["nx_lo"] + t * (case["nx_hi"] - case["nx_lo"]))))
        out.append((dict(nx=nx, ny=nx // 2, nz=nx // 2, q=19, storage=case["storage"], body="wing"), int(seed) + 7919 * k))
    return out


def _mesh(case, seed):
    """(positions, indices) on the GPU: the body, turned and scaled a little by the seed, and the grid of the body as
    it is: (dims, cell size, origin)."""
    rng = np.random.default_rng(int(seed) & 0x7FFFFFFF)
    if case["mesh"] == "aircraft":
        pos, idx = meshes.aircraft(**meshes.C5_TESSELLATION)
    elif case["mesh"] == "wing":
        pos, idx = meshes.naca_wing("2412", 96.0, 128.0, 4.0)
    else:
        pos, idx = meshes.icosphere(4, 20.0)
    grid = voxelizer.GridForMesh(pos, voxelizer.Params(targetResolution=case["resolution"]), DEV)
    a, b = np.radians(rng.uniform(-3.0, 3.0, 2))
    ra = np.array([[1, 0, 0], [0, math.cos(a), -math.sin(a)], [0, math.sin(a), math.cos(a)]])
    rb = np.array([[math.cos(b), -math.sin(b), 0], [math.sin(b), math.cos(b), 0], [0, 0, 1]])
    pos = (pos.astype(np.float64) @ ra.T @ rb.T * rng.uniform(0.9, 1.1)).astype(np.float32)
    return (torch.from_numpy(pos).to(CUDA), torch.from_numpy(idx.astype(np.int64).astype(np.int32)).to(CUDA)) + grid


def _particle_starts(case, seed):
    """Points upstream of the body, world units (grid x is world y)."""
    rng = np.random.default_rng(int(seed) & 0x7FFFFFFF)
    n = case["particles"]
    return np.stack([rng.uniform(0.2, 0.8, n) * case["ny"], rng.uniform(0.03, 0.1, n) * case["nx"],
                     rng.uniform(0.2, 0.8, n) * case["nz"]], axis=1).astype(np.float32)


SMOKE_DT, SMOKE_SCALE = 1.0 / 60.0, 300.0  # 5 cells per step and lattice unit


def _training(case, seed):
    """Normalized inputs and targets as the closure's samples have them (strain input, two invariants, wall distance,
    filter width; a heavy-tailed non-negative eddy viscosity), and the batches' rows."""
    g = torch.Generator(device=CUDA)
    g.manual_seed(int(seed))
    n = case["samples"]
    x = torch.randn((n, 5), generator=g, device=CUDA)
    x[:, 3] = torch.clamp(x[:, 3], max=0.3)
    x[:, 4] = 0.2
    y = torch.relu(0.7 * torch.tanh(x[:, 0]) + 0.3 * x[:, 1] * x[:, 2] + 0.2 * torch.randn(n, generator=g, device=CUDA))
    rows = torch.randint(0, n, (case["batches"], case["batch"]), generator=g, device=CUDA)
    return x.contiguous(), y.contiguous(), rows


def _pinned(count):
    """Page-locked host memory that the returned outputs keep alive."""
    return torch.empty(count, dtype=torch.float32, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("flow", "monitor", "smoke"):
        body = case if "body" in case else dict(case, body="sphere")
        st["s"] = _solver(body, *_problem(body, seed))
        cells = case["nx"] * case["ny"] * case["nz"]
        if kind == "flow" and case["read"] == "async":
            st["out"] = _pinned(4 * cells)
        if kind == "monitor":
            st["out"] = np.zeros(4 * cells, dtype=np.float32)
        if kind == "smoke":
            st["smoke"] = SmokeTrailSystem(st["s"])
            st["smoke"].Reset(False, case["particles"], case["trail"], seed=int(seed))
            st["smoke"].SetPositions(_particle_starts(case, seed))
    elif kind == "sweep":
        st["m"] = [_solver(c, *_problem(c, k)) for c, k in _members(case, seed)]
        st["out"] = [_pinned(4 * s.CellCount()) for s in st["m"]]
        st["batch"] = LbmBatch(st["m"])
        st["batch"].Config(0, 1)  # what the autotuner picks for such a set
    elif kind == "voxelize":
        st["mesh"] = _mesh(case, seed)
    else:
        st["x"], st["y"], rows = _training(case, seed)
        st["rows"] = [r.contiguous() for r in rows]
        st["t"] = MlpTrainer(he_init(int(seed)), DEV)
    return st


# ---- one pass ----

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "flow":
        s = st["s"]
        s.Step(None, case["steps"])
        if case["read"] == "blocking":
            return s.ReadbackField()
        s.ReadbackFieldAsync(st["out"].numpy())
        s.ReadbackWait()
        return st["out"]
    if kind == "monitor":
        s = st["s"]
        s.Step(None, case["steps"])
        a, t = s.AerodynamicForces(), s.ReadbackStats()
        bad = s.ProbeSliceHealth(case["nz"] // 2)
        s.ReadbackFieldRange(case["nz"] // 2, 1, st["out"])
        layer = case["nx"] * case["ny"] * 4
        return {"force": np.array([a.forceX, a.forceY, a.forceZ], np.float32),
                "centre": np.array(a.centerOfPressure, np.float32), "stress": a.maxStress, "bad": bool(bad),
                "density": [t.avgDensity, t.minDensity, t.maxDensity], "speed": [t.avgSpeed, t.maxSpeed],
                "cells": t.fluidCells, "slice": st["out"][case["nz"] // 2 * layer:][:layer]}
    if kind == "sweep":
        st["batch"].Step(case["steps"])
        force = np.zeros((case["members"], 3), np.float32)
        for k, s in enumerate(st["m"]):
            a = s.AerodynamicForces()
            force[k] = a.forceX, a.forceY, a.forceZ
        for s, o in zip(st["m"], st["out"]):
            s.ReadbackFieldAsync(o.numpy())
        for s in st["m"]:
            s.ReadbackWait()
        return {"force": force, "fields": st["out"]}
    if kind == "voxelize":
        g = voxelizer.VoxelizeOnGrid(*st["mesh"], device=DEV)
        return {"solid": g.solid, "sdf": g.signedDistance}
    if kind == "smoke":
        s, smoke = st["s"], st["smoke"]
        for _ in range(case["frames"]):
            s.Step(None, case["steps"])
            smoke.Step(False, SMOKE_SCALE, SMOKE_DT)
        points, lens = smoke.Trails()
        return {"points": points, "lens": lens}
    t = st["t"]
    for r in st["rows"]:
        loss, _ = t.grad(st["x"], st["y"], r)
        t.adam(1e-3)
    return {"loss": loss.float(), "grad": t.g, "params": t.p, "m": t.m, "v": t.v, "predicted": t.predict(st["x"][:case["held_out"]])}


def work(case):
    kind = case["kind"]
    if kind == "train":
        b, p = case["batches"] * case["batch"], 1281
        return {"bytes": case["batches"] * (case["batch"] * 32 + 6 * 4 * p) + case["held_out"] * 24,
                "flops": 6.0 * 1216 * b + 2.0 * 1216 * case["held_out"]}
    if kind == "voxelize":
        # the cells of the body's padded box, as a share of a cube of its longest side
        n = {"aircraft": 0.119, "wing": 0.0625, "sphere": 0.357}[case["mesh"]] * case["resolution"] ** 3
        return {"bytes": 5.0 * n, "flops": 20.0 * n}
    if kind == "sweep":
        cells = sum(c["nx"] * c["ny"] * c["nz"] for c, _ in _members(case, 0))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    q = case.get("q", 19)
    each = 2 * q * (4 if case["storage"] == "FP32" else 2)
    steps = case["steps"] * case.get("frames", 1)
    more = 16 * cells
    if kind == "monitor":
        more = cells * (each // 2 + 1) + 32 * case["nx"] * case["ny"]
    if kind == "smoke":
        more = case["particles"] * (case["frames"] * (8 * each // 2 + 32) + 12 * case["trail"])
    return {"bytes": float(each) * cells * steps + more,
            "flops": cells * steps * (12.0 * q + 100.0 + (2.0 * 1216 if case.get("closure") else 0.0))}


# ---- the same in 64 bits, in plain torch ----

_E19 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
        (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
        (0, -1, 1)]
_E15 = _E19[:7] + [(1, 1, 1), (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)]


class _Exact:
    """A lattice in 64 bits: regularized collision with a Smagorinsky (or learned) relaxation time, interpolated
    bounce-back at the body, velocity inlet, zero-gradient outlet, free-slip or no-slip sides."""

    def __init__(self, q, solid, sdf, p, field, closure=None):
        self.e = _E19 if q == 19 else _E15
        w1, w2 = (1 / 18, 1 / 36) if q == 19 else (1 / 9, 1 / 72)
        self.w = [(1 / 3 if q == 19 else 2 / 9)] + [w1] * 6 + [w2] * (q - 7)
        self.opp = [self.e.index((-a, -b, -c)) for a, b, c in self.e]
        self.p, self.q = p, q
        self.solid = solid.bool()
        self.shape = solid.shape
        ux = (-1 if p.reverseFlow else 1) * p.inletVelocity
        if field is None:
            rho = torch.full(self.shape, 1 + 1.5 * 0.75 * ux * ux, dtype=torch.float64, device=CUDA)
            u = [torch.full_like(rho, 0.5 * ux), torch.zeros_like(rho), torch.zeros_like(rho)]
        else:
            f = field.double()
            f[self.solid] = torch.tensor([1.0, 0, 0, 0], dtype=torch.float64, device=CUDA)
            rho, u = f[..., 0].clone(), [f[..., k].clone() for k in (1, 2, 3)]
        self.f = [self._eq(i, rho, u) for i in range(q)]
        self._links(sdf.double())
        self.closure = closure
        if closure is not None:
            self.wall = self._wall()

    def _eu(self, i, u):
        return sum((c * v for c, v in zip(self.e[i], u) if c), torch.zeros((), dtype=torch.float64, device=CUDA))

    def _eq(self, i, rho, u):
        eu = self._eu(i, u)
        return self.w[i] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2))

    def _at(self, t, e, sign):
        """t at every cell's neighbour cell + sign * e (wrapped around: the callers mask what is off the lattice)."""
        return torch.roll(t, shifts=(-sign * e[2], -sign * e[1], -sign * e[0]), dims=(0, 1, 2))

    def _inside(self, e, sign):
        m = torch.ones(self.shape, dtype=torch.bool, device=CUDA)
        for dim, c in zip((2, 1, 0), e):
            if sign * c > 0:
                m.select(dim, self.shape[dim] - 1).fill_(False)
            if sign * c < 0:
                m.select(dim, 0).fill_(False)
        return m

    def _links(self, sdf):
        """Per direction: the fluid cells whose upstream neighbour is solid, and what their population is made of."""
        nz, ny, nx = self.shape
        self.link = []
        for i in range(self.q):
            e = self.e[i]
            wall = ~self.solid & self._inside(e, -1) & self._at(self.solid, e, -1)
            idx = wall.reshape(-1).nonzero()[:, 0]
            off = (e[2] * ny + e[1]) * nx + e[0]
            flat = sdf.reshape(-1)
            a, b = flat[idx], flat[idx - off]
            den = a - b
            ok = torch.isfinite(a) & torch.isfinite(b) & (den > 1e-4)
            r = torch.where(ok, a / torch.where(ok, den, torch.ones_like(den)), torch.ones_like(a)).clamp(0, 1)
            ahead = (self._inside(e, 1) & ~self._at(self.solid, e, 1)).reshape(-1)[idx]
            near = ok & (r < 0.5) & ahead
            far = ok & (r >= 0.5)
            inv = 1 / (2 * r.clamp(min=0.5))
            k1 = torch.where(near, 2 * r, torch.where(far, inv, torch.ones_like(r)))
            self.link.append((idx, off, near, far, k1, 1 - k1))

    def _bounced(self, i):
        """The reflected population in direction i at the cells of link[i]."""
        idx, off, near, far, k1, k2 = self.link[i]
        back, own = self.f[self.opp[i]].reshape(-1), self.f[i].reshape(-1)
        ahead = torch.where(near, idx + off, idx)
        second = torch.where(near, back[ahead], torch.where(far, own[idx], torch.zeros_like(k2)))
        return k1 * back[idx] + k2 * second

    def _edge(self, i, oy, oz):
        e = self.e[i]
        if (oy and not self.p.freeSlipY) or (oz and not self.p.freeSlipZ):
            return self.opp[i]
        return self.e.index((e[0], -e[1] if oy else e[1], -e[2] if oz else e[2]))

    def _moments(self, f):
        rho = sum(f)
        u = []
        for k in range(3):
            u.append(sum(f[i] * self.e[i][k] for i in range(self.q) if self.e[i][k]) / rho)
        return rho, u

    def step(self, n):
        for _ in range(n):
            self._step()

    def _step(self):
        nz, ny, nx = self.shape
        g = []
        for i in range(self.q):
            e = self.e[i]
            t = self._at(self.f[i], e, -1)
            ys = None if not e[1] else (0 if e[1] > 0 else ny - 1)
            zs = None if not e[2] else (0 if e[2] > 0 else nz - 1)
            if ys is not None:
                t[:, ys] = self.f[self._edge(i, True, False)][:, ys]
            if zs is not None:
                t[zs] = self.f[self._edge(i, False, True)][zs]
            if ys is not None and zs is not None:
                t[zs, ys] = self.f[self._edge(i, True, True)][zs, ys]
            if self.link[i][0].numel():
                t.view(-1)[self.link[i][0]] = self._bounced(i)
            g.append(t)
        rho, u = self._moments(g)
        e, w = self.e, self.w
        pi = {}
        for a in range(3):
            for b in range(a, 3):
                pi[a, b] = sum(g[i] * (e[i][a] * e[i][b]) for i in range(self.q) if e[i][a] * e[i][b]) - rho * u[a] * u[b]
            pi[a, a] = pi[a, a] - rho / 3
        mag = torch.sqrt(pi[0, 0] ** 2 + pi[1, 1] ** 2 + pi[2, 2] ** 2 +
                         2 * (pi[0, 1] ** 2 + pi[0, 2] ** 2 + pi[1, 2] ** 2))
        tau = self.p.tau
        te = 0.5 * (tau + torch.sqrt(tau * tau + 18 * 2 ** 0.5 * self.p.smagorinskyCs ** 2 * mag / rho))
        if self.closure is not None:
            te = self._learned(te, pi, mag, rho)
        k = (1 - 1 / te) * 4.5
        tr = (pi[0, 0] + pi[1, 1] + pi[2, 2]) / 3
        inlet, outlet = (nx - 1, 0) if self.p.reverseFlow else (0, nx - 1)
        nb = outlet + 1 if self.p.reverseFlow else outlet - 1
        orho, ou = self._moments([t[:, :, nb] for t in self.f])
        orho = 1 + 0.999 * (orho - 1)
        one = torch.ones((nz, ny), dtype=torch.float64, device=CUDA)
        iu = [(-1 if self.p.reverseFlow else 1) * self.p.inletVelocity * one, 0 * one, 0 * one]
        for i in range(self.q):
            s = -tr
            for a in range(3):
                for b in range(a, 3):
                    c = e[i][a] * e[i][b]
                    if c:
                        s = s + (c if a == b else 2 * c) * pi[a, b]
            t = self._eq(i, rho, u) + w[i] * k * s
            t[:, :, inlet] = self._eq(i, one, iu)
            t[:, :, outlet] = self._eq(i, orho, ou)
            t[self.solid] = w[i]
            g[i] = t
        self.f = g

    def _wall(self):
        """Distance to the nearest solid cell in sixteenths of a cell: sixteen chamfer sweeps, as the input is defined."""
        d = torch.where(self.solid, 0, 255).to(torch.int32)
        for _ in range(16):
            pad = torch.nn.functional.pad(d, (1, 1, 1, 1, 1, 1), value=512)
            for a in range(3):
                for b in range(3):
                    for c in range(3):
                        m = (a != 1) + (b != 1) + (c != 1)
                        if m:
                            v = pad[a:a + self.shape[0], b:b + self.shape[1], c:c + self.shape[2]] + (16, 23, 28)[m - 1]
                            d = torch.minimum(d, v)
        return d

    def _learned(self, te, pi, mag, rho):
        c = self.closure
        det = (pi[0, 0] * (pi[1, 1] * pi[2, 2] - pi[1, 2] ** 2) - pi[0, 1] * (pi[0, 1] * pi[2, 2] - pi[1, 2] * pi[0, 2]) +
               pi[0, 2] * (pi[0, 1] * pi[1, 2] - pi[1, 1] * pi[0, 2]))
        safe = mag.clamp(min=1e-30)
        x = [torch.log2(mag / rho + 1e-12), (pi[0, 0] + pi[1, 1] + pi[2, 2]) / safe, det / safe ** 3]
        ok = ~self.solid & (self.wall >= math.ceil(c.wall_min * 16))
        for v, lo, hi in zip(x, c.lo, c.hi):
            ok &= (v >= float(lo)) & (v <= float(hi))
        idx = ok.reshape(-1).nonzero()[:, 0]
        wall = self.wall.reshape(-1)
        w = {k: torch.as_tensor(np.asarray(getattr(c, k)), dtype=torch.float64, device=CUDA)
             for k in ("w1", "b1", "w2", "b2", "w3", "mean", "std")}
        out = te.reshape(-1).clone()
        for part in idx.split(4_000_000):
            z = torch.stack([v.reshape(-1)[part] for v in x] +
                            [wall[part].double() / 16, torch.full_like(out[part], c.filter_width)], dim=1)
            z = torch.relu(((z - w["mean"]) / w["std"]) @ w["w1"] + w["b1"])
            z = torch.relu(z @ w["w2"] + w["b2"])
            out[part] = self.p.tau + 3 * torch.relu(z @ w["w3"] + c.b3) * c.out_scale
        return out.reshape(te.shape)

    def field(self):
        rho, u = self._moments(self.f)
        o = torch.stack([rho] + u, dim=-1)
        force = torch.zeros(self.shape + (4,), dtype=torch.float64, device=CUDA).reshape(-1, 4)
        for i in range(1, self.q):
            idx, off = self.link[i][:2]
            dp = self.f[self.opp[i]].reshape(-1)[idx] + self._bounced(i) - 2 * self.w[i]
            v = torch.stack([torch.full_like(dp, self.w[i])] + [-c * dp for c in self.e[i]], dim=1)
            force.index_add_(0, idx - off, v)
        mag = force[:, 1:].norm(dim=1)
        force[:, 0] = torch.where(force[:, 0] > 0, mag / (6 * force[:, 0].clamp(min=1e-30)), torch.zeros_like(mag))
        return torch.where(self.solid.reshape(-1, 1), force, o.reshape(-1, 4))


def _exact_lattice(case, seed):
    body = case if "body" in case else dict(case, body="sphere")
    solid, sdf, p, field = _problem(body, seed)
    closure = ClosureWeights.load(WEIGHTS) if case.get("closure") else None
    return _Exact(case["q"], solid, sdf, p, field, closure)


def _exact_monitor(case, seed):
    x = _exact_lattice(case, seed)
    x.step(case["steps"])
    f = x.field()
    solid = x.solid.reshape(-1)
    nz, ny, nx = x.shape
    fluid, body = f[~solid], f[solid]
    idx = solid.nonzero()[:, 0]
    # world x is grid y, world y is grid x
    at = torch.stack([(idx // nx) % ny, idx % nx, idx // (nx * ny)], dim=1).double() + 0.5
    lift = body[:, 3].abs()
    speed = fluid[:, 1:].norm(dim=1)
    loaded = body[:, 0][body[:, 0] > 0]
    layer = nx * ny
    return {"force": body[:, 1:].sum(0), "centre": (lift[:, None] * at).sum(0) / lift.sum(), "stress": float(loaded.max()),
            "bad": None, "density": [float(fluid[:, 0].mean()), float(fluid[:, 0].min()), float(fluid[:, 0].max())],
            "speed": [float(speed.mean()), float(speed.max())], "cells": None,
            "slice": f[nz // 2 * layer:][:layer].reshape(-1)}


def _exact_sweep(case, seed):
    force, fields = [], []
    for c, k in _members(case, seed):
        x = _exact_lattice(c, k)
        x.step(case["steps"])
        f = x.field()
        force.append(f[x.solid.reshape(-1), 1:].sum(0))
        fields.append(f.reshape(-1))
    return {"force": torch.stack(force), "fields": fields}


def _exact_smoke(case, seed):
    x = _exact_lattice(case, seed)
    nz, ny, nx = x.shape
    pos = torch.from_numpy(_particle_starts(case, seed)).to(CUDA).double()
    trail = [pos]
    top = torch.tensor([nx, ny, nz], device=CUDA) - 1
    for _ in range(case["frames"]):
        x.step(case["steps"])
        _, u = x._moments(x.f)
        v = torch.stack([u[1], u[0], u[2]], dim=-1)  # world components
        v[x.solid] = 0
        g = torch.stack([pos[:, 1], pos[:, 0], pos[:, 2]], dim=1) - 0.5  # grid coordinates
        base = torch.floor(g)
        t = g - base
        vel = torch.zeros_like(pos)
        for k in range(8):
            d = torch.tensor([k & 1, (k >> 1) & 1, k >> 2], device=CUDA)
            c = torch.minimum((base.long() + d).clamp(min=0), top)
            wt = torch.where(d.bool(), t, 1 - t).prod(dim=1)
            vel += wt[:, None] * v[c[:, 2], c[:, 1], c[:, 0]]
        pos = pos + vel * (SMOKE_SCALE * SMOKE_DT)
        trail.append(pos)
    trail = trail[-case["trail"]:]
    out = torch.zeros((case["particles"], case["trail"], 3), dtype=torch.float64, device=CUDA)
    out[:, :len(trail)] = torch.stack(trail, dim=1)
    return {"points": out, "lens": None}


def _exact_train(case, seed):
    x, y, rows = _training(case, seed)
    x, y = x.double(), y.double()
    p = torch.from_numpy(he_init(int(seed))).to(CUDA).double().requires_grad_(True)
    m, v = torch.zeros_like(p), torch.zeros_like(p)

    def net(z):
        z = torch.relu(z @ p[:160].view(5, 32) + p[160:192])
        z = torch.relu(z @ p[192:1216].view(32, 32) + p[1216:1248])
        return z @ p[1248:1280] + p[1280]

    for k, r in enumerate(rows):
        loss = ((net(x[r]) - y[r]) ** 2).mean()
        g, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m.mul_(0.9).add_(g, alpha=0.1)
            v.mul_(0.999).add_(g * g, alpha=0.001)
            p -= 1e-3 * (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
    with torch.no_grad():
        out = net(x[:case["held_out"]])
    return {"loss": loss.detach().reshape(1), "grad": g, "params": p.detach(), "m": m, "v": v, "predicted": out}


def exact(case, seed):
    kind = case["kind"]
    if kind == "voxelize":
        return None  # its distances, ties and signs are those of the reference's 32-bit operations, bit for bit
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if case["nx"] * case["ny"] * case["nz"] > 50_000_000:
        return None  # over 80 GB in 64 bits
    if kind == "monitor":
        return _exact_monitor(case, seed)
    if kind == "smoke":
        return _exact_smoke(case, seed)
    x = _exact_lattice(case, seed)
    x.step(case["steps"])
    return x.field().reshape(-1)
