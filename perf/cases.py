"""The work that users of this package have it do, as cases to be timed.

Every case goes through the package's public entry points: a tracking run on
a regular grid, on a tetrahedral mesh (octree or hash grid) or on scattered
nodes, an ensemble pass, a gradient, one field evaluation, or a density pass.
The flow is the ABC flow of ``jaxtrace_gb300/workloads.py`` (with a phase that
follows the seed); grids, meshes, time steps, boundaries and densities are
those of that file's configurations, with the step count cut to keep a pass
short.

A case is a dict of plain values: ``kind`` picks the builder below, the other
keys are its sizes and options.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import jaxtrace_gb300 as jt
from jaxtrace_gb300.adjoint import AdjointRK4
from jaxtrace_gb300.density import KDEEstimator, SPHDensityEstimator

UNIT = ((0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # probing a velocity field at a few thousand points (a probe line or a
        # plane), the smallest call: latency and launches count
        dict(name="sample_4k", kind="sample", nx=32, ny=32, nz=32, snapshots=16, bounds="periodic", points=4096, t=0.37),
        # the plain configuration with every row recorded, as the tracker does by default
        dict(name="plain_10k_all_rows", kind="grid", nx=32, ny=32, nz=32, snapshots=16, bounds="periodic", bc="periodic",
             integrator="rk4", storage="f32", precision="exact", particles=10_000, steps=100, dt=0.01, record="all"),
        # the precision configuration's flow and inlet at 128^3 with float32
        # snapshots, particles kept on the device
        dict(name="inlet_f32_2m", kind="grid", nx=128, ny=128, nz=128, snapshots=8, bounds="clamp", bc="inlet",
             integrator="rk4", storage="f32", precision="exact", particles=2_097_152, steps=100, dt=0.002,
             record="device"),
        # the same with bfloat16 storage at its full particle count: the largest call
        dict(name="inlet_bf16_16m", kind="grid", nx=128, ny=128, nz=128, snapshots=8, bounds="clamp", bc="inlet",
             integrator="rk4", storage="bf16", precision="exact", particles=16_777_216, steps=100, dt=0.002,
             record="device"),
        # a ragged grid with the midpoint integrator, positions and velocities
        # recorded every few steps for export
        dict(name="rk2_velocities_odd", kind="grid", nx=97, ny=65, nz=49, snapshots=12, bounds="clamp", bc="reflective",
             integrator="rk2", storage="f32", precision="exact", particles=300_007, steps=60, dt=0.005,
             record="velocities"),
        # the unstructured FEM configuration: octree point location
        dict(name="octree_1m", kind="mesh", locate="octree", cells=64, snapshots=9, particles=1_000_000, steps=64,
             dt=0.005),
        # the same mesh through the hash grid
        dict(name="hash_1m", kind="mesh", locate="hash", cells=64, snapshots=9, particles=1_000_000, steps=32,
             dt=0.005),
        # ensembles of uneven size and release time on the octree mesh
        dict(name="ensembles_24", kind="ensembles", cells=64, snapshots=17, ensembles=24, smallest=1_000,
             largest=100_000, steps=50, dt=0.005),
        # snapshots at scattered nodes, nearest node in space: the reference's default field
        dict(name="nearest_200k", kind="nearest", cells=32, snapshots=9, particles=200_003, steps=50, dt=0.005),
        # the differentiation configuration's field: final positions and both gradients
        dict(name="adjoint_1m", kind="adjoint", n=64, snapshots=16, particles=1_048_576, steps=50, dt=0.01),
        # densities of the final positions of a run, which pile up at the reflective walls
        dict(name="sph_4m", kind="sph", particles=4_000_000, h=0.02),
        dict(name="kde_3m", kind="kde", particles=3_000_017, resolution=100),
    ]


def _spread(rng, lo, hi):
    """An integer of [lo, hi], even over the logarithm."""
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["sample", "grid", "grid", "grid", "mesh", "mesh", "ensembles", "nearest", "adjoint", "sph", "kde"])
    if kind == "sample":
        return dict(kind=kind, nx=_spread(rng, 9, 96), ny=_spread(rng, 9, 96), nz=_spread(rng, 9, 96),
                    snapshots=rng.randint(2, 16), bounds=rng.choice(["clamp", "periodic"]),
                    points=_spread(rng, 1_000, 2_000_000), t=rng.uniform(0.0, 1.0))
    if kind == "grid":
        storage = rng.choice(["f32", "f32", "bf16", "f16"])
        record = rng.choice(["device", "device", "all", "velocities"])
        bc = rng.choice(["inlet", "periodic", "reflective"])
        steps = rng.randint(20, 100)
        top = 16_000_000 if record == "device" else 10_000_000 // steps
        return dict(kind=kind, nx=_spread(rng, 17, 128), ny=_spread(rng, 17, 128), nz=_spread(rng, 17, 128),
                    snapshots=rng.randint(4, 12), bounds="periodic" if bc == "periodic" else "clamp", bc=bc,
                    integrator=rng.choice(["rk4", "rk4", "rk2", "euler"]), storage=storage,
                    precision=rng.choice(["exact", "compensated"]), particles=_spread(rng, 2_000, top),
                    steps=steps, dt=rng.choice([0.002, 0.005]), record=record)
    if kind == "mesh":
        locate = rng.choice(["octree", "hash"])
        return dict(kind=kind, locate=locate, cells=_spread(rng, 12, 64), snapshots=rng.randint(4, 12),
                    particles=_spread(rng, 2_000, 1_000_000), steps=rng.randint(8, 64 if locate == "octree" else 32),
                    dt=0.005)
    if kind == "ensembles":
        return dict(kind=kind, cells=_spread(rng, 12, 64), snapshots=rng.randint(8, 17), ensembles=rng.randint(3, 32),
                    smallest=_spread(rng, 200, 2_000), largest=_spread(rng, 10_000, 100_000),
                    steps=rng.randint(10, 50), dt=0.005)
    if kind == "nearest":
        return dict(kind=kind, cells=_spread(rng, 10, 48), snapshots=rng.randint(4, 12),
                    particles=_spread(rng, 2_000, 300_000), steps=rng.randint(8, 50), dt=0.005)
    if kind == "adjoint":
        return dict(kind=kind, n=_spread(rng, 17, 64), snapshots=rng.randint(4, 16),
                    particles=_spread(rng, 10_000, 1_000_000), steps=rng.randint(10, 60), dt=0.01)
    if kind == "sph":
        return dict(kind=kind, particles=_spread(rng, 20_000, 4_000_000), h=rng.choice([0.015, 0.02, 0.03]))
    return dict(kind=kind, particles=_spread(rng, 20_000, 4_000_000), resolution=rng.choice([64, 81, 100]))


# ---------------------------------------------------------------------------
# inputs, made on the GPU from the seed
# ---------------------------------------------------------------------------
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _flow(p, t, phase, offset):
    """ABC flow at float64 points of the unit cube, slowly varying in time."""
    x, y, z = (2 * math.pi * (p + phase)).unbind(-1)
    s = 1.0 + 0.1 * math.sin(2 * math.pi * t)
    u = torch.stack([torch.sin(z) + 0.43 * torch.cos(y), 0.7 * torch.sin(x) + torch.cos(z),
                     0.43 * torch.sin(y) + 0.7 * torch.cos(x)], dim=-1) * s
    u[..., 0] += offset
    return u


def _snapshots(nodes, times, gen, offset=0.0, noise=0.0):
    """(T, N, 3) float32 snapshots on the GPU."""
    phase = torch.rand(3, generator=gen, device=DEV, dtype=F64)
    out = torch.empty((len(times), nodes.shape[0], 3), dtype=torch.float32, device=DEV)
    for k, t in enumerate(times):
        v = _flow(nodes, float(t), phase, offset)
        if noise:
            v = v + noise * torch.randn(v.shape, generator=gen, device=DEV, dtype=F64)
        out[k] = v
    return out


def _axes(case):
    """Grid axes in float32: [0, 1) without its last node on a periodic grid, else [0, 1]."""
    per = case["bounds"] == "periodic"
    return [(np.arange(n) / n if per else np.linspace(0.0, 1.0, n)).astype(np.float32)
            for n in (case["nx"], case["ny"], case["nz"])]


def _nodes(axes):
    g = torch.meshgrid(*[torch.from_numpy(a).to(DEV, F64) for a in axes], indexing="ij")
    return torch.stack([a.reshape(-1) for a in g], dim=1)


def _grid_inputs(case, seed):
    gen = _rng(seed)
    axes = _axes(case)
    end = case["steps"] * case["dt"] if "steps" in case else 1.0
    times = np.linspace(0.0, end, case["snapshots"]).astype(np.float32)
    inlet = case.get("bc") == "inlet"
    data = _snapshots(_nodes(axes), times, gen, 1.0 if inlet else 0.0, 0.01 if inlet else 0.0)
    n = case["particles"] if "particles" in case else case["points"]
    x0 = torch.rand((n, 3), generator=gen, device=DEV)
    return axes, times, data, x0


def _mesh(case, gen):
    """Nodes of a jittered lattice over the unit cube, each hexahedron split in six tetrahedra."""
    n = case["cells"]
    g = np.linspace(0.0, 1.0, n + 1)
    P = _nodes([g, g, g])
    inside = ((P > 0) & (P < 1)).all(dim=1, keepdim=True)
    P = P + inside * (torch.rand(P.shape, generator=gen, device=DEV, dtype=F64) - 0.5) * (0.4 / n)
    idx = torch.arange((n + 1) ** 3, device=DEV).reshape(n + 1, n + 1, n + 1)
    corner = torch.stack([idx[c & 1:n + (c & 1), c >> 1 & 1:n + (c >> 1 & 1), c >> 2:n + (c >> 2)].reshape(-1)
                          for c in range(8)], dim=1)
    local = torch.tensor([(0, 1, 3, 7), (0, 1, 5, 7), (0, 2, 3, 7), (0, 2, 6, 7), (0, 4, 5, 7), (0, 4, 6, 7)],
                         device=DEV)
    return P.float(), corner[:, local].reshape(-1, 4).to(torch.int32)


def _mesh_inputs(case, seed, span):
    gen = _rng(seed)
    P, tets = _mesh(case, gen)
    times = np.linspace(0.0, span, case["snapshots"]).astype(np.float32)
    return gen, P, tets, times, _snapshots(P.double(), times, gen)


def _ensemble_inputs(case, gen):
    """Seed positions per ensemble and release times; the sizes belong to the case."""
    r = np.random.default_rng(case["ensembles"])
    sizes = np.round(np.exp(r.uniform(math.log(case["smallest"]), math.log(case["largest"]), case["ensembles"])))
    release = r.uniform(0.0, 0.25, case["ensembles"])
    return [torch.rand((int(s), 3), generator=gen, device=DEV) for s in sizes], release


def _piled(n, gen):
    """Positions that pile up at the walls y = 0 and y = 1, as those of a run with reflective walls do."""
    p = torch.rand((n, 3), generator=gen, device=DEV)
    d = (-0.03 * torch.log1p(-0.999 * torch.rand(n, generator=gen, device=DEV))).clamp_(max=0.5)
    side = torch.rand(n, generator=gen, device=DEV)
    p[:, 1] = torch.where(side < 0.29, d, torch.where(side < 0.58, 1.0 - d, p[:, 1]))
    return p


def _boundary(case):
    if case["bc"] == "inlet":
        return jt.continuous_inlet_boundary_factory(UNIT, "x", "positive", "grid", {"x": 256, "y": 256, "z": 256})
    return jt.periodic_boundary(UNIT) if case["bc"] == "periodic" else jt.reflective_boundary(UNIT)


WALLS = {"x": "periodic", "y": "reflective", "z": "periodic"}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("sample", "grid"):
        axes, times, data, x0 = _grid_inputs(case, seed)
        field = jt.StructuredTimeSeriesField(data.cpu().numpy(), times, *axes, case["bounds"],
                                             storage=case.get("storage", "f32"))
        if kind == "sample":
            field.sample_at_positions(x0[:1], 0.0)
            return {"kind": kind, "field": field, "x": x0, "t": case["t"]}
        opts = {"precision": case["precision"]}
        if case["record"] == "device":
            opts["record_final_only"] = True
        elif case["record"] == "velocities":
            opts.update(record_velocities=True, record_every=10)
        tr = jt.create_tracker(case["integrator"], field, _boundary(case), **opts)
        # a first short call uploads the field, as it does once in a user's program
        tr.track_particles(x0[:64], (0.0, case["dt"]), 2, dt=case["dt"])
        x = x0 if case["record"] == "device" else x0.cpu().numpy()
        return {"kind": kind, "tracker": tr, "x": x, "case": case}
    if kind == "mesh":
        gen, P, tets, times, data = _mesh_inputs(case, seed, case["steps"] * case["dt"])
        make = jt.OctreeFEMTimeSeriesFieldOptimized if case["locate"] == "octree" else jt.FEMTimeSeriesField
        field = make(data.cpu().numpy(), times, P.cpu().numpy(), tets.cpu().numpy())
        x0 = torch.rand((case["particles"], 3), generator=gen, device=DEV)
        field.sample_at_positions(x0[:1], 0.0)
        tr = jt.create_tracker("rk4", field, jt.mixed_boundary(UNIT, WALLS), record_final_only=True)
        return {"kind": kind, "tracker": tr, "x": x0, "case": case}
    if kind == "ensembles":
        gen, P, tets, times, data = _mesh_inputs(case, seed, 0.25 + case["steps"] * case["dt"])
        field = jt.OctreeFEMTimeSeriesFieldOptimized(data.cpu().numpy(), times, P.cpu().numpy(), tets.cpu().numpy())
        xs, release = _ensemble_inputs(case, gen)
        tr = jt.create_tracker("rk4", field, jt.mixed_boundary(UNIT, WALLS))
        batch = tr.ensemble_batch([x.cpu().numpy() for x in xs], release, case["steps"] + 1, dt=case["dt"])
        return {"kind": kind, "batch": batch}
    if kind == "nearest":
        gen, P, _, times, data = _mesh_inputs(case, seed, case["steps"] * case["dt"])
        field = jt.TimeSeriesField(data.cpu().numpy(), times, P.cpu().numpy())
        x0 = torch.rand((case["particles"], 3), generator=gen, device=DEV)
        field.sample_at_positions(x0[:1], 0.0)
        tr = jt.create_tracker("rk4", field, jt.periodic_boundary(UNIT), record_final_only=True)
        return {"kind": kind, "tracker": tr, "x": x0, "case": case}
    if kind == "adjoint":
        axes, times, data, x0, cot = _adjoint_inputs(case, seed)
        solver = AdjointRK4(times, *axes, "periodic", jt.periodic_boundary(UNIT))
        n = case["n"]
        U = data.reshape(case["snapshots"], n, n, n, 3).requires_grad_(True)
        return {"kind": kind, "solver": solver, "x": x0.requires_grad_(True), "U": U, "cot": cot, "case": case}
    return {"kind": kind, "x": _piled(case["particles"], _rng(seed)), "case": case}


def _adjoint_inputs(case, seed):
    n = case["n"]
    grid = dict(nx=n, ny=n, nz=n, bounds="periodic", snapshots=case["snapshots"], steps=case["steps"], dt=case["dt"],
                particles=case["particles"])
    axes, times, data, x0 = _grid_inputs(grid, seed)
    cot = torch.randn(x0.shape, generator=_rng(seed + 1), device=DEV)
    return axes, times, data, x0, cot


def run(state):
    kind = state["kind"]
    if kind == "sample":
        return state["field"].sample_at_positions(state["x"], state["t"])
    if kind == "ensembles":
        return state["batch"].run().pos
    c = state["case"]
    if kind == "sph":
        return SPHDensityEstimator(state["x"], dimensions="3d", smoothing_length=c["h"]).evaluate(state["x"])
    if kind == "kde":
        return KDEEstimator(state["x"], resolution=c["resolution"]).evaluate_3d()
    span, rows, dt = (0.0, c["steps"] * c["dt"]), c["steps"] + 1, c["dt"]
    if kind == "adjoint":
        xT = state["solver"](state["x"], state["U"], span, rows, dt=dt)
        gx, gU = torch.autograd.grad(xT, (state["x"], state["U"]), state["cot"])
        return {"x": xT.detach(), "dx0": gx, "dU": gU}
    if kind == "grid" and c["record"] != "device":
        traj = state["tracker"].track_particles(state["x"], span, rows, dt=dt)
        out = {"positions": traj.positions}
        if c["record"] == "velocities":
            out["velocities"] = traj.velocities
        return out
    return state["tracker"].track_particles(state["x"], span, rows, dt=dt, return_device=True)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    evals = {"rk4": 4, "rk2": 2, "euler": 1}
    if kind in ("sample", "grid"):
        nodes = case["nx"] * case["ny"] * case["nz"]
        if kind == "sample":
            return {"bytes": 2 * min(nodes, 8 * case["points"]) * 12 + 24 * case["points"], "flops": 110 * case["points"]}
        n, s = case["particles"], case["steps"]
        rows = {"device": 1, "all": s + 1, "velocities": 2 * (1 + s // 10)}[case["record"]]
        value = 12 if case["storage"] == "f32" else 6
        # per evaluation: cell and weights (12), trilinear (42), both snapshots blended (54)
        return {"bytes": case["snapshots"] * nodes * value + 12 * n * (1 + rows),
                "flops": n * s * (108 * evals[case["integrator"]] + 24)}
    if kind in ("mesh", "ensembles", "nearest"):
        nodes = (case["cells"] + 1) ** 3
        if kind == "ensembles":
            lo, hi = case["smallest"], case["largest"]
            n = case["ensembles"] * (hi - lo) / math.log(hi / lo) if hi > lo else case["ensembles"] * lo
        else:
            n = case["particles"]
        tets = 0 if kind == "nearest" else 6 * case["cells"] ** 3
        # per evaluation: barycentrics (70), four corners blended (36), weighted sum (21); nearest: one corner
        flops = 20 if kind == "nearest" else 127
        return {"bytes": int(case["snapshots"] * nodes * 12 + nodes * 12 + tets * 16 + 24 * n),
                "flops": int(n * case["steps"] * (4 * flops + 24))}
    if kind == "adjoint":
        n, s, U = case["particles"], case["steps"], case["snapshots"] * case["n"] ** 3 * 12
        # forward, its recomputation, and per evaluation the vector-Jacobian product and the weighted cotangents
        return {"bytes": 2 * U + 48 * n, "flops": n * s * (2 * (4 * 108 + 24) + 4 * 260)}
    n = case["particles"]
    if kind == "sph":
        # pairs inside the support 2h of a uniform cloud, 18 operations each; the walls hold about five times as many
        pairs = 5.0 * n * n * 4.0 / 3.0 * math.pi * (2 * case["h"]) ** 3
        return {"bytes": 16 * n, "flops": int(18 * min(pairs, float(n) * n))}
    r = case["resolution"]
    h = 0.31 * n ** (-1.0 / 7.0)
    # separable: three factors per particle and axis point within 5 bandwidths, one multiply-add per grid point
    per_axis = min(10.0 * h * r, float(r))
    return {"bytes": 12 * n + 16 * r ** 3, "flops": int(n * (2.0 * per_axis ** 3 * math.pi / 6.0 + 30.0 * per_axis))}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _weights(times, t):
    """Bracketing snapshots of time t and the weight of the second."""
    T = np.asarray(times, dtype=np.float64)
    if t <= T[0]:
        return 0, 0, 0.0
    if t >= T[-1]:
        return len(T) - 1, len(T) - 1, 0.0
    r = int(np.searchsorted(T, t, side="right"))
    return r - 1, r, float((t - T[r - 1]) / (T[r] - T[r - 1]))


def _blend(data, times, t):
    a, b, w = _weights(times, t)
    return data[a].double() * (1.0 - w) + data[b].double() * w


def _cells(p, axes, periodic):
    """Lower and upper index and upper weight of each axis."""
    out = []
    for a in range(3):
        n = len(axes[a])
        f = (p[:, a] - float(axes[a][0])) / float(axes[a][1] - axes[a][0])
        f = torch.remainder(f, n) if periodic else f.clamp(0, n - 1)
        i = f.floor().clamp(max=n - 1)
        lo = i.long()
        out.append((lo, (lo + 1) % n if periodic else (lo + 1).clamp(max=n - 1), f - i))
    return out


def _corners(cells, axes):
    ny, nz = len(axes[1]), len(axes[2])
    for c in range(8):
        i, j, k = (cells[a][c >> a & 1] for a in range(3))
        w = [cells[a][2] if c >> a & 1 else 1.0 - cells[a][2] for a in range(3)]
        yield c, (i * ny + j) * nz + k, w


def _trilinear(values, p, axes, periodic, piece=1 << 22):
    out = torch.empty_like(p)
    for b in range(0, p.shape[0], piece):
        cells = _cells(p[b:b + piece], axes, periodic)
        acc = 0.0
        for _, node, w in _corners(cells, axes):
            acc = acc + (w[0] * w[1] * w[2])[:, None] * values[node]
        out[b:b + piece] = acc
    return out


def _step(velocity, integrator, x, t, dt):
    """One step with velocity(x, t); the reference's RK2 is the midpoint rule."""
    k1 = velocity(x, t)
    if integrator == "euler":
        return x + dt * k1
    k2 = velocity(x + 0.5 * dt * k1, t + 0.5 * dt)
    if integrator == "rk2":
        return x + dt * k2
    k3 = velocity(x + 0.5 * dt * k2, t + 0.5 * dt)
    k4 = velocity(x + dt * k3, t + dt)
    return x + dt / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4)


def _fold(x, reflective):
    return 1.0 - (torch.remainder(x, 2.0) - 1.0).abs() if reflective else torch.remainder(x, 1.0)


def _apply(bc, x):
    if bc == "periodic":
        return _fold(x, False)
    if bc == "reflective":
        return _fold(x, True)
    if bc == "walls":
        return torch.stack([_fold(x[:, 0], False), _fold(x[:, 1], True), _fold(x[:, 2], False)], dim=1)
    # inlet: what left through x = 1 comes back in at x = 0 on the 256^2 lattice
    out = x[:, 0] > 1.0
    snap = lambda u: (u.clamp(0, 1) * 255.0).round() / 255.0  # noqa: E731
    xs = torch.where(out, torch.zeros_like(x[:, 0]), x[:, 0])
    xs = torch.where(xs < 0, torch.full_like(xs, 0.001), xs)
    yz = torch.where(out[:, None], snap(x[:, 1:]), x[:, 1:])
    yz = torch.where(yz < 0, -yz, torch.where(yz > 1, 2.0 - yz, yz))
    return torch.cat([xs[:, None], yz], dim=1)


def _exact_grid(case, seed):
    axes, times, data, x0 = _grid_inputs(case, seed)
    per = case["bounds"] == "periodic"
    x, dt = x0.double(), case["dt"]
    every = {"device": 0, "all": 1, "velocities": 10}[case["record"]]

    def velocity(p, t):
        return _trilinear(_blend(data, times, t), p, axes, per)

    rows, vels = [x], [velocity(x, 0.0)] if case["record"] == "velocities" else []
    for s in range(case["steps"]):
        x = _apply(case["bc"], _step(velocity, case["integrator"], x, s * dt, dt))
        if every and (s + 1) % every == 0:
            rows.append(x)
            if vels:
                vels.append(velocity(x, (s + 1) * dt))
    if not every:
        return x
    out = {"positions": torch.stack(rows).cpu().numpy()}
    if vels:
        out["velocities"] = torch.stack(vels).cpu().numpy()
    return out


class _Tets:
    """P1 on the jittered mesh: barycentrics from the inverse edge matrix of every tetrahedron."""

    def __init__(self, P, tets, cells):
        self.P, self.tets, self.n = P.double(), tets.long(), cells
        v = self.P[self.tets]
        self.v0 = v[:, 0]
        self.inv = torch.linalg.inv((v[:, 1:] - v[:, :1]).transpose(1, 2))

    def hexes(self, q, spread):
        """The hexahedra within `spread` of the one that q's lattice cell is: (M, k)."""
        n = self.n
        c = (q * n).floor().long().clamp(0, n - 1)
        r = torch.arange(-spread, spread + 1, device=q.device)
        d = torch.cartesian_prod(r, r, r).reshape(-1, 3)
        h = (c[:, None] + d[None]).clamp(0, n - 1)
        return (h[..., 0] * n + h[..., 1]) * n + h[..., 2]

    def bary(self, q, ids):
        b = torch.einsum("mkij,mkj->mki", self.inv[ids], q[:, None] - self.v0[ids])
        return torch.cat([1.0 - b.sum(dim=2, keepdim=True), b], dim=2)

    def locate(self, q, spread):
        """First tetrahedron (lowest number) of the nearby hexahedra that holds q, its barycentrics, and whether there is one."""
        ids = (6 * self.hexes(q, spread)[..., None] + torch.arange(6, device=q.device)).reshape(q.shape[0], -1)
        b = self.bary(q, ids)
        held = ((b >= -1e-6) & (b <= 0.999999)).all(dim=2)
        first = torch.where(held, ids, ids.max() + 1).argmin(dim=1)
        row = torch.arange(q.shape[0], device=q.device)
        return ids[row, first], b[row, first], held.any(dim=1)

    def value(self, V, tet, b):
        return (b[..., None] * V[self.tets[tet]]).sum(dim=1)

    def octree(self, q, V, piece=1 << 20):
        """One octree leaf per hexahedron; no hit: the nearest vertex of the leaf's first tetrahedron."""
        out = torch.empty_like(q)
        for a in range(0, q.shape[0], piece):
            p = q[a:a + piece]
            tet, b, ok = self.locate(p, 0)
            four = self.tets[6 * self.hexes(p, 0)[:, 0]]
            near = ((self.P[four] - p[:, None]) ** 2).sum(dim=2).argmin(dim=1)
            vertex = four[torch.arange(p.shape[0], device=p.device), near]
            out[a:a + piece] = torch.where(ok[:, None], self.value(V, tet, b), V[vertex])
        return out

    def hashed(self, q, V, piece=1 << 20):
        """The tetrahedron that holds q anywhere in the mesh; none: the nearest node."""
        out = torch.empty_like(q)
        for a in range(0, q.shape[0], piece):
            p = q[a:a + piece]
            tet, b, ok = self.locate(p, 0)
            v = self.value(V, tet, b)
            rest = torch.nonzero(~ok)[:, 0]
            for c in range(0, rest.shape[0], piece // 8):
                k = rest[c:c + piece // 8]
                tet, b, held = self.locate(p[k], 1)
                v[k] = torch.where(held[:, None], self.value(V, tet, b), V[_nearest(p[k], self.P, self.n)])
            out[a:a + piece] = v
        return out


def _nearest(q, P, cells):
    """The node nearest to q among the 27 around its lattice point (the jitter is a fifth of a cell)."""
    c = (q * cells).round().long().clamp(0, cells)
    r = torch.arange(-1, 2, device=q.device)
    h = (c[:, None] + torch.cartesian_prod(r, r, r)[None]).clamp(0, cells)
    ids = (h[..., 0] * (cells + 1) + h[..., 1]) * (cells + 1) + h[..., 2]
    near = ((P[ids] - q[:, None]) ** 2).sum(dim=2).argmin(dim=1)
    return ids[torch.arange(q.shape[0], device=q.device), near]


def _exact_mesh(case, seed):
    kind = case["kind"]
    octree = kind == "ensembles" or case.get("locate") == "octree"
    if octree and case["cells"] & (case["cells"] - 1):
        return None  # a leaf is one hexahedron only where the lattice is a power of two
    span = case["steps"] * case["dt"] + (0.25 if kind == "ensembles" else 0.0)
    gen, P, tets, times, data = _mesh_inputs(case, seed, span)
    mesh = None if kind == "nearest" else _Tets(P, tets, case["cells"])
    Pd, dt = P.double(), case["dt"]

    def velocity(p, t):
        V = _blend(data, times, t)
        if kind == "nearest":
            return V[torch.cat([_nearest(q, Pd, case["cells"]) for q in p.split(1 << 20)])]
        return mesh.octree(p, V) if octree else mesh.hashed(p, V)

    def advance(x, t0):
        for s in range(case["steps"]):
            x = _apply("periodic" if kind == "nearest" else "walls", _step(velocity, "rk4", x, t0 + s * dt, dt))
        return x

    if kind == "ensembles":
        xs, release = _ensemble_inputs(case, gen)
        return torch.cat([advance(x.double(), float(t)) for x, t in zip(xs, release)])
    return advance(torch.rand((case["particles"], 3), generator=gen, device=DEV).double(), 0.0)


def _exact_adjoint(case, seed):
    axes, times, data, x0, cot = _adjoint_inputs(case, seed)
    h, steps = case["dt"], case["steps"]
    inv = [1.0 / float(a[1] - a[0]) for a in axes]
    dU = torch.zeros(data.shape, dtype=F64, device=DEV)

    def velocity(p, t):
        return _trilinear(_blend(data, times, t), p, axes, True)

    def back(p, t, g):
        """J^T g at p, and the share of the snapshots in dU."""
        V = _blend(data, times, t)
        cells = _cells(p, axes, True)
        out = torch.zeros_like(p)
        dV = torch.zeros_like(V)
        for c, node, w in _corners(cells, axes):
            vg = (V[node] * g).sum(dim=1)
            for a in range(3):
                s = inv[a] if c >> a & 1 else -inv[a]
                out[:, a] += s * w[(a + 1) % 3] * w[(a + 2) % 3] * vg
            dV.index_add_(0, node, (w[0] * w[1] * w[2])[:, None] * g)
        a, b, w = _weights(times, t)
        dU[a] += (1.0 - w) * dV
        dU[b] += w * dV
        return out

    x, points = x0.double(), []
    for s in range(steps):
        t = s * h
        k1 = velocity(x, t)
        x2 = x + 0.5 * h * k1
        k2 = velocity(x2, t + 0.5 * h)
        x3 = x + 0.5 * h * k2
        k3 = velocity(x3, t + 0.5 * h)
        x4 = x + h * k3
        points.append((x, x2, x3, x4))
        x = _fold(x + h / 6.0 * (k1 + 2 * k2 + 2 * k3 + velocity(x4, t + h)), False)
    lam = cot.double()
    for s in reversed(range(steps)):
        t, (p1, p2, p3, p4) = s * h, points.pop()
        g4 = h / 6.0 * lam
        l4 = back(p4, t + h, g4)
        l3 = back(p3, t + 0.5 * h, h / 3.0 * lam + h * l4)
        l2 = back(p2, t + 0.5 * h, h / 3.0 * lam + 0.5 * h * l3)
        l1 = back(p1, t, g4 + 0.5 * h * l2)
        lam = lam + l1 + l2 + l3 + l4
    n = case["n"]
    return {"x": x, "dx0": lam, "dU": dU.reshape(case["snapshots"], n, n, n, 3)}


def _exact_sph(case, seed):
    p = _piled(case["particles"], _rng(seed)).double()
    h, n = case["h"], case["particles"]
    m = int(1.0 / (2.0 * h))  # cells at least as wide as the support
    c = (p * m).long().clamp(0, m - 1)
    key = (c[:, 0] * m + c[:, 1]) * m + c[:, 2]
    order = torch.argsort(key)
    p, start = p[order], torch.searchsorted(key[order], torch.arange(m ** 3 + 1, device=DEV)).tolist()
    rho = torch.empty(n, dtype=F64, device=DEV)
    sigma = 1.0 / (math.pi * h ** 3)
    for i in range(m):
        for j in range(m):
            for k in range(m):
                cell = (i * m + j) * m + k
                a, b = start[cell], start[cell + 1]
                if a == b:
                    continue
                near = [p[start[(u * m + v) * m + max(k - 1, 0)]:start[(u * m + v) * m + min(k + 1, m - 1) + 1]]
                        for u in range(max(i - 1, 0), min(i + 2, m)) for v in range(max(j - 1, 0), min(j + 2, m))]
                near = torch.cat(near)
                size = max(1, (1 << 26) // near.shape[0])
                for u in range(a, b, size):
                    q = p[u:min(u + size, b)]
                    d2 = sum((q[:, None, e] - near[None, :, e]) ** 2 for e in range(3))
                    r = d2.sqrt_().div_(h)
                    w = torch.where(r <= 1.0, 1.0 - 1.5 * r * r + 0.75 * r ** 3, 0.25 * (2.0 - r).clamp(min=0.0) ** 3)
                    rho[u:u + q.shape[0]] = w.sum(dim=1)
    out = torch.empty_like(rho)
    out[order] = rho * sigma
    return (out / (n / float((p.amax(0) - p.amin(0)).prod()))).cpu().numpy()


def _exact_kde(case, seed):
    p = _piled(case["particles"], _rng(seed)).double()
    n, r = case["particles"], case["resolution"]
    h = float(p.std(dim=0).mean()) * n ** (-1.0 / 7.0)
    axes = [torch.linspace(float(p[:, a].min()), float(p[:, a].max()), r, dtype=F64, device=DEV) for a in range(3)]
    total = torch.zeros((r, r * r), dtype=F64, device=DEV)
    for q in p.split(1 << 16):
        e = [torch.exp(-0.5 * ((axes[a][None] - q[:, a:a + 1]) / h) ** 2) for a in range(3)]
        total += e[0].T @ (e[1][:, :, None] * e[2][:, None, :]).reshape(q.shape[0], r * r)
    X, Y, Z = torch.meshgrid(*axes, indexing="xy")
    D = total.reshape(r, r, r).transpose(0, 1) * ((2.0 * math.pi) ** -1.5 / n)
    span = math.prod(float(a[-1] - a[0]) for a in axes)
    D = D * (n / float(D.sum() * span / (r - 1) ** 3)) / (n / span)
    return tuple(a.cpu().numpy() for a in (X, Y, Z, D))


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        axes, times, data, x = _grid_inputs(case, seed)
        return _trilinear(_blend(data, times, case["t"]), x.double(), axes, case["bounds"] == "periodic")
    if kind == "grid":
        return _exact_grid(case, seed)
    if kind in ("mesh", "ensembles", "nearest"):
        return _exact_mesh(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    return _exact_sph(case, seed) if kind == "sph" else _exact_kde(case, seed)
