"""What a user of this framework has it do, as cases that can be timed.

Four kinds of call, each through the public Python API:

  flow    substeps of a scene that already holds liquid (``Solver.substep``) and the particles read
          back, as a simulation loop between two frames does it
  sdf     a triangle mesh voxelised into a signed distance field (``sdf_from_mesh``), the start of
          every run on a scanned cavity
  frame   what a run writes per frame: metrics (``MetricsCollector.record``), two previews
          (``render_slice``) and the particle positions and velocities
  batch   many small scenes from their first substep to their summary (``run_batch``), packed into
          one launch per operation or with a stream per scene

``listed`` gives the cases, ``draw`` more of the same ranges, ``prepare`` what a program holds before
the call (made from the seed), ``run`` one pass, ``work`` the bytes and operations a pass cannot do
without, ``exact`` its result in 64 bits without this package, where there is one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sdr_b200 import scene as sc
from sdr_b200 import workloads
from sdr_b200.cavity import perturbed_ellipsoid
from sdr_b200.render import SlicePlane, render_slice
from sdr_b200.serving import run_batch
from sdr_b200.solver import MetricsCollector, Solver, build_sdf, cavity_volume, sdf_from_mesh

PPC = 8              # particles per cell, the default of every scene
SETTLED_SPEED = 0.5  # m/s: the CFL speed of a pool without a jet
MESH_BOX_MM = (9.6, 25.3, 18.7)  # the box of the sdf cases' cavities
CAVITY_SEED = 2      # the real-cavity workload's cavity


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # The continuous-integration scene (2 mm): one substep, where launches and latency are all there is.
        dict(name="flow_sinus_2mm", kind="flow", cavity="sinus", dx_mm=2.0, fill=0.25, flow_ml_s=5.0, substeps=1),
        # The `sdr init` scene at 0.8 mm with the jet on: the usual desktop run, in its first second.
        dict(name="flow_sinus_0p8mm_jet", kind="flow", cavity="sinus", dx_mm=0.8, fill=0.15, flow_ml_s=4.0, substeps=8),
        # A scanned cavity at 0.5 mm, needle firing into the liquid.
        dict(name="flow_cavity_0p5mm_jet", kind="flow", cavity="ellipsoid", dx_mm=0.5, fill=0.3, flow_ml_s=4.0,
             substeps=8),
        # The same cavity with the dose in: settling, longer steps, no emission.
        dict(name="flow_cavity_0p5mm_settled", kind="flow", cavity="ellipsoid", dx_mm=0.5, fill=0.55, flow_ml_s=0.0,
             substeps=8),
        # Between the small scenes and the largest: a half-full cavity at 0.4 mm.
        dict(name="flow_sinus_0p4mm_pool", kind="flow", cavity="sinus", dx_mm=0.4, fill=0.5, flow_ml_s=6.0, substeps=2),
        # The large single scene: the 0.2 mm cavity full of liquid, 9.5 M particles, the benchmark's state.
        dict(name="flow_sinus_0p2mm_pool", kind="flow", cavity="sinus", dx_mm=0.2, fill=1.0, flow_ml_s=6.0, substeps=2),
        # A coarse mesh on a coarse grid, and the 20k-triangle cavity at the resolution it is simulated at.
        dict(name="sdf_1k_tri_1mm", kind="sdf", subdiv=3, dx_mm=1.0),
        dict(name="sdf_20k_tri_0p5mm", kind="sdf", subdiv=5, dx_mm=0.5),
        # The output of one frame: the scanned cavity, and a pool of 2.8 M particles.
        dict(name="frame_cavity_0p5mm", kind="frame", cavity="ellipsoid", dx_mm=0.5, fill=0.55, flow_ml_s=0.0, px=600),
        dict(name="frame_sinus_0p3mm", kind="frame", cavity="sinus", dx_mm=0.3, fill=1.0, flow_ml_s=6.0, px=600),
        # Scenes of the batched and served family (32^3 to 96^3 cells), from t = 0.
        dict(name="batch_packed_16", kind="batch", scenes=16, cfl_steps=40, packed=True),
        dict(name="batch_streams_16", kind="batch", scenes=16, cfl_steps=40, packed=False),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "sdf", "frame", "batch"])
    if kind in ("flow", "frame"):
        cavity = rng.choice(["sinus", "sinus", "ellipsoid"])
        # sinus: 0.25 mm holds about 5 M particles; the scanned cavity is ten times smaller
        dx = _log(rng, 0.25, 2.0) if cavity == "sinus" else _log(rng, 0.2, 0.8)
        c = dict(kind=kind, cavity=cavity, dx_mm=round(dx, 3), fill=round(rng.uniform(0.1, 1.0), 3),
                 flow_ml_s=rng.choice([0.0, round(rng.uniform(1.0, 8.0), 2)]))
        if kind == "flow":
            c["substeps"] = rng.choice([1, 2, 3]) if dx < 0.6 else rng.choice([1, 4, 8])
        else:
            c["px"] = rng.choice([300, 600, 601])
        return c
    if kind == "sdf":
        return dict(kind="sdf", subdiv=rng.choice([2, 3, 4, 5]), dx_mm=round(_log(rng, 0.5, 2.0), 3))
    return dict(kind="batch", scenes=rng.randint(3, 16), cfl_steps=rng.randint(20, 40), packed=rng.choice([True, False]))


# ---------------------------------------------------------------- inputs
def _workload(case) -> workloads.Workload:
    if case["cavity"] == "ellipsoid":
        return workloads.real_cavity(seed=CAVITY_SEED, flow_ml_s=max(case["flow_ml_s"], 1.0), dx_mm=case["dx_mm"])
    cfg = sc.SceneConfig.from_toml_str(
        f"[sim]\nresolution_mm = {case['dx_mm']}\npcg_iters = 400\npcg_tol = 1e-6\n"
        f"[needle]\nflow_rate_ml_s = {case['flow_ml_s']}\n")
    return workloads.Workload("sinus", cfg.resolve())


def _pool(dims, origin, dx, gravity, mask, fill, seed):
    """Liquid in motion: the deepest cells along gravity up to ``fill`` of the cavity, PPC particles each spread over
    the cell (nearer its centre in the cells of the wall, so that none lies behind it), one in 140 displaced into the
    cells around (so that a few per cent of the particles sit in overfull cells, as in a stirred run), a slow swirl
    about the vertical axis and some noise in the velocities. Rounded to f32."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(device=dev).manual_seed(1_000_003 + seed)
    nx, ny, nz = (int(v) for v in dims)
    cav = torch.zeros(nz + 2, ny + 2, nx + 2, dtype=torch.bool, device=dev)
    cav[1:-1, 1:-1, 1:-1] = torch.from_numpy(mask.reshape(nz, ny, nx)).to(dev) != 0
    inner = cav.clone()  # cavity cells without a wall beside them
    for axis in range(3):
        inner &= cav.roll(1, axis) & cav.roll(-1, axis)
    inner = inner[1:-1, 1:-1, 1:-1].reshape(-1)
    cells = torch.from_numpy(np.flatnonzero(mask)).to(dev)
    ijk = torch.stack([cells % nx, (cells // nx) % ny, cells // (nx * ny)], dim=1).double()
    org = torch.tensor(origin, dtype=torch.float64, device=dev)
    centre = org + (ijk + 0.5) * dx
    g = torch.tensor(gravity, dtype=torch.float64, device=dev)
    depth = centre @ (g / torch.linalg.norm(g))
    order = torch.argsort(-depth, stable=True)
    order = order[:max(1, int(len(order) * fill))]
    centre, free = centre[order], inner[cells[order]].repeat_interleave(PPC)[:, None]
    pos = centre.repeat_interleave(PPC, dim=0)
    n = len(pos)
    pos += (torch.rand(n, 3, generator=gen, device=dev, dtype=torch.float64) - 0.5) * torch.where(free, 0.998 * dx, 0.4 * dx)
    kick = torch.rand(n, 1, generator=gen, device=dev, dtype=torch.float64) < 1.0 / 140.0
    pos += (kick & free) * torch.randn(n, 3, generator=gen, device=dev, dtype=torch.float64) * (0.4 * dx)
    mid = pos.mean(dim=0)
    swirl = torch.stack([pos[:, 2] - mid[2], torch.zeros(n, device=dev, dtype=torch.float64), mid[0] - pos[:, 0]], dim=1)
    vel = 5.0 * swirl + 0.01 * torch.randn(n, 3, generator=gen, device=dev, dtype=torch.float64)
    return tuple(a.float().double().cpu().numpy() for a in (pos, vel))


def _solver(case, seed):
    """A solver holding the case's liquid, the scene's cavity volume and the step length."""
    w = _workload(case)
    sdf = build_sdf(w.res, w.tris)
    vol = w.cavity_volume if w.cavity_volume is not None else cavity_volume(w.res, sdf)
    r = w.res
    on = case["flow_ml_s"] > 0.0
    needle = sc.Needle(tip=r.needle.tip, axis=r.needle.axis, radius=r.needle.radius,
                       flow_rate=case["flow_ml_s"] * sc.ML_PER_S, inject_until=math.inf if on else 0.0)
    cells = max(vol / r.sim_dx ** 3, 1.0)
    s = Solver(sdf, r.sim_dx, r.fluid, needle, max_particles=int(cells * PPC * 1.3) + 4096)
    s.solve = sc.SolveParams(400, 1e-6)
    st = s.stats()  # no outlet: the dose stays in, and a pass does not empty the cavity for the next
    pos, vel = _pool((st.nx, st.ny, st.nz), (st.origin.x, st.origin.y, st.origin.z), float(st.dx), r.fluid.gravity,
                     s.cavity_mask(), case["fill"], seed)
    s.set_particles(pos, vel)
    return s, vol, r.sim_dx / (needle.jet_speed() if on else SETTLED_SPEED)


def _mesh(subdiv, seed):
    """A cavity of the workloads' family at a given mesh density, as triangles (T, 9) in metres, in a box of the same
    size for every seed (so that every seed has the same grid)."""
    p = perturbed_ellipsoid(seed, subdiv=subdiv).tris.reshape(-1, 3)
    lo, hi = p.min(axis=0), p.max(axis=0)
    return ((p - lo) * (np.array(MESH_BOX_MM) * sc.MM / (hi - lo))).reshape(-1, 9)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "flow":
        s, _, dt = _solver(case, seed)
        return dict(kind=kind, solver=s, dt=dt, substeps=int(case["substeps"]))
    if kind == "frame":
        s, vol, dt = _solver(case, seed)
        s.substep(dt)  # labels and pressure of a running simulation
        st = s.stats()
        mid = float(st.origin.z) + 0.5 * st.nz * float(st.dx)
        return dict(kind=kind, solver=s, metrics=MetricsCollector(s, vol), px=int(case["px"]),
                    planes=[SlicePlane.xy(mid, 1.5 * float(st.dx)),
                            SlicePlane.projected_along_gravity(s.fluid.gravity)])
    if kind == "sdf":
        return dict(kind=kind, tris=_mesh(case["subdiv"], seed), dx=case["dx_mm"] * sc.MM)
    specs = []
    for k in range(int(case["scenes"])):
        w = workloads.batch_scene(100 + seed % 1_000_000 * 16 + k, frames=1)
        spec = workloads.scene_spec(w)
        spec.frame_dt = int(case["cfl_steps"]) * spec.sim_dx / spec.needle.jet_speed()
        specs.append(spec)
    return dict(kind=kind, specs=specs, packed=bool(case["packed"]))


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "flow":
        s = state["solver"]
        for _ in range(state["substeps"]):
            s.substep(state["dt"])
        pos, vel = s.particles_f32()
        st = s.stats()
        return dict(pos=pos, vel=vel, particles=int(st.particles), drained=int(st.drained),
                    redistributed=int(st.redistributed), pcg_iters=int(st.last_pcg_iters))
    if kind == "frame":
        s = state["solver"]
        frame = state["metrics"].record(s, 0)
        images = [render_slice(s, p, state["px"]) for p in state["planes"]]
        pos, vel = s.particles_f32()
        return dict(metrics=frame, images=images, pos=pos, vel=vel)
    if kind == "sdf":
        f = sdf_from_mesh(state["tris"], state["dx"], 3.0 * state["dx"])
        return dict(origin=list(f.origin), data=f.data)
    out = run_batch(state["specs"], packed=state["packed"])
    rows = [dict(status=r.status, **r.summary, substeps=r.stats["substeps_total"]) for r in out]
    return {key: np.array([row[key] for row in rows]) for key in rows[0]}


# ---------------------------------------------------------------- floors
def _cells(case):
    """Grid cells and liquid cells of a flow or frame case, from the cavity's size."""
    dx = case["dx_mm"]
    volume_mm3, box_mm3 = (2200.0, 7500.0) if case["cavity"] == "ellipsoid" else (9520.0, 57900.0)
    return box_mm3 / dx ** 3, volume_mm3 * case["fill"] / dx ** 3


def work(case):
    kind = case["kind"]
    if kind == "flow":
        grid, liquid = _cells(case)
        n = liquid * PPC
        # per substep: particles in and out (position and velocity, 24 B each way), pressure out; the solve reads its
        # right-hand side and writes its result once. Per pass: the particles read back.
        return {"bytes": case["substeps"] * (48.0 * n + 24.0 * liquid + grid) + 24.0 * n,
                "flops": case["substeps"] * (600.0 * n + 2000.0 * liquid)}
    if kind == "frame":
        grid, liquid = _cells(case)
        n = liquid * PPC
        return {"bytes": 48.0 * n + 9.0 * grid + 6.0 * case["px"] ** 2, "flops": 20.0 * n}
    if kind == "sdf":
        tris = 20 * 4 ** case["subdiv"]
        nodes = 4540.0 / case["dx_mm"] ** 3 * 1.3
        return {"bytes": 72.0 * tris + 8.0 * nodes, "flops": 200.0 * nodes}
    cells = case["scenes"] * 62.0 ** 3
    return {"bytes": case["cfl_steps"] * cells * 1.0 + 8.0 * cells, "flops": 0.0}


# ---------------------------------------------------------------- results in 64 bits
def exact(case, seed):
    """The distance field of an sdf case. The other kinds have no such value: a substep takes branches (which neighbour
    a surplus particle goes to, the iteration the pressure solve stops at) that another rounding takes differently, and
    frames and summaries are of states reached by substeps."""
    if case["kind"] != "sdf":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    dx = case["dx_mm"] * sc.MM
    tris = torch.from_numpy(_mesh(case["subdiv"], seed)).to(dev).reshape(-1, 3, 3)
    pts = tris.reshape(-1, 3)
    lo, hi = pts.min(dim=0).values - 3.0 * dx, pts.max(dim=0).values + 3.0 * dx
    dims = [int(math.ceil(float(v))) + 1 for v in (hi - lo) / dx]
    ax = [lo[c] + torch.arange(dims[c], device=dev, dtype=torch.float64) * dx for c in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    nodes = torch.stack([x, y, z], dim=-1).reshape(-1, 3)
    a, b, c = tris[:, 0], tris[:, 1], tris[:, 2]
    out = torch.empty(len(nodes), dtype=torch.float64, device=dev)
    step = max(1, 4_000_000 // len(tris))
    for k in range(0, len(nodes), step):
        p = nodes[k:k + step, None, :]
        d2 = _distance_sq(p, a, b, c).min(dim=1).values
        va, vb, vc = a - p, b - p, c - p
        la, lb, lc = (torch.linalg.norm(v, dim=-1) for v in (va, vb, vc))
        num = (va * torch.linalg.cross(vb, vc)).sum(-1)
        den = la * lb * lc + (va * vb).sum(-1) * lc + (vb * vc).sum(-1) * la + (vc * va).sum(-1) * lb
        wind = 2.0 * torch.atan2(num, den).sum(dim=1) / (4.0 * math.pi)
        out[k:k + step] = torch.where(wind > 0.5, -d2.sqrt(), d2.sqrt())
    return dict(origin=[float(v) for v in lo], data=out.reshape(dims[2], dims[1], dims[0]).cpu().numpy())


def _distance_sq(p, a, b, c):
    """Squared distance of points to triangles: the plane's foot point if it lies inside, else the nearest edge."""
    def edge(u, v):
        e = v - u
        t = (((p - u) * e).sum(-1) / (e * e).sum(-1)).clamp(0.0, 1.0)
        d = p - (u + t[..., None] * e)
        return (d * d).sum(-1)

    n = torch.linalg.cross(b - a, c - a)
    inside = torch.ones((), dtype=torch.bool, device=a.device)
    for u, v in ((a, b), (b, c), (c, a)):
        inside = inside & ((torch.linalg.cross((v - u).expand_as(p - u), p - u) * n).sum(-1) >= 0.0)
    h = ((p - a) * n).sum(-1)
    near = torch.minimum(torch.minimum(edge(a, b), edge(b, c)), edge(c, a))
    return torch.where(inside, h * h / (n * n).sum(-1), near)
