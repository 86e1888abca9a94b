"""Performance cases: the work that programs built on this framework have it do.

Five kinds of call, each through its public entry point:

  frame    a simulation loop that keeps the scene on the device: submit a frame's
           substeps, then encode the particle snapshot a renderer draws from;
  step     a program that wants the new state on the host after every call, with a
           fixed substep count or (cfl, as the tessera3d world does) up to a
           CFL-limited time;
  batch    many uneven scenes advanced together, each read back;
  rollout  one gradient step through a differentiable rollout (forward, adjoint);
  sort     the allocation-free block binning a host engine calls inside its frame.

Sizes follow the repository's configurations (55 k and 64 k particle blocks, the
4.05 M particle dam break, the 4 k - 256 k heterogeneous batch), its tests (512
particle drop, small batches) and odd sizes between them.  `exact` restates the
substep in float64 torch operations.
"""

import ctypes
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from tessera_b200 import _native, scenes
from tessera_b200._abi import (
    MAT_ELASTIC, MAT_FLUID, MAT_NEO_HOOKEAN, MAT_SNOW, Obstacle, density_particles, make_params,
)
from tessera_b200.adjoint import Rollout, rollout
from tessera_b200.batch import Batch
from tessera_b200.session import Session

# material name -> (code, parameters, density)
MATERIALS = {
    "elastic": (MAT_ELASTIC, (1e4, 0.2), 1000.0),
    "neo_hookean": (MAT_NEO_HOOKEAN, (5e3, 0.3), 1000.0),
    "fluid": (MAT_FLUID, (1e4, 7.0, 0.01, 0.25), 1000.0),
    "snow": (MAT_SNOW, (1.4e5, 0.2, 2.5e-2, 7.5e-3, 10.0), 400.0),
}
STATE_FIELDS = ("position", "velocity", "deformation", "affine")
DT = 1e-4  # under the CFL bound of every material above at the resolutions drawn


def listed():
    return [
        # the smallest interactive scene: one body over one obstacle, a few substeps a frame
        block("frame_512_sphere", "frame", "elastic", (4, 4, 4), 20, 8, sphere=True),
        # the 55 k particle corotated block of the small configuration
        block("frame_elastic_55k", "frame", "elastic", (19, 19, 19), 64, 16),
        # plastic material (snow), whose return map carries extra state; odd sizes
        block("frame_snow_39k", "frame", "snow", (17, 17, 17), 64, 16),
        # a mid-sized flow around an obstacle: fluid and elastic bodies together
        dam("frame_dam_sphere", 0.35, 32, sphere=True),
        # the headline scene, 4.05 M particles, one full submission
        dam("frame_dam_4m", 1.0, 64),
        # world.step(dt): CFL-limited substeps, state on the host after each
        block("step_cfl_nh_9k", "cfl", "neo_hookean", (11, 7, 15), 48, 9),
        # a fixed submission whose whole state the program reads (a recording, a checkpoint)
        block("step_read_fluid_230k", "step", "fluid", (31, 29, 32), 128, 64),
        # heterogeneous batches: the batch configuration's substeps, and a handful of tiny scenes
        dict(name="batch_16", kind="batch", scenes=16, cells_min=8, cells_max=20, substeps=100),
        dict(name="batch_6_small", kind="batch", scenes=6, cells_min=4, cells_max=9, substeps=20),
        # system identification and control: gradients of a centroid loss
        dict(name="rollout_64k", kind="rollout", cells=20, substeps=256, checkpoint_every=16),
        dict(name="rollout_4k", kind="rollout", cells=8, substeps=64, checkpoint_every=8),
        # binning inside a host engine's frame
        dict(name="sort_200k", kind="sort", count=200_003, spread=1.0, resolution=96),
    ]


def block(name, kind, material, cells, resolution, substeps, sphere=False):
    return dict(name=name, kind=kind, scene="block", material=material, cx=cells[0], cy=cells[1], cz=cells[2],
                resolution=resolution, substeps=substeps, sphere=sphere)


def dam(name, scale, substeps, sphere=False):
    return dict(name=name, kind="frame", scene="dam", scale=scale, substeps=substeps, sphere=sphere)


def draw(rng):
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(["frame", "frame", "frame", "dam", "cfl", "step", "batch", "rollout", "sort"])
    if kind == "dam":
        case = dam("", round(log(0.1, 0.8), 3), rng.randint(8, 64), rng.random() < 0.4)
    elif kind == "batch":
        lo = rng.randint(4, 10)
        case = dict(kind="batch", scenes=int(log(2, 16.99)), cells_min=lo, cells_max=lo + rng.randint(0, 10),
                    substeps=rng.randint(5, 100))
    elif kind == "rollout":
        case = dict(kind="rollout", cells=rng.randint(5, 20), substeps=rng.randint(17, 160),
                    checkpoint_every=rng.randint(5, 16))
    elif kind == "sort":
        case = dict(kind="sort", count=int(log(1_000, 262_144)), spread=round(log(0.05, 1.0), 3),
                    resolution=rng.randint(32, 400))
    else:
        edge = int(log(4, 36.99))
        cells = [max(3, edge + rng.randint(-edge // 4, edge // 4)) for _ in range(3)]
        material = "neo_hookean" if kind == "cfl" else rng.choice(["elastic", "neo_hookean", "fluid", "snow"])
        case = block("", kind, material, cells, min(100 if kind == "cfl" else 128, 3 * max(cells) + rng.randint(4, 12)),
                     rng.randint(2, 9) if kind == "cfl" else rng.randint(4, 64), kind == "frame" and rng.random() < 0.3)
    case.pop("name", None)
    return case


# ------------------------------------------------------------------ scenes


def _block_scene(case, seed):
    """A jittered block of cx x cy x cz cells (8 particles each) two cells above the
    floor of the unit cube, moving down; `sphere` puts an obstacle under its corner."""
    rng = np.random.default_rng(seed)
    code, prm, density = MATERIALS[case["material"]]
    h = 1.0 / case["resolution"]
    r = h / 4.0
    cells = np.array([case["cx"], case["cy"], case["cz"]])
    lo = np.array([(case["resolution"] - cells[0]) // 2, (case["resolution"] - cells[1]) // 2, 2]) * h
    obstacles = []
    if case["sphere"]:
        lo[2] += 3 * h
        obstacles = [Obstacle.sphere((lo[0] + 1.3 * h, lo[1] + 1.1 * h, 2.2 * h), 2.05 * h, friction=0.3)]
    pos = scenes.lattice(lo, lo + cells * h, 2.0 * r, rng, 0.5)
    vel = np.array([rng.uniform(-0.2, 0.2), rng.uniform(-0.2, 0.2), -rng.uniform(0.3, 0.6)])
    parts = density_particles(pos, r, density, code, prm, velocity=vel)
    params = make_params(h, max_substep=1e-3, bounds=((0, 0, 0), (1, 1, 1)))
    return params, parts, DT, obstacles


def _scene(case, seed):
    if case["scene"] == "block":
        return _block_scene(case, seed)
    sc = scenes.dam_break(seed=seed, scale=case["scale"])
    if case["sphere"]:  # half a cell in front of the column's face, near the floor
        h, r = sc.params.cell_width, 0.09
        sc.obstacles = [Obstacle.sphere((0.4 * case["scale"] + r + 0.5 * h, 0.4 * case["scale"], r + h), r, friction=0.3)]
    return sc.params, sc.particles, sc.dt, sc.obstacles


def _batch_scenes(case, seed):
    # the sizes belong to the case; positions, jitter and materials to the seed
    cells = np.random.default_rng(case["scenes"]).integers(case["cells_min"], case["cells_max"] + 1, case["scenes"])
    rng = np.random.default_rng(seed)
    return [scenes.batch_scene(int(rng.integers(1 << 30)), cells=int(c)) for c in cells]


def _rollout_inputs(case, seed):
    sc = scenes.adjoint_block(seed=seed, cells=case["cells"], dt=DT, substeps=case["substeps"])
    rng = np.random.default_rng(seed + 1)
    young = 5e3 * np.exp(rng.uniform(-0.2, 0.2, sc.particles.count))
    return sc, young, np.asarray(sc.info["target"])


def _sort_positions(case, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.0, case["spread"], (3, case["count"])).astype(np.float32)


# ------------------------------------------------------------------ calls


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "step", "cfl"):
        params, parts, dt, obstacles = _scene(case, seed)
        # a long run of the headline scene pins the launch configuration measured best for it
        shape = 3 if case["scene"] == "dam" and case["scale"] == 1.0 else None
        session = Session(params, parts, dt, obstacles=obstacles, launch_shape=shape)
        state = dict(case=case, session=session)
        if kind == "frame":
            state["snapshot"] = torch.empty((parts.count, 2, 4), device="cuda")
        return state
    if kind == "batch":
        batch = Batch()
        ids = [batch.add_scene(s.params, s.particles, s.dt) for s in _batch_scenes(case, seed)]
        return dict(case=case, batch=batch, ids=ids)
    if kind == "rollout":
        sc, young, target = _rollout_inputs(case, seed)
        sim = Rollout(sc.params, sc.particles, sc.dt, case["substeps"], case["checkpoint_every"])
        return dict(case=case, sim=sim, v0=torch.from_numpy(sc.particles.velocity.copy()).cuda().requires_grad_(),
                    young=torch.from_numpy(young).cuda().requires_grad_(), target=torch.from_numpy(target).cuda())
    pos = torch.from_numpy(_sort_positions(case, seed)).cuda()
    order = torch.empty(case["count"], dtype=torch.int32, device="cuda")
    return dict(case=case, pos=pos, order=order, keys=torch.empty_like(order), lib=_native.lib())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        session, out = state["session"], state["snapshot"]
        session.submit_steps(case["substeps"])
        session.encode_particle_snapshot(out.data_ptr(), out.numel() * 4)
        return {"position_mass": out[:, 0], "velocity_volume": out[:, 1]}
    if kind == "step":
        state["session"].step(case["substeps"])
        return state["session"].read(STATE_FIELDS)
    if kind == "cfl":
        state["session"].step_cfl((case["substeps"] - 0.5) * 1e-3)
        return state["session"].read(STATE_FIELDS)
    if kind == "batch":
        batch, ids = state["batch"], state["ids"]
        batch.run({i: case["substeps"] for i in ids})
        return {str(k): batch.read(i) for k, i in enumerate(ids)}
    if kind == "rollout":
        v0, young = state["v0"], state["young"]
        v0.grad = young.grad = None
        x = rollout(state["sim"], v0, young)
        ((x.mean(0) - state["target"]) ** 2).sum().backward()
        return {"x": x.detach(), "v0_grad": v0.grad, "young_grad": young.grad}
    n = case["count"]
    st = state["lib"].tmpm_sort_by_block_noalloc(
        ctypes.c_void_p(state["pos"].data_ptr()), n, n, 1.0 / case["resolution"],
        ctypes.c_void_p(state["order"].data_ptr()), ctypes.c_void_p(state["keys"].data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if st != 0:
        raise RuntimeError(state["lib"].tmpm_last_error().decode())
    return {"order": state["order"], "keys": state["keys"]}


# ------------------------------------------------------------------ figures


def _particles(case):
    if case["kind"] == "batch":
        mid = (case["cells_min"] + case["cells_max"]) / 2.0
        return case["scenes"] * 8 * mid ** 3
    if case["kind"] == "rollout":
        return 8 * case["cells"] ** 3
    if case["kind"] == "sort":
        return case["count"]
    if case["scene"] == "block":
        return 8 * case["cx"] * case["cy"] * case["cz"]
    return 4.01e6 * case["scale"] ** 2 + 38_000


def work(case):
    n = _particles(case)
    if case["kind"] == "sort":
        return {"bytes": n * (12 + 4 + 4), "flops": 6 * n}
    s = case["substeps"]
    # 27-node gather and scatter of 12 and 8 multiply-adds, update and stress
    flops = 1400
    if case["kind"] == "rollout":  # forward, then the adjoint's replay and reverse sweep
        return {"bytes": n * (4 * 26 + 8 * 7), "flops": n * s * 4.5 * flops}
    # position, velocity, affine, F (24 floats) read and written and the class word:
    # once a call where the state fits on the chip, else once a substep
    state = 2 * 96 + 4
    passes = 1 if n * state < 120e6 else s
    out = {"frame": 32, "batch": 48}.get(case["kind"], 192)
    return {"bytes": n * (passes * state + out), "flops": n * s * flops}


def tolerance(case):
    if case["kind"] == "sort":
        return "exact"
    if case["kind"] == "rollout":
        # gradients of a centroid loss: 32-bit sums carried back through every substep
        return {"rel": 4e-3}
    if case.get("material") == "snow":
        # yielding switches on 32-bit stretches: velocities measured 2e-4 from float64
        return {"rel": 1e-3, "max": 0.02}
    # velocities and affine matrices of stiff materials: the stress is a small
    # difference of 32-bit deformations, so last-bit changes grow over the substeps
    return {"rel": 2e-4, "max": 0.02}


# ------------------------------------------------------------------ float64 restatement


def _lame(young, nu):
    return young * nu / ((1 + nu) * (1 - 2 * nu)), young / (2 * (1 + nu))


def _polar(F):
    R = F
    for _ in range(9):
        R = 0.5 * (R + torch.linalg.inv(R).transpose(-1, -2))
    return R


def _det(F):
    return (F[:, :, 0] * torch.linalg.cross(F[:, :, 1], F[:, :, 2])).sum(-1)


def _stress(mat, F, C, jp):
    """Kirchhoff stress; `mat` holds the kind's name and parameter tensors."""
    eye = torch.eye(3, dtype=F.dtype, device=F.device)
    J = _det(F)
    FT = F.transpose(1, 2)
    if mat["kind"] == MAT_NEO_HOOKEAN:
        return mat["mu"] * (F @ FT - eye) + (mat["lam"] * torch.log(J.clamp_min(1e-10)))[:, None, None] * eye
    if mat["kind"] == MAT_FLUID:
        bulk, gamma, visc, tensile = mat["fluid"]
        sj = J.clamp_min(1e-6)
        p = torch.where(sj <= 1, bulk * (sj ** -gamma - 1), -bulk * tensile * (sj - 1))
        rate = 0.5 * (C + C.transpose(1, 2))
        dev = rate - rate.diagonal(dim1=1, dim2=2).sum(1)[:, None, None] / 3 * eye
        return (2 * visc * sj)[:, None, None] * dev - (p * sj)[:, None, None] * eye
    lam, mu = mat["lam"], mat["mu"]
    if mat["kind"] == MAT_SNOW:
        f = torch.exp(mat["harden"] * (1 - jp)).clamp(0.01, 100.0)
        lam, mu = lam * f, mu * f
    two_mu = (2 * mu)[:, None, None] if torch.is_tensor(mu) else 2 * mu
    return two_mu * ((F - _polar(F)) @ FT) + (lam * (J - 1) * J)[:, None, None] * eye


def _contact(vel, n, friction):
    ns = (vel * n).sum(1, keepdim=True)
    t = vel - n * ns
    ts = t.norm(dim=1, keepdim=True)
    scale = torch.where(ts > 1e-12, (1 + friction * ns / ts.clamp_min(1e-12)).clamp_min(0), torch.zeros_like(ts))
    return torch.where(ns >= 0, vel, t * scale)


def _substep(x, v, C, F, jp, mats, sc):
    """One MLS-MPM substep of all particles; `mats`: (row slice, material) pairs."""
    h, dt, dev = sc["h"], sc["dt"], x.device
    base = torch.floor(x.detach() / h - 0.5)
    f = x / h - base
    axis = torch.arange(3, dtype=x.dtype, device=dev)
    offset = torch.stack(torch.meshgrid(axis, axis, axis, indexing="ij"), -1)
    w = [0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2]
    lo = base.amin(0)
    dim = (base.amax(0) - lo + 3).long().tolist()
    cell = (base - lo).long()
    row = (cell[:, 0] * dim[1] + cell[:, 1]) * dim[2] + cell[:, 2]
    tau = torch.cat([_stress(m, F[s], C[s], jp[s]) for s, m in mats])
    A = -dt * 4 / h ** 2 * sc["vol"][:, None, None] * tau + sc["mass"][:, None, None] * C
    mv = sc["mass"][:, None] * v
    grid = torch.zeros((dim[0] * dim[1] * dim[2], 4), dtype=x.dtype, device=dev)

    def stencil():
        for a in range(3):
            for b in range(3):
                for c in range(3):
                    yield ((a * dim[1] + b) * dim[2] + c, (w[a][:, 0] * w[b][:, 1] * w[c][:, 2])[:, None],
                           (offset[a, b, c] - f) * h)

    for o, wt, d in stencil():
        mom = wt * (mv + (A @ d[:, :, None])[:, :, 0])
        grid = grid.index_add(0, row + o, torch.cat([wt * sc["mass"][:, None], mom], 1))
    used = grid[:, :1] > 0
    vel = torch.where(used, grid[:, 1:] / torch.where(used, grid[:, :1], torch.ones_like(grid[:, :1])), 0.0)
    vel = vel + used * (dt * sc["g"])
    idx = torch.arange(dim[0] * dim[1] * dim[2], device=dev)
    node = torch.stack([idx // (dim[1] * dim[2]), idx // dim[2] % dim[1], idx % dim[2]], 1) + lo
    p = node * h
    vel = torch.where((p <= sc["bmin"] + h) & (vel < 0) | (p >= sc["bmax"] - h) & (vel > 0), 0.0, vel)
    for center, radius, friction in sc["spheres"]:
        rel = p - center
        n = rel / rel.norm(dim=1, keepdim=True).clamp_min(1e-12)
        near = (rel.norm(dim=1, keepdim=True) - radius <= h) & used
        vel = torch.where(near, _contact(vel, n, friction), vel)
    nv, nC = torch.zeros_like(x), torch.zeros_like(C)
    for o, wt, d in stencil():
        g = wt * vel[row + o]
        nv = nv + g
        nC = nC + 4 / h ** 2 * g[:, :, None] * d[:, None, :]
    nx = x + dt * nv
    r = sc["radius"][:, None]
    low, high = nx < sc["bmin"] + r, nx > sc["bmax"] - r
    nv = torch.where(low, nv.clamp_min(0), torch.where(high, nv.clamp_max(0), nv))
    nx = torch.where(low, sc["bmin"] + r, torch.where(high, sc["bmax"] - r, nx))
    for center, radius, friction in sc["spheres"]:
        rel = nx - center
        dist = rel.norm(dim=1, keepdim=True)
        n = rel / dist.clamp_min(1e-12)
        hit = dist - radius < r
        nv = torch.where(hit, _contact(nv, n, friction), nv)
        nx = torch.where(hit, nx + n * (r - (dist - radius)), nx)
    nF = F + dt * nC @ F
    parts, jps = [], []
    for s, m in mats:
        Fs, js = nF[s], jp[s]
        if m["kind"] == MAT_FLUID:
            eye = torch.eye(3, dtype=F.dtype, device=dev)
            Fs = _det(Fs).clamp_min(1e-9).pow(1 / 3)[:, None, None] * eye
        elif m["kind"] == MAT_SNOW:
            U, sg, Vh = torch.linalg.svd(Fs)
            cl = sg.clamp(1 - m["compress"], 1 + m["stretch"])
            js = (js * sg.prod(1) / cl.prod(1).clamp_min(1e-12)).clamp(0.1, 4.0)
            Fs = U @ (cl[:, :, None] * Vh)
        parts.append(Fs)
        jps.append(js)
    return nx, nv, nC, torch.cat(parts), torch.cat(jps)


def _exact_scene(params, parts, obstacles, young=None):
    """(state tensors, materials, scene constants) on the GPU in float64."""
    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()

    n = parts.count
    mats, start = [], 0
    kinds, prm = parts.material, parts.material_params
    cuts = [0] + [i + 1 for i in np.nonzero((kinds[1:] != kinds[:-1]) | (prm[1:] != prm[:-1]).any(1))[0]] + [n]
    for start, end in zip(cuts[:-1], cuts[1:]):
        q = prm[start]
        m = dict(kind=int(kinds[start]))
        if m["kind"] == MAT_FLUID:
            m["fluid"] = tuple(float(a) for a in q[:4])
        else:
            m["lam"], m["mu"] = _lame(float(q[0]) if young is None else young, float(q[1]))
        if m["kind"] == MAT_SNOW:
            m.update(compress=float(q[2]), stretch=float(q[3]), harden=float(q[4]))
        mats.append((slice(int(start), int(end)), m))
    sc = dict(h=float(params.cell_width), g=t(list(params.gravity)), bmin=t(list(params.bounds_min)),
              bmax=t(list(params.bounds_max)), mass=t(parts.mass), vol=t(parts.rest_volume), radius=t(parts.radius),
              spheres=[(t(o.center), float(o.dims[0]), float(o.friction)) for o in obstacles])
    F = t(parts.deformation).reshape(n, 3, 3).transpose(1, 2)
    C = t(parts.affine).reshape(n, 3, 3).transpose(1, 2)
    return [t(parts.position), t(parts.velocity), C, F, t(parts.plastic[:, 0])], mats, sc


def _advance(params, parts, dts, obstacles):
    state, mats, sc = _exact_scene(params, parts, obstacles)
    for dt in dts:
        state = _substep(*state, mats, dict(sc, dt=dt))
    return state, sc


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        return None  # whole numbers
    if kind in ("frame", "step", "cfl"):
        if _particles(case) * case["substeps"] > 8e7:
            return None  # minutes in float64
        params, parts, dt, obstacles = _scene(case, seed)
        dts = [dt] * case["substeps"]
        if kind == "cfl":  # whole steps of max_substep, below the CFL bound of these scenes, and half a one
            dts = [1e-3] * (case["substeps"] - 1) + [0.5e-3]
        with torch.no_grad():
            (x, v, C, F, _), sc = _advance(params, parts, dts, obstacles)
        if kind == "frame":
            return {"position_mass": torch.cat([x, sc["mass"][:, None]], 1),
                    "velocity_volume": torch.cat([v, sc["vol"][:, None]], 1)}
        return {"position": x, "velocity": v, "deformation": F.transpose(1, 2).reshape(-1, 9),
                "affine": C.transpose(1, 2).reshape(-1, 9)}
    if kind == "batch":
        out = {}
        with torch.no_grad():
            for k, s in enumerate(_batch_scenes(case, seed)):
                (x, v, _, _, _), _ = _advance(s.params, s.particles, [s.dt] * case["substeps"], [])
                out[str(k)] = {"position": x, "velocity": v}
        return out
    sc, young, target = _rollout_inputs(case, seed)
    E = torch.from_numpy(young).cuda().requires_grad_()
    v0 = torch.from_numpy(sc.particles.velocity.copy()).cuda().requires_grad_()
    state, mats, const = _exact_scene(sc.params, sc.particles, [], young=E)
    const["dt"] = sc.dt
    state[1] = v0
    for _ in range(case["substeps"]):
        state = checkpoint(lambda *s: _substep(*s, mats, const), *state, use_reentrant=False)
    ((state[0].mean(0) - torch.from_numpy(target).cuda()) ** 2).sum().backward()
    return {"x": state[0].detach(), "v0_grad": v0.grad, "young_grad": E.grad}
