"""The work that programs built on this framework have it do, as timed cases.

Every case is one call sequence of the public binding (femstep.py) with what such a
program has in hand before it: a resident solver or pool for the stepping cases, the
requests themselves for the served one.

  tet    one tet mesh in a TetSolver: `steps` steps, then positions and velocities back
         (the reference's FemGpuSolver run / readback loop), and the plastic state where
         the program looks at it; the drop-in float step, the FP64 step and the two FP32 ones
  pool   many meshes of uneven size resident in a TetPool in the batched schedule:
         `steps` steps of all of them, then the whole batch read back
  serve  a group of solves with step counts of their own through a resident TetPool:
         admitted, stepped in chunks, read back and released as they finish
  shell  one solid-shell zone in a ShellSolver: `steps` steps, then positions and
         velocities back, and the points' plastic state where the program looks at it

The FP32 steps hold velocity, plastic strain and energy densities in single precision;
where the binding widens them on the way out, the program keeps them as float32.

`exact` restates each step in torch float64.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("sinking-simulator_b200"))
import femstep as F  # noqa: E402
import meshes as M  # noqa: E402
import workloads as W  # noqa: E402

E_TET, E_SHELL, NU, RHO, YIELD, HARD = 210e9, 206e9, 0.3, 7850.0, 235e6, 1e9
GRAVITY = 9.80665
SWIFT = dict(hardening=F.SHELL_SWIFT, strength_coefficient=600e6, reference_strain=0.02, hardening_exponent=0.18)


def listed():
    return [
        # the reference's tet driver at its smallest mesh (960 tets): a frame's worth of
        # steps, bound by latency and launches
        dict(name="spike-960", kind="tet", mode="ref32", nx=40, ny=2, nz=2, steps=200, load=0.0, plastic=False),
        # the same driver at its largest mesh (491,520 tets)
        dict(name="spike-491520", kind="tet", mode="ref32", nx=320, ny=16, nz=16, steps=200, load=0.0, plastic=False),
        # the plain single-mesh FP64 step on the 3,840-tet cantilever
        dict(name="cantilever-f64", kind="tet", mode="f64", nx=40, ny=4, nz=4, steps=400, load=1.5, plastic=True),
        # a small ragged part in the compensated FP32 step (4,830 tets, no size a power of two)
        dict(name="part-f32k", kind="tet", mode="f32k", nx=23, ny=7, nz=5, steps=400, load=1.5, plastic=True),
        # the precision study's 480,000-tet beam, compensated FP32 and FP64
        dict(name="beam-f32k", kind="tet", mode="f32k", nx=200, ny=20, nz=20, steps=300, load=1.0, plastic=False),
        dict(name="beam-f64", kind="tet", mode="f64", nx=200, ny=20, nz=20, steps=60, load=1.0, plastic=False),
        # the headline batch: 256 uneven meshes of 2e3 to 2e5 tets
        dict(name="batch-256", kind="pool", count=256, lo=2e3, hi=2e5, mix=20261203, steps=600),
        # a small batch of small parts, where launches and tails count
        dict(name="batch-24-small", kind="pool", count=24, lo=1e3, hi=2e4, mix=7, steps=400),
        # a served group: 1e3 to 5e5 tets, each solve with its own step count
        dict(name="serve-12", kind="serve", count=12, lo=1e3, hi=5e5, mix=20261204, steps=600, chunk=64),
        # a zone of the size the ship code cuts out of its plating, Swift hardening
        dict(name="zone-swift", kind="shell", nx=64, ny=32, thickness=0.012, law="swift", peak=6e6, steps=400,
             plastic=True),
        # one bay of the stiffened panel (28,600 elements)
        dict(name="bay", kind="shell", nx=200, ny=143, thickness=0.012, law="linear", peak=1.5e6, steps=200,
             plastic=False),
        # the whole stiffened panel (2,000,000 elements, 4 million nodes)
        dict(name="panel", kind="shell", nx=2000, ny=1000, thickness=0.012, law="linear", peak=1.5e6, steps=80,
             plastic=False),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["tet", "tet", "pool", "serve", "shell", "shell"])
    if kind == "tet":
        mode = rng.choice(["ref32", "f64", "f32k", "f32k", "f32"])
        cells = log(150, 80000)
        slender = rng.uniform(1.0, 12.0)
        k = max(1, round((cells / slender) ** (1 / 3)))
        j = max(1, k + rng.choice([-1, 0, 0, 1]))
        nx = max(2, round(cells / (j * k)))
        steps = round(log(100, 400) if nx * j * k < 20000 else log(30, 100))
        return dict(kind="tet", mode=mode, nx=nx, ny=j, nz=k, steps=steps, load=0.0 if mode == "ref32" else
                    round(rng.uniform(0.5, 2.0), 2), plastic=nx * j * k < 5000 and mode != "ref32")
    if kind == "pool":
        lo, hi = rng.choice([(1e3, 2e4), (2e3, 1e5), (2e3, 2e5)])
        return dict(kind="pool", count=round(log(6, 120)), lo=lo, hi=hi, mix=rng.randrange(1, 1 << 30),
                    steps=round(log(100, 400)))
    if kind == "serve":
        return dict(kind="serve", count=round(log(2, 24)), lo=1e3, hi=rng.choice([2e4, 2e5, 5e5]),
                    mix=rng.randrange(1, 1 << 30), steps=round(log(100, 600)), chunk=rng.choice([32, 64]))
    elements = log(200, 300000)
    ny = max(3, round(math.sqrt(elements / rng.uniform(1.0, 3.0))))
    nx = max(3, round(elements / ny))
    law = rng.choice(["linear", "linear", "swift"])
    return dict(kind="shell", nx=nx, ny=ny, thickness=round(rng.uniform(0.006, 0.014), 4), law=law,
                peak=round(rng.uniform(1e6, 5e6)), steps=round(log(60, 300) if elements < 50000 else 40),
                plastic=elements < 5000)


# ---- inputs ------------------------------------------------------------------------


@functools.lru_cache(maxsize=4)
def _box(nx, ny, nz):
    h = 0.025
    pos, idx = M.box_tet_mesh(h * nx, h * ny, h * nz, nx, ny, nz)
    return pos, idx, F.csr(pos.size // 3, idx, 4)


@functools.lru_cache(maxsize=2)
def _mix(count, lo, hi, mix):
    return [W.build(s) for s in W.batch_meshes(count, lo, hi, seed=mix)]


@functools.lru_cache(maxsize=2)
def _plate(nx, ny, thickness):
    """The panel's 10 mm cells, clamped edges, pinned stiffener lines every 143 cells."""
    rest, index = M.plate_mesh(0.01 * nx, 0.01 * ny, thickness, nx, ny)
    i = np.arange(rest.size // 3) // (2 * (ny + 1))
    j = (np.arange(rest.size // 3) // 2) % (ny + 1)
    held = (i == 0) | (i == nx) | (j == 0) | (j == ny) | ((j % 143 == 0) & (ny > 200))
    # the consistent load of a unit pressure on the flat plate: a cell's area / 4 a corner
    cells = ((i > 0).astype(float) + (i < nx)) * ((j > 0).astype(float) + (j < ny))
    top = (np.arange(rest.size // 3) % 2) == 1
    return rest, index, np.repeat(held, 3).astype(np.uint8), -0.25e-4 * cells * top


def _jitter(pos, cell, rng):
    """As-built imperfection: 2 % of a cell on every node."""
    return (pos + rng.uniform(-0.02, 0.02, pos.size).reshape(pos.shape) * cell).astype(np.float32)


def _tet_dt(cell, youngs=E_TET):
    """0.8 of the element bound 2 / omega of the six Kuhn tets of one (hx, hy, hz) cell."""
    p, idx = M.box_tet_mesh(*cell, 1, 1, 1)
    worst = 0.0
    lam, mu = youngs * NU / ((1 + NU) * (1 - 2 * NU)), youngs / (2 * (1 + NU))
    C = np.diag([2 * mu] * 3 + [mu] * 3)
    C[:3, :3] += lam
    for t in idx.reshape(-1, 4):
        x = p.reshape(-1, 3)[t].astype(np.float64)
        g = np.linalg.inv((x[1:] - x[0]).T)
        g = np.vstack([-g.sum(0), g])
        B = np.zeros((6, 12))
        for c in range(4):
            a, b, d = g[c]
            B[:, 3 * c:3 * c + 3] = [[a, 0, 0], [0, b, 0], [0, 0, d], [b, a, 0], [0, d, b], [d, 0, a]]
        worst = max(worst, 4 / RHO * np.linalg.eigvalsh(B.T @ C @ B)[-1])
    return 0.8 * 2 / math.sqrt(worst)


def _tet_inputs(case, seed):
    rng = np.random.default_rng([seed, 1])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = 0.025
    flat, idx, (offset, entry) = _box(nx, ny, nz)
    pos = _jitter(flat, h, rng)
    x0, x = flat.reshape(-1, 3)[:, 0], pos.reshape(-1, 3)
    fixed = (x0 < 0.5 * h).astype(np.uint32)
    tip = x0 > h * (nx - 0.5)
    ext = np.zeros(x.shape)
    if case["load"]:
        ly, lz, length = h * ny, h * nz, h * nx
        total = case["load"] * rng.uniform(0.8, 1.2) * W.LOCKING * YIELD * ly * lz * lz / 6.0 / length
        ext[tip, 2] = -total / tip.sum()
    params = dict(youngs=E_TET * rng.uniform(0.97, 1.0), poisson=NU, dt=_tet_dt((h, h, h)), gravity=GRAVITY, damping=1.0)
    if case["mode"] != "ref32":
        params.update(yield_strength=YIELD * rng.uniform(1.0, 1.5), hardening=HARD * rng.uniform(0.5, 2.0),
                      ramp_steps=max(1, case["steps"] // 2))
    vel = np.zeros(x.shape, np.float32)
    if case["mode"] == "ref32":  # struck: the drop-in step takes no nodal load
        vel[:, 2] = -rng.uniform(5.0, 20.0) * (x0 / (h * nx)) ** 2
    return dict(pos=pos, idx=idx, offset=offset, entry=entry, fixed=fixed, ext=ext.reshape(-1), vel=vel.reshape(-1),
                params=params)


def _tet_rest(pos, idx):
    """TetMesh::restInv (column-major per tet), restVolume and the lumped mass, as the
    reference's mesh generator hands them over (float)."""
    x = pos.reshape(-1, 3).astype(np.float64)[idx.reshape(-1, 4)]
    d = np.transpose(x[:, 1:] - x[:, :1], (0, 2, 1))
    inv = np.linalg.inv(d)
    vol = np.abs(np.linalg.det(d)) / 6.0
    mass = np.bincount(idx, weights=np.repeat(RHO * vol / 4, 4), minlength=pos.size // 3)
    return np.transpose(inv, (0, 2, 1)).reshape(-1).astype(np.float32), vol.astype(np.float32), mass.astype(np.float32)


def _batch_inputs(case, seed):
    """The mix's meshes with this seed's imperfections, plates, loads and step counts."""
    rng = np.random.default_rng([seed, 2])
    out, steps = [], []
    for b in _mix(case["count"], case["lo"], case["hi"], case["mix"]):
        s = b.spec
        cell = [s.size[a] / s.cells[a] for a in range(3)]
        y, f = rng.uniform(235e6, 355e6), rng.uniform(0.7, 1.4)
        out.append(dict(position=_jitter(b.position.reshape(-1, 3), cell, rng).reshape(-1), index=b.index, fixed=b.fixed,
                        external_force=b.external_force * (f * y / s.yield_strength), density=RHO, youngs=E_TET,
                        poisson=NU, yield_strength=y, hardening=rng.uniform(0.5e9, 2e9), gravity=GRAVITY,
                        dt=0.0 if case["kind"] == "serve" else _tet_dt(cell), ramp_steps=max(1, case["steps"] // 2)))
        steps.append(int(rng.integers(max(1, case["steps"] // 4), case["steps"] + 1)))
    return out, steps


def _shell_inputs(case, seed):
    rng = np.random.default_rng([seed, 3])
    nx, ny, t = case["nx"], case["ny"], case["thickness"]
    flat, index, pinned, unit = _plate(nx, ny, t)
    rest = flat.reshape(-1, 3).copy()
    rest[:, 2] += np.repeat(rng.normal(0.0, 5e-4, rest.shape[0] // 2), 2)  # both faces alike
    lx, ly = 0.01 * nx, 0.01 * ny
    cx, cy, radius = lx * rng.uniform(0.4, 0.6), ly * rng.uniform(0.4, 0.6), 0.3 * min(lx, ly)
    r2 = (rest[:, 0] - cx) ** 2 + (rest[:, 1] - cy) ** 2
    load = np.zeros_like(rest)
    load[:, 2] = unit * case["peak"] * rng.uniform(0.8, 1.2) * np.exp(-r2 / (2 * radius ** 2))
    c = math.sqrt(E_SHELL * (1 - NU) / ((1 + NU) * (1 - 2 * NU) * RHO))
    dt = 0.95 / (c * math.sqrt(2 / 0.01 ** 2 + 1 / t ** 2))
    params = dict(youngs=E_SHELL, poisson=NU, yield_strength=355e6, hardening=HARD, dt=dt,
                  rise_time=0.5 * case["steps"] * dt, damping=1.0, max_iterations=12, compensated=True)
    if case["law"] == "swift":
        params.update(material=SWIFT, damping=0.9999)
    return dict(rest=rest.reshape(-1), index=index, pinned=pinned, load=load.reshape(-1), params=params)


# ---- prepare / run -----------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "tet":
        a = _tet_inputs(case, seed)
        if case["mode"] == "ref32":
            inv, vol, mass = _tet_rest(a["pos"], a["idx"])
            s = F.TetSolver(a["pos"], a["idx"], mode="ref32", velocity=a["vel"], mass=mass, fixed=a["fixed"],
                            rest_inv=inv, rest_volume=vol, adjacency_offset=a["offset"], adjacency_entry=a["entry"])
        else:
            s = F.TetSolver(a["pos"], a["idx"], mode=case["mode"], fixed=a["fixed"], external_force=a["ext"],
                            density=RHO)
        return dict(case=case, solver=s, params=a["params"])
    if kind == "shell":
        a = _shell_inputs(case, seed)
        s = F.ShellSolver(a["rest"], a["index"], pinned=a["pinned"], load=a["load"], density=RHO)
        return dict(case=case, solver=s, params=a["params"])
    meshes, steps = _batch_inputs(case, seed)
    tets = sum(m["index"].size // 4 for m in meshes)
    nodes = sum(m["position"].size // 3 + 1 for m in meshes)
    pool = F.TetPool(tets, nodes, max_meshes=case["count"], tile=128)
    if kind == "serve":  # the serving loop's schedule: its mix changes at every chunk
        pool.set_schedule(128, F.POOL_GRAPH_STAGED)
        return dict(case=case, pool=pool, meshes=meshes, steps=steps)
    pool.set_schedule(128, F.POOL_GRAPH_TILED)  # what the autotuner picks on the batch
    ids = pool.admit_many(meshes, [1 << 40] * len(meshes))
    pool.prepare()
    return dict(case=case, pool=pool, ids=ids)


def _joined(results):
    return dict(position=np.concatenate([p for p, _ in results]),
                velocity=np.concatenate([v for _, v in results], dtype=np.float32, casting="same_kind"))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "tet":
        s = state["solver"]
        s.run(case["steps"], **state["params"])
        wide = case["mode"] == "f64"
        p, v = s.readback64() if wide else s.readback()
        out = dict(position=p, velocity=v)
        if case["plastic"]:
            out["plastic"] = s.plastic() if wide else s.plastic().astype(np.float32)
            out["energy"] = s.energy() if wide else s.energy().astype(np.float32)
        return out
    if kind == "shell":
        s = state["solver"]
        s.run(case["steps"], **state["params"])
        p, v = s.readback()
        out = dict(position=p, velocity=v.astype(np.float32))
        if case["plastic"]:  # the points' plastic strain and eq. plastic strain
            points = s.state()[:, :120].reshape(-1, 8, 15)
            out["plastic"] = points[:, :, [0, 1, 2, 3, 4, 5, 12]].astype(np.float32)
            out["energy"] = s.energy().astype(np.float32)
        return out
    pool = state["pool"]
    if kind == "pool":
        pool.run(case["steps"])
        return _joined(pool.readback_many(state["ids"]))
    ids = pool.admit_many(state["meshes"], state["steps"])
    place = {i: k for k, i in enumerate(ids)}
    results = [None] * len(ids)
    while place:
        pool.run(case["chunk"])
        done = pool.finished()
        for i, r in zip(done, pool.readback_many(done)):
            results[place.pop(i)] = r
            pool.release(i)
    return _joined(results)


# ---- what a pass cannot do without ---------------------------------------------------


def work(case):
    """Per step: every element's rest data, state and connectivity read once (and, where
    it yields, its state written), every node's state read and written once."""
    if case["kind"] == "shell":
        e, n = case["nx"] * case["ny"], 2 * (case["nx"] + 1) * (case["ny"] + 1)
        # J0^-1 and mode scales, 8 points x 7 of plastic state, alpha, node ids; per node
        # rest in double, load, displacement and compensation and velocity both ways
        return dict(bytes=case["steps"] * (e * (64 + 224 + 64 + 32) + n * (24 + 12 + 8 + 1 + 2 * 36)),
                    flops=case["steps"] * e * 16700)
    if case["kind"] == "tet":
        t = 6 * case["nx"] * case["ny"] * case["nz"]
        n = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        real = 8 if case["mode"] == "f64" else 4
        elem = 16 + real * (10 + (0 if case["mode"] == "ref32" else 7))
        node = real * (12 + 2 + (6 if case["mode"] == "f32k" else 0) + (0 if case["mode"] == "ref32" else 3)) + 1
        return dict(bytes=case["steps"] * (t * elem + n * node), flops=case["steps"] * t * 500)
    b = _mix(case["count"], case["lo"], case["hi"], case["mix"])
    t, n = sum(x.spec.tets for x in b), sum(x.spec.nodes for x in b)
    steps = case["steps"] if case["kind"] == "pool" else 0.625 * case["steps"]
    return dict(bytes=steps * (t * 84 + n * 93), flops=steps * t * 500)


# ---- the same in 64 bits ---------------------------------------------------------------


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, kind=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(_dev(), kind)


def _cof(a):
    """Cofactor matrices of (..., 3, 3)."""
    c0, c1, c2 = a[..., 0], a[..., 1], a[..., 2]
    cross = torch.linalg.cross
    return torch.stack([cross(c1, c2), cross(c2, c0), cross(c0, c1)], -1)


def _polar(f, rounds=5):
    for _ in range(rounds):
        c = _cof(f)
        f = 0.5 * (f + c / (f[..., 0] * c[..., 0]).sum(-1)[..., None, None])
    return f


def _voigt(s):
    return torch.stack([s[..., 0, 0], s[..., 1, 1], s[..., 2, 2], s[..., 0, 1], s[..., 1, 2], s[..., 2, 0]], -1)


def _matrix(v):
    return torch.stack([v[..., 0], v[..., 3], v[..., 5], v[..., 3], v[..., 1], v[..., 4], v[..., 5], v[..., 4], v[..., 2]],
                       -1).reshape(*v.shape[:-1], 3, 3)


def _return_map(strain, ps, mu, kappa, flow, slope):
    """J2 radial return (engineering shears in): stress, plastic increment, eq. plastic
    increment, flow direction and the tangent's theta, theta-bar, dissipation density."""
    el = strain - ps[..., :6]
    tr = el[..., :3].sum(-1, keepdim=True)
    dev = torch.cat([2 * mu * (el[..., :3] - tr / 3), mu * el[..., 3:]], -1)
    norm = (dev[..., :3].square().sum(-1, keepdim=True) + 2 * dev[..., 3:].square().sum(-1, keepdim=True)).sqrt()
    r23 = math.sqrt(2 / 3)
    p0 = ps[..., 6:7]
    excess = norm - r23 * flow(p0)
    gamma = torch.clamp(excess, min=0) / (2 * mu)
    on = excess > 0
    for _ in range(8):
        res = norm - 2 * mu * gamma - r23 * flow(p0 + r23 * gamma)
        gamma = torch.where(on, gamma + res / (2 * mu + 2 / 3 * slope(p0 + r23 * gamma)), 0.0)
    n = dev / torch.where(norm > 0, norm, 1.0)
    dp = gamma * torch.cat([n[..., :3], 2 * n[..., 3:]], -1)
    s = dev - 2 * mu * gamma * n
    sigma = torch.cat([s[..., :3] + kappa * tr, s[..., 3:]], -1)
    theta = 1 - torch.where(on, 2 * mu * gamma / torch.where(norm > 0, norm, 1.0), 0.0)
    bar = torch.where(on, 1 / (1 + slope(p0 + r23 * gamma) / (3 * mu)) - (1 - theta), 0.0)
    return sigma, dp, r23 * gamma, n, theta, bar, (sigma * dp).sum(-1)


def _strain_energy(s, mu, kappa):
    tr = s[..., :3].sum(-1)
    d = s[..., :3] - tr[..., None] / 3
    dev = d.square().sum(-1) + 2 * s[..., 3:].square().sum(-1)
    return 0.5 * (dev / (2 * mu) + tr.square() / (9 * kappa))


def _tet_exact(pos, idx, fixed, ext, steps, youngs, dt, yield_strength, hardening, ramp, mass=None, vel=None):
    """The union of the meshes at once: the material per tet, dt and ramp per node."""
    x, free = _t(pos).reshape(-1, 3), (_t(fixed, torch.int64) == 0)[:, None]
    i = _t(idx, torch.int64).reshape(-1, 4)
    d = (x[i[:, 1:]] - x[i[:, :1]]).transpose(1, 2)
    inv, vol = torch.linalg.inv(d), torch.linalg.det(d).abs() / 6
    n = x.shape[0]
    if mass is None:
        mass = torch.zeros(n, dtype=torch.float64, device=x.device)
        mass.index_add_(0, i.reshape(-1), (RHO * vol / 4).repeat_interleave(4))
    mass = mass[:, None]
    mu, kappa = youngs / (2 * (1 + NU)), youngs / (3 * (1 - 2 * NU))
    u, v = torch.zeros_like(x), torch.zeros_like(x) if vel is None else torch.where(free, _t(vel).reshape(-1, 3), 0.0)
    ps = torch.zeros(i.shape[0], 7, dtype=torch.float64, device=x.device)
    ext = _t(ext).reshape(-1, 3)
    g = torch.tensor([0.0, 0.0, -GRAVITY], dtype=torch.float64, device=x.device)
    work, diss, gwork = (torch.zeros((), dtype=torch.float64, device=x.device) for _ in range(3))
    eye = torch.eye(3, dtype=torch.float64, device=x.device)
    for k in range(steps):
        h = (u[i[:, 1:]] - u[i[:, :1]]).transpose(1, 2) @ inv
        r = _polar(eye + h)
        s = r.transpose(1, 2) @ (eye + h)
        e = _voigt(0.5 * (s + s.transpose(1, 2)) - eye)
        e = torch.cat([e[:, :3], 2 * e[:, 3:]], 1)
        sig, dp, deq, _, _, _, de = _return_map(e, ps, mu, kappa, lambda p: yield_strength + hardening * p,
                                                lambda p: hardening)
        ps = ps + torch.cat([dp, deq], 1)
        hf = -vol[:, None, None] * (r @ _matrix(sig) @ inv.transpose(1, 2))
        f = torch.cat([-hf.sum(2, keepdim=True), hf], 2).transpose(1, 2).reshape(-1, 3)
        a = torch.zeros_like(x).index_add_(0, i.reshape(-1), f)
        fe = ext * min(1.0, (k + 1.0) / ramp) if ramp else ext
        v = torch.where(free, v + ((a + fe) / mass + g) * dt, 0.0)
        u = u + v * dt
        work += (torch.where(free, fe, 0.0) * v * dt).sum()
        gwork += (mass * g * v * dt).sum()
        diss += (vol * de).sum()
    w = (vol * _strain_energy(sig, mu, kappa).reshape(-1) if not torch.is_tensor(mu) else
         vol * _strain_energy(sig, mu[:, 0], kappa[:, 0])).sum()
    return x + u, v, ps, torch.stack([work, diss, w, 0.5 * (mass * v.square()).sum(), gwork])


_XI = torch.tensor([[(1 if g & 1 else -1), (1 if g & 2 else -1), (1 if g & 4 else -1)] for g in range(8)],
                   dtype=torch.float64) / math.sqrt(3)
_CX, _CY = (-1.0, 1.0, 1.0, -1.0), (-1.0, -1.0, 1.0, 1.0)


def _transform(a):
    """Voigt (engineering) transform of eps = a^T E a for (..., 3, 3) a: (..., 6, 6)."""
    pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0))
    rows = []
    for r, c in pairs:
        row = []
        for k, l in pairs:
            t = a[..., k, r] * a[..., l, c] + (a[..., l, r] * a[..., k, c] if k != l else 0.0)
            row.append(t * (1.0 if r == c else 2.0) * (1.0 if k == l else 0.5))
        rows.append(torch.stack(row, -1))
    return torch.stack(rows, -2)


def _shell_operators(x):
    """B (E, 8, 6, 24), G (E, 8, 6, 7), weights (E, 8) and J0^-1 of corner sets (E, 8, 3)."""
    E = x.shape[0]
    bot, D = x[:, :4], x[:, 4:] - x[:, :4]
    B = torch.zeros(E, 8, 6, 24, dtype=torch.float64, device=x.device)
    w = torch.zeros(E, 8, dtype=torch.float64, device=x.device)
    G = torch.zeros(E, 8, 6, 7, dtype=torch.float64, device=x.device)

    def base(xi, eta, zeta):
        ps = [0.25 * (1 + xi * _CX[c]) * (1 + eta * _CY[c]) for c in range(4)]
        px = [0.25 * _CX[c] * (1 + eta * _CY[c]) for c in range(4)]
        py = [0.25 * _CY[c] * (1 + xi * _CX[c]) for c in range(4)]
        hi = 0.5 * (1 + zeta)
        lv = bot + hi * D
        gx = sum(px[c] * lv[:, c] for c in range(4))
        gy = sum(py[c] * lv[:, c] for c in range(4))
        gz = 0.5 * sum(ps[c] * D[:, c] for c in range(4))
        return ps, px, py, hi, lv, torch.stack([gx, gy, gz], -1)  # J: columns the base vectors

    J0 = base(0.0, 0.0, 0.0)[-1]
    J0i = torch.linalg.inv(J0)
    T0 = _transform(J0i)
    det0 = torch.linalg.det(J0)
    for g in range(8):
        xi, eta, zeta = (float(q) for q in _XI[g])
        ps, px, py, hi, lv, J = base(xi, eta, zeta)
        lo = 1 - hi
        gx, gy = J[..., 0], J[..., 1]
        N = torch.zeros(E, 6, 8, 3, dtype=torch.float64, device=x.device)
        for c in range(4):
            for node, f in ((c, lo), (c + 4, hi)):
                N[:, 0, node] += px[c] * f * gx
                N[:, 1, node] += py[c] * f * gy
                N[:, 3, node] += f * (py[c] * gx + px[c] * gy)
            N[:, 2, c + 4] += 0.25 * ps[c] * D[:, c]
            N[:, 2, c] -= 0.25 * ps[c] * D[:, c]
        for row, m, p, f in ((4, 0, 3, 0.5 * (1 - xi)), (4, 1, 2, 0.5 * (1 + xi)), (5, 0, 1, 0.5 * (1 - eta)),
                             (5, 3, 2, 0.5 * (1 + eta))):
            dx, dd = lv[:, p] - lv[:, m], D[:, m] + D[:, p]
            for c in (m, p):
                N[:, row, c + 4] += f / 8 * dx
                N[:, row, c] -= f / 8 * dx
            for c, sign in ((p, 1.0), (m, -1.0)):
                N[:, row, c + 4] += sign * f / 8 * hi * dd
                N[:, row, c] += sign * f / 8 * lo * dd
        B[:, g] = _transform(torch.linalg.inv(J)) @ N.reshape(E, 6, 24)
        w[:, g] = torch.linalg.det(J)
        for j, (mode, k) in enumerate(zip((xi, eta, zeta, xi * zeta, eta * zeta, xi, eta), (0, 1, 2, 2, 2, 3, 3))):
            G[:, g, :, j] = (det0 / w[:, g])[:, None] * mode * T0[..., k]
    return B, G, w, J0i


def _shell_exact(a, steps, law):
    p = a["params"]
    x = _t(a["rest"]).reshape(-1, 3)
    i = _t(a["index"], torch.int64).reshape(-1, 8)
    E, dev, f64 = i.shape[0], x.device, torch.float64
    mu, kappa = E_SHELL / (2 * (1 + NU)), E_SHELL / (3 * (1 - 2 * NU))
    if law == "swift":
        ks, e0, m = SWIFT["strength_coefficient"], SWIFT["reference_strain"], SWIFT["hardening_exponent"]
        flow, slope = (lambda q: ks * (e0 + q) ** m), (lambda q: ks * m * (e0 + q) ** (m - 1))
    else:
        flow, slope = (lambda q: p["yield_strength"] + p["hardening"] * q), (lambda q: torch.full_like(q, p["hardening"]))
    parts = [_shell_operators(x[i[c:c + 65536]]) for c in range(0, E, 65536)]
    B, G, w, J0i = (torch.cat([q[k] for q in parts]) for k in range(4))
    del parts
    shape = torch.tensor([[0.125 * (1 + g[0] * sx) * (1 + g[1] * sy) * (1 + g[2] * sz) for sx, sy, sz in
                           [(_CX[c % 4], _CY[c % 4], -1.0 if c < 4 else 1.0) for c in range(8)]] for g in _XI.tolist()],
                         dtype=f64, device=dev)
    mass = torch.zeros(x.shape[0], dtype=f64, device=dev)
    mass = mass.index_add_(0, i.reshape(-1), (RHO * w @ shape).reshape(-1))[:, None]
    grad0 = torch.tensor([[0.125 * s for s in (_CX[c % 4], _CY[c % 4], -1.0 if c < 4 else 1.0)] for c in range(8)],
                         dtype=f64, device=dev)
    C = torch.diag(torch.tensor([2 * mu] * 3 + [mu] * 3, dtype=f64, device=dev))
    C[:3, :3] += kappa - 2 * mu / 3
    K = torch.zeros(E, 7, 7, dtype=f64, device=dev)
    for g in range(8):
        K += w[:, g, None, None] * (G[:, g].transpose(1, 2) @ (C @ G[:, g]))
    K0i = torch.linalg.inv(K)
    del K
    dev6 = torch.diag(torch.tensor([1.0] * 3 + [0.5] * 3, dtype=f64, device=dev))
    dev6[:3, :3] -= 1 / 3
    one = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=f64, device=dev)
    eye = torch.eye(3, dtype=f64, device=dev)
    u, v = torch.zeros_like(x), torch.zeros_like(x)
    alpha = torch.zeros(E, 7, dtype=f64, device=dev)
    ps = torch.zeros(E, 8, 7, dtype=f64, device=dev)
    free = _t(a["pinned"], torch.int64).reshape(-1, 3) == 0
    load = _t(a["load"]).reshape(-1, 3)
    work, diss = torch.zeros((), dtype=f64, device=dev), torch.zeros((), dtype=f64, device=dev)
    B48, G56 = B.reshape(E, 48, 24), G.reshape(E, 48, 7)
    dX = x[i] - x[i[:, :1]]
    dt, damping = p["dt"], p["damping"]
    for k in range(steps):
        du = u[i] - u[i[:, :1]]
        r = _polar(eye + (du.transpose(1, 2) @ grad0) @ J0i)
        loc = (dX + du) @ r - dX
        base = (B48 @ loc.reshape(E, 24, 1)).reshape(E, 8, 6)
        for it in range(12):
            sig, dp, deq, nrm, theta, bar, de = _return_map(base + (G56 @ alpha[:, :, None]).reshape(E, 8, 6), ps, mu, kappa,
                                                            flow, slope)
            res = (G56.transpose(1, 2) @ (w[..., None] * sig).reshape(E, 48, 1))[..., 0]
            rest_of = res.square().sum(1).sqrt() > 1e-13 * p["yield_strength"] * w.sum(1)
            if it == 11 or not bool(rest_of.any()):
                break
            step = (K0i @ res[..., None])[..., 0]
            yielded = (theta < 1).reshape(E, 8).any(1) & rest_of
            if bool(yielded.any()):
                q = yielded.nonzero()[:, 0]
                Cq = kappa * one[:, None] * one + 2 * mu * theta[q][..., None] * dev6 - \
                    2 * mu * bar[q][..., None] * nrm[q][..., :, None] * nrm[q][..., None, :]
                Kq = (G[q].transpose(2, 3) @ (w[q][..., None, None] * (Cq @ G[q]))).sum(1)
                step[q] = torch.linalg.solve(Kq, res[q])
            alpha = torch.where(rest_of[:, None], alpha - step, alpha)
        ps = ps + torch.cat([dp, deq], -1)
        f = -(B48.transpose(1, 2) @ (w[..., None] * sig).reshape(E, 48, 1)).reshape(E, 8, 3) @ r.transpose(1, 2)
        force = torch.zeros_like(x).index_add_(0, i.reshape(-1), f.reshape(-1, 3))
        fe = load * min(1.0, (k + 1) * dt / p["rise_time"])
        v = torch.where(free, v + (force + fe) / mass * dt, 0.0) * damping
        u = u + v * dt
        work += (fe * v * dt).sum()
        diss += (w * de).sum()
    energy = torch.stack([work, diss, (w * _strain_energy(sig, mu, kappa)).sum(), 0.5 * (mass * v.square()).sum()])
    return x + u, v, ps, energy


def exact(case, seed):
    if work(case)["flops"] > (3e13 if case["kind"] == "shell" else 1e12):
        return None
    if case["kind"] == "shell":
        x, v, ps, energy = _shell_exact(_shell_inputs(case, seed), case["steps"], case["law"])
        out = dict(position=x.reshape(-1), velocity=v.reshape(-1))
        return dict(out, plastic=ps, energy=energy) if case["plastic"] else out
    if case["kind"] == "tet":
        a = _tet_inputs(case, seed)
        p = a["params"]
        mass = None
        if case["mode"] == "ref32":
            mass = _t(_tet_rest(a["pos"], a["idx"])[2])
        x, v, ps, energy = _tet_exact(a["pos"], a["idx"], a["fixed"], a["ext"], case["steps"], p["youngs"], p["dt"],
                                      p.get("yield_strength", 1e30), p.get("hardening", 0.0), p.get("ramp_steps", 0), mass,
                                      a["vel"])
        out = dict(position=x.reshape(-1), velocity=v.reshape(-1))
        return dict(out, plastic=ps, energy=energy) if case["plastic"] else out
    if case["kind"] == "serve":
        return None  # each solve takes its own bound as its time step, formed by the pool
    meshes, _ = _batch_inputs(case, seed)
    first = np.cumsum([0] + [m["position"].size // 3 for m in meshes[:-1]])

    def per_tet(key):
        return _t(np.repeat([m[key] for m in meshes], [m["index"].size // 4 for m in meshes]))[:, None]

    dt = _t(np.repeat([m["dt"] for m in meshes], [m["position"].size // 3 for m in meshes]))[:, None]
    x, v, _, _ = _tet_exact(np.concatenate([m["position"] for m in meshes]),
                            np.concatenate([m["index"].astype(np.int64) + o for m, o in zip(meshes, first)]),
                            np.concatenate([m["fixed"] for m in meshes]),
                            np.concatenate([m["external_force"] for m in meshes]), case["steps"], per_tet("youngs"), dt,
                            per_tet("yield_strength"), per_tet("hardening"), meshes[0]["ramp_steps"])
    return dict(position=x.reshape(-1), velocity=v.reshape(-1))
