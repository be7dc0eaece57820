"""The workloads this library is measured on.

Each case is something a user has the library do through its public entry
points (``mps_solvers_b200.capi``): stepping a scene and reading its state
back, stepping a batch, extracting the free surface, a training step of the
learned preconditioner, and the device-pointer cell sort.  ``listed()`` names
them, ``draw()`` makes more of the same ranges, ``prepare()`` builds the
handle and the buffers a program holds, ``run()`` is one pass, ``work()`` the
bytes and operations a pass cannot do without, and ``exact()`` the same
outputs in 64 bits from plain torch.

Scenes are closed tanks (two wall and two dummy layers, ``scene.py``) with a
column of water in the middle of a flow: lattice positions displaced by
``jitter`` spacings, a velocity of about ``speed`` m/s into the corner of the
tank, so that the water there is compressed, and a hydrostatic pressure.
Time steps, kernel radii and spacings are those of the workloads of
``scene.py``.
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from mps_solvers_b200 import capi, precond_weights, scene

GRAVITY = 9.81


def listed():
    return [
        # a few thousand particles, the reference's exact arithmetic: the
        # smallest scene people step, ten steps between two reads of the state
        {"name": "explicit tank", "kind": "step", "method": "explicit", "arith": "exact", "nx": 14, "ny": 6, "nz": 12,
         "fx": 5, "fy": 4, "fz": 8, "l0": 0.02, "steps": 10},
        # the 70,912-particle explicit dam break
        {"name": "explicit dam break", "kind": "step", "method": "explicit", "arith": "exact", "nx": 80, "ny": 20,
         "nz": 50, "fx": 20, "fy": 10, "fz": 40, "l0": 0.02, "steps": 10},
        # the same at 310,912 particles with the fast arithmetic
        {"name": "explicit fast", "kind": "step", "method": "explicit", "arith": "fast", "nx": 160, "ny": 40,
         "nz": 100, "fx": 40, "fy": 25, "fz": 80, "l0": 0.02, "steps": 5},
        # a semi-implicit tank of odd sizes with the default options (exact
        # arithmetic, diagonally scaled CG): few rows for the solver's grid
        {"name": "semi tank", "kind": "step", "method": "semi", "arith": "exact", "nx": 41, "ny": 13, "nz": 29,
         "fx": 17, "fy": 13, "fz": 23, "l0": 0.01, "steps": 2},
        # the semi-implicit dam break the headline metric is quoted on
        {"name": "semi dam break", "kind": "step", "method": "semi", "arith": "fast", "nx": 160, "ny": 40, "nz": 100,
         "fx": 40, "fy": 25, "fz": 80, "l0": 0.01, "steps": 2},
        # the same with the learned preconditioner
        {"name": "semi learned", "kind": "step", "method": "semi", "arith": "fast", "learned": True, "nx": 160,
         "ny": 40, "nz": 100, "fx": 40, "fy": 25, "fz": 80, "l0": 0.01, "steps": 2},
        # a viscous fluid: Crank-Nicolson viscosity, three more solves a step
        {"name": "semi viscous", "kind": "step", "method": "semi", "arith": "fast", "implicit_visc": True, "nx": 80,
         "ny": 31, "nz": 50, "fx": 33, "fy": 25, "fz": 40, "l0": 0.01, "steps": 1},
        # a large single scene with the learned preconditioner
        {"name": "semi large", "kind": "step", "method": "semi", "arith": "fast", "learned": True, "nx": 300, "ny": 90,
         "nz": 150, "fx": 90, "fy": 90, "fz": 110, "l0": 0.005, "steps": 1},
        # uneven scenes in one launch, learned preconditioner
        {"name": "batch", "kind": "batch", "scenes": 6, "pick": 3, "learned": True, "steps": 1},
        # the free surface of a flow on a rendering grid
        {"name": "surface", "kind": "surface", "nx": 160, "ny": 40, "nz": 100, "fx": 40, "fy": 25, "fz": 80,
         "l0": 0.01, "gx": 256, "gy": 64, "gz": 128},
        # loss and gradients of the learned preconditioner on one PPE system
        {"name": "training", "kind": "train", "nx": 80, "ny": 25, "nz": 60, "fx": 33, "fy": 25, "fz": 50,
         "l0": 0.01},
        # the neighbour-search rebuild on device arrays
        {"name": "cell sort", "kind": "sort", "n": 500000, "nx": 67, "ny": 33, "nz": 41},
    ]


def _tank(rng, lo, hi):
    """Sizes of a tank with about `lo`..`hi` fluid particles (log-uniform)."""
    nf = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    fy = max(4, int(round(nf ** (1 / 3) * rng.uniform(0.5, 0.9))))
    fx = max(4, int(round(math.sqrt(nf / fy) * rng.uniform(0.6, 0.95))))
    fz = max(6, int(round(nf / (fx * fy))))
    return {"nx": max(12, int(fx * rng.uniform(1.5, 3.5))), "ny": fy + rng.choice([0, 0, 1, 5]),
            "nz": int(fz * 1.25) + 2, "fx": fx, "fy": fy, "fz": fz}


def draw(rng):
    kind = rng.choice(["explicit", "semi", "semi", "semi", "learned", "viscous", "batch", "surface", "train", "sort"])
    if kind == "explicit":
        c = {"kind": "step", "method": "explicit", "arith": rng.choice(["exact", "exact", "fast"]), "l0": 0.02,
             "steps": rng.choice([1, 3, 10])}
        return {**c, **_tank(rng, 200, 60000)}
    if kind in ("semi", "learned", "viscous"):
        c = {"kind": "step", "method": "semi", "arith": rng.choice(["exact", "fast", "fast"]), "l0": 0.01,
             "steps": rng.choice([1, 2, 3])}
        if kind == "learned":
            return {**c, "learned": True, **_tank(rng, 4000, 200000)}
        if kind == "viscous":
            return {**c, "implicit_visc": True, **_tank(rng, 2000, 60000)}
        return {**c, **_tank(rng, 400, 250000)}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.choice([1, 2, 3, 5]), "pick": rng.randrange(1000),
                "learned": rng.choice([True, False]), "steps": rng.choice([1, 2])}
    if kind == "surface":
        t = _tank(rng, 3000, 80000)
        return {"kind": "surface", "l0": 0.01, "gx": rng.randint(40, 256), "gy": rng.randint(20, 64),
                "gz": rng.randint(30, 128), **t}
    if kind == "train":
        return {"kind": "train", "l0": 0.01, **_tank(rng, 4000, 60000)}
    return {"kind": "sort", "n": int(math.exp(rng.uniform(math.log(1000), math.log(1000000)))),
            "nx": rng.randint(4, 90), "ny": rng.randint(4, 60), "nz": rng.randint(4, 60)}


# ---- inputs


def _params(case):
    """input.dat's values as the library holds them (lengths times the spacing)."""
    l0 = case["l0"]
    semi = case.get("method") == "semi" or case["kind"] == "train"
    dt = (5e-4 if l0 >= 0.01 else 2.5e-4) if semi else 1e-4
    niu = 0.01 if case.get("implicit_visc") else 1e-6
    p = capi.mps_params()
    p.dim = 3
    for k, v in dict(rho=1000.0, niu=niu, dp=l0, rzero=2.1 * l0, rlap=4.0 * l0, beta=0.97, cs=20.0, cfl=0.2,
                     col_dis=0.8 * l0, col_rate=2.0, dt_max=dt, dt_min=1e-3 * dt, tt=1.0, tout=1e9,
                     max_dis=l0).items():
        setattr(p, k, v)
    return p


def _scene(case):
    return scene.Scene(l0=case["l0"], interior=(case["nx"], case["ny"], case["nz"]),
                       fluid=[scene.Box(0, 0, 0, case["fx"], case["fy"], case["fz"])], jitter=0.0)


def _flow(sc, seed, jitter=2e-4, speed=0.8):
    """Positions, velocities and pressures of the scene in the middle of a flow
    that runs into the corner of its tank."""
    pos, nb2, nb1 = scene.build(sc)
    rng = np.random.default_rng(seed)
    l0 = np.float32(sc.l0)
    pos = pos + (rng.random(pos.shape, dtype=np.float32) * 2 - 1) * np.float32(jitter) * l0
    b = sc.fluid[0]
    s = 2 * sc.wall_layers
    f = pos[nb2 + nb1:]
    x = (f[:, 0] / l0 - s) / b.nx
    z = (f[:, 2] / l0 - s) / b.nz
    u = np.float32(speed * rng.uniform(0.75, 1.25))
    vel = np.zeros_like(pos)
    vel[nb2 + nb1:, 0] = -u * (0.25 + 0.75 * x)
    vel[nb2 + nb1:, 2] = -u * (0.25 + 0.75 * z)
    press = np.zeros(len(pos), np.float32)
    press[nb2 + nb1:] = np.maximum(0, 1000.0 * GRAVITY * (1 - z) * b.nz * l0)
    return pos, vel, press, nb2, nb1


def _batch_scenes(case):
    out = []
    for sc, amp, freq in scene.batch_scenes(case["scenes"], case["pick"]):
        out.append((scene.Scene(l0=sc.l0, interior=sc.interior, fluid=sc.fluid, jitter=0.0, params=sc.params), amp,
                    freq))
    return out


def _options(case):
    semi = case.get("method") == "semi" or case["kind"] in ("train", "batch")
    o = {"method": capi.METHOD_SEMI_IMPLICIT if semi else capi.METHOD_EXPLICIT}
    if case.get("arith", "fast") == "fast":
        o["arith"] = capi.ARITH_FAST
    if case.get("learned"):
        o["precond"] = capi.PRECOND_LEARNED
    if case.get("implicit_visc"):
        o["visc_implicit"] = 1
    return o


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()


def _sort_grid(case):
    g = capi.mps_grid()
    g.left = g.back = g.bottom = 0.0
    g.cell_size = 0.04
    g.cdx, g.cdy, g.cdz = case["nx"], case["ny"], case["nz"]
    g.ncells = case["nx"] * case["ny"] * case["nz"]
    g.dim = 3
    return g


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        ext = torch.tensor([case["nx"], case["ny"], case["nz"], 1], device="cuda") * 0.04
        pos = torch.rand((case["n"], 4), device="cuda", generator=gen) * (0.999 * ext)
        i32 = lambda k: torch.empty(k, dtype=torch.int32, device="cuda")
        g = _sort_grid(case)
        return {"case": case, "pos": pos, "grid": g, "perm": i32(case["n"]), "cell": i32(case["n"]),
                "start": i32(g.ncells), "end": i32(g.ncells), "inside": i32(1)}
    if kind == "batch":
        scenes = _batch_scenes(case)
        with tempfile.TemporaryDirectory() as d:
            dirs = []
            for k, (sc, _, _) in enumerate(scenes):
                dirs.append(os.path.join(d, str(k)))
                os.makedirs(dirs[-1])
                pos, vel, press, nb2, nb1 = _flow(sc, seed * 1000 + k)
                scene.write_input_dat(os.path.join(dirs[-1], "input.dat"), sc.params)
                scene.write_geo_dat(os.path.join(dirs[-1], "GEO.dat"), pos, nb2, nb1, vel, press)
            sim = capi.Simulation.batch(dirs, accel=[(a, f) for _, a, f in scenes], **_options(case))
    else:
        pos, vel, press, nb2, nb1 = _flow(_scene(case), seed)
        sim = capi.Simulation.from_arrays(_params(case), pos, nb2, nb1, vel, press, **_options(case))
    if case.get("learned") or kind == "train":
        sim.set_precond_params(precond_weights.load())
    n = sim.counts()["np"]
    s = {"case": case, "sim": sim, "pos": _pinned(n, 3), "vel": _pinned(n, 3), "press": _pinned(n)}
    if kind == "surface":
        shape = (case["gx"], case["gy"], case["gz"])
        origin, spacing = scene.surface_grid(_scene(case), shape)
        sim.surface_setup(shape, origin, spacing, 4 * shape[0] * shape[1] + 200000)
    if kind == "train":
        sim.step(1)  # the system the network is trained on
        s["seed"] = seed
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sort":
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        st = capi.lib().mps_cell_sort_dev(p(state["pos"]), case["n"], ctypes.byref(state["grid"]), p(state["perm"]),
                                          p(state["cell"]), p(state["start"]), p(state["end"]), p(state["inside"]),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st:
            raise capi.MPSError(st, "cell sort")
        return {k: state[k] for k in ("perm", "cell", "start", "end", "inside")}
    sim = state["sim"]
    if kind == "surface":
        sim.surface_extract()
        pos, nrm = sim.surface_triangles()
        return {"pos": pos, "nrm": nrm}
    if kind == "train":
        loss, grad = sim.precond_loss_grad(state["seed"])
        return {"loss": loss, "grad": grad}
    sim.step(case["steps"])
    sim.get_state_into(state["pos"], state["vel"], state["press"], capi.ORDER_BY_ID)
    return {"pos": state["pos"], "vel": state["vel"], "press": state["press"]}


# ---- the least a pass moves and computes


def _counts(sc):
    nx, ny, nz = sc.interior
    s = 2 * sc.wall_layers
    tank = nx * ny * nz
    fluid = sum(b.nx * b.ny * b.nz for b in sc.fluid)
    return (nx + 2 * s) * (ny + 2 * s) * (nz + 2 * s) - tank + fluid, fluid


def work(case):
    kind = case["kind"]
    if kind == "sort":
        n, cells = case["n"], case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 24 * n + 8 * cells, "flops": 6 * n}
    if kind == "surface":
        n, f = _counts(_scene(case))
        v = case["gx"] * case["gy"] * case["gz"]
        return {"bytes": 12 * f + 4 * v, "flops": 30 * 16 * f}
    if kind == "train":
        # forward and backward of two rounds of 64-wide layers over the rows
        # (three 64 x 64 layers) and the 32 neighbours of each
        n, f = _counts(_scene(case))
        return {"bytes": 16 * f * 32, "flops": 6.0 * f * (3 * 64 * 64 + 32 * 2 * 8 * 64)}
    scenes = [sc for sc, _, _ in _batch_scenes(case)] if kind == "batch" else [_scene(case)]
    nb = fl = 0.0
    for sc in scenes:
        n, f = _counts(sc)
        # the state in and out and to the host; pair terms of the stages:
        # number density (32 pairs), viscosity (256), collision, gradient
        b, w = 56.0 * n, f * (32 * 10 + 256 * 16 + 32 * 20 + 32 * 18)
        if kind == "batch" or case["method"] == "semi":
            # 30 CG iterations over the fluid's rows: the vectors live on
            # chip, the stencil of 160 neighbours is evaluated each time
            w += 30.0 * f * 160 * 2
            b += 24.0 * f
        nb += b * case["steps"]
        fl += w * case["steps"]
    return {"bytes": nb, "flops": fl}


# ---- the same results in 64 bits


def _pairs(pos, radius):
    """(i, j) of all pairs closer than radius, j != i, both directions."""
    lo = pos.min(0).values
    c = ((pos - lo) / radius).long()
    dim = c.max(0).values + 3
    key = ((c[:, 2] + 1) * dim[1] + (c[:, 1] + 1)) * dim[0] + c[:, 0] + 1
    key_s, order = key.sort(stable=True)
    p = pos[order]
    out_i, out_j = [], []
    idx = torch.arange(len(pos), device=pos.device)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            # the three cells along x are one run of the sorted order
            k = key_s + (dz * dim[1] + dy) * dim[0]
            a = torch.searchsorted(key_s, k - 1)
            cnt = torch.searchsorted(key_s, k + 2) - a
            for part in torch.split(idx, 100000):
                n = cnt[part]
                i = torch.repeat_interleave(part, n)
                j = torch.arange(len(i), device=pos.device) - torch.repeat_interleave(n.cumsum(0) - n, n)
                j = j + torch.repeat_interleave(a[part], n)
                d = p[j] - p[i]
                keep = ((d * d).sum(1) < radius * radius) & (i != j)
                out_i.append(order[i[keep]])
                out_j.append(order[j[keep]])
    return torch.cat(out_i), torch.cat(out_j)


def _pair_geometry(pos, radius):
    i, j = _pairs(pos, radius)
    d = pos[j] - pos[i]
    r = (d * d).sum(1).sqrt()
    return i, j, d, r, radius / r - 1


def _sum_to(n, i, v):
    return torch.zeros((n,) + tuple(v.shape[1:]), dtype=v.dtype, device=v.device).index_add_(0, i, v)


def _cg(i, j, w, diag, b, x):
    """Diagonally scaled CG to 1e-13 on A = diag + (w at (i, j))."""
    n = len(b)
    a = torch.sparse_coo_tensor(torch.stack([i, j]), w, (n, n)).to_sparse_csr()
    mul = lambda v: diag * v + torch.mv(a, v)
    r = b - mul(x)
    z = r / diag
    p = z.clone()
    rz = torch.dot(r, z)
    stop = 1e-13 * b.norm()
    for _ in range(2000):
        if r.norm() <= stop:
            break
        q = mul(p)
        alpha = rz / torch.dot(p, q)
        x = x + alpha * p
        r = r - alpha * q
        z = r / diag
        rz, old = torch.dot(r, z), rz
        p = z + (rz / old) * p
    return x


def _steps64(prm, pos, vel, press, nb2, nb1, semi, steps, accel=(0.0, 0.0)):
    g = lambda name: float(getattr(prm, name))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
    pos, vel, press = t64(pos), t64(vel), t64(press)
    n = len(pos)
    kind = torch.zeros(n, dtype=torch.long, device=dev)
    kind[:nb2 + nb1] = 1
    kind[:nb2] = 2
    fluid, solid = kind == 0, kind != 2
    r0, rlap, beta, rho = g("rzero"), g("rlap"), g("beta"), g("rho")
    i, j, d, r, w = _pair_geometry(pos, r0)
    dens = _sum_to(n, i, w)
    top = int(dens.argmax())
    n0 = float(dens[top])
    near = i == top
    lam = float((r[near] ** 2 * w[near]).sum()) / n0
    c_lap = 6.0 / (n0 * lam)
    alpha = 1.0 / (rho * g("cs") ** 2)
    wall_of = torch.arange(n, device=dev)
    if not semi:
        i, j, d, r, w = _pair_geometry(pos, math.sqrt(2.0) * r0)
        m = (kind[i] == 2) & (kind[j] == 1)
        i, j, r = i[m], j[m], r[m]
        best = torch.full((n,), math.inf, dtype=torch.float64, device=dev).scatter_reduce_(0, i, r, "amin")
        hit = r == best[i]
        wall_of[i[hit]] = j[hit]
    time = 0.0
    dt_max = g("dt_max")
    gvec = t64([0.0, 0.0, -float(np.float32(GRAVITY))])
    for _ in range(steps):
        dt = min(dt_max, g("cfl") * g("dp") / max(float(vel.norm(dim=1).max()), 1e-300))
        force = gvec.clone()
        force[0] -= accel[0] * math.sin(2 * math.pi * accel[1] * time)
        # viscosity and gravity
        i, j, d, r, w = _pair_geometry(pos, rlap)
        m = fluid[i]
        lap = _sum_to(n, i[m], w[m, None] * (vel[j[m]] - vel[i[m]]))
        t = vel + dt * (g("niu") * c_lap * lap + force)
        vel = torch.where(fluid[:, None], t, vel)
        pos = torch.where(fluid[:, None], pos + dt * t, pos)
        # collision
        i, j, d, r, w = _pair_geometry(pos, g("col_dis"))
        va = (0.5 * (vel[j] - vel[i]) * d).sum(1) / r
        m = fluid[i] & (va <= 0)
        t = _sum_to(n, i[m], (g("col_rate") * va / r)[m, None] * d[m])
        vel, pos = vel + t, pos + dt * t
        # number density and pressure
        i, j, d, r, w = _pair_geometry(pos, r0)
        dens = _sum_to(n, i, w)
        if semi:
            row = solid & (dens >= beta * n0)
            li, lj, _, _, lw = _pair_geometry(pos, rlap)
            m = row[li] & solid[lj]
            diag = -_sum_to(n, li[m], lw[m]) - rho * lam * alpha * n0 / (6.0 * dt * dt)
            num = torch.cumsum(row.long(), 0) - 1
            m = m & row[lj]
            b = lam * rho / (6.0 * dt_max * dt_max) * (n0 - dens)
            x = _cg(num[li[m]], num[lj[m]], lw[m], diag[row], b[row], press[row])
            press = torch.zeros_like(press)
            press[row] = x.clamp(min=0)
            m = fluid[i] & solid[j]
        else:
            p = (rho * g("cs") ** 2 * (dens - n0) / n0).clamp(min=0)
            press = torch.where(solid, p, press)
            press = torch.where(solid, press, press[wall_of])
            m = fluid[i]
        # pressure gradient
        hs = solid[j]
        hat = press.clone().scatter_reduce_(0, i[hs], press[j[hs]], "amin")
        k = (press[j] - hat[i]) / (r * r) * w
        t = -dt / rho * 3.0 / n0 * _sum_to(n, i[m], k[m, None] * d[m])
        vel = torch.where(fluid[:, None], vel + t, vel)
        pos = torch.where(fluid[:, None], pos + dt * t, pos)
        time += dt
    return {"pos": pos, "vel": vel, "press": press}


def exact(case, seed):
    if case["kind"] == "step" and not case.get("implicit_visc"):
        n, _ = _counts(_scene(case))
        if n > 600000:
            return None
        pos, vel, press, nb2, nb1 = _flow(_scene(case), seed)
        return _steps64(_params(case), pos, vel, press, nb2, nb1, case["method"] == "semi", case["steps"])
    if case["kind"] == "batch":
        got = []
        for k, (sc, amp, freq) in enumerate(_batch_scenes(case)):
            pos, vel, press, nb2, nb1 = _flow(sc, seed * 1000 + k)
            prm = _params({"kind": "batch", "method": "semi", "l0": sc.l0})
            got.append(_steps64(prm, pos, vel, press, nb2, nb1, True, case["steps"], (amp, freq)))
        return {f: torch.cat([g[f] for g in got]) for f in ("pos", "vel", "press")}
    return None
