"""What the engine is measured on: the calls a program makes, over the range of sizes it makes them with.

Kinds of case:

* ``steps``    records uploaded from pinned memory, a number of substeps, records downloaded
               (GpuSolver.upload / step / download). One substep per pass is the transfer pattern
               of a program with a per-substep callback; ten are one output frame at the default
               simulation_scale of 0.1.
* ``batch``    the same over many independent scenes in one solver (GpuSolver.batched).
* ``learned``  the same with learned steps in place of plain substeps (learned.step_learned).
* ``forward``  the stepper's network on standardised rows in device memory (Mlp.forward).
* ``grads``    one training pass: loss and gradients (Mlp.gradients).
* ``sort``     the allocation-free key sort on device buffers (clsph_gpu_sort_keys_noalloc).

Every pass uploads its records (or reads inputs that no pass writes), so a pass is the same work however
often it is repeated.
"""

import math

import numpy as np
import torch

from libclsph_gb300 import workloads as W
from libclsph_gb300.layout import PARTICLE, particles_from_arrays

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"

# a viscous fluid with a bouncing wall response (restitution 0.5) and 40 particles within the radius
MUCUS = {"fluid_density": 1000, "dynamic_viscosity": 36, "restitution": 0.5, "k": 5,
         "surface_tension_threshold": 5, "surface_tension": 6, "particles_inside_influence_radius": 40}
FLUIDS = {"water": {}, "mucus": MUCUS}
H = 1.0 / 64.0  # smoothing radius of every scene (through the particle mass)


def listed():
    return [
        # a callback every substep on a small scene: launches, copies and synchronisation count
        {"name": "callback_4k", "kind": "steps", "n": 4096, "state": "pool", "fluid": "water", "substeps": 1,
         "graph": False, "tune": False},
        # a callback every substep on the large scene: half of the pass is the host link
        {"name": "callback_1m", "kind": "steps", "n": 1048576, "state": "pool", "fluid": "water", "substeps": 1,
         "graph": False, "tune": False},
        # a frame of an interactive-sized scene, tuned once as a long-running program does
        {"name": "frame_32k", "kind": "steps", "n": 32768, "state": "pool", "fluid": "water", "substeps": 10,
         "graph": True, "tune": True},
        # a frame of an ordinary scene of an odd size, with a fluid that bounces off the walls
        {"name": "frame_150k_mucus", "kind": "steps", "n": 150001, "state": "pool", "fluid": "mucus",
         "substeps": 10, "graph": True, "tune": False},
        # a frame of the large scene in the middle of a run: ragged cells, particles on walls and floor
        {"name": "frame_1m", "kind": "steps", "n": 1048576, "state": "pool", "fluid": "water", "substeps": 10,
         "graph": True, "tune": False},
        # the first frame of the large dam break: the column as released, in lattice order
        {"name": "dam_break_1m", "kind": "steps", "n": 1048576, "state": "column", "fluid": "water",
         "substeps": 10, "graph": True, "tune": False},
        # a large body of fluid landing on a heightfield of 131,072 triangles
        {"name": "pour_4m", "kind": "steps", "n": 4194304, "state": "pour", "fluid": "water", "substeps": 4,
         "graph": True, "tune": False},
        # 256 independent scenes of 2,048 to 65,536 particles in one solver
        {"name": "batch_256", "kind": "batch", "scenes": 256, "n_max": 65536, "substeps": 4, "graph": True,
         "tune": True},
        # the learned stepper: each step covers four plain time steps
        {"name": "learned_1m", "kind": "learned", "n": 1048576, "state": "pool", "fluid": "water", "steps": 4,
         "graph": True},
        # the stepper's network by itself, one row per particle, ragged last tile
        {"name": "forward_1m", "kind": "forward", "rows": 1048577},
        # one training batch of the stepper's network
        {"name": "grads_64k", "kind": "grads", "rows": 65536},
        # the key sort for callers that own every allocation, at the substep's key width
        {"name": "sort_1m", "kind": "sort", "n": 1048576, "bits": 22},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["batch", "learned", "forward", "grads", "sort"])
    if kind == "steps":
        state = rng.choice(["pool", "pool", "column", "pour"])
        return {"kind": kind, "n": _log_int(rng, 2000, 3000000) if state == "pour" else _log_int(rng, 500, 1100000),
                "state": state, "fluid": rng.choice(["water", "water", "mucus"]),
                "substeps": rng.choice([1, 2, 3, 10]) if state != "pour" else rng.choice([1, 2, 4]),
                "graph": rng.random() < 0.5, "tune": rng.random() < 0.25}
    if kind == "batch":
        return {"kind": kind, "scenes": _log_int(rng, 3, 200), "n_max": _log_int(rng, 4096, 65536),
                "substeps": rng.choice([1, 2, 4]), "graph": rng.random() < 0.5, "tune": rng.random() < 0.25}
    if kind == "learned":
        return {"kind": kind, "n": _log_int(rng, 20000, 1000000), "state": "pool", "fluid": "water",
                "steps": rng.choice([1, 3, 4]), "graph": rng.random() < 0.5}
    if kind == "forward":
        return {"kind": kind, "rows": _log_int(rng, 1000, 4000000)}
    if kind == "grads":
        return {"kind": kind, "rows": 2048 * rng.randint(1, 60)}
    return {"kind": kind, "n": _log_int(rng, 1000, 1 << 20), "bits": rng.choice([8, 16, 20, 24, 30, 32])}


# ------------------------------------------------------------------------------------------- inputs


def _mesh_height(mesh, quads, width, x, z):
    """Height of the heightfield over (x, z), bilinear between its vertices."""
    y = mesh["vertices"].reshape(-1, 3)[:, 1].reshape(quads + 1, quads + 1).astype(np.float64)
    u, w = np.clip(x / width * quads, 0, quads - 1e-6), np.clip(z / width * quads, 0, quads - 1e-6)
    i, k = u.astype(np.int64), w.astype(np.int64)
    a, b = u - i, w - k
    return ((y[i, k] * (1 - b) + y[i, k + 1] * b) * (1 - a) + (y[i + 1, k] * (1 - b) + y[i + 1, k + 1] * b) * a)


def _scene(case, seed):
    """(params, terms, mesh, records, h) of one scene, from the seed alone."""
    rng = np.random.default_rng(1000003 * seed + 17)
    n, fluid = case["n"], FLUIDS[case["fluid"]]
    st = W.water_settings(n, mass=0.05, **fluid)
    st = W.water_settings(n, mass=0.05 * (H / float(st.params["h"])) ** 3, **fluid)  # h scales with the cube root
    h = float(st.params["h"])
    k = 40 if case["fluid"] == "mucus" else 20
    if case["state"] == "column":
        # a 2 : 2 : 1 column (the large dam break's shape) at spacing h/2 in the left quarter of its box
        c = max(1, round((n / 4) ** (1 / 3)))
        nz, nx = c, 2 * c
        ny = -(-n // (nx * nz))
        s = h / 2
        pos = W.lattice((nx, ny, nz), s, (0.0, 0.0, 0.0), 0.01, rng)
        pos = pos[np.sort(np.argsort(pos[:, 1], kind="stable")[:n])]
        vel = np.zeros_like(pos)
        mesh = W.box_mesh((0, 0, 0), (4 * nx * s, 2 * ny * s, 2 * nz * s))
    elif case["state"] == "pool":
        # fluid spread over the floor between three walls: uneven spacing (closer at the bottom), waves,
        # a little spray, a swirl with per-particle noise; records in the cell order a run leaves them in
        s = (0.54 if k == 20 else 0.46) * h
        c = max(1, round((n / 8) ** (1 / 3)))
        nx, nz = 4 * c, 2 * c
        ny = -(-n // (nx * nz))
        g = rng.random((n, 3))
        i = np.arange(n)
        pos = np.stack([i % nx, i // (nx * nz), (i // nx) % nz], 1) + 0.5 + (g - 0.5) * 0.6
        top = ny * s
        pos *= s
        pos[:, 1] *= 0.85 + 0.15 * pos[:, 1] / top
        pos[:, 1] *= 1 + 0.08 * np.sin(6.0 * pos[:, 0] / (nx * s)) + 0.08 * np.cos(9.0 * pos[:, 2] / (nz * s))
        spray = rng.random(n) < 0.01
        pos[spray, 1] = top * (1.2 + 0.8 * rng.random(int(spray.sum())))
        box = (2 * nx * s, max(4 * ny, 8) * s, nz * s)
        vel = rng.normal(0.0, 0.05, (n, 3))
        vel[:, 0] += 0.5 * np.sin(3.0 * pos[:, 1] / box[1]) + 0.2 * np.cos(7.0 * pos[:, 2] / box[2])
        vel[:, 1] += 0.3 * np.sin(5.0 * pos[:, 0] / box[0]) - 0.2
        vel[:, 2] += 0.2 * np.sin(4.0 * pos[:, 0] / box[0])
        mesh = W.box_mesh((0, 0, 0), box)
        pos = pos.astype(np.float32)
        order = np.argsort(_keys(pos, np.float32(h))[0], kind="stable")
        pos, vel = pos[order], vel[order].astype(np.float32)
    else:
        # a sheet of fluid just above a heightfield, falling on it at 2 m/s
        quads, s = 256, h / 2
        layers = 16 if n >= 65536 else 4
        side = max(2, math.ceil(math.sqrt(n / layers)))
        width = max(4.0, side * s)
        field = W.heightfield_mesh((0.0, 0.0), (width, width), quads, 0.25, 0.2, 3)
        mesh = W.merge_meshes(field, W.box_mesh((0, 0, 0), (width, 2.0, width)))
        g = rng.random((n, 3)).astype(np.float32)
        i = np.arange(n)
        x = (i % side + 0.5 + 0.2 * (g[:, 0] - 0.5)) * s + (width - side * s) / 2
        z = ((i // side) % side + 0.5 + 0.2 * (g[:, 2] - 0.5)) * s + (width - side * s) / 2
        y = _mesh_height(field, quads, width, x, z) + (i // (side * side) + 0.3 + 0.2 * g[:, 1]) * s
        pos = np.stack([x, y, z], 1).astype(np.float32)
        vel = np.zeros_like(pos)
        vel[:, 1] = -2.0 * (0.95 + 0.1 * rng.random(n))
    return st.params, st.terms, mesh, particles_from_arrays(pos, vel, vel), h


def _pinned(records):
    keep = torch.empty(records.nbytes, dtype=torch.uint8, pin_memory=torch.cuda.is_available())
    view = keep.numpy().view(PARTICLE)
    view[:] = records
    return view, keep


def _solver_state(gpu, records, case):
    src, keep_src = _pinned(records)
    out, keep_out = _pinned(np.zeros_like(records))
    if case["graph"]:
        gpu.set_graph(True)
    if case.get("tune"):
        gpu.upload(src)
        gpu.autotune(3)
    return {"kind": case["kind"], "gpu": gpu, "in": src, "out": out, "keep": (keep_src, keep_out),
            "count": case.get("substeps", case.get("steps"))}


def _rows(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed * 7919 + 5)
    return torch.randn(case["rows"], 32, device=DEVICE, generator=g).clamp_(-6, 6), g


def _blob():
    from libclsph_gb300 import learned as Lm

    with np.load(Lm.default_weights_path()) as z:
        return np.asarray(z["blob"], dtype=np.float32)


def prepare(case, seed):
    from libclsph_gb300.gpu import GpuSolver, load_library

    kind = case["kind"]
    if kind in ("steps", "learned"):
        params, terms, mesh, records, _ = _scene(case, seed)
        state = _solver_state(GpuSolver(params, terms, case["n"], mesh), records, case)
        if kind == "learned":
            from libclsph_gb300 import learned as Lm

            state["mlp"] = Lm.Mlp.load()
        return state
    if kind == "batch":
        # the set of scenes is the case's; the seed moves every particle a little and gives it a velocity
        scenes = W.batched_dam_breaks(case["scenes"], n_max=case["n_max"])
        gpu = GpuSolver.batched([s.params for s in scenes], [s.terms for s in scenes], [s.n for s in scenes],
                                [s.mesh for s in scenes])
        records = np.zeros(gpu.n, dtype=PARTICLE)
        np.concatenate([s.particles for s in scenes], out=records)
        rng = np.random.default_rng(seed)
        records["position"][:, :3] += rng.uniform(0.0, 0.02 * H, (gpu.n, 3)).astype(np.float32)
        records["velocity"][:, :3] = rng.uniform(-0.1, 0.1, (gpu.n, 3))
        records["intermediate_velocity"] = records["velocity"]
        return _solver_state(gpu, records, case)
    if kind in ("forward", "grads"):
        from libclsph_gb300 import learned as Lm

        x, g = _rows(case, seed)
        mlp = Lm.Mlp.load()
        if kind == "forward":
            return {"kind": kind, "mlp": mlp, "x": x.to(torch.bfloat16),
                    "y": torch.empty(case["rows"], 4, device=DEVICE), "rows": case["rows"]}
        x, y = _raw(x, g)
        return {"kind": kind, "mlp": mlp, "x": x, "y": y, "rows": case["rows"]}
    keys = _sort_keys(case, seed)
    return {"kind": kind, "lib": load_library(), "keys": keys, "n": case["n"], "out": torch.empty_like(keys),
            "perm": torch.empty_like(keys)}


def _raw(x, g):
    """Raw training rows from standardised ones: features and targets in the network's own units."""
    t = torch.from_numpy(_blob()).to(DEVICE)
    mu, sigma, ymu, ysigma = t[-72:-40], t[-40:-8], t[-8:-4], t[-4:]
    y = torch.randn(len(x), 4, device=DEVICE, generator=g) * 0.5 + torch.tanh(x[:, :4])
    return (x * sigma + mu).contiguous(), (y * ysigma + ymu).contiguous()


def _sort_keys(case, seed):
    """Keys of a nearly sorted state: runs of equal keys in ascending order, a few per cent out of place."""
    rng = np.random.default_rng(seed)
    n, bits = case["n"], case["bits"]
    cells = np.sort(rng.integers(0, 1 << bits, max(1, n // 50), dtype=np.uint64))
    keys = cells[np.minimum(np.arange(n) // 50, len(cells) - 1)]
    stray = rng.random(n) < 0.03
    keys[stray] = cells[rng.integers(0, len(cells), int(stray.sum()))]
    return torch.from_numpy(keys.astype(np.uint32).view(np.int32)).to(DEVICE)


# ------------------------------------------------------------------------------------------- a pass


def _fields(out):
    return {"position": out["position"][:, :3], "velocity": out["velocity"][:, :3],
            "intermediate_velocity": out["intermediate_velocity"][:, :3], "density": out["density"],
            "pressure": out["pressure"], "grid_index": out["grid_index"].view(np.int32)}


def run(state):
    kind = state["kind"]
    if kind in ("steps", "batch", "learned"):
        gpu = state["gpu"]
        gpu.upload(state["in"])
        if kind == "learned":
            from libclsph_gb300 import learned as Lm

            Lm.step_learned(gpu, state["mlp"], state["count"], check=False)
        else:
            gpu.step(state["count"])
        return _fields(gpu.download(state["out"]))
    if kind == "forward":
        state["mlp"].forward(state["x"].data_ptr(), state["rows"], state["y"].data_ptr())
        return state["y"]
    if kind == "grads":
        grads, loss = state["mlp"].gradients(state["x"].data_ptr(), state["y"].data_ptr(), state["rows"])
        return {"gradients": grads, "loss": loss}
    rc = state["lib"].clsph_gpu_sort_keys_noalloc(state["keys"].data_ptr(), state["out"].data_ptr(),
                                                  state["perm"].data_ptr(), state["n"],
                                                  torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(f"sort_keys_noalloc: {rc}")
    return {"keys": state["out"], "perm": state["perm"]}


# ------------------------------------------------------------------------------------------- work


def work(case):
    kind = case["kind"]
    # a substep reads position, half-step velocity and velocity of each particle and writes them (72 B); about
    # 28 neighbours each cost 16 (density) and 65 (forces) operations
    step_bytes, step_flops = 72, 28 * 81 + 30
    mlp = 2 * (32 * 256 + 256 * 256 + 256 * 4)
    if kind in ("steps", "batch"):
        n = case["n"] if kind == "steps" else int(case["scenes"] * (case["n_max"] - 2048) / math.log(case["n_max"] / 2048))
        return {"bytes": n * (160 + step_bytes * case["substeps"]), "flops": n * step_flops * case["substeps"]}
    if kind == "learned":
        return {"bytes": case["n"] * (160 + step_bytes * case["steps"]),
                "flops": case["n"] * (step_flops + mlp) * case["steps"]}
    if kind == "forward":
        return {"bytes": case["rows"] * (64 + 16), "flops": case["rows"] * mlp}
    if kind == "grads":
        return {"bytes": case["rows"] * 144 + 2 * 4 * 75268, "flops": case["rows"] * (3 * mlp - 2 * 32 * 256)}
    return {"bytes": case["n"] * 12, "flops": 0}


# ------------------------------------------------------------------------------------------- in 64 bits


def _keys(pos, h):
    """Morton key of every particle as the substep defines it, in its own 32-bit arithmetic (the cell a
    particle falls into, and so the order of the records, is a decision in 32 bits)."""
    cell = np.float32(h * np.float32(2))
    lo = pos.min(0) - np.float32(cell * np.float32(2))
    c = ((pos - lo) / cell).astype(np.uint32).astype(np.uint64)

    def spread(v):
        v = (v | (v << 16)) & 0x030000FF
        v = (v | (v << 8)) & 0x0300F00F
        v = (v | (v << 4)) & 0x030C30C3
        return (v | (v << 2)) & 0x09249249

    return (spread(c[:, 0]) | (spread(c[:, 1]) << 1) | (spread(c[:, 2]) << 2)).astype(np.uint32), c


def _pairs(pos, h, visit):
    """visit(i, j, d, r) for all pairs with r < h (i == j among them), in slices; torch, 64 bits."""
    c = torch.floor((pos - pos.min(0).values) / h).long() + 1
    dims = c.max(0).values + 2
    flat = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    order = torch.argsort(flat)
    count = torch.bincount(flat, minlength=int(dims.prod()))
    start = torch.cumsum(count, 0) - count
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                f = flat + (dz * dims[1] + dy) * dims[0] + dx
                s, k = start[f], count[f]
                for m in range(int(k.max())):
                    i = torch.nonzero(k > m).flatten()
                    j = order[s[i] + m]
                    d = pos[i] - pos[j]
                    r = d.square().sum(1).sqrt()
                    near = r < h
                    visit(i[near], j[near], d[near], r[near])


def _collide(pos, vel, a, dt, vmax, restitution, mesh):
    """Leapfrog and collision loop against every face of a small mesh; torch, 64 bits."""
    v = torch.from_numpy(mesh["vertices"].reshape(-1, 3)).to(pos)
    tri = v[torch.from_numpy(mesh["indices"].astype(np.int64).reshape(-1, 3)).to(pos.device)]
    normals = torch.from_numpy(mesh["face_normals"].reshape(-1, 3)).to(pos)
    out_p, out_v = pos.clone(), vel.clone()
    live = torch.arange(len(pos), device=pos.device)
    left = torch.full((len(pos),), dt, dtype=pos.dtype, device=pos.device)
    for _ in range(64):
        p0, nv, rem = out_p[live], out_v[live] + a[live] * left[live, None], left[live]
        sp = nv.norm(dim=1, keepdim=True)
        nv = torch.where(sp > vmax, nv / sp * vmax, nv)
        p1 = p0 + nv * rem[:, None]
        d = p1 - p0
        best = torch.full_like(rem, math.inf)
        hit_p, hit_n = p1.clone(), torch.zeros_like(p1)
        for f in range(len(tri)):
            n = normals[f].expand_as(d)
            n = torch.where(((n * d).sum(1) <= 0)[:, None], -n, n)
            den = (n * d).sum(1)
            t = (n * (tri[f, 0] - p0)).sum(1) / den
            at = p0 + t[:, None] * d
            u, w, q = tri[f, 1] - tri[f, 0], tri[f, 2] - tri[f, 0], at - tri[f, 0]
            uu, uv, vv = u @ u, u @ w, w @ w
            qu, qv = q @ u, q @ w
            e = uv * uv - uu * vv
            s1, s2 = (uv * qv - vv * qu) / e, (uv * qu - uu * qv) / e
            dist = (at - p0).norm(dim=1)
            ok = (den != 0) & (t >= 0) & (t <= 1) & (s1 >= 0) & (s2 >= 0) & (s1 + s2 <= 1) & (dist <= best)
            best = torch.where(ok, dist, best)
            hit_p = torch.where(ok[:, None], at, hit_p)
            hit_n = torch.where(ok[:, None], n, hit_n)
        hit = torch.isfinite(best)
        depth = (p1 - hit_p).norm(dim=1)
        k = (1 + restitution * depth / (rem * nv.norm(dim=1))) * (nv * hit_n).sum(1)
        np_ = torch.where(hit[:, None], hit_p - 0.001 * hit_n, p1)
        nv = torch.where(hit[:, None], nv - k[:, None] * hit_n, nv)
        gone = torch.where(hit, rem * (np_ - p0).norm(dim=1) / d.norm(dim=1), rem)
        out_p[live], out_v[live], left[live] = np_, nv, rem - gone
        a[live] = 0.0
        live = live[hit]
        if not len(live):
            break
    return out_p, out_v


def _exact_substep(case, seed):
    params, terms, mesh, records, _ = _scene(case, seed)
    keys, _c = _keys(records["position"][:, :3], params["h"])
    order = np.argsort(keys, kind="stable")
    rec = records[order]

    def t64(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE).double()

    pos, vel, ivel = (t64(rec[f][:, :3]) for f in ("position", "velocity", "intermediate_velocity"))
    h, m, rho0 = float(params["h"]), float(params["particle_mass"]), float(params["fluid_density"])
    n = len(pos)
    rho = torch.zeros(n, dtype=torch.float64, device=pos.device)

    def density(i, j, d, r):
        rho.index_add_(0, i, m * float(terms["poly_6"]) * (h * h - r * r) ** 3)

    _pairs(pos, h, density)
    prs = float(params["K"]) * ((rho / rho0) ** 7 - 1)
    q = prs / rho ** 2
    P, V, N = (torch.zeros(n, 3, dtype=torch.float64, device=pos.device) for _ in range(3))
    L = torch.zeros_like(rho)

    def forces(i, j, d, r):
        mj, z = m / rho[j], h * h - r * r
        N.index_add_(0, i, mj[:, None] * float(terms["poly_6_gradient"]) * d * (z * z)[:, None])
        L.index_add_(0, i, mj * float(terms["poly_6_laplacian"]) * z * (3 * h * h - 7 * r * r))
        o = i != j
        i, j, d, r, mj = i[o], j[o], d[o], r[o], mj[o]
        P.index_add_(0, i, ((q[i] + q[j]) * m * float(terms["spiky"]) * (h - r) ** 2 / r)[:, None] * d)
        V.index_add_(0, i, (mj * float(terms["viscosity"]) * (h - r))[:, None] * (vel[j] - vel[i]))

    _pairs(pos, h, forces)
    total = V * float(params["dynamic_viscosity"]) - rho[:, None] * P
    nl = N.norm(dim=1, keepdim=True)
    surface = -float(params["surface_tension"]) * L[:, None] * N / nl
    total = total + torch.where(nl > float(params["surface_tension_threshold"]), surface, torch.zeros_like(N))
    g = t64(np.array(params["constant_acceleration"])[:3])
    dt = float(params["time_delta"]) * float(params["simulation_scale"])
    p1, v1 = _collide(pos, ivel, total / rho[:, None] + g, dt, float(params["max_velocity"]),
                      float(params["restitution"]), mesh)
    host = [x.cpu().numpy() for x in (p1, (ivel + v1) / 2, v1, rho, prs)]
    return dict(zip(("position", "velocity", "intermediate_velocity", "density", "pressure"), host),
                grid_index=keys[order].view(np.int32))


def _exact_mlp(x, blob):
    t = torch.from_numpy(blob).to(DEVICE).double()
    cuts = np.cumsum([32 * 256, 256, 256 * 256, 256, 256 * 4, 4])
    w1, b1, w2, b2, w3, b3 = (t[a:b].clone().requires_grad_(True) for a, b in zip(np.r_[0, cuts[:-1]], cuts))
    act = torch.nn.functional.gelu
    h1 = act(x @ w1.view(32, 256) + b1, approximate="tanh")
    h2 = act(h1 @ w2.view(256, 256) + b2, approximate="tanh")
    return h2 @ w3.view(256, 4) + b3, (w1, b1, w2, b2, w3, b3)


def exact(case, seed):
    kind = case["kind"]
    if kind == "steps" and case["substeps"] == 1 and case["state"] != "pour":
        return _exact_substep(case, seed)
    if kind == "forward":
        x, _ = _rows(case, seed)
        x, blob = x.to(torch.bfloat16), _blob()
        with torch.no_grad():
            y = torch.cat([_exact_mlp(c.double(), blob)[0] for c in x.split(65536)])
        return y * torch.from_numpy(blob[-4:]).to(y) + torch.from_numpy(blob[-8:-4]).to(y)
    if kind == "grads":
        x, g = _rows(case, seed)
        x, y = _raw(x, g)
        blob = _blob()
        t = torch.from_numpy(blob).to(DEVICE).double()
        std = ((x.double() - t[-72:-40]) / t[-40:-8]).clamp(-6, 6)
        out, parts = _exact_mlp(std, blob)
        loss = (out - (y.double() - t[-8:-4]) / t[-4:]).square().sum(1).mean()
        loss.backward()
        return {"gradients": torch.cat([p.grad.reshape(-1) for p in parts]).cpu().numpy(), "loss": float(loss.detach())}
    # sorted keys and permutations are whole numbers. After several substeps the records' order follows from
    # decisions in 32 bits at cell borders, so an exact state has no counterpart record by record; a collision
    # with a heightfield of 131,072 faces is out of reach of a plain restatement
    return None
