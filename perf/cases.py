"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public entry points of `libfluid_gb300.solver`:

  frame      `SphSolver.advance`: the drop-in, one frame on the caller's own host arrays, in place
  records    `SphSolver.advance_records`: the same on an array of particle records, with cell queries
  resident   `Batch.step` on one resident scene, some steps and one readback
  batched    `Batch.step` on several scenes of different sizes at once, and their readbacks
  surface    `Batch.step`, `Batch.surface` and `weld`: one step, its mesh, and the mesh as an index buffer

A scene is a block of particles at the corner of a box (a dam break), at rest or already in motion.
The state moves on with every pass, as it does in a program that runs a simulation.
"""
import numpy as np
import torch

from libfluid_gb300 import capi, scenes
from libfluid_gb300.solver import Batch, SphSolver
from libfluid_gb300.weld import weld

H = 0.1
#: neighbours within h of a particle at rest density, for the operation counts
NEIGHBOURS = 34
BOX = (2.0, 1.5, 1.5)  # the box, in block extents


def _case(kind, nx, ny, nz, profile="baseline", steps=1, iterations=4, moving=False, sphere=False, obstacles=0,
          wells=0, surface=False, queries=0, count=1, tuned=False):
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "profile": profile, "steps": steps, "iterations": iterations,
            "moving": moving, "sphere": sphere, "obstacles": obstacles, "wells": wells, "surface": surface,
            "queries": queries, "scenes": count, "tuned": tuned}


def listed():
    return [
        # the smallest frames: an interactive toy scene, where latency and launches count
        {"name": "frame_4k", **_case("frame", 16, 16, 16)},
        # the drop-in as a libfluid application has it by default: the reference's constants, five
        # iterations and a surface every frame, with obstacles and a gravity well; an odd size
        {"name": "frame_ref_50k", **_case("frame", 37, 37, 37, "ref", iterations=5, obstacles=13, wells=1,
                                          surface=True)},
        # the benchmark's dam break onto a sphere, host arrays in and out every frame
        {"name": "frame_1m", **_case("frame", 128, 64, 128, sphere=True)},
        # the C++ adapter's path: records in place, with cell queries, a flow in motion, an odd size
        {"name": "records_ref_250k", **_case("records", 63, 63, 63, "ref", iterations=5, moving=True, queries=8)},
        # a small resident scene read back every sixteen steps: bound by the launches of a step
        {"name": "resident_14k", **_case("resident", 24, 24, 24, steps=16)},
        # an ordinary resident scene in violent motion, with obstacles among the fluid
        {"name": "resident_262k", **_case("resident", 64, 64, 64, steps=8, moving=True, obstacles=29)},
        # the benchmark's scene resident on the device, launch shapes tuned first as a long run does
        {"name": "resident_1m", **_case("resident", 128, 64, 128, steps=8, sphere=True, tuned=True)},
        # the reference's constants on a resident scene: the fluid clumps, rows of neighbours are long
        {"name": "resident_ref_120k", **_case("resident", 61, 43, 47, "ref", steps=6, iterations=5, moving=True)},
        # many scenes of a simulation service stepped together, sizes log-uniform
        {"name": "batched_16", **_case("batched", 20, 0, 64, steps=5, count=16)},
        # one step and its mesh as an index buffer, as a renderer takes it
        {"name": "surface_205k", **_case("surface", 59, 59, 59, moving=True, surface=True)},
        # the largest: a scene whose arrays exceed the L2 cache
        {"name": "resident_4m", **_case("resident", 128, 128, 256, steps=2)},
    ]


def draw(rng):
    kind = rng.choice(["frame", "frame", "records", "resident", "resident", "resident", "batched", "surface"])
    ref = kind == "records" or rng.random() < 0.35
    lo, hi = {"frame": (12, 100), "records": (16, 90), "resident": (16, 128), "batched": (16, 56),
              "surface": (16, 64)}[kind]

    def side():
        return int(round(lo * (hi / lo) ** rng.random()))

    n = side()
    dims = [max(lo, min(hi, int(round(n * 2.0 ** rng.uniform(-0.7, 0.7))))) for _ in range(3)]
    if kind == "batched":
        dims = [lo, 0, max(lo + 4, dims[2])]
    return _case(kind, *dims, profile="ref" if ref else "baseline",
                 steps=rng.choice([1, 2, 3, 5]) if kind in ("resident", "batched") else 1,
                 iterations=rng.choice([2, 3, 4, 4, 5, 5, 6]), moving=rng.random() < 0.5,
                 sphere=not ref and kind != "batched" and rng.random() < 0.4,
                 obstacles=rng.choice([0, 0, 7, 13, 29]), wells=rng.choice([0, 0, 1, 3]),
                 surface=kind == "surface" or (kind in ("frame", "records") and rng.random() < 0.3),
                 queries=rng.choice([0, 3, 8]) if kind == "records" else 0,
                 count=rng.choice([2, 5, 9, 16]) if kind == "batched" else 1)


# ---------------------------------------------------------------- inputs


def _scene_sides(case, rng):
    """Block dimensions of a case's scenes (particles a side)."""
    if case["kind"] != "batched":
        return [(case["nx"], case["ny"], case["nz"])]
    lo, hi = case["nx"], case["nz"]
    u = (np.arange(case["scenes"]) + 0.5) / case["scenes"]  # log-uniform cubes, a fixed spread of sizes
    sides = np.rint(lo * (hi / lo) ** u).astype(int)
    return [(int(s), int(s), int(s)) for s in rng.permutation(sides)]


def _particles(case, dims, rng):
    """A lattice block of fluid with jitter; in motion: a swirl and noise on its velocities."""
    n = dims[0] * dims[1] * dims[2]
    axes = [(np.arange(d, dtype=np.float32) + np.float32(0.5)) * np.float32(scenes.SPACING) for d in dims]
    pos = np.stack(np.meshgrid(*axes, indexing="ij"), axis=-1).reshape(n, 3)
    jitter = 0.012 if case["moving"] else scenes.JITTER
    pos += (rng.random((n, 3), np.float32) * np.float32(2) - np.float32(1)) * np.float32(jitter)
    if case["moving"]:
        k = np.float32(2 * np.pi / (max(dims) * scenes.SPACING))
        swirl = np.stack([np.sin(k * pos[:, 1]), np.sin(2 * k * pos[:, 2]), np.cos(k * pos[:, 0])], axis=1)
        vel = (swirl + np.float32(0.3) * (rng.random((n, 3), np.float32) - np.float32(0.5))).astype(np.float32)
    else:
        vel = np.zeros((n, 3), np.float32)
    kind = np.full(n, capi.TYPE_FLUID, np.int32)
    if case["obstacles"]:
        kind[:: case["obstacles"]] = capi.TYPE_OBSTACLE
    return {"id": np.arange(n, dtype=np.uint64), "type": kind, "mass": np.full(n, scenes.MASS, np.float32),
            "position": pos.ravel(), "velocity": vel.ravel(),
            "colour": rng.integers(0, 1 << 32, n, dtype=np.uint32)}


def _config(case, dims):
    ext = [d * scenes.SPACING for d in dims]
    box = [max(b * e, e + 0.4) for b, e in zip(BOX, ext)]
    sphere = (1.25 * ext[0], 0.15 * ext[1], 0.5 * ext[2], 0.15 * min(ext)) if case["sphere"] else None
    profile = capi.PROFILE_REF if case["profile"] == "ref" else capi.PROFILE_BASELINE
    cfg = scenes.config((0.0, 0.0, 0.0), box, sphere, case["iterations"], 1 if case["surface"] else 0, profile)
    cfg.n_wells = case["wells"]
    for w in range(case["wells"]):
        cfg.wells[w].centre[:] = ((0.3 + 0.2 * w) * box[0], 0.5 * box[1], 0.4 * box[2])
        cfg.wells[w].force = 2.0 + w
    return cfg


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    return [(_particles(case, d, rng), _config(case, d)) for d in _scene_sides(case, rng)]


def prepare(case, seed):
    profile = capi.PROFILE_REF if case["profile"] == "ref" else capi.PROFILE_BASELINE
    solver = SphSolver(h=H, profile=profile)
    s = {"case": case, "solver": solver}
    made = _inputs(case, seed)
    if case["surface"]:  # the buffers a renderer fills frame after frame, larger than any mesh of the scene
        room = 4096 + sum(len(parts["mass"]) for parts, _ in made)
        s["vertices"], s["mesh_colours"] = np.zeros((room, 18), np.float32), np.zeros((room, 3), np.int32)
        s["index"], s["welded"] = np.zeros(3 * room, np.int32), np.zeros((3 * room, 3), np.float32)
        s["filled"] = {}
    if case["kind"] == "frame":
        s["particles"], s["config"] = made[0]
    elif case["kind"] == "records":
        parts, s["config"] = made[0]
        s["records"] = capi.to_records(parts)
        p = parts["position"].reshape(-1, 3)
        pick = np.random.default_rng(seed + 1).integers(0, len(p), case["queries"])
        s["queries"] = [(int(i), tuple(float(c) for c in p[i])) for i in pick]
    else:
        s["batch"] = batch = Batch(solver, made)
        if case["tuned"]:
            batch.autotune()
            for k, (parts, _) in enumerate(made):
                batch.upload(k, parts)
    return s


# ---------------------------------------------------------------- one pass


def _fill(s, name, rows):
    """`rows` into the front of the state's buffer, which is zero behind them."""
    buffer, before = s[name], s["filled"].get(name, 0)
    buffer[: len(rows)] = rows
    buffer[len(rows) : before] = 0
    s["filled"][name] = len(rows)
    return buffer


def _signed(fields):
    """The same bytes as signed integers where they are unsigned."""
    return {k: v.view(v.dtype.str.replace("u", "i")) if v.dtype.kind == "u" else v for k, v in fields.items()}


def run(s):
    case = s["case"]
    if case["kind"] == "frame":
        mesh = s["solver"].advance(s["config"], s["particles"])
        out = {"particles": _signed(s["particles"])}
    elif case["kind"] == "records":
        mesh, found = s["solver"].advance_records(s["config"], s["records"], queries=s["queries"])
        rec = s["records"]
        out = {"particles": _signed({f: rec[f] for f in rec.dtype.names})}
        answers = np.zeros((case["queries"], 3), np.int64)
        answers[: len(found)] = np.array([(q, n, c) for q, _, n, c in found], np.int64).reshape(-1, 3)
        out["queries"] = answers
    else:
        batch = s["batch"]
        batch.step(case["steps"])
        mesh = batch.surface(0) if case["surface"] else None
        got = [batch.download(k) for k in range(batch.n_scenes)]
        out = {"particles": _signed(got[0] if len(got) == 1 else scenes.concat(got))}
        if mesh is not None:
            index, vertices = weld(mesh)
            out["index"], out["welded"] = _fill(s, "index", index.view(np.int32)), _fill(s, "welded", vertices)
    if mesh is not None:
        out["vertices"] = _fill(s, "vertices", mesh[:, :18])
        out["colours"] = _fill(s, "mesh_colours", mesh[:, 18:].view(np.int32))
    return out


def work(case):
    """Each particle's state in and out once, and the pair sums of a step over the neighbours within h."""
    if case["kind"] == "batched":
        dims = _scene_sides(case, np.random.default_rng(0))
    else:
        dims = [(case["nx"], case["ny"], case["nz"])]
    n = sum(a * b * c for a, b, c in dims)
    pair = 52 * case["iterations"] + (0 if case["profile"] == "ref" else 60)
    return {"bytes": 88 * n, "flops": n * case["steps"] * NEIGHBOURS * pair}


# ---------------------------------------------------------------- the same in 64 bits


def _cells32(p, cfg):
    """Grid cells of predicted positions, decided in 32 bits as the interface defines them."""
    h = np.float32(H)
    cell = np.empty(p.shape, np.int64)
    ext = []
    for a in range(3):
        mn = np.float32(cfg.min_bound[a]) / np.float32(cfg.scale) - h * np.float32(2)
        mx = np.float32(cfg.max_bound[a]) / np.float32(cfg.scale) + h * np.float32(2)
        e = int((mx - mn) / h)
        cell[:, a] = np.clip(np.trunc((p[:, a] - mn) / h), 0, e).astype(np.int64)
        ext.append(e)
    return cell, ext


def _morton(cell):
    key = np.zeros(len(cell), np.int64)
    for b in range(10):
        for a in range(3):
            key |= ((cell[:, a] >> b) & 1) << (3 * b + a)
    return key


def _predict(parts, cfg, ref, t):
    """Predicted positions in the type `t`, in the reference's order of operations."""
    dt, scale = t(cfg.dt), t(cfg.scale)
    x, v = parts["position"].reshape(-1, 3).astype(t), parts["velocity"].reshape(-1, 3).astype(t)
    m = parts["mass"].astype(t)[:, None]
    f = np.array(list(cfg.constant_force), np.float32).astype(t)[None, :] * (m if ref else np.ones_like(m))
    for w in range(cfg.n_wells):
        c = np.array(list(cfg.wells[w].centre), np.float32).astype(t)
        u = c - x
        d = x - c
        dist = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])[:, None]
        with np.errstate(all="ignore"):
            pull = (u / dist) * t(cfg.wells[w].force)
            pull = (pull * m if ref else pull) / (dist * dist)
        f = f + np.where(dist < t(75), np.clip(pull, t(-10), t(10)), t(0))
    p = (f * dt + v) * dt + x / scale
    return np.where((parts["type"] == capi.TYPE_OBSTACLE)[:, None], x / scale, p)


class _Pairs:
    """Every ordered pair (a, b) of particles in neighbouring cells, an offset of cells at a time."""

    def __init__(self, cell, ext, dev):
        size = [e + 1 for e in ext]
        flat = (cell[:, 0] * size[1] + cell[:, 1]) * size[2] + cell[:, 2]
        self.dev = dev
        self.cell, self.size = torch.from_numpy(cell).to(dev), size
        self.flat, self.order = torch.sort(torch.from_numpy(flat).to(dev))

    def __iter__(self):
        c = self.cell
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    q = c + torch.tensor([dx, dy, dz], device=self.dev)
                    ok = ((q >= 0) & (q < torch.tensor(self.size, device=self.dev))).all(1)
                    at = torch.where(ok, (q[:, 0] * self.size[1] + q[:, 1]) * self.size[2] + q[:, 2], -1)
                    lo, hi = torch.searchsorted(self.flat, at), torch.searchsorted(self.flat, at, right=True)
                    count = torch.where(ok, hi - lo, torch.zeros_like(lo))
                    a = torch.repeat_interleave(torch.arange(len(c), device=self.dev), count)
                    first = torch.cumsum(count, 0) - count
                    b = self.order[torch.arange(len(a), device=self.dev) - first[a] + lo[a]]
                    yield a, b


def _step64(parts, cfg, profile):
    """One step in 64 bits: (order, positions, velocities), sorted as the step returns them."""
    ref = profile == "ref"
    prm = capi.default_params(capi.PROFILE_REF if ref else capi.PROFILE_BASELINE, H)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    h = float(np.float32(H))
    hh, dt, scale = h * h, float(cfg.dt), float(cfg.scale)
    poly, spiky = 315 / (64 * np.pi * h ** 9), -45 / (np.pi * h ** 6)
    rho0, cfm, dq = float(prm.rho0), float(prm.cfm_epsilon), float(prm.corr_delta_q) * h
    wdq = (hh - dq * dq) ** 3
    corr_k = float(prm.corr_k) * (1 if ref else hh)
    cell, ext = _cells32(_predict(parts, cfg, ref, np.float32), cfg)
    order = np.argsort(_morton(cell), kind="stable")
    pairs = _Pairs(cell, ext, dev)
    put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)  # noqa: E731
    p = put(_predict(parts, cfg, ref, np.float64))
    x, v = put(parts["position"].reshape(-1, 3).astype(np.float64)), put(parts["velocity"].reshape(-1, 3).astype(np.float64))
    m = put(parts["mass"].astype(np.float64))
    fluid = put(parts["type"] != capi.TYPE_OBSTACLE)
    lo, hi = (torch.tensor(list(b), dtype=torch.float64, device=dev) for b in (cfg.min_bound, cfg.max_bound))
    n = len(m)

    def near(p):
        for a, b in pairs:
            d = p[a] - p[b]
            r2 = (d * d).sum(1)
            keep = r2 <= hh
            a, b, d, r2 = a[keep], b[keep], d[keep], r2[keep]
            r = r2.sqrt()
            s = torch.where(r >= 1e-8, (h - r) ** 2 / r.clamp_min(1e-8), torch.zeros_like(r))
            yield a, b, d, (hh - r2) ** 3, s

    zeros = lambda *k: torch.zeros(n, *k, dtype=torch.float64, device=dev)  # noqa: E731
    for _ in range(cfg.iterations):
        rho, g, g2 = zeros(), zeros(3), zeros()
        for a, b, d, w, s in near(p):
            rho.index_add_(0, a, (m[a] if ref else m[b]) * poly * w)
            k = (s if ref else m[b] * s) * (spiky / rho0)
            g.index_add_(0, a, k[:, None] * d)
            if not ref:
                g2.index_add_(0, a, k * k * (d * d).sum(1))
        lam = torch.where(fluid, -(rho / rho0 - 1) / ((g * g).sum(1) + g2 + cfm), zeros())
        move = zeros(3)
        for a, b, d, w, s in near(p):
            c = -corr_k * (w / wdq) ** float(prm.corr_n)
            k = (1 if ref else m[b]) * s * (spiky / rho0) * (lam[a] + lam[b] + c)
            move.index_add_(0, a, k[:, None] * d)
        q = (p + move) * scale
        if cfg.sphere_enabled and not ref:
            centre = torch.tensor(list(cfg.sphere)[:3], dtype=torch.float64, device=dev)
            away = q - centre
            dist = away.norm(dim=1, keepdim=True)
            q = torch.where(dist < cfg.sphere[3], centre + away * (cfg.sphere[3] / dist), q)
        q = torch.minimum(torch.maximum(q, lo), hi) / scale
        p = torch.where(fluid[:, None], q, p)
    shift = (p - x / scale) / dt
    if ref:
        vel = (shift + v) * float(prm.velocity_damping)
    else:
        vel = torch.where(fluid[:, None], shift, v)
        xs, om = zeros(3), zeros(3)
        for a, b, d, w, s in near(p):
            live = (fluid[b]).double()
            u = vel[b] - vel[a]
            xs.index_add_(0, a, (live * m[b] * w)[:, None] * u)
            om.index_add_(0, a, (live * m[b] * s)[:, None] * torch.linalg.cross(u, d))
        om = torch.where(fluid[:, None], -om * (spiky / rho0), zeros(3))
        size = om.norm(dim=1)
        eta = zeros(3)
        for a, b, d, w, s in near(p):
            eta.index_add_(0, a, (fluid[b].double() * m[b] * s * (size[b] - size[a]))[:, None] * d)
        eta = eta * (spiky / rho0)
        length = eta.norm(dim=1, keepdim=True)
        eta = torch.where(length > 0, eta / length, zeros(3))
        vel = vel + float(prm.xsph_c) * xs * (poly / rho0) + dt * float(prm.vorticity_epsilon) * torch.linalg.cross(eta, om)
    vel = torch.where(fluid[:, None], vel, v)
    pos = torch.where(fluid[:, None], p * scale, x)
    return order, pos.cpu().numpy()[order], vel.cpu().numpy()[order]


def exact(case, seed):
    """Positions and velocities after one step.  Over several steps the flow is chaotic and the order is
    decided in 32 bits at each; a mesh's triangles come from comparisons with the iso level: no value for those."""
    if case["steps"] != 1:
        return None
    done = [_step64(parts, cfg, case["profile"]) for parts, cfg in _inputs(case, seed)]
    pos, vel = (np.concatenate([d[k] for d in done]) for k in (1, 2))
    if case["kind"] != "records":
        pos, vel = pos.ravel(), vel.ravel()
    return {"particles": {"position": pos, "velocity": vel}}
