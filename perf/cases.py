"""Performance cases of the FLIP step: what programs that use this framework run, through its
public Python entry points, from the smallest scenes to the largest.

Kinds of case:
- ``step``: a simulation loop, one ``Batch.step(1)`` and the particles of that frame in pinned
  host buffers (``download_state``), a dam break at grid size ``n``.  A pass is one frame of a
  running simulation, so repeated passes go through successive frames.
- ``sphere``: the same loop on a dam break around a solid sphere, dt 1/480, with resampling and
  reseeding on every 5th frame.
- ``batch``: the loop over ``k`` scenes of uneven sizes stepped together.
- ``viewer``: ``FlipSim.Step`` and ``GetParticles`` with the default parameters (the reference's
  fp32 solver and stopping rule), as an interactive viewer calls them.
- ``solve``: the pressure solve as a solver call: a divergence field in, the pressure out, from a
  zero start; the cell types and liquid level set belong to the handle.
- ``transfer``: particles from pinned host buffers onto the staggered grid (sort and splat), and
  the face velocities back.
- ``levelset``: the level set of a frame's liquid surface, as an exporter takes it.
- ``serve``: requests through the request server until all are done, and their results.

Grid sizes, fill fractions and solver settings are those of the repository's workloads
(32^3-256^3, blocks filling 20-50% of the domain, 8 particles per cell, tolerance 1e-5 or 1e-7).
"""
import math

import numpy as np
import torch

from ariel_b200 import _abi as A
from ariel_b200 import workloads
from ariel_b200.flipsim import Batch, FlipSim, Server

PRECISIONS = {"ref32": A.PREC_REF32, "fp64": A.PREC_FP64, "mixed": A.PREC_MIXED}


def listed():
    return [
        # the smallest scene of the batch workload, alone: latency and launches
        {"name": "step-32-mixed", "kind": "step", "n": 32, "precision": "mixed", "hx": 0.4, "hy": 0.6},
        # the 64^3 dam break (0.5 M particles)
        {"name": "step-64-mixed", "kind": "step", "n": 64, "precision": "mixed", "hx": 0.4, "hy": 0.6},
        # an odd grid size on the plain double-precision path
        {"name": "step-77-fp64", "kind": "step", "n": 77, "precision": "fp64", "hx": 0.55, "hy": 0.5},
        # the 128^3 dam break (4 M particles), the benchmark's default line
        {"name": "step-128-mixed", "kind": "step", "n": 128, "precision": "mixed", "hx": 0.4, "hy": 0.6},
        # the 256^3 scene with the sphere (25 M particles): the largest single scene
        {"name": "sphere-256-mixed", "kind": "sphere", "n": 256, "precision": "mixed"},
        # eight uneven scenes in one launch per stage
        {"name": "batch-8-mixed", "kind": "batch", "k": 8, "set": 7, "precision": "mixed"},
        # an interactive viewer with the default parameters
        {"name": "viewer-48-ref32", "kind": "viewer", "n": 48, "hx": 0.4, "hy": 0.6},
        # the pressure solve alone, mixed precision at the usual tolerance
        {"name": "solve-64-mixed", "kind": "solve", "n": 64, "precision": "mixed", "tol": 1e-5, "hx": 0.5, "hy": 0.6},
        # the pressure solve alone, double precision at the tight tolerance
        {"name": "solve-120-fp64", "kind": "solve", "n": 120, "precision": "fp64", "tol": 1e-7, "hx": 0.45, "hy": 0.6},
        # particles to grid, host to host
        {"name": "transfer-96", "kind": "transfer", "n": 96, "hx": 0.45, "hy": 0.6},
        # the liquid surface of a frame for an exporter
        {"name": "levelset-96", "kind": "levelset", "n": 96, "hx": 0.45, "hy": 0.6},
        # a handful of small requests through the server
        {"name": "serve-6", "kind": "serve", "set": 11, "count": 6, "n_lo": 32, "n_hi": 64, "steps": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["sphere", "batch", "viewer", "solve", "solve", "transfer", "levelset", "serve"])
    fill = rng.uniform(0.2, 0.5)
    hy = round(rng.uniform(0.4, 0.8), 3)
    hx = round(min(0.95, fill / hy), 3)
    if kind == "step":
        return {"kind": kind, "n": _log_int(rng, 24, 160), "precision": rng.choice(["mixed", "mixed", "mixed", "fp64"]),
                "hx": hx, "hy": hy}
    if kind == "sphere":
        return {"kind": kind, "n": _log_int(rng, 48, 192), "precision": rng.choice(["mixed", "mixed", "fp64"])}
    if kind == "batch":
        case = {"kind": kind, "k": rng.randint(2, 8), "precision": rng.choice(["mixed", "mixed", "fp64"])}
        while True:  # a set of scenes of at most the largest listed case's particles
            case["set"] = rng.randrange(100000)
            if _batch_totals(case)[0] <= 24e6:
                return case
    if kind == "viewer":
        return {"kind": kind, "n": _log_int(rng, 24, 72), "hx": hx, "hy": hy}
    if kind == "solve":
        return {"kind": kind, "n": _log_int(rng, 32, 128), "precision": rng.choice(["mixed", "fp64"]),
                "tol": rng.choice([1e-5, 1e-7]), "hx": hx, "hy": hy}
    if kind in ("transfer", "levelset"):
        return {"kind": kind, "n": _log_int(rng, 32, 128), "hx": hx, "hy": hy}
    lo = rng.randint(24, 48)
    return {"kind": kind, "set": rng.randrange(100000), "count": rng.randint(2, 6), "n_lo": lo, "n_hi": lo + rng.randint(8, 32), "steps": rng.randint(6, 16)}


def _params(precision, tol=1e-5, **kw):
    p = A.params_default()
    p.precision = PRECISIONS[precision]
    p.stop_rule = A.STOP_REL
    p.tol = tol
    for k, v in kw.items():
        setattr(p, k, v)
    return p


def _frame_buffers(batch):
    """Pinned host buffers for every scene's frame, kept by the program between frames."""
    out = []
    for s in range(batch.k):
        m = batch.count(s)
        out.append(tuple(torch.empty((m, 3), dtype=torch.float32, pin_memory=True) for _ in range(2)))
    return [(p.numpy(), v.numpy(), p, v) for p, v in out]


def _running(descs, params, frames):
    """A simulation in progress: initialised and stepped past its first frames."""
    b = Batch(descs, params)
    b.init()
    b.step(frames)
    b.synchronize()
    return {"sim": b, "frame": _frame_buffers(b)}


def _block_particles(n, hx, hy, seed):
    """An evolved-looking liquid block: 8 particles per cell displaced by up to half a cell, a
    wavy free surface, a smooth velocity field with noise.  Unit coordinates, float32."""
    g = torch.Generator().manual_seed(seed)
    h = 0.5 / n
    ax = [torch.arange(int(round(2 * n * e)), dtype=torch.float64) for e in (hx, hy, 1.0)]
    p = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    p = (p + 0.5 + torch.rand(p.shape, generator=g, dtype=torch.float64) * 2.0 - 1.0) * h
    wave = hy * (0.9 + 0.1 * torch.sin(9.0 * p[:, 0] + 7.0 * p[:, 2] + 0.01 * seed))
    p = p[p[:, 1] < wave]
    p = p.clamp(1.0 / n, 1.0 - 1.0 / n)
    v = torch.stack([torch.sin(3 * p[:, 1]) + p[:, 0], -2.0 * p[:, 1], 0.5 * torch.cos(5 * p[:, 0])], -1)
    v = v + 0.1 * torch.randn(v.shape, generator=g, dtype=torch.float64)
    return p.float(), v.float()


def _fed(case, seed):
    """A handle whose particles come from the program."""
    pos, vel = _block_particles(case["n"], case["hx"], case["hy"], seed)
    b = Batch([workloads.dambreak(case["n"])], _params("mixed"))
    m = len(pos)
    b.set_particles(pos.numpy(), vel.numpy(), np.ones(m, np.float32), np.full(m, A.FLUID, np.int32))
    return b, pos, vel


def _pressure_problem(case, seed):
    """Cell types, liquid level set and negated divergence of a block of liquid with a wavy
    surface falling onto the floor, with turbulent noise.  (n, n, n) arrays."""
    n = case["n"]
    g = torch.Generator().manual_seed(seed)
    c = (torch.arange(n, dtype=torch.float64) + 0.5) / n
    x, y, z = torch.meshgrid(c, c, c, indexing="ij")
    depth_y = case["hy"] * (0.9 + 0.1 * torch.sin(9.0 * x + 7.0 * z + 0.01 * seed)) - y
    depth = torch.minimum(depth_y, case["hx"] - x) * n
    fluid = depth > 0
    # 1.6 in empty cells, below zero where particles are: -6.4 in the bulk, less at the surface
    lset = torch.where(fluid, -6.4 * (0.1 + depth).clamp(max=1.0), torch.full_like(depth, 1.6)).float()
    noise = torch.randn((n, n, n), generator=g, dtype=torch.float64)
    fall = torch.zeros_like(noise)
    fall[:, 0, :] = 9.8 / 240.0 * n
    div = torch.where(fluid, 0.02 * n * noise + fall, torch.zeros_like(noise)).float()
    return fluid, lset, div


def _serve_scenes(case, seed):
    rng = np.random.default_rng(case["set"])  # sizes and blocks; the seed only moves the particles
    out = []
    for i in range(case["count"]):
        hy = float(rng.uniform(0.4, 0.8))
        hx = float(min(0.95, rng.uniform(0.2, 0.5) / hy))
        out.append(A.scene_dambreak(int(rng.integers(case["n_lo"], case["n_hi"] + 1)), liquid_hi=(hx, hy, 1.0),
                                    seed=int(seed) * 100 + i))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        d = A.scene_dambreak(case["n"], liquid_hi=(case["hx"], case["hy"], 1.0), seed=seed + 1)
        s = _running([d], _params(case["precision"]), 6)
    elif kind == "sphere":
        s = _running([workloads.sphere_dambreak(case["n"], seed=seed + 1)],
                     _params(case["precision"], resample_every=5, reseed_every=5), 6)
    elif kind == "batch":
        # the set gives the scenes' sizes and blocks; the seed only moves their particles
        descs = workloads.uneven_batch(case["k"], seed=case["set"])
        for i, d in enumerate(descs):
            d.seed = seed * 1000 + i + 1
        s = _running(descs, _params(case["precision"]), 3)
    elif kind == "viewer":
        d = A.scene_dambreak(case["n"], liquid_hi=(case["hx"], case["hy"], 1.0), seed=seed + 1)
        sim = FlipSim(case["n"], 0.5, 1.0 / 240.0, d)
        sim.Init()
        for _ in range(6):
            sim.Step(False, False, False)
        s = {"sim": sim}
    elif kind == "solve":
        fluid, lset, div = _pressure_problem(case, seed)
        d = A.scene_dambreak(case["n"])
        d.n_liquid = 0
        b = Batch([d], _params(case["precision"], case["tol"]))
        b.init()
        b.set_grid(A.GRID_A, fluid.to(torch.int32).numpy())
        b.set_grid(A.GRID_L, lset.numpy())
        s = {"sim": b, "div": div.numpy(), "zero": np.zeros(div.shape, np.float64)}
    elif kind == "transfer":
        b, pos, vel = _fed(case, seed)
        s = {"sim": b, "pos": pos.pin_memory(), "vel": vel.pin_memory()}
    elif kind == "levelset":
        s = {"sim": _fed(case, seed)[0]}
    else:
        s = {"sim": Server(_params("mixed")), "scenes": _serve_scenes(case, seed), "steps": case["steps"]}
    s["kind"] = kind
    return s


def run(state):
    kind, sim = state["kind"], state["sim"]
    if kind in ("step", "sphere", "batch"):
        sim.step(1)
        for i, (p, v, _, _) in enumerate(state["frame"]):
            sim.download_state(p, v, i)
        return [(p, v) for _, _, p, v in state["frame"]]
    if kind == "viewer":
        sim.Step(False, False, False)
        return sim.GetParticles()
    if kind == "solve":
        sim.set_grid(A.GRID_D, state["div"])
        sim.set_grid(A.GRID_P64, state["zero"])
        sim.stage(A.STAGE_SOLVE)
        return sim.get_grid(A.GRID_P)
    if kind == "transfer":
        sim.upload_state(state["pos"].numpy(), state["vel"].numpy())
        sim.stage(A.STAGE_SORT)
        sim.stage(A.STAGE_P2G)
        return [sim.get_grid(g) for g in (A.GRID_UX, A.GRID_UY, A.GRID_UZ)]
    if kind == "levelset":
        return sim.level_set()
    ids = [sim.submit(d, state["steps"]) for d in state["scenes"]]
    for r in ids:
        sim.wait(r)
    out = [sim.fetch(r) for r in ids]
    for r in ids:
        sim.release(r)
    return out


def _liquid(n, hx, hy):
    """(particles, liquid cells) of a block at 8 particles per cell."""
    cells = hx * hy * n ** 3
    return 8.0 * cells, cells


def _batch_totals(case):
    """(particles, liquid cells, grid cells) of a batch case's scenes."""
    tot = [0.0, 0.0, 0.0]
    for d in workloads.uneven_batch(case["k"], seed=case["set"]):
        m, cells = _liquid(d.dim, d.liquid[0].hi[0], d.liquid[0].hi[1])
        tot = [tot[0] + m, tot[1] + cells, tot[2] + d.dim ** 3]
    return tot


def work(case):
    """Bytes: particle state in and out (24 bytes each way), what a stage hands to the next one
    through memory once, host results once.  Flops: the particle neighbourhoods (about 64 pairs a
    particle within two cells' reach of the density kernel's half, 30 of the splat) and, for a
    solve, 20 operations a liquid cell and iteration at 2 n iterations."""
    kind = case["kind"]

    def step(m, cells, n):
        return 96.0 * m + 60.0 * n ** 3, 1500.0 * m + 20.0 * cells * 2.0 * n

    if kind in ("step", "viewer"):
        m, cells = _liquid(case["n"], case["hx"], case["hy"])
        b, f = step(m, cells, case["n"])
    elif kind == "sphere":
        m, cells = _liquid(case["n"], 0.35, 0.5)
        b, f = step(m, cells, case["n"])
    elif kind == "batch":
        m, cells, grid = _batch_totals(case)
        b, f = step(m, cells, grid ** (1.0 / 3.0))
    elif kind == "solve":
        _, cells = _liquid(case["n"], case["hx"], case["hy"])
        b, f = 24.0 * case["n"] ** 3, 20.0 * cells * 2.0 * case["n"]
    elif kind == "transfer":
        m, cells = _liquid(case["n"], case["hx"], case["hy"])
        b, f = 24.0 * m + 12.0 * case["n"] ** 3, 1000.0 * m
    elif kind == "levelset":
        m, cells = _liquid(case["n"], case["hx"], case["hy"])
        b, f = 12.0 * m + 4.0 * (case["n"] + 5) ** 3, 300.0 * m
    else:
        n = 0.5 * (case["n_lo"] + case["n_hi"])
        m, cells = _liquid(n, 0.58, 0.6)
        b, f = step(m, cells, n)
        b, f = b * case["count"] * case["steps"], f * case["count"] * case["steps"]
    return {"bytes": b, "flops": f}


# ---- the same results in 64 bits, by torch alone --------------------------------------------
def _exact_solve(case, seed):
    """Conjugate gradients on the 7-point operator to 1e-12: liquid neighbours off the diagonal,
    walls left out, air neighbours at the ghost-fluid distance."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    fluid, lset, div = (t.to(dev) for t in _pressure_problem(case, seed))
    n = case["n"]
    lset, b = lset.double(), torch.where(fluid, div.double(), torch.zeros((), dtype=torch.float64, device=dev))

    def shifted(t, dim, by, fill):
        out = torch.full_like(t, fill)
        src, dst = [slice(None)] * 3, [slice(None)] * 3
        src[dim], dst[dim] = (slice(1, None), slice(None, -1)) if by > 0 else (slice(None, -1), slice(1, None))
        out[tuple(dst)] = t[tuple(src)]
        return out

    diag = torch.zeros_like(lset)
    sides = [(d, s) for d in range(3) for s in (-1, 1)]
    inside = torch.ones_like(fluid)
    for d, s in sides:
        there = shifted(inside, d, s, False)
        wet = shifted(fluid, d, s, False)
        air = there & ~wet
        diag += there.double()
        diag -= torch.where(air, shifted(lset, d, s, 0.0) / torch.clamp(lset, max=1e-6), torch.zeros_like(diag))

    def apply(v):
        out = diag * v
        for d, s in sides:
            out = out - shifted(v, d, s, 0.0)
        return torch.where(fluid, out * float(n) ** 2, torch.zeros_like(v))

    inv = torch.where(fluid, 1.0 / diag, torch.zeros_like(diag))
    x = torch.zeros_like(b)
    r = b.clone()
    z = r * inv
    p = z.clone()
    rz = (r * z).sum()
    stop = 1e-24 * (b * b).sum()
    for it in range(20 * n):
        q = apply(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if it % 16 == 15 and bool((r * r).sum() <= stop):
            break
        z = r * inv
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x.cpu()


def _exact_transfer(case, seed):
    """Face velocities: the Sharpen-weighted mean over the particles within 1.4 cells of the face
    centre, of the two cell layers that share the face."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = case["n"]
    pos, vel = (t.to(dev).double() for t in _block_particles(n, case["hx"], case["hy"], seed))
    gp = (pos * n).clamp(0.0, float(n))
    cell = (pos.float() * n).long().clamp(0, n - 1)  # cells are defined by the fp32 product
    out = []
    for axis in range(3):
        ext = [n + (a == axis) for a in range(3)]
        num = torch.zeros(ext[0] * ext[1] * ext[2], dtype=torch.float64, device=dev)
        den = torch.zeros_like(num)
        offs = [[(o, 0.0) for o in (0, 1)] if a == axis else [(o, 0.5) for o in (-2, -1, 0, 1, 2)] for a in range(3)]
        for ox, cx in offs[0]:
            for oy, cy in offs[1]:
                for oz, cz in offs[2]:
                    f = [cell[:, 0] + ox, cell[:, 1] + oy, cell[:, 2] + oz]
                    r2 = sum((gp[:, a] - (f[a].double() + c)) ** 2 for a, c in zip(range(3), (cx, cy, cz)))
                    w = (1.4 * 1.4 / r2.clamp(min=1e-5) - 1.0).clamp(min=0.0)
                    ok = w > 0
                    for a in range(3):
                        ok &= (f[a] >= 0) & (f[a] < ext[a])
                    idx = ((f[0] * ext[1] + f[1]) * ext[2] + f[2])[ok]
                    num.index_add_(0, idx, (w * vel[:, axis])[ok])
                    den.index_add_(0, idx, w[ok])
        out.append(torch.where(den > 0, num / den, torch.zeros_like(num)).reshape(ext).cpu())
    return out


def _exact_levelset(case, seed):
    """Distance to the nearest particle less half a cell, up to 1.5, on the grid points padded by
    two cells."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = case["n"]
    N = n + 5
    q = _block_particles(n, case["hx"], case["hy"], seed)[0].to(dev).double() * n
    phi = torch.full((N * N * N,), 1.5, dtype=torch.float64, device=dev)
    base = torch.floor(q).long()
    for i in range(-2, 4):
        for j in range(-2, 4):
            for k in range(-2, 4):
                g = base + torch.tensor([i, j, k], device=dev)
                d = ((g.double() - q) ** 2).sum(1).sqrt()
                at = g + 2
                ok = (d < 2.0) & ((at >= 0) & (at < N)).all(1)
                idx = (at[:, 0] * N + at[:, 1]) * N + at[:, 2]
                phi.scatter_reduce_(0, idx[ok], d[ok] - 0.5, "amin")
    return phi.reshape(N, N, N).cpu()


def exact(case, seed):
    """64-bit results where the inputs are given numbers; a running simulation's next frame
    depends on its whole history and has none."""
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "transfer":
        return _exact_transfer(case, seed)
    if case["kind"] == "levelset":
        return _exact_levelset(case, seed)
    return None
