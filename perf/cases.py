"""The workloads this engine is timed on, through its public entry points.

Seven of them advance a PUFFY run the way a host program does that keeps its own
fields: the host's p, u and flags go up, the engine takes some steps (the CFL dt,
or a dt given by the caller), the diagnostics row is read, and p, u and flags come
back. They go from the 32x30 grid of the regression scenario to the 192x180x64
wedge, with the step eager and as a graph, plain FP64 and mixed, with and without
the bisection warm start. The others are the batched implicit solve over
independent cells, the batched conserved -> primitive inversion, a restart from a
checkpoint, and the start of a new run.
"""
import importlib.util
import math
import os

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NV, NFLAGS = 13, 6
PER_CELL, SORTED, ITERS = 0, 3, 5  # forms of the batched implicit solve
GAM = 5.0 / 3.0

_engine = None


def engine():
    global _engine
    if _engine is None:
        spec = importlib.util.spec_from_file_location("koralcuda", os.path.join(ROOT, "koral-zig_b200", "koralcuda.py"))
        _engine = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(_engine)
    return _engine


# ---- the cases ---------------------------------------------------------------


def _steps(name, nx, ny, nz, steps, graph=True, mixed=False, bisect=True, forced=False):
    case = {"kind": "steps", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "graph": graph, "mixed": mixed,
            "bisect": bisect, "forced": forced}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the regression scenario's grid: the smallest run there is, all launches and latency
        _steps("run_2d_32x30", 32, 30, 1, 8),
        # a ragged 2D grid stepped eagerly with the caller's dt, as a comparison against another code does
        _steps("run_2d_101x75_eager", 101, 75, 1, 4, graph=False, forced=True),
        # the 2D production grid
        _steps("run_2d_384x360", 384, 360, 1, 6),
        # the small 3D wedge of the step goldens, eager (a short run never replays a graph)
        _steps("run_3d_32x30x4_eager", 32, 30, 4, 4, graph=False),
        # a ragged 3D wedge in the mixed form
        _steps("run_3d_97x61x13_mixed", 97, 61, 13, 4, mixed=True),
        # a medium wedge with the solve started from the pre-solve state
        _steps("run_3d_128x96x24_nobisect", 128, 96, 24, 4, bisect=False),
        # the 3D wedge that the engine is built for
        _steps("run_3d_192x180x64", 192, 180, 64, 4),
        # the implicit solve over independent cells resident on the device: as many as the reference's battery
        # has records, where a call lasts as long as its slowest cell
        {"name": "solve_336", "kind": "solve", "n": 336, "mode": PER_CELL},
        # and as many as fill the device, in the form made for them
        {"name": "solve_65537_iters", "kind": "solve", "n": 65537, "mode": ITERS},
        # the inversion of conserved variables over host arrays
        {"name": "invert_100003", "kind": "invert", "n": 100003},
        # a restart: load a checkpoint, fill the ghosts, report, write the next checkpoint
        {"name": "restart_192x180x8", "kind": "restart", "nx": 192, "ny": 180, "nz": 8},
        # a new run: torus, atmosphere, field and normalisation on an existing handle
        {"name": "start_192x180x4", "kind": "start", "nx": 192, "ny": 180, "nz": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, most):
    """A grid of at most `most` cells: sizes over their logarithm, 2D and 3D alike often."""
    while True:
        nx, ny = _log(rng, 24, 384), _log(rng, 20, 360)
        nz = 1 if rng.random() < 0.5 else _log(rng, 4, 64)
        if nx * ny * nz <= most:
            return nx, ny, nz


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["solve", "solve", "invert", "restart", "start"])
    if kind == "steps":
        nx, ny, nz = _grid(rng, 192 * 180 * 64)
        steps = rng.randint(1, 4)
        return _steps(None, nx, ny, nz, steps, graph=rng.random() < 0.6, mixed=rng.random() < 0.25,
                      bisect=rng.random() < 0.75, forced=rng.random() < 0.25)
    if kind == "solve":
        return {"kind": "solve", "n": _log(rng, 1, 40000), "mode": rng.choice([PER_CELL, SORTED, ITERS])}
    if kind == "invert":
        return {"kind": "invert", "n": _log(rng, 1, 300000)}
    nx, ny, nz = _grid(rng, 192 * 180 * 8)
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}


# ---- what a program has in hand ------------------------------------------------


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _download(sim, p, u, flags):
    lib, h = engine().lib(), sim._h
    sim._check(lib.kc_download_prims(h, p.ctypes.data))
    sim._check(lib.kc_download_cons(h, u.ctypes.data))
    sim._check(lib.kc_download_flags(h, flags.ctypes.data))


def _upload(sim, p, u, flags):
    lib, h = engine().lib(), sim._h
    sim._check(lib.kc_upload_prims(h, p.ctypes.data))
    sim._check(lib.kc_upload_cons(h, u.ctypes.data))
    sim._check(lib.kc_upload_flags(h, flags.ctypes.data))


def _host_fields(sim):
    return (_pinned((sim.ncell, NV), torch.float64), _pinned((sim.ncell, NV), torch.float64),
            _pinned((sim.ncell, NFLAGS), torch.int32))


def _sim(case, seed, **options):
    """A handle holding the perturbed torus two steps into its run."""
    kc = engine()
    sim = kc.Sim(kc.puffy_grid(case["nx"], case["ny"], case["nz"]), kc.puffy_options(**options))
    sim.initPuffy(1e-3, 1e-3, seed)
    for _ in range(2):
        sim.step()
    return sim


def _metric(r, th):
    """The 23 geometry numbers of the batch entry points at radius r and polar angle th around a
    non-rotating hole in Kerr-Schild coordinates, and the two metrics as [n][4][4]."""
    n = r.size
    f = 2.0 / r
    gg, up = np.zeros((n, 4, 4)), np.zeros((n, 4, 4))
    gg[:, 0, 0], gg[:, 0, 1], gg[:, 1, 0], gg[:, 1, 1] = f - 1.0, f, f, 1.0 + f
    gg[:, 2, 2], gg[:, 3, 3] = r * r, (r * np.sin(th)) ** 2
    up[:, 0, 0], up[:, 0, 1], up[:, 1, 0], up[:, 1, 1] = -1.0 - f, f, f, 1.0 - f
    up[:, 2, 2], up[:, 3, 3] = 1.0 / gg[:, 2, 2], 1.0 / gg[:, 3, 3]
    i, j = np.triu_indices(4)
    rest = np.stack([r * r * np.sin(th), 1.0 / np.sqrt(1.0 + f), f], axis=1)  # sqrt(-g), lapse, 1 + g_tt
    return np.ascontiguousarray(np.concatenate([gg[:, i, j], up[:, i, j], rest], axis=1)), gg, up


def _velocity(rng, gg, gamma):
    """Relative four-velocities u~^i of the Lorentz factors gamma in random directions."""
    d = rng.uniform(-1.0, 1.0, (gamma.size, 3))
    q = np.einsum("ni,nij,nj->n", d, gg[:, 1:, 1:], d)
    return d * np.sqrt((gamma * gamma - 1.0) / q)[:, None]


def _loguniform(rng, lo, hi, n):
    return np.exp(rng.uniform(math.log(lo), math.log(hi), n))


def _inversion(case, seed):
    """Cells of a thin hot flow: their geometry, primitives and conserveds (plain numpy)."""
    n = case["n"]
    rng = np.random.default_rng([seed, 4])
    geom, gg, up = _metric(_loguniform(rng, 3.0, 50.0, n), rng.uniform(0.3, math.pi - 0.3, n))
    rho = _loguniform(rng, 1e-6, 1.0, n)
    ugas = rho * _loguniform(rng, 1e-4, 1e-1, n)
    erad = ugas * _loguniform(rng, 1e-2, 1e2, n)
    v = _velocity(rng, gg, 1.0 / np.sqrt(1.0 - rng.uniform(0.0, 0.81, n)))
    B = _velocity(rng, gg, np.sqrt(1.0 + 2.0 * (GAM - 1.0) * ugas / _loguniform(rng, 1.0, 1e3, n)))
    F = _velocity(rng, gg, rng.uniform(1.0, 2.0, n))
    entr = rho * np.log(((GAM - 1.0) * ugas) ** 1.5 / rho**2.5)
    pp = np.concatenate([np.stack([rho, ugas], 1), v, entr[:, None], B, erad[:, None], F], axis=1)

    def four_velocity(w):
        q = np.einsum("ni,nij,nj->n", w, gg[:, 1:, 1:], w)
        ag = np.sqrt((1.0 + q) / -up[:, 0, 0])  # lapse x Lorentz factor
        con = -ag[:, None] * up[:, 0, :]
        con[:, 1:] += w
        return con, np.einsum("nij,nj->ni", gg, con), q, ag

    gdet = geom[:, 20]
    con, cov, q, ag = four_velocity(v)
    b0 = np.einsum("ni,ni->n", B, cov[:, 1:])
    bcon = np.concatenate([b0[:, None], (B + b0[:, None] * con[:, 1:]) / con[:, :1]], axis=1)
    bcov = np.einsum("nij,nj->ni", gg, bcon)
    bsq = np.einsum("ni,ni->n", bcon, bcov)
    pre = (GAM - 1.0) * ugas
    eta = rho + ugas + pre + bsq
    ut = con[:, 0]
    # T^t_nu + rho u^t delta^t_nu, with 1 + u_t formed without cancellation
    alpha2 = geom[:, 21] ** 2
    beta2 = np.einsum("ni,ni->n", gg[:, 0, 1:], up[:, 0, 1:])
    utp1 = np.einsum("ni,ni->n", v, gg[:, 0, 1:]) + (geom[:, 22] - alpha2 * (beta2 + q)) / (1.0 + ag)
    mom = (eta * ut)[:, None] * cov[:, 1:] - bcon[:, :1] * bcov[:, 1:]
    ene = (ugas + pre + bsq) * ut * cov[:, 0] + rho * ut * utp1 + pre + 0.5 * bsq - bcon[:, 0] * bcov[:, 0]
    rcon, _, _, _ = four_velocity(F)
    rtop = 4.0 / 3.0 * (erad * rcon[:, 0])[:, None] * rcon + 1.0 / 3.0 * erad[:, None] * up[:, 0, :]
    rad = np.einsum("nij,nj->ni", gg, rtop)
    uu = gdet[:, None] * np.concatenate([np.stack([rho * ut, ene], 1), mom, (entr * ut)[:, None], B, rad], axis=1)
    # the inversion starts from the primitives of the step before
    before = pp * (1.0 + 1e-2 * rng.uniform(-1.0, 1.0, pp.shape))
    return geom, np.ascontiguousarray(uu), np.ascontiguousarray(before), pp


def prepare(case, seed):
    kc = engine()
    kind = case["kind"]
    if kind == "steps":
        sim = _sim(case, seed, precision=kc.KC_MIXED if case["mixed"] else kc.KC_PLAIN_FP64,
                   radimp_start_with_bisect=int(case["bisect"]))
        p, u, flags = _host_fields(sim)
        _download(sim, p, u, flags)
        counters = sim.counters()
        dt = 0.8 * counters["dt"] if case["forced"] else None
        if case["graph"]:
            sim.set_graph(True)  # a run of any length replays the captured step
            for _ in range(2):
                sim.step(dt)
        return {"kind": kind, "sim": sim, "host": (p, u, flags), "out": _host_fields(sim), "counters": counters,
                "dt": dt, "steps": case["steps"]}
    if kind == "solve":
        opt = kc.puffy_options()
        geom, dt, pp = (torch.from_numpy(a).cuda() for a in kc.synth_implicit_cells(opt, case["n"], seed))
        return {"kind": kind, "opt": opt, "n": case["n"], "mode": case["mode"], "geom": geom, "dt": dt, "start": pp,
                "pp": torch.empty_like(pp), "res": torch.zeros((case["n"], 6), dtype=torch.int32, device="cuda")}
    if kind == "invert":
        geom, uu, before, _ = _inversion(case, seed)
        return {"kind": kind, "opt": kc.puffy_options(), "geom": geom, "uu": uu, "before": before}
    if kind == "restart":
        sim = _sim(case, seed)
        return {"kind": kind, "sim": sim, "checkpoint": sim.kdmp_write(7)}
    sim = kc.Sim(kc.puffy_grid(case["nx"], case["ny"], case["nz"]), kc.puffy_options())
    return {"kind": kind, "sim": sim, "seed": seed, "out": _host_fields(sim)}


# ---- one pass --------------------------------------------------------------------


def run(state):
    kc = engine()
    kind = state["kind"]
    if kind == "steps":
        sim = state["sim"]
        _upload(sim, *state["host"])
        sim.set_counters(**state["counters"])
        for _ in range(state["steps"]):
            dt = sim.step(state["dt"])
        row = sim.scalars(dt)
        p, u, flags = state["out"]
        _download(sim, p, u, flags)
        return {"p": p, "u": u, "flags": flags, "row": row, "counters": sim.counters()}
    if kind == "solve":
        state["pp"].copy_(state["start"])
        kc.implicit_batch_device(state["opt"], state["n"], state["geom"].data_ptr(), state["dt"].data_ptr(),
                                 state["pp"].data_ptr(), state["res"].data_ptr(),
                                 torch.cuda.current_stream().cuda_stream, mode=state["mode"])
        return {"pp": state["pp"], "res": state["res"]}
    if kind == "invert":
        pp, flags = kc.u2p_batch(state["opt"], state["geom"], state["uu"], state["before"])
        return {"pp": pp, "flags": flags}
    sim = state["sim"]
    if kind == "restart":
        head = sim.kdmp_load(state["checkpoint"])
        sim.set_counters(t=head["t"], nstep=head["nstep"])
        sim.finishInit()
        row = sim.scalars()
        again = sim.kdmp_write(8)
        return {"u": sim.u, "row": row, "checkpoint": np.frombuffer(again, dtype=np.uint8)}
    fac = sim.initPuffy(1e-3, 1e-3, state["seed"])
    p, u, flags = state["out"]
    _download(sim, p, u, flags)
    return {"p": p, "u": u, "flags": flags, "fac": fac, "counters": sim.counters()}


# ---- what a pass cannot do without, and how far results may be off ----------------


def work(case):
    kind = case["kind"]
    if kind == "solve":
        # geometry 23, dt, p in; p and six 32-bit results out. About 116 Newton iterations a cell on these
        # states, each five evaluations of the residual of some 1,200 FP64 operations.
        return {"bytes": case["n"] * ((23 + 1 + 2 * NV) * 8 + 24), "flops": case["n"] * 116 * 5 * 1200}
    if kind == "invert":
        # geometry, u, p in; p and three flags out. Three Newton steps, floors and the M1 closure.
        return {"bytes": case["n"] * ((23 + 3 * NV) * 8 + 12), "flops": case["n"] * 1500}
    cells = case["nx"] * case["ny"] * case["nz"]
    fields = cells * (2 * NV * 8 + NFLAGS * 4)  # p, u and the flags of the domain
    if kind == "restart":
        return {"bytes": cells * NV * 8 * 4 + cells * 28 * 8, "flops": cells * 600}
    if kind == "start":
        # per (r, theta) column a torus solve with its quadrature, per cell the field
        return {"bytes": fields + cells * 28 * 8, "flops": case["nx"] * case["ny"] * 40000 + cells * 1500}
    # a step: p and u in and out, the metric (28) and the connection (40) of the cell and the metric of its
    # faces (28 each); two implicit solves of about 15,000 FP64 operations and 12,000 for the explicit half
    dims = 2 + (case["nz"] > 1)
    per_step = (4 * NV + 28 + 40 + 28 * dims) * 8
    return {"bytes": 2 * fields + case["steps"] * cells * per_step, "flops": case["steps"] * cells * 42000}


def tolerance(case):
    # Every value here is a fixed sequence of IEEE operations on one point, an ordered sum or a maximum: the
    # engine promises the reference's bits (and the FP32 pieces of the mixed form are such sequences too), so
    # the same inputs give the same bits in every form and at every block size.
    return "exact"


def exact(case, seed):
    """The inversion has a closed answer: the primitives that the conserveds were formed from. The others
    have none that plain code gives in seconds (iterations to a tolerance, whole time steps)."""
    if case["kind"] != "invert":
        return None
    _, _, _, pp = _inversion(case, seed)
    return {"pp": pp, "flags": np.zeros((case["n"], 3), dtype=np.int32)}
