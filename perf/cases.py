"""What this framework is timed on: the calls its users make, over the sizes they make them at.

Every case goes through the public entry points of the Python mirror of the C-ABI (api.Context, serve.Server, the
CSR solvers): contexts with the tuned solver options, host state in, host state out.  The kinds:

  step     production steps of one solitary-wave beach scene and the read-back of its state
  batch    steps of many uneven beach scenes in one context (the parameter study), each scene read back
  aquifer  steps of the reference's own scene with the reference's own solver settings and its open-boundary zones
  lattice  the stand-alone neighbour search + PPE assembly + solve of a jittered lattice with a given source
  serve    requests joining a running batch (admission, priming, ten steps, result)
  csr      a linear solve of the caller's own CSR system (host arrays, or device arrays without allocation)
"""
import math

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()

from beachslope_gb300 import abi, api, aquifer, scene, serve  # noqa: E402

FIXED, GHOST, FLUID = abi.TID_WALL, abi.TID_GHOST, abi.TID_FLUID


def listed():
    return [
        # The everyday scene (dx = 10 mm, 13 k particles): thousands of short steps, bound by latency and launches.
        {"name": "step_13k_mixed", "kind": "step", "n": 12989, "mixed": True, "wcsph": False, "steps": 1},
        # The same as the FP64 drop-in of a host program that keeps its own precision.
        {"name": "step_13k_fp64", "kind": "step", "n": 12989, "mixed": False, "wcsph": False, "steps": 1},
        # A medium refinement (dx = 2.5 mm), both forms.
        {"name": "step_182k_mixed", "kind": "step", "n": 182395, "mixed": True, "wcsph": False, "steps": 1},
        {"name": "step_182k_fp64", "kind": "step", "n": 182395, "mixed": False, "wcsph": False, "steps": 1},
        # The refined scene of the benchmark (dx = 1.25 mm): the largest single scene.
        {"name": "step_712k_mixed", "kind": "step", "n": 712460, "mixed": True, "wcsph": False, "steps": 1},
        # The parameter study: 64 scenes of 3.9 k to 47 k particles (dx 5 to 20 mm) in one context, ISPH and WCSPH.
        {"name": "batch_64_isph", "kind": "batch", "scenes": 64, "study": 20261203, "mixed": True, "wcsph": False,
         "steps": 2},
        {"name": "batch_64_wcsph", "kind": "batch", "scenes": 64, "study": 20261203, "mixed": True, "wcsph": True,
         "steps": 8},
        # The reference's aquifer tank as its main program settles it: its FGMRES (150 columns, 1e-3 of the first
        # residual, no preconditioner), FP64, the buffer zones set.
        {"name": "aquifer_reference", "kind": "aquifer", "steps": 2},
        # Search + PPE of a million particles with a given source (the stand-alone solve of the benchmark).
        {"name": "lattice_1m_mixed", "kind": "lattice", "side": 1000, "mixed": True},
        # Three requests of different sizes that arrive while the others run.
        {"name": "serve_3_requests", "kind": "serve", "sizes": "7000 21000 52000", "steps": 10},
        # A host program's own matrix: the no-allocation BiCGStab on device arrays, near its largest size, and the
        # FGMRES call on host arrays.
        {"name": "csr_device_bicgstab", "kind": "csr", "n": 60025, "solver": "bicgstab_device"},
        {"name": "csr_host_fgmres", "kind": "csr", "n": 9801, "solver": "fgmres_host"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "batch", "lattice", "serve", "csr", "csr"])
    mixed = rng.random() < 0.6
    if kind == "step":
        return {"kind": kind, "n": int(_log(rng, 3900, 700000)), "mixed": mixed, "wcsph": rng.random() < 0.2,
                "steps": rng.choice([1, 1, 2])}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 63), "study": rng.randrange(1 << 20), "mixed": mixed,
                "wcsph": rng.random() < 0.5, "steps": rng.choice([1, 2])}
    if kind == "lattice":
        return {"kind": kind, "side": int(_log(rng, 40, 990)), "mixed": mixed}
    if kind == "serve":
        return {"kind": kind, "sizes": " ".join(str(int(_log(rng, 5000, 30000))) for _ in range(rng.randint(1, 3))),
                "steps": rng.randint(3, 10)}
    solver = rng.choice(["bicgstab_device", "bicgstab_device", "fgmres_host", "bicgstab_host"])
    return {"kind": kind, "n": int(_log(rng, 60, 65000 if solver == "bicgstab_device" else 20000)), "solver": solver}


# ---------------------------------------------------------------- inputs
def _stir(st, rng):
    """The seed's part of a beach scene: the wave's velocities up to a tenth faster or slower, and the fluid's own
    motion of the size that a run has after its first steps."""
    fl = st["tid"] == FLUID
    scale = rng.uniform(0.9, 1.1)
    for k in ("vx", "vy"):
        st[k] = np.where(fl, scale * st[k] + 2e-3 * rng.standard_normal(len(fl)), st[k])
    return st


def _beach(n, mixed, wcsph, rng):
    """A beach scene of about n particles (the benchmark's wave, slope and bed)."""
    p, st, gr = scene.beach_scene(dx=scene.dx_for_particles(n), wcsph=wcsph,
                                  precision=abi.PREC_MIXED if mixed else abi.PREC_FP64)
    return p, _stir(st, rng), gr


def _system(n, seed):
    """A CSR system like the PPE's: the points of a ragged 2-D grid (the last row of it partly filled), each coupled
    to those within 2.6 spacings, weights that fall off with the distance, unsymmetric by a third, rows scaled to a
    unit diagonal with 1 % to spare.  Returns (row_ptr, col, val, b, x): A x = b."""
    rng = np.random.default_rng(seed)
    w = int(math.ceil(math.sqrt(n)))
    i = np.arange(n)
    r, c = i // w, i % w
    cols, vals, rows = [], [], []
    for dr in range(-2, 3):
        for dc in range(-2, 3):
            d2 = dr * dr + dc * dc
            if d2 == 0 or d2 > 6.76:
                continue
            j = (r + dr) * w + c + dc
            ok = (r + dr >= 0) & (c + dc >= 0) & (c + dc < w) & (j < n)
            rows.append(i[ok])
            cols.append(j[ok])
            vals.append(-math.exp(-d2 / 2.0) * rng.uniform(0.67, 1.33, int(ok.sum())))
    rows, cols, vals = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    total = -np.bincount(rows, weights=vals, minlength=n)
    rows, cols = np.concatenate([rows, i]), np.concatenate([cols, i])
    vals = np.concatenate([vals, np.where(total > 0, 1.01 * total, 1.0)])
    vals = vals / np.where(total > 0, 1.01 * total, 1.0)[rows]
    order = np.lexsort((cols, rows))
    rows, cols, vals = rows[order], cols[order], vals[order]
    ptr = np.zeros(n + 1, np.int32)
    ptr[1:] = np.cumsum(np.bincount(rows, minlength=n))
    x = rng.standard_normal(n)
    b = np.bincount(rows, weights=vals * x[cols], minlength=n)
    return ptr, cols.astype(np.int32), vals, b, x


def _lattice(case, seed):
    p, st, _ = scene.lattice_scene(n=case["side"], dx=1e-3, seed=seed)
    p.precision = abi.PREC_MIXED if case["mixed"] else abi.PREC_FP64
    p.ppe_tol = 1e-8
    return p, st, np.random.default_rng(seed + 7).standard_normal(len(st["x"]))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = {"case": case}
    if kind == "step":
        p, st, gr = _beach(case["n"], case["mixed"], case["wcsph"], rng)
        ctx = api.Context([p], [st], [gr], tuning="auto")
        ctx.prime()
        state.update(ctx=ctx, out=[api.pinned_state(len(st["x"]))])
    elif kind == "batch":
        scenes = scene.batch_scenes(case["scenes"], seed=case["study"], wcsph=case["wcsph"],
                                    precision=abi.PREC_MIXED if case["mixed"] else abi.PREC_FP64)
        P, S, G = (list(v) for v in zip(*scenes))
        S = [_stir(st, rng) for st in S]
        ctx = api.Context(P, S, G, tuning="auto")
        ctx.prime()
        state.update(ctx=ctx, out=[api.pinned_state(len(s["x"])) for s in S])
    elif kind == "aquifer":
        p, st, gr, zones, _ = aquifer.aquifer_scene()
        # the settling water is not at rest: velocities of the settling phase's size
        fl = (st["tid"] == FLUID) & ((st["flags"] & abi.FLAG_BUFFER) == 0)
        for k in ("vx", "vy"):
            st[k] = np.where(fl, 1e-3 * rng.standard_normal(len(fl)), st[k])
        ctx = api.Context([p], [st], [gr], capacity=[len(st["x"]) + 2048])
        for z, zone in enumerate(zones):
            ctx.set_inflow(z, zone)
        ctx.prime_setup()
        state.update(ctx=ctx, out=[api.pinned_state(len(st["x"]) + 2048)])
    elif kind == "lattice":
        p, st, b = _lattice(case, seed)
        ctx = api.Context([p], [st], [None], tuning="auto")
        state.update(ctx=ctx, b=b, out=[api.pinned_state(len(b))])
    elif kind == "serve":
        sizes = [int(v) for v in case["sizes"].split()]
        reqs = []
        for k, n in enumerate(sizes):
            reqs.append(serve.Request(k, 2.0 * k, *_beach(n, True, False, rng)))
        # the slots' templates: the finest scenes they take (their grids bound the requests' grids)
        t64, t16 = (scene.beach_scene(dx=scene.dx_for_particles(v), precision=abi.PREC_MIXED) for v in (70000, 16000))
        slots = [(t[0], int(1.2 * len(t[1]["x"])), int(1.6 * len(t[2]["x"])) + 64) for t in (t64, t64, t64, t16)]
        state.update(server=serve.Server(slots, tuning="auto"), requests=reqs)
    else:
        ptr, col, val, b, _ = _system(case["n"], seed)
        state.update(host=(ptr, col, val, b), x0=np.zeros(len(b)))
        if case["solver"] == "bicgstab_device":
            dev = [torch.from_numpy(a).cuda() for a in (ptr, col, val, b)]
            state.update(dev=dev, x=torch.zeros(len(b), dtype=torch.float64, device="cuda"))
    return state


# ---------------------------------------------------------------- one pass
def _read(ctx, out):
    return [ctx.download(s, full=False, out=o) for s, o in enumerate(out)]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "batch"):
        ctx = state["ctx"]
        (ctx.wcsph_step if case["wcsph"] else ctx.step)(case["steps"])
        got = _read(ctx, state["out"])
        if kind == "step":
            return got[0]
        # one array per field, scene after scene
        return {k: np.concatenate([g[k] for g in got]) for k in got[0]}
    if kind == "aquifer":
        state["ctx"].step_flags(case["steps"], abi.STEP_BUFFERS)
        return _read(state["ctx"], state["out"])[0]
    if kind == "lattice":
        ctx = state["ctx"]
        ctx.set_fields({"p": np.zeros(len(state["b"]))})   # the first guess, the same on every call
        ctx.search()
        ctx.porosity()
        ctx.int_vel()
        ctx.ppe_assemble()
        ctx.set_rhs(state["b"])
        ctx.ppe_solve()
        got = _read(ctx, state["out"])[0]
        return {"p": got["p"], "pid": got["pid"]}
    if kind == "serve":
        got = state["server"].run(state["requests"], case["steps"], clock="steps")
        got = [got[k]["state"] for k in sorted(got)]
        return {k: np.concatenate([g[k] for g in got]) for k in got[0]}
    if case["solver"] == "bicgstab_device":
        ptr, col, val, b = state["dev"]
        x = state["x"].zero_()
        stream = torch.cuda.current_stream().cuda_stream
        rc, _, _ = api.bicgstab_csr_noalloc(len(b), ptr.data_ptr(), col.data_ptr(), val.data_ptr(), b.data_ptr(),
                                            x.data_ptr(), tol=1e-12, maxit=2000, stream=stream)
    elif case["solver"] == "bicgstab_host":
        rc, x, _, _ = api.bicgstab_csr(*state["host"], state["x0"], tol=1e-12, maxit=2000)
    else:
        rc, x, _, _ = api.fgmres_csr(*state["host"], state["x0"], tol=1e-11, maxit=600, restart=150,
                                     rule=abi.STOP_RELRES)
    if rc != 0:
        raise RuntimeError("solve failed: %d" % rc)
    return {"x": x}


# ---------------------------------------------------------------- what a pass cannot do without
STATE_BYTES = 10 * 8 + 2 * 4 + 1    # one particle's state, read or written
PAIRS = 20                          # neighbours of an inner particle at h = 1.3 dx
STEP_FLOPS = PAIRS * 250 + 400      # the sweeps of a step, per particle


def work(case):
    kind = case["kind"]
    if kind == "step":
        n, steps = case["n"], case["steps"]
    elif kind == "batch":   # dx log-uniform in 5 to 20 mm
        n, steps = case["scenes"] * scene.BEACH_N_DX2 * 0.5 * (0.005 ** -2 - 0.02 ** -2) / math.log(4.0), case["steps"]
    elif kind == "aquifer":
        n, steps = 13681, case["steps"]
    elif kind == "serve":
        n, steps = sum(int(v) for v in case["sizes"].split()), case["steps"]
    elif kind == "lattice":
        n = (case["side"] + 4.5) ** 2
        # positions, types, source and first guess in; pressure out
        return {"bytes": n * (7 * 8 + 2 * 4 + 2), "flops": n * PAIRS * 120.0}
    else:
        nnz = case["n"] * 21.0
        return {"bytes": nnz * 12 + case["n"] * 20.0, "flops": 2 * nnz}
    return {"bytes": 2.0 * STATE_BYTES * n * steps, "flops": float(n * steps * STEP_FLOPS)}


# ---------------------------------------------------------------- the same in 64 bits, from the formulas
def exact(case, seed):
    if case["kind"] == "csr":
        return {"x": _system(case["n"], seed)[4]}
    if case["kind"] == "lattice":
        return _exact_lattice(case, seed)
    return None   # a time step is pinned by the repository's tests; no second implementation of it here


def _grad_over_d(r, h):
    """F of the kernel gradient F (x_i - x_j), with the reference's single-precision constants."""
    a1 = 0.1 * 10.0 / (float(np.float32(28.0) * np.float32(3.14)) * h * h)
    a2 = 0.9 / (float(np.float32(3.0) * np.float32(3.14)) * h * h)
    far = -(3.0 / (r * h)) * (2.0 - r / h) ** 2
    return torch.where(r < h, a1 * (9.0 * r / h ** 3 - 12.0 / h ** 2) + a2 * (3.0 * r / h ** 3 - 6.0 / (r * h)),
                       (a1 + a2) * far)


def _exact_lattice(case, seed):
    """Pairs, corrected gradients and the Jacobi-scaled PPE rows by the formulas in plain torch, solved by BiCGStab
    to 1e-12."""
    p, st, b = _lattice(case, seed)
    h, lam, cw = p.h, 0.001 * p.h * p.h, 4.0 * p.h
    # the library's order: cell by cell (column-major, from the bottom row up), walls first, then as given
    col, up = (np.searchsorted(np.arange(m) * cw, st[k], side="right") for k, m in (("x", p.cellx), ("y", p.celly)))
    order = np.lexsort((st["tid"] == FLUID, col * p.celly - up))
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    x, y, mass, rho, oden = (torch.tensor(st[k][order], device=dev) for k in ("x", "y", "mass", "rho", "oden"))
    tid = torch.tensor(st["tid"][order], device=dev)
    n = len(x)
    i, j, r = _pairs(x, y, 2.0 * h)
    dx, dy = x[i] - x[j], y[i] - y[j]
    F = _grad_over_d(r, h)
    z1, z2, vol = F * dx, F * dy, mass / rho

    def total(v):
        return torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, i, v)

    # gradient correction matrix; the unit matrix where it cannot be inverted
    m = [total(z * vol[j] * d) for d in (-dx, -dy) for z in (z1, z2)]
    div, det = m[0] + m[3], m[0] * m[3] - m[1] * m[2]
    ok = det.abs() >= float(np.float32(1e-5))
    one, zero = torch.ones_like(det), torch.zeros_like(det)
    C = [torch.where(ok, v / det, w) for v, w in ((m[3], one), (-m[1], zero), (-m[2], zero), (m[0], one))]
    free = (tid == FLUID) & (div <= p.lamfs * p.maxdivr)
    ti, tj = tid[i], tid[j]
    pd = 1.0 / (r * r + lam)

    def term(c, v):
        return 2.0 * v * ((c[0] * z1 + c[1] * z2) * dx + (c[2] * z1 + c[3] * z2) * dy) * pd

    fluid_row = term([c[i] for c in C], vol[j])
    wall_fluid = term([c[j] for c in C], vol[i])
    plain = 2.0 * vol[j] * (z1 * dx + z2 * dy) * pd
    t = torch.where(ti == FLUID, fluid_row, torch.where((ti == FIXED) & (tj == FLUID), wall_fluid, plain))
    t = torch.where((ti == GHOST) & (tj == FLUID), torch.zeros_like(t), t)
    dia = total(t * torch.where(free[i] & (tj == FLUID), 1.0 + oden[j] / (p.rho * p.rel_den), torch.ones_like(t)))
    # a ghost row whose first neighbour is a fluid particle keeps the row initialiser's 1
    first = torch.full((n,), n, dtype=torch.int64, device=dev).scatter_reduce_(0, i, j, "amin")
    keep = (tid == GHOST) & (first < torch.arange(n, device=dev))
    keep &= tid[first.clamp(max=n - 1)] == FLUID
    diag = torch.where(keep, 1.0 + 1.0 / dia, one)
    counts = torch.bincount(i, minlength=n)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    ptr[1:] = torch.cumsum(counts, 0)
    A = torch.sparse_csr_tensor(ptr, j, -t / dia[i], size=(n, n))
    rhs = torch.tensor(b, device=dev)
    sol = _bicgstab(lambda v: diag * v + A @ v, rhs, torch.tensor(st["p"][order], device=dev), 1e-12, 40000)
    return {"p": sol.cpu().numpy(), "pid": None}


def _pairs(x, y, reach):
    """All ordered pairs (i, j), i ascending, closer than reach, and their distances."""
    n = len(x)
    ny = int(y.max() / reach) + 3
    key = (torch.floor(x / reach).long() + 1) * ny + torch.floor(y / reach).long() + 1
    bins = int(key.max()) + ny + 2
    order = torch.argsort(key, stable=True)
    count = torch.bincount(key, minlength=bins)
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    me = torch.arange(n, device=x.device)
    found = []
    for a in (-1, 0, 1):
        for c in (-1, 0, 1):
            other = key + a * ny + c
            for q in range(most):
                j = order[(start[other] + q).clamp(max=n - 1)]
                r = torch.sqrt((x - x[j]) ** 2 + (y - y[j]) ** 2)
                ok = (q < count[other]) & (r < reach) & (j != me)
                found.append((me[ok], j[ok], r[ok]))
    i, j, r = (torch.cat(v) for v in zip(*found))
    at = torch.argsort(i * n + j)
    return i[at], j[at], r[at]


def _bicgstab(mul, b, x, tol, most):
    r = b - mul(x)
    shadow, rho = r.clone(), r @ r
    p = r.clone()
    stop = float(tol * torch.linalg.norm(b))
    for k in range(most):
        v = mul(p)
        alpha = rho / (shadow @ v)
        s = r - alpha * v
        t = mul(s)
        omega = (t @ s) / (t @ t)
        x = x + alpha * p + omega * s
        r = s - omega * t
        if k % 25 == 0 and float(torch.linalg.norm(r)) <= stop:
            break
        new = shadow @ r
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
    return x
