"""The work a user of this framework has it do, as measurable cases.

Kinds of case:

  run    one registered box: upload its state, step it on the device
         (rhyme_gpu_run), read the result back: in plain FP64 the dt trace and
         the whole state (into a CUDA tensor), in mixed precision the FP32
         level output (what a run writes to its snapshot).
  batch  many uneven boxes stepped together (rhyme_gpu_batch), one level.
  loop   the host-driven loop of src/main.f90:106-177 on a box whose state
         lives in host memory: upload, dt, ghost fill, solve with the host
         write-back, download, per step.
  serve  requests of uneven sizes and lengths given to the continuous-batching
         server at once, painted on the device, each returning its level
         output.

Inputs are drawn from the seed: two-state Riemann problems, the shear slab
and boxes with spheres in a flow of a few long waves, as the repository's
benchmark workloads have them (rhyme_gb300/ic.py, rhyme_gb300/serving.py),
with states that stay clear of vacuum.
"""
import math

import numpy as np
import torch

from rhyme_gb300 import drawing, gpu
from rhyme_gb300.params import (CPU_INTENSIVE, FP64, LIMITERS, MEMORY_INTENSIVE, MIXED, OUTFLOW, PERIODIC,
                                REFLECTIVE, hydro_params)

GAMMA = 5.0 / 3.0
BC = {"periodic": PERIODIC, "outflow": OUTFLOW, "reflective": REFLECTIVE}
COURANT = (0.8, 0.4, 0.3)


def listed():
    return [
        # the smallest call: the 1-D shock tube of the tests and the benchmark, plain FP64
        dict(name="tube1d_512_fp64", kind="run", ndim=1, n1=512, n2=1, n3=1, precision="fp64", limiter="van_leer",
             bc="outflow", order="memory", omega=0.0, init="tube", steps=60),
        # a long 1-D tube of odd length in mixed precision
        dict(name="tube1d_4001_mixed", kind="run", ndim=1, n1=4001, n2=1, n3=1, precision="mixed",
             limiter="superbee", bc="reflective", order="memory", omega=0.0, init="tube", steps=100),
        # the 2-D shear slab of the benchmark, plain FP64 (the precision it is quoted in)
        dict(name="slab2d_256_fp64", kind="run", ndim=2, n1=256, n2=256, n3=1, precision="fp64", limiter="minmod",
             bc="periodic", order="memory", omega=0.0, init="slab", steps=20),
        # a ragged 2-D box in mixed precision
        dict(name="flow2d_1003x333_mixed", kind="run", ndim=2, n1=1003, n2=333, n3=1, precision="mixed",
             limiter="van_leer", bc="outflow", order="memory", omega=0.0, init="flow", steps=24),
        # a small ragged 3-D box, plain FP64, the cpu-intensive order
        dict(name="flow3d_37x61x29_fp64", kind="run", ndim=3, n1=37, n2=61, n3=29, precision="fp64",
             limiter="van_albada", bc="reflective", order="cpu", omega=0.25, init="flow", steps=6),
        # an ordinary 3-D box, plain FP64: what the drop-in runs by default
        dict(name="flow3d_128_fp64", kind="run", ndim=3, n1=128, n2=128, n3=128, precision="fp64",
             limiter="superbee", bc="periodic", order="memory", omega=0.0, init="flow", steps=2),
        # an ordinary 3-D box in mixed precision
        dict(name="flow3d_64_mixed", kind="run", ndim=3, n1=64, n2=64, n3=64, precision="mixed", limiter="superbee",
             bc="periodic", order="memory", omega=0.0, init="flow", steps=24),
        # the headline size of the benchmark: 3-D 256^3 spheres, mixed precision
        dict(name="flow3d_256_mixed", kind="run", ndim=3, n1=256, n2=256, n3=256, precision="mixed",
             limiter="superbee", bc="periodic", order="memory", omega=0.0, init="flow", steps=10),
        # a level of uneven boxes (edges 8..64, as the many-box workload), mixed precision
        dict(name="batch_96_mixed", kind="batch", ndim=3, nboxes=96, edge=64, shape_seed=0, precision="mixed",
             limiter="van_albada", bc="mixed", order="memory", omega=0.0, init="mixed", steps=8),
        # a small level of uneven boxes, plain FP64
        dict(name="batch_16_fp64", kind="batch", ndim=3, nboxes=16, edge=64, shape_seed=1, precision="fp64",
             limiter="van_albada", bc="mixed", order="memory", omega=0.0, init="mixed", steps=2),
        # the host-driven loop with the state in host memory, mixed precision
        dict(name="loop3d_160_mixed", kind="loop", ndim=3, n1=160, n2=160, n3=160, precision="mixed",
             limiter="van_leer", bc="periodic", order="memory", omega=0.0, init="waves", steps=2),
        # a burst of requests to the server (1-, 2- and 3-D, uneven sizes and lengths), mixed precision
        dict(name="serve_32_mixed", kind="serve", nreq=32, max_cells=64 ** 3, shape_seed=2, max_steps=60,
             precision="mixed"),
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "batch", "loop", "serve"])
    precision = rng.choice(["fp64", "mixed"])
    limiter = rng.choice(sorted(LIMITERS))
    order = rng.choice(["memory", "memory", "cpu"]) if precision == "fp64" else "memory"
    omega = rng.choice([0.0, 0.0, 0.25])
    if kind == "serve":
        return dict(kind=kind, nreq=rng.randint(4, 32), max_cells=_logint(rng, 24 ** 3, 64 ** 3),
                    shape_seed=rng.randint(0, 1 << 20), max_steps=rng.randint(8, 60), precision="mixed")
    if kind == "batch":
        mixed = precision == "mixed"
        edge = rng.choice([32, 48, 64])
        return dict(kind=kind, ndim=3, nboxes=_logint(rng, 4, 96 if mixed else 16), edge=edge,
                    shape_seed=rng.randint(0, 1 << 20), precision=precision, limiter=limiter, bc="mixed",
                    order=order, omega=omega, init="mixed", steps=rng.randint(1, 8 if mixed else 2))
    ndim = rng.choice([1, 2, 3])
    # cells of the box and cell updates of a pass, below the listed extremes
    if precision == "mixed":
        top, updates = (20000, 600000, 256 ** 3)[ndim - 1], 10 * 256 ** 3
    else:
        top, updates = (8000, 256 * 256, 128 ** 3)[ndim - 1], 2 * 128 ** 3
    if kind == "loop":
        ndim = max(ndim, 2)
        top = (256 * 256 if precision == "fp64" else 600000) if ndim == 2 else 96 ** 3 if precision == "fp64" else 160 ** 3
    cells = _logint(rng, (100, 400, 1000)[ndim - 1], int(0.8 * top))
    n = [1, 1, 1]
    base = cells ** (1.0 / ndim)
    for a in range(ndim):
        n[a] = max(4, int(base * rng.uniform(0.75, 1.2) + 0.5))
    total = n[0] * n[1] * n[2]
    steps = max(1, min(2 if kind == "loop" else 60, int(0.8 * updates / total)))
    steps = rng.randint(1, steps)
    init = "waves" if kind == "loop" else rng.choice((("tube", "flow"), ("tube", "slab", "flow"), ("tube", "ball", "flow"))[ndim - 1])
    bc = "periodic" if init == "slab" else rng.choice(sorted(BC))
    return dict(kind=kind, ndim=ndim, n1=n[0], n2=n[1], n3=n[2], precision=precision, limiter=limiter, bc=bc,
                order=order, omega=omega, init=init, steps=steps)


# ---- inputs ------------------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cons(rho, vel, p):
    s = sum(v * v for v in vel)
    return torch.stack([rho] + [rho * v for v in vel] + [0.5 * rho * s + p / (GAMMA - 1.0)])


def _field(init, n, rng):
    """Interior conserved state (NDIM+2, [n3,] [n2,] n1) as an FP64 tensor."""
    D = len(n)
    dev = _dev()
    shape = tuple(n[::-1])
    x = []  # cell centres along each axis, broadcastable
    for a in range(D):
        view = [1] * D
        view[D - 1 - a] = n[a]
        x.append(torch.arange(n[a], dtype=torch.float64, device=dev).add(0.5).reshape(view))
    one = torch.ones(shape, dtype=torch.float64, device=dev)
    if init == "mixed":
        init = "tube" if rng.random() < 0.5 else "ball"
    if init == "tube":  # two states split at the mid-plane of an axis
        axis = int(rng.integers(0, D))
        rho, p = 10.0 ** rng.uniform(-0.5, 0.5, 2), 10.0 ** rng.uniform(-0.5, 0.5, 2)
        u = rng.uniform(-0.4, 0.4, 2)
        left = (x[axis] < n[axis] // 2) & (one > 0)
        vel = [torch.where(left, u[0], u[1]) * one if a == axis else 0.0 * one for a in range(D)]
        return _cons(torch.where(left, rho[0], rho[1]) * one, vel, torch.where(left, p[0], p[1]) * one)
    if init == "ball":  # a dense centred sphere at rest
        r = rng.uniform(0.15, 0.4) * min(n)
        dens = 10.0 ** rng.uniform(0.3, 1.5)
        d2 = sum((x[a] - n[a] / 2.0) ** 2 for a in range(D))
        return _cons(torch.where(d2 < r * r, dens, 1.0) * one, [0.0 * one] * D, one)
    if init == "slab":  # the shear slab (rhyme_drawing_smoothed_slab_2d.f90), seeded phase
        sigma, yc, rs = 2.0 * n[1] / 256.0, n[1] / 2.0, n[1] / 4.0
        ramp = 0.25 * (1 + torch.tanh((rs - (x[1] - yc)) / sigma)) * (1 + torch.tanh((rs + (x[1] - yc)) / sigma))
        v = 0.01 * torch.cos(2 * math.pi * x[0] / (n[0] / 4.0) + rng.uniform(0, 2 * math.pi))
        return _cons((1.0 + ramp) * one, [(-0.5 + ramp) * one, v * one], 2.5 * one)
    # a flow of a few long waves in every field; "flow" adds dense moving spheres
    def waves(amp):
        f = 0.0 * one
        for _ in range(4):
            k = [int(rng.integers(1, 4)) for _ in range(D)]
            ph = rng.uniform(0, 2 * math.pi)
            f = f + amp / 2.0 * torch.cos(sum(2 * math.pi * k[a] * x[a] / n[a] for a in range(D)) + ph)
        return f
    rho, p = 1.0 + 0.3 * torch.tanh(waves(0.5)), 1.0 + 0.3 * torch.tanh(waves(0.5))
    vel = [waves(0.2) for _ in range(D)]
    if init == "flow":
        for _ in range(12):
            c = [rng.uniform(0, n[a]) for a in range(D)]
            r = rng.uniform(0.04, 0.12) * min(n)
            dens, bulk = 10.0 ** rng.uniform(0.0, 0.8), rng.uniform(-0.15, 0.15, D)
            d2 = 0.0
            for a in range(D):
                d = (x[a] - c[a]).abs()
                d2 = d2 + torch.minimum(d, n[a] - d) ** 2
            m = d2 < r * r
            rho = torch.where(m, dens, rho)
            vel = [torch.where(m, vel[a] + float(bulk[a]), vel[a]) for a in range(D)]
    return _cons(rho, vel, p)


def _box_array(field):
    """The reference's ghosted array (ghosts zero) of an interior state, on the host."""
    shape = (field.shape[0],) + tuple(s + 4 for s in field.shape[1:])
    full = torch.zeros(shape, dtype=torch.float64, device=field.device)
    full[(slice(None),) + (slice(2, -2),) * (field.dim() - 1)] = field
    return np.ascontiguousarray(full.cpu().numpy())


def _boxes(case, seed):
    """[(n, bc list, interior state)] of a case's boxes."""
    rng = np.random.default_rng([int(seed), 1])
    if case["kind"] == "batch":
        shapes = np.random.default_rng([case["shape_seed"], 7])
        edges = list(range(8, case["edge"] + 1, 8))
        out = []
        for _ in range(case["nboxes"]):
            n = [int(shapes.choice(edges)) for _ in range(3)]
            bc = [int(shapes.choice([REFLECTIVE, OUTFLOW])) for _ in range(6)]
            out.append((n, bc, _field(case["init"], n, rng)))
        return out
    n = [case["n1"], case["n2"], case["n3"]][:case["ndim"]]
    return [(n, [BC[case["bc"]]] * 6, _field(case["init"], n, rng))]


def _requests(case, seed):
    """The server's requests: sizes from the case, states from the seed."""
    shapes, rng = np.random.default_rng([case["shape_seed"], 8]), np.random.default_rng([int(seed), 2])
    out = []
    for _ in range(case["nreq"]):
        D = int(shapes.integers(1, 4))
        total = math.exp(shapes.uniform(math.log(256.0), math.log(float(case["max_cells"]))))
        total = min(total, (20000.0, 1e6, 1e9)[D - 1])
        n = [max(4, int(round(total ** (1.0 / D) * f))) for f in shapes.uniform(0.8, 1.25, D)]
        bc = [int(shapes.choice([REFLECTIVE, OUTFLOW])) for _ in range(2 * D)] + [OUTFLOW] * (6 - 2 * D)
        steps, limiter = int(shapes.integers(4, case["max_steps"] + 1)), int(shapes.integers(1, 5))
        rho, p, u = 10.0 ** rng.uniform(-0.5, 0.5, 2), 10.0 ** rng.uniform(-0.5, 0.5, 2), rng.uniform(-0.4, 0.4, 2)
        axis = int(rng.integers(0, D))
        w = [[rho[i]] + [u[i] if a == axis else 0.0 for a in range(3)] + [p[i]] for i in (0, 1)]
        out.append(dict(D=D, n=n, bc=bc, steps=steps, limiter=limiter, axis=axis, w=w, dx=[1.0 / max(n)] * D))
    return out


def _params(case, bc, ndim):
    return hydro_params(ndim, limiter=LIMITERS[case.get("limiter", "van_leer")], bc=bc, gamma=GAMMA,
                        courant=COURANT[ndim - 1], omega=case.get("omega", 0.0),
                        solver_type=CPU_INTENSIVE if case.get("order") == "cpu" else MEMORY_INTENSIVE,
                        precision=MIXED if case["precision"] == "mixed" else FP64)


def _dx(n):
    return [1.0 / max(n)] * len(n)


def _pinned(count):
    t = torch.empty(int(count), dtype=torch.float32, pin_memory=torch.cuda.is_available())
    return t.numpy()


class _Program:
    """What a user's program holds: the context or server, its boxes and arrays."""


def prepare(case, seed):
    s = _Program()
    s.case = case
    mixed = case["precision"] == "mixed"
    if case["kind"] == "serve":
        s.requests = _requests(case, seed)
        for q in s.requests:
            lengths = [q["n"][a] if a != q["axis"] else q["n"][a] // 2 for a in range(q["D"])]
            q["shapes"] = [drawing.canvas(q["w"][1]), drawing.sharp_cuboid([1] * q["D"], lengths, q["w"][0])]
            q["cells"] = np.zeros((q["D"] + 2,) + tuple(k + 4 for k in q["n"][::-1]))
            q["size"] = (q["D"] + 2) * int(np.prod(q["n"]))
        s.out = _pinned(sum(q["size"] for q in s.requests))
        s.server = gpu.Server(hydro_params(3, gamma=GAMMA, precision=MIXED if mixed else FP64), COURANT)
        return s
    boxes = _boxes(case, seed)
    s.ctx = gpu.Context(_params(case, boxes[0][1], case["ndim"]))
    s.boxes, s.dxs, size = [], [], 0
    for n, bc, field in boxes:
        b = s.ctx.register_box(_box_array(field))
        if len(boxes) > 1:
            s.ctx.set_box_params(b, bc=bc)
        s.boxes.append(b)
        s.dxs.append([1.0 / 64] * 3 if case["kind"] == "batch" else _dx(n))
        size += (case["ndim"] + 2) * int(np.prod(n))
    if case["kind"] == "batch":
        s.batch = s.ctx.batch(s.boxes, s.dxs)
    if mixed:
        s.out = _pinned(size)
    else:
        s.out = [torch.empty(s.ctx.rows_shape(b, b.cells.shape[1]), dtype=torch.float64, device=_dev())
                 for b in s.boxes]
    if case["kind"] == "loop":
        s.ctx.set_host_writeback(s.boxes[0])
    return s


def _result(s):
    """The mixed form's level output, or every box's whole FP64 state."""
    if s.case["precision"] == "mixed":
        s.ctx.output_level(s.boxes, out=s.out)
        s.ctx.output_wait()
        return s.out
    return [s.ctx.get_rows(b, 0, b.cells.shape[1], out=o) for b, o in zip(s.boxes, s.out)]


def run(s):
    case = s.case
    if case["kind"] == "serve":
        at = 0
        for q in s.requests:
            s.server.submit(q["cells"], q["steps"], q["dx"], q["limiter"], q["bc"], shapes=q["shapes"],
                            output=s.out[at:at + q["size"]])
            at += q["size"]
        while any(s.server.tick()):
            pass
        return s.out
    if case["kind"] == "batch":
        for b in s.boxes:
            s.ctx.sync_to_device(b)
        s.batch.run(case["steps"])
        return _result(s)
    b, dx = s.boxes[0], s.dxs[0]
    if case["kind"] == "loop":
        for _ in range(case["steps"]):
            s.ctx.sync_to_device(b)
            dt = s.ctx.cfl_time_step(b, dx)
            s.ctx.set_boundaries(b)
            s.ctx.muscl_hancock_solve(b, dx, dt)
            s.ctx.sync_to_host(b)
        return _result(s)
    s.ctx.sync_to_device(b)
    dts = s.ctx.run(b, dx, case["steps"], trace=case["precision"] == "fp64")
    r = _result(s)
    return r if dts is None else [dts] + r


# ---- what a pass cannot do without ---------------------------------------------

def work(case):
    """Bytes: per cell update the conserved state read once and written once
    in FP64 (48, 64 or 80 B in 1-, 2- or 3-D). Operations: per cell and axis
    about 120 for the limited slopes and half step and 200 for the exact
    Riemann problem and its flux, a power or a root counted as one."""
    if case["kind"] == "serve":
        todo = [(q["D"], int(np.prod(q["n"])), q["steps"]) for q in _requests(case, 0)]
    elif case["kind"] == "batch":
        shapes = np.random.default_rng([case["shape_seed"], 7])
        edges = list(range(8, case["edge"] + 1, 8))
        todo = []
        for _ in range(case["nboxes"]):
            n = [int(shapes.choice(edges)) for _ in range(3)]
            [shapes.choice([REFLECTIVE, OUTFLOW]) for _ in range(6)]
            todo.append((3, n[0] * n[1] * n[2], case["steps"]))
    else:
        todo = [(case["ndim"], case["n1"] * case["n2"] * case["n3"], case["steps"])]
    return {"bytes": float(sum(c * k * (D + 2) * 16 for D, c, k in todo)),
            "flops": float(sum(c * k * D * 320 for D, c, k in todo))}


# ---- the same steps in plain torch, 64 bits --------------------------------------

TINY = np.finfo(np.float64).tiny
G1, GP = GAMMA - 1.0, GAMMA + 1.0


def _pressure(u):
    s = sum(u[c] * u[c] for c in range(1, u.shape[0] - 1))
    return u[0] * (u[-1] / u[0] - 0.5 * s / (u[0] * u[0])) * G1


def _flux(u, a):
    p = _pressure(u)
    vn = u[1 + a] / u[0]
    f = [u[1 + a]] + [u[c] * vn for c in range(1, u.shape[0] - 1)] + [vn * (u[-1] + p)]
    f[1 + a] = f[1 + a] + p
    return torch.stack(f)


def _slope(limiter, w, um, u, up):
    dl, dr = u - um, up - u
    d = 0.5 * (1 + w) * dl + 0.5 * (1 + w) * dr
    zero = dr.abs() < TINY
    r = torch.where(zero, 0.0, dl / torch.where(zero, 1.0, dr))
    xi = 2.0 / (1.0 - w + (1.0 + w) * r)
    one = torch.ones_like(r)
    if limiter == "van_leer":
        phi = torch.minimum(2 * r / (1 + r), xi)
    elif limiter == "minmod":
        phi = torch.where(r > 1, torch.minimum(one, xi), r)
    elif limiter == "van_albada":
        phi = torch.minimum(r * (1 + r) / (1 + r * r), xi)
    else:
        phi = torch.where(r > 1, torch.minimum(torch.minimum(r, xi), 2 * one), torch.where(r > 0.5, one, 2 * r))
    return torch.where(r > 0, phi * d, 0.0)


def _wave(p, rho, pk, cs):
    shock = p > pk
    bp = G1 / GP * pk + p
    q = torch.sqrt(2.0 / (GP * rho) / bp)
    y = p / pk
    f = torch.where(shock, (p - pk) * q, 2 * cs / G1 * (y ** (G1 / (2 * GAMMA)) - 1))
    df = torch.where(shock, q * (1 - (p - pk) / (2 * bp)), y ** (-GP / (2 * GAMMA)) / (rho * cs))
    return f, df


def _riemann(l, r, a):
    """The state at x/t = 0 of the exact Riemann problem (no vacuum)."""
    rl, rr = l[0], r[0]
    vl, vr = l[1 + a] / rl, r[1 + a] / rr
    pl, pr = _pressure(l), _pressure(r)
    cl, cr = torch.sqrt(GAMMA * pl / rl), torch.sqrt(GAMMA * pr / rr)
    ppv = (0.5 * (pl + pr) + 0.125 * (vl - vr) * (rl + rr) * (cl + cr)).clamp(min=0.0)
    lo, hi = torch.minimum(pl, pr), torch.maximum(pl, pr)
    z = G1 / (2 * GAMMA)
    pq = (pl / pr) ** z
    um = (pq * vl / cl + vr / cr + 2 / G1 * (pq - 1)) / (pq / cl + 1 / cr)
    p2r = 0.5 * (pl * (1 + G1 / 2 * (vl - um) / cl).clamp(min=TINY) ** (1 / z)
                 + pr * (1 + G1 / 2 * (um - vr) / cr).clamp(min=TINY) ** (1 / z))
    gl, gr = torch.sqrt(2 / GP / rl / (G1 / GP * pl + ppv)), torch.sqrt(2 / GP / rr / (G1 / GP * pr + ppv))
    p2s = (gl * pl + gr * pr - (vr - vl)) / (gl + gr)
    p = torch.where((hi <= 2 * lo) & (lo < ppv) & (ppv < hi), ppv, torch.where(ppv < lo, p2r, p2s)).clamp(min=TINY)
    done = torch.zeros_like(p, dtype=torch.bool)
    fl = fr = torch.zeros_like(p)
    for _ in range(100):
        nl, dl = _wave(p, rl, pl, cl)
        nr, dr = _wave(p, rr, pr, cr)
        q = (p - (nl + nr + (vr - vl)) / (dl + dr)).clamp(min=TINY)
        fl, fr = torch.where(done, fl, nl), torch.where(done, fr, nr)
        stop = 2 * (q - p).abs() / (q + p) < 1e-6
        p = torch.where(done, p, q)
        done = done | stop
        if bool(done.all()):
            break
    us = 0.5 * ((vr + vl) + (fr - fl))
    right = us < 0
    # the sampled side, mirrored to the left
    sg = torch.where(right, -1.0, 1.0)
    rho, pk, cs, v = (torch.where(right, x, y) for x, y in ((rr, rl), (pr, pl), (cr, cl), (vr, vl)))
    v, us = sg * v, sg * us
    y = p / pk
    shock = p > pk
    rs = torch.where(shock, rho * (G1 / GP + y) / (G1 / GP * y + 1), rho * y ** (1 / GAMMA))
    head = torch.where(shock, v - cs * torch.sqrt(GP / (2 * GAMMA) * y + z), v - cs)
    tail = torch.where(shock, head, us - cs * y ** z)
    base = (2 / GP + G1 / GP / cs * v).clamp(min=TINY)
    fan = (rho * base ** (2 / G1), 2 / GP * (cs + G1 / 2 * v), pk * base ** (1 / z))
    star, out = tail < 0, head >= 0
    rho, vn, pp = (torch.where(star, x, torch.where(out, y_, f))
                   for x, y_, f in ((rs, rho, fan[0]), (us, v, fan[1]), (p, pk, fan[2])))
    vel = [torch.where(right, r[1 + b] / rr, l[1 + b] / rl) if b != a else sg * vn for b in range(l.shape[0] - 2)]
    s = sum(x * x for x in vel)
    return torch.stack([rho] + [rho * x for x in vel] + [0.5 * rho * s + pp / G1])


def _ghosts(U, n, bc):
    D = len(n)
    for a in range(D):
        dim = 1 + D - 1 - a
        V = U.movedim(dim, -1)
        inner = V[(slice(None),) + (slice(2, -2),) * (D - 1)]  # a view: transverse interior, whole axis
        N = n[a]
        for side in (0, 1):
            kind = bc[2 * a + side]
            g = (1, 0) if side == 0 else (N + 2, N + 3)
            if kind == PERIODIC:
                src = (N + 1, N) if side == 0 else (2, 3)
            else:
                src = (2, 3) if side == 0 else (N + 1, N)
            for i, j in zip(g, src):
                v = inner[..., j].clone()
                if kind == REFLECTIVE:
                    v[1 + a] = -v[1 + a]
                inner[..., i] = v


def _steps(field, n, bc, limiter, omega, order, courant, dx, steps):
    """(dts, ghosted state) after `steps` steps."""
    D = len(n)
    U = torch.zeros((D + 2,) + tuple(k + 4 for k in n[::-1]), dtype=torch.float64, device=field.device)
    inside = (slice(None),) + (slice(2, -2),) * D
    U[inside] = field
    dts = []
    for _ in range(steps):
        u = U[inside]
        s = sum(u[c] * u[c] for c in range(1, D + 1))
        speed = torch.sqrt(s) / u[0] + torch.sqrt(GAMMA * _pressure(u) / u[0])
        dt = courant * min(dx) / float(speed.max())
        dts.append(dt)
        _ghosts(U, n, bc)
        diffs = []
        for a in range(D):
            dim = 1 + D - 1 - a
            V = U.movedim(dim, -1)[(slice(None),) + (slice(2, -2),) * (D - 1)].contiguous()
            um, u0, up = V[..., :-2], V[..., 1:-1], V[..., 2:]
            d = 0.5 * _slope(limiter, omega, um, u0, up)
            l, r = u0 - d, u0 + d
            half = 0.5 * dt / dx[a] * (_flux(l, a) - _flux(r, a))
            l, r = l + half, r + half
            F = _flux(_riemann(r[..., :-1], l[..., 1:], a), a)
            diffs.append((dt / dx[a] * (F[..., :-1] - F[..., 1:])).movedim(-1, dim))
        new = U.clone()
        new[inside] = sum(diffs, U[inside]) if order == "cpu" else U[inside] + sum(diffs[1:], diffs[0])
        U = new
    return np.array(dts), U


def exact(case, seed):
    mixed = case["precision"] == "mixed"
    if case["kind"] == "serve":
        todo = _requests(case, seed)
        names = {v: k for k, v in LIMITERS.items()}
        if sum(q["steps"] * q["D"] for q in todo) > 4000:
            return None
        out = []
        for q in todo:
            D, n = q["D"], q["n"]
            idx = torch.arange(n[q["axis"]], device=_dev())
            view = [1] * D
            view[D - 1 - q["axis"]] = n[q["axis"]]
            left = (idx < n[q["axis"]] // 2).reshape(view).expand(tuple(n[::-1]))
            w = [torch.where(left, float(x), float(y)).double() for x, y in zip(*q["w"])]
            U = _steps(_cons(w[0], w[1:1 + D], w[4]), n, q["bc"], names[q["limiter"]], 0.0, "memory",
                       COURANT[D - 1], q["dx"], q["steps"])[1]
            out.append(U[(slice(None),) + (slice(2, -2),) * D].reshape(-1))
        return torch.cat(out)
    boxes = _boxes(case, seed)
    if len(boxes) * case["steps"] * case["ndim"] > 4000:
        return None
    done = []
    for n, bc, field in boxes:
        dx = [1.0 / 64] * 3 if case["kind"] == "batch" else _dx(n)
        done.append(_steps(field, n, bc, case["limiter"], case["omega"], case["order"], COURANT[len(n) - 1], dx,
                           case["steps"]))
    if mixed:
        return torch.cat([U[(slice(None),) + (slice(2, -2),) * (U.dim() - 1)].reshape(-1) for _, U in done])
    states = [U for _, U in done]
    return states if case["kind"] != "run" else [done[0][0]] + states
