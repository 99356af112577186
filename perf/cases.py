"""The calls that users of fluidgb make, with their sizes and options, for timing and for checking results.

A case is a dict of plain values.  `op` says which entry point it calls:

  step      resume from a checkpoint in device memory, run one substep, read the particles, ids and pressure
            (fl_load_state_device, fl_step, fl_copy_pressure_device, fl_get_particles_device)
  frame     the same with the four substeps of a 30 Hz frame at dt = 1/120
  inplace   one substep on the caller's own device buffer, pressure from a cold start (fl_step_device)
  adjoint   resume, record one substep on a tape and pull a gradient back through it (fl_step_record, fl_step_adjoint)
  poisson   the stand-alone pressure solve on host arrays (fl_solve_pressure)
  relax     the reference's relaxation solvers on host arrays (fl_relax_pressure)
  noalloc   the pressure solve on device arrays without allocation (fl_solve_pressure_noalloc)

Particles are a liquid region of the tank in motion: eight jittered particles per cell, displaced by a third of a cell
(so that cells hold unequal numbers and the surface is rough), with a smooth swirl and some noise as velocity, and a
hydrostatic pressure as the previous substep's.  `exact` is the same step in 64 bits in plain torch.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluid-simulation_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from fluidgb import _abi, scenes  # noqa: E402

DT = float(np.float32(1.0 / 120.0))
GRAVITY = float(np.float32(-9.81))
RHO = 1000.0


def _grid(nx, ny=None, nz=None):
    return {"nx": nx, "ny": ny or nx, "nz": nz or nx}


def _fluid(x=1.0, y=1.0, z=1.0, drop=0.0):
    """Liquid below (x, y, z) of the tank's extent, with a sphere of radius `drop` above it if that is not 0."""
    return {"x": x, "y": y, "z": z, "drop": drop}


def _opts(iters=200, tol=1e-5, precision=0, solver=0, advect=1, friction=0.0, dilation=0, flip=0.95):
    return {"iters": iters, "tol": tol, "precision": precision, "solver": solver, "advect": advect,
            "friction": friction, "dilation": dilation, "flip": flip}


def listed():
    return [
        # a frame of the small interactive tank: every launch and every wait counts
        dict(name="frame_dam32", op="frame", **_grid(32), **_fluid(0.4, 0.6), **_opts(iters=40, tol=1e-4)),
        # the differentiable-rollout scene's forward step
        dict(name="step_block64", op="step", **_grid(64), **_fluid(0.5, 0.4), **_opts()),
        # the headline: a 128^3 dam break with two million particles
        dict(name="step_dam128", op="step", **_grid(128), **_fluid(0.5, 0.5, 0.5), **_opts()),
        # the full-depth dam with the extended-precision reductions
        dict(name="step_dam128_f64", op="step", **_grid(128), **_fluid(0.5, 0.5), **_opts(precision=1)),
        # the largest grid of the configurations, 18 million particles
        dict(name="step_block256", op="step", **_grid(256), **_fluid(0.4, 0.35), **_opts()),
        # sphere into a pool through the multigrid-preconditioned solver
        dict(name="step_pool128_mg", op="step", **_grid(128), **_fluid(1.0, 0.3, 1.0, drop=0.12), **_opts(solver=1)),
        # a caller's own buffer in a tank of odd sizes, with the midpoint advection, wall friction and dilation
        # and the settings' default of thirty iterations without a tolerance
        dict(name="inplace_odd", op="inplace", **_grid(97, 61, 83), **_fluid(0.6, 0.5),
             **_opts(iters=30, tol=0.0, advect=2, friction=0.1, dilation=1, flip=0.9)),
        # one recorded substep and its adjoint: a control loop's gradient at 64^3, plain CG
        dict(name="adjoint_block64", op="adjoint", **_grid(64), **_fluid(0.5, 0.4), **_opts()),
        # the same at the headline size, adjoint systems through the multigrid preconditioner
        dict(name="adjoint_dam128", op="adjoint", **_grid(128), **_fluid(0.5, 0.5, 0.5), **_opts(), adj_solver=1),
        # a host program's pressure projection
        dict(name="poisson_96", op="poisson", **_grid(96, 80, 72), **_opts()),
        # the reference's fallback smoother as a solver
        dict(name="relax_rbgs_64", op="relax", **_grid(64, 64, 64), method=1, sweeps=100),
        # a plug-in's solve in a frame loop without allocation
        dict(name="noalloc_48", op="noalloc", **_grid(48, 40, 56), **_opts(iters=100, tol=1e-4)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["frame", "step", "step", "step", "inplace", "adjoint", "poisson", "relax", "noalloc"])
    lo, hi = {"frame": (20, 56), "step": (32, 224), "inplace": (32, 160), "adjoint": (32, 128), "poisson": (24, 128),
              "relax": (24, 128), "noalloc": (20, 60)}[op]
    nx = _log_int(rng, lo, hi)
    case = dict(op=op, **_grid(nx, max(16, int(nx * rng.uniform(0.7, 1.05))), max(16, int(nx * rng.uniform(0.7, 1.05)))))
    if op == "relax":
        case.update(method=rng.randrange(2), sweeps=_log_int(rng, 10, 150))
        return case
    opts = _opts(iters=rng.choice([30, 60, 120, 200]), tol=rng.choice([1e-3, 1e-4, 1e-5]), precision=rng.randrange(2))
    if op in ("frame", "step", "inplace", "adjoint"):
        case.update(_fluid(rng.uniform(0.3, 0.9), rng.uniform(0.2, 0.5), rng.uniform(0.4, 1.0)))
        opts.update(flip=rng.choice([0.9, 0.95, 0.99]), dilation=rng.randrange(2))
        if op == "frame":
            opts["precision"] = 0
        if op == "step":
            opts["solver"] = rng.choice([0, 0, 1])
        if op == "inplace":
            opts.update(advect=rng.choice([1, 2]), friction=rng.choice([0.0, 0.1]))
        if op == "adjoint":
            case["adj_solver"] = rng.randrange(2)
            opts["dilation"] = 0
    case.update(opts)
    return case


# ---------------------------------------------------------------------------
# inputs


def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


def _dims(c):
    return c["nx"], c["ny"], c["nz"]


def _params(c):
    p = scenes.params_for(c["nx"], flip=c["flip"], iters=c["iters"], tol=c["tol"], precision=c["precision"],
                          warm_start=c["op"] != "inplace", advect_order=c["advect"], ny=c["ny"], nz=c["nz"])
    p.phys[3] = c["friction"]
    p.cls[1] = float(c["dilation"])
    p.pressure_solver = c["solver"]
    return p


def _wet(c, dev):
    """(nz, ny, nx) mask of the interior cells whose centre is in the liquid region."""
    nx, ny, nz = _dims(c)
    x = ((torch.arange(nx, device=dev) + 0.5) / nx).view(1, 1, nx)
    y = ((torch.arange(ny, device=dev) + 0.5) / ny).view(1, ny, 1)
    z = ((torch.arange(nz, device=dev) + 0.5) / nz).view(nz, 1, 1)
    m = (x < c["x"]) & (y < c["y"]) & (z < c["z"])
    if c["drop"] > 0:
        m = m | ((x - 0.5) ** 2 + (y - 0.75) ** 2 + (z - 0.5) ** 2 < c["drop"] ** 2)
    m = m.clone()
    m[0], m[-1], m[:, 0], m[:, -1], m[:, :, 0], m[:, :, -1] = False, False, False, False, False, False
    return m


def _scene(c, seed):
    """Particles (N, 8) and the previous substep's pressure (C), both float32."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    nx, ny, nz = _dims(c)
    h = 1.0 / nx
    wet = _wet(c, dev)
    cell = wet.nonzero()  # z, y, x
    n = cell.shape[0] * 8
    sub = torch.tensor([[s & 1, (s >> 1) & 1, s >> 2] for s in range(8)], device=dev, dtype=torch.float32)
    pos = cell.flip(1).to(torch.float32).repeat_interleave(8, 0) + 0.5 * sub.repeat(cell.shape[0], 1)
    pos += 0.5 * torch.rand((n, 3), generator=g, device=dev)
    pos += 0.33 * torch.randn((n, 3), generator=g, device=dev)
    pos *= h
    top = torch.tensor([nx * h, ny * h, nz * h], device=dev)
    pos = torch.minimum(torch.clamp(pos, min=1.06 * h), top - 1.06 * h)
    phase = 2 * math.pi * torch.rand(6, generator=g, device=dev)
    k = 2 * math.pi * pos / top
    vel = 0.05 * torch.randn((n, 3), generator=g, device=dev)
    vel[:, 0] += 0.4 * torch.sin(k[:, 1] + phase[0]) + 0.2 * torch.sin(k[:, 2] + phase[1])
    vel[:, 1] += 0.3 * torch.sin(k[:, 2] + phase[2]) + 0.2 * torch.sin(k[:, 0] + phase[3])
    vel[:, 2] += 0.3 * torch.sin(k[:, 0] + phase[4]) + 0.2 * torch.sin(k[:, 1] + phase[5])
    parts = torch.zeros((n, 8), device=dev, dtype=torch.float32)
    parts[:, 0:3] = pos
    parts[:, 4:7] = vel
    y = ((torch.arange(ny, device=dev) + 0.5) * h).view(1, ny, 1)
    depth = torch.clamp(c["y"] * ny * h - y, min=0.0).expand(nz, ny, nx)
    p0 = -RHO * GRAVITY * depth * (1.0 + 0.05 * torch.randn((nz, ny, nx), generator=g, device=dev))
    p0 = torch.where(wet, p0, torch.zeros_like(p0)).to(torch.float32).contiguous()
    return parts, p0.reshape(-1)


def _field(c, seed):
    """Cell types (uint8) and divergence (float32) of a stand-alone solve, (nz, ny, nx): a tank three fifths full under
    a wavy surface, a few solid blocks in it, and a divergence with large and small scales."""
    nx, ny, nz = _dims(c)
    rs = np.random.RandomState(int(seed) % (1 << 32))
    x, z = np.arange(nx)[None, :] / nx, np.arange(nz)[:, None] / nz
    a = rs.uniform(0, 2 * np.pi, 4)
    level = ny * (0.6 + 0.08 * np.sin(2 * np.pi * x + a[0]) + 0.08 * np.sin(4 * np.pi * z + a[1]))
    ct = np.where(np.arange(ny)[None, :, None] < level[:, None, :], 1, 2).astype(np.uint8)
    for _ in range(3):
        o = [rs.randint(1, max(2, n - n // 6 - 1)) for n in (nz, ny, nx)]
        ct[o[0]:o[0] + nz // 6, o[1]:o[1] + ny // 6, o[2]:o[2] + nx // 6] = 0
    ct[0], ct[-1], ct[:, 0], ct[:, -1], ct[:, :, 0], ct[:, :, -1] = 0, 0, 0, 0, 0, 0
    div = np.sin(2 * np.pi * x[:, None, :] + a[2]) * np.cos(2 * np.pi * np.arange(ny)[None, :, None] / ny + a[3])
    div = div + 0.5 * rs.standard_normal((nz, ny, nx))
    return ct, np.where(ct == 1, div, 0.0).astype(np.float32)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    op = case["op"]
    if op in ("poisson", "relax", "noalloc"):
        s.ct, s.div = _field(case, seed)
        s.h = float(np.float32(1.0 / case["nx"]))
        if op == "noalloc":
            dev = _device()
            s.lib = _abi.load_library()
            s.ct = torch.from_numpy(s.ct).to(dev)
            s.div = torch.from_numpy(s.div).to(dev)
            s.p = torch.zeros_like(s.div)
            s.stream = torch.cuda.Stream(dev)
            torch.cuda.current_stream().synchronize()
        return s
    dev = _device()
    s.parts, p0 = _scene(case, seed)
    n = s.parts.shape[0]
    s.n = n
    s.stream = torch.cuda.Stream(dev)
    s.fluid = _abi.Fluid(_params(case), n)
    s.fluid.set_stream(s.stream.cuda_stream)
    s.out = torch.empty((n, 8), dtype=torch.float32, device=dev)
    torch.cuda.current_stream().synchronize()
    if op == "inplace":
        return s
    # the state a program checkpoints: these particles, and p0 as the pressure of the substep before
    s.fluid.set_particles_device(s.parts.data_ptr(), n)
    s.fluid.step_replay(p0.data_ptr())
    s.fluid.set_particles_device(s.parts.data_ptr(), n)
    s.size = s.fluid.state_size()
    s.blob = torch.empty(s.size, dtype=torch.uint8, device=dev)
    s.fluid.save_state_device(s.blob.data_ptr(), s.size)
    s.ids = torch.empty(n, dtype=torch.int32, device=dev)
    if op == "adjoint":
        s.g_out, s.g_in = _gradient(case, seed, n), torch.empty((n, 8), dtype=torch.float32, device=dev)
        s.tape = s.fluid.tape(1)
        if case.get("adj_solver"):
            s.tape.set_adjoint_solver(_abi.FL_SOLVER_MGPCG)
    else:
        s.pressure = torch.empty(p0.shape, dtype=torch.float32, device=dev)
    torch.cuda.current_stream().synchronize()
    s.fluid.sync()
    s.parts = None
    return s


def _gradient(case, seed, n):
    """dL/d(particles after the substep): a loss on positions and velocities, unequal over the particles."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) + 77)
    out = torch.zeros((n, 8), device=dev, dtype=torch.float32)
    out[:, 0:3] = 1.0 + 0.5 * torch.randn((n, 3), generator=g, device=dev)
    out[:, 4:7] = 0.05 * torch.randn((n, 3), generator=g, device=dev)
    return out


def run(s):
    c, op = s.case, s.case["op"]
    if op == "poisson":
        return _abi.solve_pressure(s.ct, s.div, _dims(c), s.h, RHO, DT, c["iters"], tolerance=c["tol"],
                                   precision=c["precision"])[0]
    if op == "relax":
        return _abi.relax_pressure(s.ct, s.div, _dims(c), s.h, RHO, DT, c["method"], c["sweeps"])
    if op == "noalloc":
        st = s.lib.fl_solve_pressure_noalloc(*_dims(c), s.ct.data_ptr(), s.div.data_ptr(), s.p.data_ptr(), s.h, RHO, DT,
                                             c["iters"], 0, c["tol"], c["precision"], s.stream.cuda_stream, None)
        if st != 0:
            raise RuntimeError(s.lib.fl_last_error(None).decode())
        return s.p
    f = s.fluid
    if op == "inplace":
        with torch.cuda.stream(s.stream):
            s.out.copy_(s.parts)
        f.step_device(s.out.data_ptr(), s.n)
        return s.out
    f.load_state_device(s.blob.data_ptr(), s.size)
    if op == "adjoint":
        s.tape.clear()
        s.tape.record()
        f.get_particles_device(s.out.data_ptr())
        grav = s.tape.adjoint(s.g_out.data_ptr(), s.g_in.data_ptr(), 1000, 1e-6)
        return {"particles": s.out, "gradient": s.g_in, "gravity": np.array(grav, np.float32)}
    f.step(4 if op == "frame" else 1)
    f.copy_pressure_device(s.pressure.data_ptr())
    f.get_particles_device(s.out.data_ptr(), s.ids.data_ptr())
    return {"particles": s.out, "ids": s.ids, "pressure": s.pressure}


def work(case):
    c, op = case, case["op"]
    cells = c["nx"] * c["ny"] * c["nz"]
    if op == "relax":
        liquid = 0.6 * cells
        return {"bytes": 9 * cells, "flops": 9 * liquid * c["sweeps"]}
    if op in ("poisson", "noalloc"):
        liquid = 0.6 * cells
        return {"bytes": 9 * cells, "flops": 21 * liquid * c["iters"]}
    liquid = min(1.0, c["x"] * c["y"] * c["z"] + 4.19 * c["drop"] ** 3) * cells
    n = 8 * liquid
    # particles and ids in and out; the pressure in and out; per particle 24 taps each way; per liquid cell the
    # iterations' stencil, products and updates (the multigrid solver: about a tenth of them, each ten times dearer)
    steps = 4 if op == "frame" else 1
    w = {"bytes": steps * (72 * n + 8 * cells), "flops": steps * (500 * n + 21 * liquid * c["iters"])}
    if op == "adjoint":
        w = {"bytes": w["bytes"] + 64 * n, "flops": 3 * w["flops"]}
    return w


# ---------------------------------------------------------------------------
# the same results in 64 bits


def _neighbours(x):
    """-x, +x, -y, +y, -z, +z of a (nz, ny, nx) field (used where the outer layer is solid)."""
    return [torch.roll(x, sh, d) for d in (2, 1, 0) for sh in (1, -1)]


class _Poisson:
    """Count of non-solid neighbours times x minus the sum of liquid neighbours, on the liquid cells."""

    def __init__(self, ct):
        self.liquid = ct == 1
        self.masks = [(t == 1) & self.liquid for t in _neighbours(ct)]
        self.count = sum((t != 0).double() for t in _neighbours(ct)) * self.liquid

    def apply(self, x):
        s = torch.zeros_like(x)
        for m, t in zip(self.masks, _neighbours(x)):
            s = s + torch.where(m, t, 0.0)
        return self.count * x - s

    def solve(self, rhs, x0, iters, tol):
        x = torch.where(self.liquid, x0, 0.0)
        r = torch.where(self.liquid, rhs - self.apply(x), 0.0)
        d, rs = r.clone(), float((r * r).sum())
        stop = tol * tol * rs
        for _ in range(iters):
            q = self.apply(d)
            dq = float((d * q).sum())
            alpha = rs / dq if abs(dq) > 1e-30 else 0.0
            x = x + alpha * d
            r = r - alpha * q
            new = float((r * r).sum())
            if new <= stop and tol > 0:
                break
            d = r + (new / rs if rs > 1e-30 else 0.0) * d
            rs = new
        return x


class _Solve(torch.autograd.Function):
    @staticmethod
    def forward(ctx, rhs, op, x0, iters, tol):
        ctx.op = op
        return op.solve(rhs, x0, iters, tol)

    @staticmethod
    def backward(ctx, g):
        g = torch.where(ctx.op.liquid, g, 0.0)
        return ctx.op.solve(g, torch.zeros_like(g), 3000, 1e-11), None, None, None, None


def _tap(q, axis, dims):
    """Base cell and fractions of the trilinear stencil of the faces of `axis` (x, y, z order)."""
    g = q - 0.5
    g = torch.stack([q[:, b] if b == axis else g[:, b] for b in range(3)], 1)
    base = torch.floor(g.detach())
    return base.long(), g - base


def _taps(q, axis, dims):
    """For each of the eight taps: face coordinates, flat index (clamped), in-range mask and weight."""
    base, t = _tap(q, axis, dims)
    dim = [dims[b] + (b == axis) for b in range(3)]
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                f = [base[:, 0] + di, base[:, 1] + dj, base[:, 2] + dk]
                ok = torch.ones_like(f[0], dtype=torch.bool)
                for b in range(3):
                    ok &= (f[b] >= 0) & (f[b] < dim[b])
                i, j, k = (f[b].clamp(0, dim[b] - 1) for b in range(3))
                w = (t[:, 0] if di else 1 - t[:, 0]) * (t[:, 1] if dj else 1 - t[:, 1]) * (t[:, 2] if dk else 1 - t[:, 2])
                yield f, i + dim[0] * (j + dim[1] * k), ok, w


def _near_wall(f, axis, dims):
    m = torch.zeros_like(f[0], dtype=torch.bool)
    for b in range(3):
        m |= (f[b] <= (1 if b == axis else 0)) | (f[b] >= dims[b] - 1)
    return m


def _gather(fields, q, axis, dims):
    sums, ws = [0.0] * len(fields), 0.0
    for f, idx, ok, w in _taps(q, axis, dims):
        w = torch.where(ok & ~_near_wall(f, axis, dims), w, 0.0)
        sums = [s + w * v.reshape(-1)[idx] for s, v in zip(sums, fields)]
        ws = ws + w
    return [torch.where(ws > 0, s / torch.where(ws > 0, ws, 1.0), 0.0) for s in sums]


def _cap(v, most):
    sp = torch.sqrt((v * v).sum(1) + 1e-300)
    return v * torch.where(sp > most, most / sp, torch.ones_like(sp))[:, None]


def _substep(c, parts, p0, gravity=None, smooth=False):
    """One substep in double: particles after it (in bin order), the order, and the pressure.  smooth: the P2G sums
    unrounded, as the adjoint linearises them."""
    dims = _dims(c)
    nx, ny, nz = dims
    dev = parts.device
    h32 = np.float32(1.0) / np.float32(nx)
    h, inv_h, flip = float(h32), float(np.float32(1.0) / h32), float(np.float32(c["flip"]))
    pos, vel = parts[:, 0:3], parts[:, 4:7]
    # bins by the float32 quotient, as the binning is defined
    key32 = torch.floor(pos.detach().float() / torch.tensor(h32, device=dev)).long()
    key = [key32[:, b].clamp(0, dims[b] - 1) for b in range(3)]
    key = key[0] + nx * (key[1] + ny * key[2])
    perm = torch.sort(key, stable=True).indices
    count = torch.bincount(key, minlength=nx * ny * nz).view(nz, ny, nx)
    liquid = count >= 1
    if c["dilation"]:
        base = liquid
        for t in _neighbours(base):
            liquid = liquid | t
    ct = torch.where(liquid, 1, 2)
    ct[0], ct[-1], ct[:, 0], ct[:, -1], ct[:, :, 0], ct[:, :, -1] = 0, 0, 0, 0, 0, 0
    pos, vel = pos[perm], vel[perm]
    q = pos * inv_h
    scale = 65536.0
    grav = gravity if gravity is not None else torch.tensor([0.0, GRAVITY, 0.0], device=dev, dtype=torch.float64)
    saved, face, low, high, shapes = [], [], [], [], []
    for a in range(3):
        shape = [nz + (a == 2), ny + (a == 1), nx + (a == 0)]
        num = torch.zeros(shape[0] * shape[1] * shape[2], dtype=torch.float64, device=dev)
        den = torch.zeros_like(num)
        for _, idx, ok, w in _taps(q, a, dims):
            w = torch.where(ok, w, 0.0)
            if smooth:
                num, den = num.index_add(0, idx, w * vel[:, a]), den.index_add(0, idx, w)
            else:
                num.index_add_(0, idx, torch.round(w * vel[:, a] * scale))
                den.index_add_(0, idx, torch.round(w * scale))
        v = torch.where(den > 0, num / torch.where(den > 0, den, 1.0), 0.0).view(shape)
        d = 2 - a
        solid = torch.zeros_like(ct.narrow(d, 0, 1))
        lo, hi = torch.cat([solid, ct], d), torch.cat([ct, solid], d)
        saved.append(v)
        v = v + torch.where((lo == 1) | (hi == 1), grav[a] * DT, 0.0)
        face.append(torch.where((lo == 0) | (hi == 0), 0.0, v))
        low.append(lo)
        high.append(hi)
    div = sum(face[a].narrow(2 - a, 1, dims[a]) - face[a].narrow(2 - a, 0, dims[a]) for a in range(3)) * inv_h
    drift = torch.clamp(float(np.float32(0.45)) * torch.clamp(count - 8.0, min=0.0) / 8.0, max=0.5)
    div = div - drift
    op = _Poisson(ct)
    rhs = torch.where(op.liquid, -(RHO * h * h / DT) * div, 0.0)
    # the reference's CG to its own stopping test; the multigrid solver and the adjoint: the solution
    exact_solve = c["solver"] == 1 or smooth
    p = _Solve.apply(rhs, op, p0, 3000 if exact_solve else c["iters"], 1e-11 if exact_solve else float(np.float32(c["tol"])))
    final = []
    zero = torch.zeros(1, dtype=torch.float64, device=dev)
    for a in range(3):
        d = 2 - a
        pad = zero.expand(p.narrow(d, 0, 1).shape)
        on = (low[a] != 0) & (high[a] != 0) & ((low[a] == 1) | (high[a] == 1))
        dp = torch.cat([p, pad], d) - torch.cat([pad, p], d)
        final.append(face[a] - torch.where(on, DT / RHO / h * dp, 0.0))
    got = [_gather([final[a], saved[a]], q, a, dims) for a in range(3)]
    pic, old = torch.stack([g[0] for g in got], 1), torch.stack([g[1] for g in got], 1)
    most = 2.0 * h / DT
    new = _cap(pic * (1 - flip) + (vel + pic - old) * flip, most)
    lo = torch.full((3,), 1.05 * h, dtype=torch.float64, device=dev)
    hi = torch.tensor([n * h for n in dims], dtype=torch.float64, device=dev) - 1.05 * h
    fr = float(np.float32(c["friction"]))
    if fr > 0:
        band = 2.5 * h
        near = torch.clamp(1 - torch.minimum((pos - lo) / band, (hi - pos) / band), 0.0, 1.0)
        most_of = torch.stack([torch.maximum(near[:, (b + 1) % 3], near[:, (b + 2) % 3]) for b in range(3)], 1)
        new = new * (1 - fr * most_of)
    if c["advect"] == 2:
        mid = (pos + _cap(pic, most) * (0.5 * DT)) * inv_h
        at = pos + _cap(torch.stack([_gather([final[a]], mid, a, dims)[0] for a in range(3)], 1), most) * DT
    else:
        at = pos + new * DT
    out_of = (at < lo) | (at > hi)
    new = torch.where(out_of, 0.0, new)
    at = torch.minimum(torch.maximum(at, lo), hi)
    z = torch.zeros((at.shape[0], 1), dtype=torch.float64, device=dev)
    return torch.cat([at, z, new, z], 1), perm, p.reshape(-1)


def exact(case, seed):
    c, op = case, case["op"]
    dev = _device()
    if op == "frame":
        return None  # after the first substep, rounding decides which particle is in which bin
    if op in ("poisson", "relax", "noalloc"):
        ct, div = (torch.from_numpy(v).to(dev) for v in _field(c, seed))
        h = float(np.float32(1.0 / c["nx"]))
        A = _Poisson(ct.long())
        b = torch.where(A.liquid, -(RHO * h * h / DT) * div.double(), 0.0)
        x = torch.zeros_like(b)
        if op == "relax":
            i = [torch.arange(n, device=dev) for n in ct.shape]
            odd = (i[0].view(-1, 1, 1) + i[1].view(1, -1, 1) + i[2].view(1, 1, -1)) % 2
            n = torch.where(A.count > 0, A.count, 1.0)
            for _ in range(c["sweeps"]):
                for phase in ((0, 1) if c["method"] else (None,)):
                    y = torch.where(A.liquid & (A.count > 0), (b + A.count * x - A.apply(x)) / n, 0.0)
                    x = y if phase is None else torch.where(odd == phase, y, x)
        else:
            x = A.solve(b, x, c["iters"], float(np.float32(c["tol"])))
        return x if op == "noalloc" else x.reshape(ct.shape)
    parts, p0 = _scene(c, seed)
    parts = parts.double()
    p0 = p0.double().view(c["nz"], c["ny"], c["nx"])
    if op == "inplace":
        return _substep(c, parts, torch.zeros_like(p0))[0]
    if op == "step":
        out, perm, p = _substep(c, parts, p0)
        return {"particles": out, "ids": perm.to(torch.int32), "pressure": p}
    out = _substep(c, parts, p0)[0]
    parts.requires_grad_(True)
    grav = torch.tensor([0.0, GRAVITY, 0.0], device=dev, dtype=torch.float64, requires_grad=True)
    end = _substep(c, parts, p0, grav, smooth=True)[0]
    g, gg = torch.autograd.grad(end, [parts, grav], _gradient(c, seed, parts.shape[0]).double())
    return {"particles": out.detach(), "gradient": g, "gravity": gg}
