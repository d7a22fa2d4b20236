"""Measured cases of the flux-advection library: what a program that uses it has it do.

Every case goes through the public Python entry points of `fia` (a mirror of the C ABI in
include/fia.h) on a device-resident session, as the reference's main loop calls them: a density
step, a velocity step, a projection, a whole smoke step, a training step of the learned
preconditioner.  Sizes are those of the repository's benchmark configurations, tests and report
scripts (16^3, 64^3, 128^3, 256^3, ragged grids), and `draw` spreads over the ranges between.

`prepare` fills a session with seeded fields: a divergence-free Fourier flow, Gaussian blobs, the
plume.  `run` puts the inputs back into the session's fields (a step replaces them) and makes one
call; its outputs are views of the session's fields.  `exact` restates the scheme in 64 bits with
plain torch operations.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "flux-interpolated-advection_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import fia  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"
MAX_DT = 1.0 / 60.0     # one step per movie frame, the default of fia_step


def listed():
    def case(name, kind, nx, ny, nz, **kw):
        c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": "fp32c", "cfl": 2.0,
             "interp": "WENO6", "split": "xz-CellFaceAligned", "k": 3, "zero_velocity_passes": True,
             "maccormack": False}
        c.update(kw)
        return c

    return [
        # the smallest call: a preview grid, where launches and host latency count
        case("density_16", "density", 16, 16, 16),
        # the isolated advection operator of the benchmark: its grid, CFL number and defaults
        case("density_128", "density", 128, 128, 128),
        # the same call on a production grid
        case("density_256", "density", 256, 256, 256),
        # the drop-in call of a program that keeps its grid in (pinned) host memory
        case("density_128_host", "host", 128, 128, 128),
        # velocity self-advection of all three components on a ragged box
        case("velocity_ragged", "velocity", 120, 161, 77, cfl=1.5),
        # the flux MacCormack option with a finer Gauss rule, odd sizes, long faces
        case("maccormack_ragged", "density", 70, 97, 51, maccormack=True, k=5, cfl=3.0),
        # the cheap options: linear interpolation, one pass, another split, Gauss midpoint
        case("linear_tall", "density", 96, 250, 101, interp="linear", k=1, zero_velocity_passes=False,
             split="x-CellFaceAligned_z-AxisAligned", cfl=1.0),
        # the plain double-precision form, which a user picks as the reference run (a 64^3 plume)
        case("density_fp64_64", "density", 64, 64, 64, precision="fp64", cfl=1.0),
        # projection with the default solver
        case("projection_128", "projection", 128, 128, 128, tol=1e-6, spheres=0),
        # projection with the learned preconditioner, at the size from which it is the faster one
        case("projection_learned_256", "learned", 256, 256, 256, tol=1e-6, spheres=0),
        # a whole smoke step of a 64^3 plume at CFL 1 with a tight pressure tolerance
        case("step_64", "step", 64, 64, 64, cfl=1.0, tol=1e-8),
        # one training step (forward, backward, Adam) of the preconditioner
        case("train_64", "train", 64, 64, 64, batch=4),
    ]


def draw(rng):
    def grid(lo, hi):
        """three sizes whose product is spread over its logarithm between lo^3 and hi^3"""
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        a, b = math.exp(rng.uniform(-0.4, 0.4)), math.exp(rng.uniform(-0.4, 0.4))
        return {d: max(8, int(round(v))) for d, v in (("nx", n * a), ("ny", n * b), ("nz", n / (a * b)))}

    kind = rng.choice(["density"] * 5 + ["host", "velocity", "velocity", "projection", "learned", "step", "train"])
    c = {"kind": kind, "precision": "fp32c", "cfl": round(rng.uniform(0.5, 4.0), 2), "interp": "WENO6",
         "split": "xz-CellFaceAligned", "k": rng.choice([1, 3, 3, 5]), "zero_velocity_passes": rng.random() < 0.8,
         "maccormack": False}
    if kind == "density":
        c["precision"] = rng.choice(["fp32c", "fp32c", "fp64"])
        c["interp"] = rng.choice(["WENO6", "WENO6", "WENO6", "linear"])
        c["split"] = rng.choice(sorted(fia.SPLIT))
        c["maccormack"] = rng.random() < 0.25
        big = 150 if c["maccormack"] or c["k"] == 5 else 200
        c.update(grid(16, 48 if c["precision"] == "fp64" else big))
    elif kind == "host":
        c.update(grid(16, 180))
    elif kind == "velocity":
        c["precision"] = rng.choice(["fp32c", "fp32c", "fp64"])
        c.update(grid(12, 32 if c["precision"] == "fp64" else 110))
    elif kind == "projection":
        c["precision"] = rng.choice(["fp32c", "fp64"])
        c.update(grid(16, 110), tol=rng.choice([1e-6, 1e-8]), spheres=rng.choice([0, 0, 3]))
    elif kind == "learned":
        c.update(grid(64, 200), tol=1e-6, spheres=0)
    elif kind == "step":
        c.update(grid(16, 80), tol=rng.choice([1e-6, 1e-8]), cfl=rng.choice([1.0, 2.0]))
    else:
        c.update(grid(24, 80), batch=rng.choice([1, 2, 4]))
    return c


# ------------------------------------------------------------------------------------
# inputs: seeded fields in 64 bits, made on the GPU
# ------------------------------------------------------------------------------------
def _h(case):
    return 1.0 / max(case["nx"], case["ny"], case["nz"])


def _flow(shape, h, rng):
    """The discrete curl of 16 Fourier modes (wavenumbers 1-8) under a window that vanishes on the
    walls: divergence-free, zero through the walls, the largest face velocity 1."""
    modes = []
    while len(modes) < 16:
        k = rng.integers(-8, 9, size=3)
        kn = float(np.sqrt((k * k).sum()))
        if 1 <= kn <= 8:
            modes.append((k, rng.normal(size=3) / kn, rng.uniform(0, 2 * np.pi)))
    kv = torch.tensor(np.array([m[0] for m in modes]), dtype=torch.float64, device=DEV)
    amp = torch.tensor(np.array([m[1] for m in modes]), dtype=torch.float64, device=DEV)
    ph = torch.tensor([m[2] for m in modes], dtype=torch.float64, device=DEV)
    node = [torch.arange(n + 1, dtype=torch.float64, device=DEV) * h for n in shape]
    mid = [(torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) * h for n in shape]

    def potential(c, *x):
        e = [torch.exp(2j * math.pi * kv[:, d, None] * x[d]) for d in range(3)]
        left = torch.einsum("m,mx,my->xym", amp[:, c] * torch.exp(1j * ph), e[0], e[1])
        a = torch.matmul(left, e[2]).imag
        for d in range(3):
            s = torch.sin(math.pi * x[d] / (shape[d] * h))
            a = a * s.reshape([-1 if q == d else 1 for q in range(3)])
        return a

    ax, ay, az = (potential(c, *[mid[d] if d == c else node[d] for d in range(3)]) for c in range(3))
    u = (az[:, 1:] - az[:, :-1]) / h - (ay[:, :, 1:] - ay[:, :, :-1]) / h
    v = (ax[:, :, 1:] - ax[:, :, :-1]) / h - (az[1:] - az[:-1]) / h
    w = (ay[1:] - ay[:-1]) / h - (ax[:, 1:] - ax[:, :-1]) / h
    m = max(float(f.abs().max()) for f in (u, v, w))
    return [f / m for f in (u, v, w)]


def _blobs(shape, h, rng):
    """32 Gaussian blobs of widths 0.02 to 0.08"""
    g = []
    ctr, sig, amp = rng.uniform(0.15, 0.85, size=(32, 3)), rng.uniform(0.02, 0.08, size=32), rng.uniform(0.5, 1.0, size=32)
    for d in range(3):
        x = (torch.arange(shape[d], dtype=torch.float64, device=DEV) + 0.5) * h
        c = torch.tensor(ctr[:, d] * shape[d] * h, device=DEV)
        s = torch.tensor(sig, device=DEV)
        g.append(torch.exp(-0.5 * ((x - c[:, None]) / s[:, None]) ** 2))
    left = torch.einsum("b,bx,by->xyb", torch.tensor(amp, device=DEV), g[0], g[1])
    return torch.matmul(left, g[2])


def _inputs(case, seed):
    """(density, u, v, w, dt) in 64 bits, rounded to what a session of the case's precision holds"""
    rng = np.random.Generator(np.random.PCG64(seed))
    shape, h = (case["nx"], case["ny"], case["nz"]), _h(case)
    u, v, w = _flow(shape, h, rng)
    dt = case["cfl"] * h
    if case["kind"] == "step":
        # the plume source in a developed flow that reaches the CFL number at the frame's length
        x = [(torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) * h for n in shape]
        r2 = (x[0][:, None, None] - 0.5) ** 2 + (x[1][None, :, None] - 0.15) ** 2 + (x[2] - 0.5) ** 2
        rho, dt = (r2 <= 0.01).double() + 0.5 * _blobs(shape, h, rng), MAX_DT
        u, v, w = (f * (case["cfl"] * h / MAX_DT) for f in (u, v, w))
    else:
        rho = _blobs(shape, h, rng)
    if case["kind"] in ("projection", "learned"):
        # what a projection is given: a flow after advection and buoyancy, no longer divergence-free
        v = v.clone()
        v[:, 1:-1] += 0.25 * (rho[:, 1:] + rho[:, :-1])
    if case["precision"] == "fp32c":
        rho, u, v, w = (f.float().double() for f in (rho, u, v, w))
    return rho, u, v, w, dt


# ------------------------------------------------------------------------------------
# sessions
# ------------------------------------------------------------------------------------
class _Memory:
    """a session's field for torch.as_tensor, which keeps this object, and so the session, as long
    as a tensor on it lives"""

    def __init__(self, grid, ptr, shape, kind):
        self.grid = grid
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": kind, "version": 2}


class _State:
    def __init__(self, case, seed):
        self.kind = case["kind"]
        n = (case["nx"], case["ny"], case["nz"])
        self.shapes = {"density": n, "pressure": n, "u": (n[0] + 1, n[1], n[2]), "v": (n[0], n[1] + 1, n[2]),
                       "w": (n[0], n[1], n[2] + 1)}
        fp32 = case["precision"] == "fp32c"
        self.typestr = "<f4" if fp32 else "<f8"
        self.grid = fia.Grid3D(*n, _h(case), precision=fia.FIA_FP32C if fp32 else fia.FIA_FP64)
        self.stream = torch.cuda.ExternalStream(self.grid.stream())
        self.views = {}
        self.params = fia.advect_params(interpolation_method=case["interp"], split_method=case["split"],
                                        num_gauss_quadrature_point_for_integrate_density=case["k"],
                                        enable_eliminate_zero_velocity_false_diffusion=case["zero_velocity_passes"],
                                        use_MacCormack_scheme=case["maccormack"])
        rho, u, v, w, self.dt = _inputs(case, seed)
        t = torch.float32 if fp32 else torch.float64
        self.given = {k: f.to(t).contiguous() for k, f in (("density", rho), ("u", u), ("v", v), ("w", w))}
        torch.cuda.synchronize()
        self.put(*self.given)

    def view(self, name):
        """the session's field as a tensor (a step exchanges the buffers behind a field)"""
        p = self.grid.device_ptr(name)
        t = self.views.get(p)
        if t is None or t.shape != self.shapes[name]:
            t = self.views[p] = torch.as_tensor(_Memory(self.grid, p, self.shapes[name], self.typestr), device="cuda")
        return t

    def put(self, *names):
        with torch.cuda.stream(self.stream):
            for k in names:
                self.view(k).copy_(self.given[k])


def _smooth_pair(shape, rng):
    """a training pair B p = r: p smooth noise, r its 7-point operator with zero-flux walls and
    the last cell pinned"""
    p = torch.tensor(rng.normal(size=shape), device=DEV)
    for d in range(3):
        n = shape[d]
        x = torch.arange(n, dtype=torch.float64, device=DEV)
        g = torch.exp(-0.5 * ((x[:, None] - x) / 3.0) ** 2)
        p = torch.movedim(torch.tensordot(g / g.sum(1, keepdim=True), p, dims=([1], [d])), 0, d).contiguous()
    p.view(-1)[-1] = 0.0
    r = torch.zeros_like(p)
    for d in range(3):
        diff = torch.diff(p, dim=d)
        z = torch.zeros_like(p.narrow(d, 0, 1))
        r += torch.cat([z, diff], d) - torch.cat([diff, z], d)
    r.view(-1)[-1] = 0.0
    return r.float().cpu().numpy(), p.float().cpu().numpy()


def prepare(case, seed):
    s = _State(case, seed)
    g = s.grid
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    if s.kind == "host":
        s.host = {}
        for k, f in s.given.items():
            s.host[k] = torch.empty(f.shape, dtype=f.dtype, pin_memory=True)
            s.host[k].copy_(f)
        s.ptrs = [s.host[k].data_ptr() for k in ("density", "u", "v", "w")]
    if s.kind in ("projection", "learned", "step"):
        s.solver = dict(tol=case["tol"], max_iter=20000)
    if case.get("spheres"):
        ext = np.array([case["nx"], case["ny"], case["nz"]]) * _h(case)
        g.set_solid_spheres(rng.uniform(0.2, 0.8, size=(case["spheres"], 3)) * ext,
                            rng.uniform(0.05, 0.12, size=case["spheres"]))
    if s.kind == "learned":
        g.learned_set_weights(np.fromfile(os.path.join(PKG, "weights", "unet_precond.f32"), dtype="<f4"))
        s.solver.update(method=fia.FIA_SOLVER_FCG_LEARNED)
    if s.kind in ("projection", "learned"):
        s.solver = fia.solver_params(**s.solver)
    if s.kind == "step":
        s.step = fia.step_params(cfl=case["cfl"], frame=1, solver=s.solver)
        s.step.advect = s.params
    if s.kind == "train":
        g.learned_set_weights(np.fromfile(os.path.join(PKG, "weights", "unet_precond.f32"), dtype="<f4"))
        for _ in range(case["batch"]):
            g.learned_add_pair(*_smooth_pair(s.shapes["density"], rng))
        s.pairs = list(range(case["batch"]))
    g.synchronize()
    return s


def run(s):
    g = s.grid
    if s.kind == "density":
        s.put("density")
        g.move_substances_3D(s.dt, s.params)
        return s.view("density")
    if s.kind == "velocity":
        s.put("u", "v", "w")
        g.advect_velocity_xyz_flux_advection_3D(s.dt, s.params)
        return {k: s.view(k) for k in "uvw"}
    if s.kind == "host":
        # the density is advected in place, pass after pass, like the grid of the reference's loop
        fia._check(g.lib.fia_move_substances_3D_host(g.s, fia.FIA_HOST_F32, *s.ptrs, s.dt, ctypes.byref(s.params)),
                   "move_substances_3D_host")
        return s.host["density"]
    if s.kind in ("projection", "learned"):
        s.put("u", "v", "w")
        g.calc_pressure_gradient_term_3D(s.solver)
        return {k: s.view(k) for k in ("u", "v", "w", "pressure")}
    if s.kind == "step":
        s.put("density", "u", "v", "w")
        rep = g.step(s.step)
        return {"dt": rep.dt, **{k: s.view(k) for k in ("density", "u", "v", "w", "pressure")}}
    # the learning rate of the end of the cosine schedule: weights of a run's last steps
    losses = g.learned_train_step(s.pairs, 1e-5)
    return {"losses": losses, "weights": g.learned_get_weights()}


def work(case):
    """bytes: the fields in and out, once.  flops: the 1D WENO6 evaluations of about three pieces
    per face that no sharing between pieces removes, 93 operations each; the network's products;
    some 60 operations a cell for a direct Poisson solve."""
    cells = case["nx"] * case["ny"] * case["nz"]
    size = 4 if case["precision"] == "fp32c" else 8
    kind, k = case["kind"], case["k"]
    per_piece = (42 + 7 * 1.5 * k) if case["interp"] == "WENO6" else 12.0
    piece_work = per_piece * (93 if case["interp"] == "WENO6" else 8)
    advect = 9.0 * cells * piece_work * (2 if case["maccormack"] else 1)
    solve = 60.0 * cells
    net = 2 * 27.0 * cells / 8 * (16 + 256 + 768 + 256 + 16 + (512 + 1024 + 2560 + 1024) / 8 + 11520 / 64 + 7168 / 512)
    if kind in ("density", "host"):
        return {"bytes": 5 * size * cells, "flops": advect}
    if kind == "velocity":
        return {"bytes": 6 * size * cells, "flops": 3 * advect}
    if kind == "projection":
        return {"bytes": 7 * size * cells, "flops": solve}
    if kind == "learned":
        return {"bytes": 7 * size * cells, "flops": net}
    if kind == "step":
        return {"bytes": 9 * size * cells, "flops": 4 * advect + solve}
    return {"bytes": 2 * size * cells * case["batch"], "flops": 3 * net * case["batch"]}


# ------------------------------------------------------------------------------------
# the scheme in 64 bits, in units of the cell length, with plain torch
# ------------------------------------------------------------------------------------
def _snap(x):
    """values within 8 units in the last place of an integer are that integer"""
    r = torch.round(x)
    return torch.where((x - r).abs() <= 8 * 2.220446049250313e-16 * x.abs().clamp(min=1.0), r, x)


def _weno(f, s):
    """the 1D sixth-order WENO interpolant of six samples at s in [0, 1) past the third"""
    t = [s + (2 - i) for i in range(6)]
    d = [f[i + 1] - f[i] for i in range(5)]
    p = [f[i] + d[i] * t[i] + (d[i + 1] - d[i]) * (t[i] * t[i + 1] / 2)
         + (d[i + 2] - 2 * d[i + 1] + d[i]) * (t[i] * t[i + 1] * t[i + 2] / 6) for i in range(3)]
    b = [244 * d[0] ** 2 - 1171 * d[0] * d[1] + 683 * d[0] * d[2] + 1561 * d[1] ** 2 - 1951 * d[1] * d[2] + 814 * d[2] ** 2,
         244 * d[1] ** 2 - 781 * d[1] * d[2] + 293 * d[1] * d[3] + 961 * d[2] ** 2 - 781 * d[2] * d[3] + 244 * d[3] ** 2,
         814 * d[2] ** 2 - 1951 * d[2] * d[3] + 683 * d[2] * d[4] + 1561 * d[3] ** 2 - 1171 * d[3] * d[4] + 244 * d[4] ** 2]
    c = [t[4] * t[5] / 20, -t[5] * t[0] / 10, t[0] * t[1] / 20]
    a = [c[i] / (1e-6 + b[i] / 180) ** 2 for i in range(3)]
    return (a[0] * p[0] + a[1] * p[1] + a[2] * p[2]) / (a[0] + a[1] + a[2])


def _stencil(x, off, m, width):
    """fractional offset and clamped node indices of a stencil along one axis"""
    b = torch.floor(x - off)
    first = b.long() - (2 if width == 6 else 0)
    return x - off - b, [(first + i).clamp(0, m - 1) for i in range(width)]


def _interp(method, a, off, x, y, z):
    """the field a, its node 0 at `off` cells, at points given in cells"""
    mx, my, mz = a.shape
    flat = a.reshape(-1)
    if method == "1Dy-linear":
        ix = torch.floor(_snap(x - off[0] + 0.5)).long().clamp(0, mx - 1)
        iz = torch.floor(_snap(z - off[2] + 0.5)).long().clamp(0, mz - 1)
        s, j = _stencil(y, off[1], my, 2)
        return (1 - s) * flat[(ix * my + j[0]) * mz + iz] + s * flat[(ix * my + j[1]) * mz + iz]
    n = 6 if method == "WENO6" else 2
    one = _weno if n == 6 else (lambda f, s: (1 - s) * f[0] + s * f[1])
    out = []
    for c in range(0, x.numel(), 1 << 21):
        p = slice(c, c + (1 << 21))
        (sx, i), (sy, j), (sz, k) = (_stencil(q[p], off[d], a.shape[d], n) for d, q in enumerate((x, y, z)))
        out.append(one([one([one([flat[(ii * my + jj) * mz + kk] for kk in k], sz) for jj in j], sy) for ii in i], sx))
    return torch.cat(out) if out else x


def _gauss(k):
    x, w = np.polynomial.legendre.leggauss(k)
    return list(zip(x.tolist(), (w / 2).tolist()))


def _psi(a, off, method, k, h):
    """running y-integral of a, on the y-faces"""
    mx, my, mz = a.shape
    if method == "plain":
        inc = a * h
    else:
        i, j, q = (t.reshape(-1).double() for t in torch.meshgrid(*[torch.arange(m, device=a.device) for m in a.shape], indexing="ij"))
        x, z, lo = i + off[0], q + off[2], j + off[1] - 0.5
        inc = torch.zeros_like(x)
        if method == "WENO6":
            cols = a.movedim(1, 2).reshape(mx, mz, my)
            for half in (0.0, 0.5):
                for t, wt in _gauss(k):
                    s, jj = _stencil(lo + half + 0.25 * (1 + t), off[1], my, 6)
                    col = (i.long() * mz + q.long()) * my
                    inc += _weno([cols.reshape(-1)[col + c] for c in jj], s) * (0.5 * h * wt)
        else:
            for dy in (0.25, 0.75):
                inc += _interp("linear", a, off, x, lo + dy, z) * (0.5 * h)
        inc = inc.reshape(a.shape)
    return torch.cat([torch.zeros_like(inc[:, :1]), torch.cumsum(inc, 1)], 1)


def _clip(face, color):
    """Pieces of quads cut at the integer iso-lines of two colours (first all of the first colour,
    smallest first, then of the second).  face: (n, 4, 3) corners; color: their two offsets.
    Returns per piece its face, centroid (3) and the y component of its scaled normal, and per
    face whether a line crossed a polygon more than twice."""
    n, dev, V = face.shape[0], face.device, 16
    col = torch.stack([_snap(face[:, :, 0] - color[0]), _snap(face[:, :, 2] - color[1])], 2)
    quad = torch.tensor([[0, 0], [1, 0], [1, 1], [0, 1]], dtype=torch.float64, device=dev)
    poly = torch.zeros(n, V, 4, dtype=torch.float64, device=dev)
    poly[:, :4] = torch.cat([quad.expand(n, 4, 2), col], 2)
    num = torch.full((n,), 4, device=dev)
    owner, dim = torch.arange(n, device=dev), torch.zeros(n, dtype=torch.long, device=dev)
    multi = torch.zeros(n, dtype=torch.bool, device=dev)
    done = []
    while owner.numel():
        valid = torch.arange(V, device=dev) < num[:, None]
        c = torch.where(dim[:, None] == 0, poly[:, :, 2], poly[:, :, 3])
        mn = torch.where(valid, c, c[:, :1]).amin(1)
        mx = torch.where(valid, c, c[:, :1]).amax(1)
        start, end = torch.floor(mn) + 1, torch.ceil(mx) - 1
        cut = start <= end
        fin = ~cut & (dim == 1)
        done.append((owner[fin], poly[fin], num[fin]))
        keep = ~cut & (dim == 0)
        batch = [(poly[keep], num[keep], owner[keep], torch.ones_like(dim[keep]))]
        poly, num, owner, dim, c, iso = poly[cut], num[cut], owner[cut], dim[cut], c[cut], start[cut]
        r = torch.arange(owner.numel(), device=dev)
        head = torch.zeros(r.numel(), V + 2, 4, dtype=torch.float64, device=dev)
        part = torch.zeros(r.numel(), 4, V + 2, 4, dtype=torch.float64, device=dev)
        head[:, 0] = poly[:, 0]
        h0, far = torch.ones_like(owner), torch.zeros_like(owner, dtype=torch.bool)
        h1 = torch.zeros(r.numel(), 4, dtype=torch.long, device=dev)
        nch = torch.zeros_like(owner)

        def near(mask, v):
            q = r[mask]
            head[q, h0[q]] = v[q]
            h0[q] += 1

        def away(mask, v):
            q = r[mask]
            part[q, nch[q], h1[q, nch[q]]] = v[q]
            h1[q, nch[q]] += 1

        for e in range(int(num.max()) if num.numel() else 0):
            on = e < num
            m = torch.where(e + 1 == num, 0, e + 1).clamp(max=V - 1)
            a, b = poly[:, e], poly[r, m]
            v0, v1 = c[:, e] - iso, c[r, m] - iso
            x = on & ((v0 < 0) != (v1 < 0))
            t0 = torch.where(x, v1 / torch.where(x, v1 - v0, 1.0), 0.0)
            t1 = torch.where(x, -v0 / torch.where(x, v1 - v0, 1.0), 0.0)
            X = t0[:, None] * a + t1[:, None] * b
            X[:, 2] = torch.where(dim == 0, iso, _snap(X[:, 2]))
            X[:, 3] = torch.where(dim == 1, iso, _snap(X[:, 3]))
            leave, back = x & ~far, x & far
            near(leave, X)
            away(leave & (t1 < 1), X)
            away(back, X)
            nch = nch + back.long()
            near(back & (t1 < 1), X)
            far = far ^ x
            near(on & (e + 1 < num) & ~far, b)
            away(on & (e + 1 < num) & far, b)
        multi[owner[nch > 1]] = True
        batch.append((head[:, :V], h0, owner, dim))
        for q in range(4):
            has = nch > q
            batch.append((part[has, q, :V], h1[has, q], owner[has], dim[has]))
        poly, num, owner, dim = (torch.cat(t) for t in zip(*batch))
    owner, poly, num = (torch.cat(t) for t in zip(*done))
    ok = num >= 3
    owner, xi, num = owner[ok], poly[ok][:, :, :2], num[ok]
    valid = torch.arange(V, device=dev) < num[:, None]
    xi = torch.where(valid[:, :, None], xi, xi[:, :1])      # repeated first vertex: adds no area
    q = xi - xi[:, :1]
    nx = torch.roll(q, -1, 1)
    cr = q[:, :, 0] * nx[:, :, 1] - nx[:, :, 0] * q[:, :, 1]
    area2 = cr.sum(1)
    ok = area2 != 0
    ctr = xi[:, 0] + (cr[:, :, None] * (q + nx)).sum(1) / (3 * torch.where(ok, area2, 1.0))[:, None]

    def bilinear(f, p):
        v = [f[:, i].reshape(f.shape[0], *([1] * (p.dim() - 2)), 3) for i in range(4)]
        a, b = p[..., :1], p[..., 1:]
        return v[0] + a * (v[1] - v[0]) + b * (v[3] - v[0]) + a * b * (v[0] - v[1] + v[2] - v[3])

    f = face[owner]
    cp = bilinear(f, ctr)
    p3 = bilinear(f, xi) - cp[:, None]
    n3 = torch.roll(p3, -1, 1)
    ny = 0.5 * (p3[:, :, 2] * n3[:, :, 0] - p3[:, :, 0] * n3[:, :, 2]).sum(1)
    ok = ok & (ny != 0)
    return owner[ok], cp[ok], ny[ok], multi


def _faces_flux(face, color, a, off, psi, poff, oy, method, integral, k, h):
    """flux through each quad seen from its lower and from its upper cell, per cell volume"""

    def flux(quads):
        own, c, ny, multi = _clip(quads, color)
        x, y, z = c.unbind(1)
        F = torch.zeros_like(ny)
        if integral:
            r = _snap(y - oy)
            fl = torch.floor(r)
            f, y0 = r - fl, fl + oy
            two = f >= 0.5
            for t, wt in _gauss(k):
                L = torch.where(two, 0.5, y - y0)
                F += _interp(method, a, off, x, L / 2 * t + L / 2 + y0, z) * (ny * torch.where(two, 0.5, f) * wt)
                L = f[two] - 0.5
                F[two] += _interp(method, a, off, x[two], L / 2 * t + L / 2 + y0[two] + 0.5, z[two]) * (ny[two] * L * wt)
            y = y0
        F += _interp(method, psi, poff, x, y, z) * (ny / h)
        return torch.zeros(quads.shape[0], dtype=F.dtype, device=F.device).index_add_(0, own, F), multi

    low, high = [], []
    for part in face.split(1 << 20):
        lo, multi = flux(part)
        up = -lo
        if multi.any():
            up[multi] = flux(part[multi][:, [0, 3, 2, 1]])[0]
        low.append(lo)
        high.append(up)
    return torch.cat(low), torch.cat(high)


def _pass(a, comp, vel, dt, h, n, method, integral, psi_mode, moving, color, k, maccormack):
    """one flux pass: the advected cell averages of a"""
    off = [0.0 if d == comp else 0.5 for d in range(3)]
    poff = [off[0], off[1] - 0.5, off[2]]
    psi = _psi(a, off, psi_mode, k, h)
    dev = a.device
    ext = [0.5 if d == comp else 0.0 for d in range(3)]
    grids = torch.meshgrid(*[torch.arange(m + 1, device=dev) for m in a.shape], indexing="ij")
    rest = torch.stack([g.double() - e for g, e in zip(grids, ext)], -1)
    lo = torch.tensor([-e for e in ext], dtype=torch.float64, device=dev)
    hi = torch.tensor([m + e for m, e in zip(n, ext)], dtype=torch.float64, device=dev)
    pinned = torch.zeros(rest.shape[:3], dtype=torch.bool, device=dev)
    if comp >= 0:
        pinned = (grids[comp] <= 1) | (grids[comp] >= n[comp])

    def trace(p, sign):
        x, y, z = p.reshape(-1, 3).unbind(1)
        step = [_interp(method, f, [0.0 if d == c else 0.5 for d in range(3)], x, y, z) for c, f in enumerate(vel)]
        step = torch.stack(step, 1).reshape(p.shape) * (sign * dt / h)
        p = p + torch.where(pinned[..., None], 0.0, step)
        return torch.minimum(torch.maximum(p, lo), hi)

    sets = [(rest, 1.0)]
    if moving:
        back = trace(rest, -1.0)
        sets = [(rest, 0.5), (back, 1.0), (trace(back, 1.0), -0.5)] if maccormack else [(back, 1.0)]
    out = torch.zeros_like(a)
    order = {0: [(0, 0, 0), (0, 1, 0), (0, 1, 1), (0, 0, 1)], 1: [(0, 0, 0), (0, 0, 1), (1, 0, 1), (1, 0, 0)],
             2: [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0)]}
    for fam in range(3):
        m = [a.shape[d] + (d == fam) for d in range(3)]
        for pts, weight in sets:
            if not moving and fam != 1:
                continue            # faces at rest along x and z have no y-normal
            quad = torch.stack([pts[o[0]:o[0] + m[0], o[1]:o[1] + m[1], o[2]:o[2] + m[2]] for o in order[fam]], 3)
            low, up = _faces_flux(quad.reshape(-1, 4, 3), color, a, off, psi, poff, 0.0 - ext[1], method, integral, k, h)
            low, up = low.reshape(m), up.reshape(m)
            out += weight * (low.narrow(fam, 1, a.shape[fam]) + up.narrow(fam, 0, a.shape[fam]))
    return out


_SPLIT = {"xz-CellFaceAligned": (0.5, 0.5), "xz-AxisAligned": (0.0, 0.0),
          "x-CellFaceAligned_z-AxisAligned": (0.5, 0.0), "x-AxisAligned_z-CellFaceAligned": (0.0, 0.5)}


def _advect(case, a, comp, vel, dt):
    h, n = _h(case), (case["nx"], case["ny"], case["nz"])
    main = _SPLIT[case["split"]] if comp < 0 else (0.0 if comp == 0 else 0.5, 0.0 if comp == 2 else 0.5)
    err = (0.0, 0.0) if comp < 0 or comp == 1 else (0.5 - main[0], 0.5 - main[1])
    k, mc, method = case["k"], case["maccormack"], case["interp"]
    out = _pass(a, comp, vel, dt, h, n, method, True, method, True, main, k, mc)
    if case["zero_velocity_passes"]:
        left = a - _pass(a, comp, vel, dt, h, n, method, False, "plain", False, main, k, False)
        out += _pass(left, comp, vel, dt, h, n, "1Dy-linear", False, "plain", True, err, k, mc)
    return out


def _project(u, v, w, h):
    """the projection by cosine transforms: the zero-flux Poisson problem of the divergence with
    the last cell held at zero (its own equation is dropped, so the right-hand side is made to
    sum to zero there)"""
    r = -h * (torch.diff(u, dim=0) + torch.diff(v, dim=1) + torch.diff(w, dim=2))
    r.view(-1)[-1] -= r.sum()
    eig, mats = [], []
    for m in r.shape:
        q = torch.arange(m, dtype=torch.float64, device=r.device)
        c = torch.cos(math.pi * q[:, None] * (q + 0.5) / m) * math.sqrt(2.0 / m)
        c[0] /= math.sqrt(2.0)
        mats.append(c)
        eig.append(2 - 2 * torch.cos(math.pi * q / m))
    p = r
    for d in range(3):
        p = torch.movedim(torch.tensordot(mats[d], p, dims=([1], [d])), 0, d)
    lam = eig[0][:, None, None] + eig[1][None, :, None] + eig[2]
    lam[0, 0, 0] = 1.0
    p = p / lam
    p[0, 0, 0] = 0.0
    for d in range(3):
        p = torch.movedim(torch.tensordot(mats[d].T, p, dims=([1], [d])), 0, d)
    p = p - p.reshape(-1)[-1]
    out = []
    for d, f in enumerate((u, v, w)):
        f = f.clone()
        f.narrow(d, 1, f.shape[d] - 2).sub_(torch.diff(p, dim=d) / h)
        out.append(f)
    return out + [p]


def exact(case, seed):
    """None: the whole step (a chain of the calls that have values here); the training step (a
    BF16 network); the learned solve, whose flexible iteration ends somewhere below its
    tolerance, and solids, which the transforms cannot take; and grids of which the advection
    takes longer than some 20 seconds."""
    kind = case["kind"]
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind in ("density", "host", "velocity"):
        cost = cells * (3 if kind == "velocity" else 1) * (3 if case["maccormack"] else 1) * (case["k"] + 1)
        if cost > 6e7:
            return None
        rho, u, v, w, dt = _inputs(case, seed)
        vel = (u, v, w)
        if kind == "velocity":
            return {k: _advect(case, f, c, vel, dt) for c, (k, f) in enumerate(zip("uvw", vel))}
        return _advect(case, rho, -1, vel, dt)
    if kind == "projection" and not case["spheres"]:
        _, u, v, w, _ = _inputs(case, seed)
        return dict(zip(("u", "v", "w", "pressure"), _project(u, v, w, _h(case))))
    return None
