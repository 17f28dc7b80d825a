"""Work that users of this package have it do, as cases that can be timed and checked.

A case is one way of calling the solver at one size (``path``):

* ``resident``: a program that keeps its state in HBM and advances it by a number of steps per call
  (DeviceSolver.solve_steps), the state read where it lies (DeviceSolver.strip_view). Every call
  goes on from where the last one ended. An FP64 state comes back as its nine double planes. An
  FP32-mixed state comes back as its nine hi planes, which are the state rounded to float32.
* ``host``: the drop-in call on host arrays: upload, solve to t_end, download.
* ``noalloc``: the allocation-free solve on a caller's own device tensors.
* ``batch``: uneven independent solves admitted together, advanced, downloaded and removed, as the
  serving loop does it; the results are kept in float32, the accuracy of the FP32-mixed form.

``exact`` computes the same in float64 with plain torch.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from mhd_gpu_solver_b200 import _capi
from mhd_gpu_solver_b200.batch import BatchSolver, fixed_params

LIMITERS = {"minmod": _capi.MINMOD, "mc": _capi.MC, "vanleer": _capi.VANLEER}
BCS = {"periodic": _capi.BC_PERIODIC, "outflow": _capi.BC_OUTFLOW}
NOALLOC_CELLS = 233016  # the allocation-free solve's limit


def _case(path, nx, ny, steps, *, name=None, precision="fp64", limiter="vanleer", bc_x="periodic",
          bc_y="periodic", init="fourier", nonideal=False, mask=False, solves=0):
    c = {"path": path, "nx": nx, "ny": ny, "steps": steps, "precision": precision,
         "limiter": limiter, "bc_x": bc_x, "bc_y": bc_y, "init": init, "nonideal": nonideal,
         "mask": mask, "solves": solves}
    return c if name is None else {"name": name, **c}


def listed():
    both_out = {"bc_x": "outflow", "bc_y": "outflow"}
    masked = {"nonideal": True, "mask": True, "bc_x": "outflow"}
    return [
        # the plain method at its reference size: four quadrants, outflow, minmod, 200 steps
        _case("resident", 128, 128, 200, name="fp64_128_quadrants", limiter="minmod",
              init="quadrants", **both_out),
        # a short wide channel with resistivity, Hall and ambipolar terms
        _case("resident", 700, 180, 50, name="fp64_700x180_nonideal", limiter="mc", nonideal=True,
              bc_y="outflow"),
        # the smooth periodic field at the two sizes it is quoted on, in both precision forms
        _case("resident", 1024, 1024, 20, name="fp64_1024"),
        _case("resident", 4096, 4096, 8, name="fp64_4096"),
        _case("resident", 1024, 1024, 40, name="mixed_1024", precision="fp32"),
        _case("resident", 4096, 4096, 16, name="mixed_4096", precision="fp32"),
        # reflective walls with non-ideal terms, in both precision forms
        _case("resident", 2048, 2048, 12, name="fp64_2048_masked", **masked),
        _case("resident", 2048, 2048, 24, name="mixed_2048_masked", precision="fp32", **masked),
        # a small ragged grid, as single requests are
        _case("resident", 301, 173, 100, name="mixed_301x173", precision="fp32", limiter="mc",
              init="quadrants", **both_out),
        # the reference's own way in: host arrays, a solve to a time, host arrays
        _case("host", 512, 512, 100, name="host_fp64_512", limiter="mc"),
        # a caller that owns the device memory
        _case("noalloc", 321, 257, 50, name="noalloc_fp64_321x257", limiter="minmod"),
        # independent solves of uneven sizes, sides log-uniform in [64, 1024]
        _case("batch", 1024, 1024, 60, name="batch_16_uneven", precision="fp32", solves=16),
    ]


def draw(rng):
    path = rng.choices(("resident", "host", "noalloc", "batch"), (12, 2, 3, 3))[0]

    def log_uniform(a, b):
        return int(math.exp(rng.uniform(math.log(a), math.log(b + 1))))

    nx, ny = log_uniform(48, 4096), log_uniform(48, 4096)
    if path == "host":
        nx, ny = log_uniform(48, 1024), log_uniform(48, 1024)
    elif path == "noalloc":
        nx = log_uniform(32, 480)
        ny = min(log_uniform(32, 480), NOALLOC_CELLS // nx)
    elif path == "batch":
        nx = ny = 1024
    solves = rng.randint(4, 16) if path == "batch" else 0
    cells = solves * 120_000 if path == "batch" else nx * ny
    steps = max(4, min(200, int(rng.uniform(0.5, 1.0) * 3e7 / cells)))
    alone = path == "resident"
    return _case(path, nx, ny, steps,
                 precision=rng.choice(("fp64", "fp32")) if alone else
                 "fp32" if path == "batch" else "fp64",
                 limiter=rng.choice(("minmod", "mc", "vanleer", "vanleer")),
                 bc_x=rng.choice(("periodic", "outflow")), bc_y=rng.choice(("periodic", "outflow")),
                 init=rng.choice(("fourier", "fourier", "quadrants")),
                 nonideal=rng.random() < 0.3, mask=alone and rng.random() < 0.25, solves=solves)


# ------------------------------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _centers(nx, ny):
    x = (torch.arange(nx, dtype=torch.float64, device=_device()) + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64, device=_device()) + 0.5) / ny
    return x, y


def _fourier(nx, ny, seed, kmax=8):
    """Smooth periodic primitives: modes 1 <= |k| <= 8, amplitude |k|^-2, seeded phases; v and
    B = curl A_z of rms 1, rho = 1 + clip(0.2 f1, 0.2), p = 1 + clip(0.1 f2, 0.2)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    modes = [(kx, ky) for kx in range(kmax + 1) for ky in range(-kmax, kmax + 1)
             if not (kx == 0 and ky <= 0) and 1.0 <= math.hypot(kx, ky) <= kmax]
    x, y = _centers(nx, ny)
    kxs = torch.arange(kmax + 1, device=x.device, dtype=torch.float64)
    kys = torch.arange(-kmax, kmax + 1, device=x.device, dtype=torch.float64)
    two_pi = 2.0 * math.pi
    ex = torch.exp(1j * two_pi * kxs[:, None] * x[None, :])
    ey = torch.exp(1j * two_pi * kys[:, None] * y[None, :])

    def coefficients():
        phases = rng.uniform(0.0, two_pi, size=len(modes))
        c = np.zeros((2 * kmax + 1, kmax + 1), dtype=np.complex128)
        for (kx, ky), ph in zip(modes, phases):
            c[ky + kmax, kx] = math.hypot(kx, ky) ** -2.0 * np.exp(1j * ph)
        return torch.from_numpy(c).to(x.device)

    def synth(c):
        return (ey.T @ (c @ ex)).real

    def rms_one(a, b):
        s = 1.0 / torch.sqrt((a * a + (0 if b is None else b * b)).mean())
        return a * s, None if b is None else b * s

    cvx, cvy, caz, cf1, cf2 = (coefficients() for _ in range(5))
    vx, vy = rms_one(synth(cvx), synth(cvy))
    bx, by = rms_one(synth(caz * (1j * two_pi * kys[:, None])),
                     -synth(caz * (1j * two_pi * kxs[None, :])))
    f1, f2 = rms_one(synth(cf1), None)[0], rms_one(synth(cf2), None)[0]
    zero = torch.zeros_like(vx)
    return torch.stack([1.0 + (0.2 * f1).clamp(-0.2, 0.2), vx, vy, zero,
                        1.0 + (0.1 * f2).clamp(-0.2, 0.2), bx, by, zero, zero])


def _quadrant_values(seed):
    """rho, p ~ U[0.1, 2], vx, vy, By ~ U[-1, 1] of the four quadrants."""
    rng = np.random.Generator(np.random.PCG64(seed))
    return np.array([[rng.uniform(0.1, 2.0), rng.uniform(0.1, 2.0), rng.uniform(-1.0, 1.0),
                      rng.uniform(-1.0, 1.0), rng.uniform(-1.0, 1.0)] for _ in range(4)])


def _quadrants(nx, ny, seed):
    x, y = _centers(nx, ny)
    which = (x[None, :] >= 0.5).long() + 2 * (y[:, None] >= 0.5).long()
    v = torch.from_numpy(_quadrant_values(seed)).to(x.device)[which]
    zero = torch.zeros_like(v[..., 0])
    return torch.stack([v[..., 0], v[..., 2], v[..., 3], zero, v[..., 1],
                        torch.full_like(zero, 0.75), v[..., 4], zero, zero])


def _initial(init, nx, ny, seed, gamma):
    """Conserved interior state (9, ny, nx)."""
    w = (_fourier if init == "fourier" else _quadrants)(nx, ny, seed)
    u = w.clone()
    u[1:4] = w[0] * w[1:4]
    u[4] = (w[4] / (gamma - 1.0) + 0.5 * w[0] * (w[1:4] ** 2).sum(0) + 0.5 * (w[5:8] ** 2).sum(0))
    return u


def _mask(nx, ny, seed):
    """Twelve solid circles and six solid rectangles at seeded places; 1 = fluid."""
    rng = np.random.Generator(np.random.PCG64(seed + 1_000_003))
    xs, ys = (np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny
    mask = np.ones((ny, nx), dtype=np.uint8)
    for _ in range(12):
        cx, cy, r = rng.uniform(0, 1), rng.uniform(0, 1), rng.uniform(0.02, 0.08)
        mask[(xs[None, :] - cx) ** 2 + (ys[:, None] - cy) ** 2 <= r * r] = 0
    for _ in range(6):
        x0, y0 = rng.uniform(0, 1), rng.uniform(0, 1)
        w, h = rng.uniform(0.02, 0.15), rng.uniform(0.02, 0.15)
        mask[((ys >= y0) & (ys <= y0 + h))[:, None] & ((xs >= x0) & (xs <= x0 + w))[None, :]] = 0
    return mask


def _ghosts(u, bc_x, bc_y, ng=2):
    """The state with its ghost cells: periodic wrap or the nearest interior cell."""
    def index(n, bc):
        i = torch.arange(-ng, n + ng, device=u.device)
        return i % n if bc == "periodic" else i.clamp(0, n - 1)
    return u[:, index(u.shape[1], bc_y)][:, :, index(u.shape[2], bc_x)]


def _physics(case):
    d = {"limiter": LIMITERS[case["limiter"]], "gamma": 5.0 / 3.0}
    if case["nonideal"]:
        d |= {"ohmic": True, "hall": True, "ambipolar": True, "eta_ohm": 1e-3, "eta_hall": 1e-2,
              "eta_ambipolar": 1e-3}
    return d


def _solves(case, seed):
    """The batch's solves: sides log-uniform in [64, nx] x [64, ny], a seed and a gamma each."""
    rng = np.random.Generator(np.random.PCG64(4242))  # sizes and order belong to the case
    out = []
    for i in range(case["solves"]):
        nx = int(64.0 * (case["nx"] / 64.0) ** rng.uniform())
        ny = int(64.0 * (case["ny"] / 64.0) ** rng.uniform())
        out.append((nx, ny, 1000 * seed + i, float(rng.uniform(1.4, 5.0 / 3.0))))
    return out


def _t_end(case):
    """A time that takes about `steps` steps of a state with signal speeds around 4."""
    h = 1.0 / max(case["nx"], case["ny"])
    dt = 0.4 / (4.0 * case["nx"] + 4.0 * case["ny"])
    return case["steps"] * (min(dt, 0.4 * h * h / 0.04) if case["nonideal"] else dt)


# ------------------------------------------------------------------------------- prepare, run


class _Planes:
    """Device memory of a solver as an array other libraries can alias; whoever holds the alias
    holds the solver too."""

    def __init__(self, owner, address, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (address, False), "shape": shape,
                                         "strides": strides, "typestr": typestr, "version": 3}


def _state_tensor(dev):
    v = dev.strip_view()
    e = v.elem_bytes
    planes = _Planes(dev, v.state, (9, dev.ny, dev.nx), (v.plane * e, v.pitch * e, e),
                     "<f8" if e == 8 else "<f4")
    # torch keeps `planes` as long as the tensor lives
    return torch.as_tensor(planes, device="cuda")


def prepare(case, seed):
    nx, ny, path = case["nx"], case["ny"], case["path"]
    bc = (BCS[case["bc_x"]], BCS[case["bc_y"]])
    s = {"case": case, "path": path, "bc": bc, "steps": case["steps"]}
    if path == "batch":
        init = {"fourier": _capi.InitSpec.fourier, "quadrants": _capi.InitSpec.quadrants}
        s["batch"] = BatchSolver(_capi.FP32)
        s["requests"] = []
        s["out"] = []
        for w, h, one, gamma in _solves(case, seed):
            p = fixed_params(case["steps"], **(_physics(case) | {"gamma": gamma}))
            s["requests"].append((w, h, init[case["init"]](one), p))
            s["out"].append(torch.empty((9, h + 4, w + 4), dtype=torch.float32))
        most = max(t.numel() for t in s["out"])
        s["landing"] = torch.empty(most, dtype=torch.float64, pin_memory=True)
        return s
    u = _initial(case["init"], nx, ny, seed, 5.0 / 3.0)
    if path == "noalloc":
        s["grid"] = _capi.Grid(nx, ny, 2, 0.0, 1.0, 0.0, 1.0)
        s["params"] = _capi.make_params(**_physics(case))
        s["u_in"], s["u_out"] = u.contiguous(), torch.empty_like(u)
        return s
    s["dev"] = _capi.DeviceSolver(
        nx, ny, precision=_capi.FP64 if case["precision"] == "fp64" else _capi.FP32)
    s["dev"].configure(*bc, _mask(nx, ny, seed) if case["mask"] else None)
    host = _ghosts(u, case["bc_x"], case["bc_y"]).cpu().numpy()
    if path == "host":
        s["params"] = _capi.make_params(t_end=_t_end(case), **_physics(case))
        s["in"], s["out"] = host, np.empty_like(host)
    else:
        s["params"] = _capi.make_params(**_physics(case))
        s["dev"].upload(host)
    return s


def run(s):
    if s["path"] == "resident":
        r = s["dev"].solve_steps(s["params"], s["steps"])
        return {"state": _state_tensor(s["dev"]), "t": r.t, "steps": r.steps, "c_h": r.c_h}
    if s["path"] == "host":
        dev = s["dev"]
        dev.upload(s["in"])
        r = dev.solve(s["params"])
        return {"state": dev.download(s["out"]), "t": r.t, "steps": r.steps, "c_h": r.c_h}
    if s["path"] == "noalloc":
        r = _capi.Result()
        _capi.raise_for(_capi.lib.mhdb_solve_steps_noalloc_f64(
            ctypes.byref(s["grid"]), *s["bc"], ctypes.byref(s["params"]), s["steps"],
            ctypes.c_void_p(s["u_in"].data_ptr()), ctypes.c_void_p(s["u_out"].data_ptr()),
            ctypes.byref(r), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), None)
        return {"state": s["u_out"], "t": r.t, "steps": r.steps, "c_h": r.c_h}
    b = s["batch"]
    ids = [b.add_generated(w, h, init, p, s["bc"], fixed_steps=True)
           for w, h, init, p in s["requests"]]
    b.step(s["steps"])
    steps = []
    for sid, out in zip(ids, s["out"]):
        steps.append(b.status(sid)[0].steps)
        landing = s["landing"][:out.numel()].view(out.shape)
        b.download(sid, landing.numpy())
        out.copy_(landing)
        b.remove(sid)
    return {"state": s["out"], "steps": steps}


def work(case):
    """Bytes: the state read and written once per step where it is larger than the L2 cache, else
    once per pass. Flops of a step of a cell: two stages of two slopes, two HLL faces, the
    primitives, the divergence and the update."""
    if case["path"] == "batch":
        cells = sum(nx * ny for nx, ny, _, _ in _solves(case, 0))
    else:
        cells = case["nx"] * case["ny"]
    passes = case["steps"] if cells * 72 > 126e6 else 1
    per_cell = 2.0 * (2 * 45 + 2 * 230 + 25 + 45 + (120 if case["nonideal"] else 0)) + 45
    return {"bytes": 144.0 * cells * passes, "flops": per_cell * cells * case["steps"]}


# -------------------------------------------------------------------------------------- exact


def _limit(kind, a, b):
    same = a * b > 0
    if kind == "vanleer":
        return torch.where(same, 2.0 * a * b / torch.where(same, a + b, 1.0), 0.0)
    small = torch.where(a.abs() < b.abs(), a, b)
    if kind == "mc":
        m = 0.5 * (a + b)
        small = torch.where(m.abs() < 2.0 * small.abs(), m, 2.0 * small)
    return torch.where(same, small, 0.0)


def _primitives(u, gamma):
    w = u.clone()
    w[1:4] = u[1:4] / u[0]
    w[4] = (gamma - 1.0) * (u[4] - 0.5 * (u[1:4] ** 2).sum(0) / u[0] - 0.5 * (u[5:8] ** 2).sum(0))
    return w


def _fast(w, bn, gamma):
    cs2, va2, vn2 = gamma * w[4] / w[0], (w[5:8] ** 2).sum(0) / w[0], w[bn] ** 2 / w[0]
    t = cs2 + va2
    return (0.5 * (t + (t * t - 4.0 * cs2 * vn2).clamp_min(0).sqrt())).clamp_min(0).sqrt()


def _flux(w, n, gamma, c_h):
    """Conserved values and flux along axis n (0: x, 1: y) of primitives w."""
    rho, p, psi = w[0], w[4], w[8]
    v, b = w[1:4], w[5:8]
    b2, vb = (b * b).sum(0), (v * b).sum(0)
    e = p / (gamma - 1.0) + 0.5 * rho * (v * v).sum(0) + 0.5 * b2
    u = torch.cat([rho[None], rho * v, e[None], b, psi[None]])
    ps = p + 0.5 * b2
    f = torch.empty_like(u)
    f[0] = rho * v[n]
    f[1:4] = rho * v[n] * v - b[n] * b
    f[1 + n] += ps
    f[4] = (e + ps) * v[n] - b[n] * vb + psi * b[n]
    f[5:8] = v[n] * b - v * b[n]
    f[5 + n] = psi
    f[8] = c_h * c_h * b[n]
    return u, f


def _rhs(ug, case, gamma, c_h, dx, dy):
    """-dF/dx - dG/dy and the psi damping of a state with two ghost layers."""
    ny, nx = ug.shape[1] - 4, ug.shape[2] - 4
    w = _primitives(ug, gamma)
    if case["nonideal"]:
        b = w[5:8]
        ddx = (b[:, 1:-1, 2:] - b[:, 1:-1, :-2]) / (2.0 * dx)
        ddy = (b[:, 2:, 1:-1] - b[:, :-2, 1:-1]) / (2.0 * dy)
        j = torch.stack([ddy[2], -ddx[2], ddx[1] - ddy[0]])
    total = None
    for n, (size, other, h) in enumerate(((nx, ny, dx), (ny, nx, dy))):
        dim = 2 - n
        c = w.narrow(3 - dim, 2, other)  # the rows (or columns) that own faces
        d = c.narrow(dim, 1, size + 3) - c.narrow(dim, 0, size + 3)
        s = 0.5 * _limit(case["limiter"], d.narrow(dim, 0, size + 2), d.narrow(dim, 1, size + 2))
        wl, wr = c.narrow(dim, 1, size + 1), c.narrow(dim, 2, size + 1)
        left, right = wl + s.narrow(dim, 0, size + 1), wr - s.narrow(dim, 1, size + 1)
        ok = (left[0] > 0) & (left[4] > 0) & (right[0] > 0) & (right[4] > 0)
        left, right = torch.where(ok, left, wl), torch.where(ok, right, wr)
        cl, cr = _fast(left, 5 + n, gamma), _fast(right, 5 + n, gamma)
        sl = torch.minimum(left[1 + n] - cl, right[1 + n] - cr).clamp_max(-c_h)
        sr = torch.maximum(left[1 + n] + cl, right[1 + n] + cr).clamp_min(c_h)
        (ul, fl), (ur, fr) = _flux(left, n, gamma, c_h), _flux(right, n, gamma, c_h)
        f = (sr * fl - sl * fr + sl * sr * (ur - ul)) / (sr - sl)
        if case["nonideal"]:
            jc = j.narrow(3 - dim, 1, other)
            jf = 0.5 * (jc.narrow(dim, 0, size + 1) + jc.narrow(dim, 1, size + 1))
            bf = 0.5 * (wl[5:8] + wr[5:8])
            b2 = (bf * bf).sum(0)
            big = b2 >= 1e-14
            x1 = torch.linalg.cross(jf, bf, dim=0)
            x2 = torch.linalg.cross(x1, bf, dim=0)
            b2 = torch.where(big, b2, 1.0)
            e = 1e-3 * jf + torch.where(big, 1e-2 * x1 / b2.sqrt() + 1e-3 * x2 / b2, 0.0)
            if n == 0:
                f[6] -= e[2]
                f[7] += e[1]
                f[4] += bf[1] * e[2] - bf[2] * e[1]
            else:
                f[5] += e[2]
                f[7] -= e[0]
                f[4] += bf[2] * e[0] - bf[0] * e[2]
        term = -(f.narrow(dim, 1, size) - f.narrow(dim, 0, size)) / h
        total = term if total is None else total + term
    total[8] -= c_h * 0.1 / min(dx, dy) * w[8, 2:-2, 2:-2]
    return total


def _fill(u, mask, gamma):
    """Solid cells of u as the mirror of their first fluid neighbour (+x, -x, +y, -y)."""
    out, left = u.clone(), ~mask
    ny, nx = mask.shape
    for di, dj in ((1, 0), (-1, 0), (0, 1), (0, -1)):
        i = torch.arange(nx, device=u.device) + di
        j = torch.arange(ny, device=u.device) + dj
        inside = ((j >= 0) & (j < ny))[:, None] & ((i >= 0) & (i < nx))[None, :]
        i, j = i.clamp(0, nx - 1), j.clamp(0, ny - 1)
        use = left & inside & mask[j][:, i]
        w = _primitives(u[:, j][:, :, i], gamma)
        w[1 if di else 2] *= -1.0
        w[0], w[4] = w[0].clamp_min(1e-12), w[4].clamp_min(1e-12)
        v = w.clone()
        v[1:4] = w[0] * w[1:4]
        v[4] = w[4] / (gamma - 1.0) + 0.5 * w[0] * (w[1:4] ** 2).sum(0) + 0.5 * (w[5:8] ** 2).sum(0)
        out = torch.where(use, v, out)
        left = left & ~use
    rest = torch.zeros(9, dtype=u.dtype, device=u.device)
    rest[0], rest[4] = 1.0, 1.0 / (gamma - 1.0)
    return torch.where(left, rest[:, None, None], out)


def _advance(u, case, gamma, steps, t_end, mask):
    """`steps` steps, or as many as reach t_end; returns the state, t, steps and the last c_h."""
    ny, nx = u.shape[1:]
    dx, dy = 1.0 / nx, 1.0 / ny
    t, done, c_h = 0.0, 0, 0.0

    def filled(v):
        return v if mask is None else _fill(v, mask, gamma)

    def slope(v, c):
        g = _ghosts(v, case["bc_x"], case["bc_y"])  # ghosts hold the values before the fill
        f = filled(v)
        g[:, 2:-2, 2:-2] = f
        r = _rhs(g, case, gamma, c, dx, dy)
        return f, r if mask is None else torch.where(mask, r, 0.0)

    while done < steps if t_end is None else t < t_end:
        w = _primitives(u, gamma)
        speed = torch.maximum(w[1].abs() + _fast(w, 5, gamma), w[2].abs() + _fast(w, 6, gamma))
        c_h = float((speed if mask is None else speed[mask]).max())
        dt = 0.4 / (c_h / dx + c_h / dy)
        if case["nonideal"]:
            dt = min(dt, 0.4 * min(dx, dy) ** 2 / (4.0 * 1e-2))
        if t_end is not None:
            dt = min(dt, t_end - t)
        f, r = slope(u, c_h)
        first = f if mask is None else torch.where(mask, u, f)
        star = first + dt * r
        f, r = slope(star, c_h)
        base = u if mask is None else torch.where(mask, u, star)
        u = 0.5 * (base + f) + 0.5 * dt * r
        t, done = t + dt, done + 1
    return u, t, done, c_h


def exact(case, seed):
    if case["path"] == "batch":
        one = [(gamma, _initial(case["init"], nx, ny, s, gamma))
               for nx, ny, s, gamma in _solves(case, seed)]
        out = [_advance(u, case, gamma, case["steps"], None, None)[0] for gamma, u in one]
        return {"state": [_ghosts(u, case["bc_x"], case["bc_y"]) for u in out],
                "steps": [case["steps"]] * len(out)}
    u = _initial(case["init"], case["nx"], case["ny"], seed, 5.0 / 3.0)
    mask = None
    if case["mask"]:
        mask = torch.from_numpy(_mask(case["nx"], case["ny"], seed)).to(u.device) != 0
    t_end = _t_end(case) if case["path"] == "host" else None
    u, t, steps, c_h = _advance(u, case, 5.0 / 3.0, case["steps"], t_end, mask)
    if case["path"] == "host":
        u = _ghosts(u, case["bc_x"], case["bc_y"])
    return {"state": u, "t": t, "steps": steps, "c_h": c_h}
