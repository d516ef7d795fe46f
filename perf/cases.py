"""The work that users have this framework do, as cases that can be timed and checked.

A case is a dict of plain values: what is run (`kind`), on which workload, at which size and
with which options.  `prepare` makes what a program holds before the call (the solver context
with its RK table, planes and masks, the state in device memory), `run` makes one pass through
the public entry points (`Solver`, `Net`, the C-ABI), `exact` states the same result in 64 bits
with plain torch where that is practical, and `work` counts the bytes and operations a pass
cannot do without.

Kinds:
  step        one time step from a state in device memory, as a restarted run makes it: the
              state's five arrays copied in, contorno(1), step(), the five arrays copied out
  level_set   transport, reinitialisation, normals, curvature, Heaviside of the level set
  momentum    Smagorinsky viscosity and the momentum right-hand side (visco, convdiff)
  projection  one pressure solve from zero pressure and the projection (graddin, posdin)
  train       loss and parameter gradient of the pressure-guess network (Net.loss_grad)

The Poisson solves stop where the benchmark's and the tests' cases stop them: at a relative FP64
residual of 1e-8 to 1e-10 (`tol`), the sloshing tank also at max |div u| <= 1e-8.
"""
import ctypes
import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parent.parent
DEV = "cuda:0"
F64 = torch.float64


def _package():
    if "suli_b200" not in sys.modules:
        d = ROOT / "suli-openmp_b200"
        spec = importlib.util.spec_from_file_location("suli_b200", d / "__init__.py",
                                                      submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["suli_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["suli_b200"]


pkg = _package()


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the reference's compiled default case (25 x 50 x 45 cells, x periodic, RK2): the smallest
        # real run, where every launch and every CG iteration's latency counts; odd sizes
        {"name": "step_default_fp64", "kind": "step", "preset": "default", "nx": 25, "ny": 50, "nz": 45,
         "precision": 0, "net": 0, "tol": 1e-10},
        # the dam break the tests run, plain FP64 path, RK3, no-slip walls
        {"name": "step_dam_fp64", "kind": "step", "preset": "dam", "nx": 64, "ny": 32, "nz": 48,
         "precision": 0, "net": 0, "tol": 1e-10},
        # a small tank on the mixed path: short kernels, the multigrid's coarse levels dominate
        {"name": "step_tank_small_mixed", "kind": "step", "preset": "sloshing", "nx": 64, "ny": 32, "nz": 32,
         "precision": 1, "net": 0, "tol": 1e-8},
        # an ordinary dam break on the mixed path, with sizes that are not powers of two
        {"name": "step_dam_mixed", "kind": "step", "preset": "dam", "nx": 144, "ny": 80, "nz": 112,
         "precision": 1, "net": 0, "tol": 1e-8},
        # the benchmark's sloshing tank, mixed path: the time step production runs repeat
        {"name": "step_sloshing_mixed", "kind": "step", "preset": "sloshing", "nx": 256, "ny": 128, "nz": 128,
         "precision": 1, "net": 0, "tol": 1e-8},
        # the same tank on the plain FP64 path (the reference's own algorithm)
        {"name": "step_sloshing_fp64", "kind": "step", "preset": "sloshing", "nx": 256, "ny": 128, "nz": 128,
         "precision": 0, "net": 0, "tol": 1e-8},
        # the benchmark's headline path: the network's initial guess in front of the mixed solve
        {"name": "step_sloshing_learned", "kind": "step", "preset": "sloshing", "nx": 256, "ny": 128, "nz": 128,
         "precision": 1, "net": 1, "tol": 1e-8},
        # the LES channel over a bump: the largest configuration (inflow, outflow, periodic y,
        # obstacle columns), mixed path
        {"name": "step_les_mixed", "kind": "step", "preset": "les", "nx": 512, "ny": 256, "nz": 256,
         "precision": 1, "net": 0, "tol": 1e-9},
        # level-set stage alone, FP64, odd sizes
        {"name": "level_set_fp64", "kind": "level_set", "nx": 191, "ny": 97, "nz": 113, "precision": 0},
        # viscosity and momentum right-hand side alone, FP64, centred scheme, ragged sizes
        {"name": "momentum_fp64", "kind": "momentum", "nx": 150, "ny": 133, "nz": 90, "precision": 0, "der": 2},
        # one pressure solve of a random tank from zero pressure (the training data's generator
        # and the per-solve comparison make thousands of them)
        {"name": "projection_mixed", "kind": "projection", "nx": 128, "ny": 128, "nz": 128, "precision": 1,
         "tol": 1e-8},
        # one gradient of the network's training (128^3 tanks)
        {"name": "train_128", "kind": "train", "nx": 128, "ny": 128, "nz": 128},
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mg_sizes(rng, most):
    """A grid the multigrid takes: it halves down to at most 1024 cells."""
    while True:
        c = [rng.randint(4, 16) for _ in range(3)]
        k = rng.randint(2, 4)
        n = [v << k for v in c]
        if c[0] * c[1] * c[2] <= 1024 and 16000 <= n[0] * n[1] * n[2] <= most:
            return n


def draw(rng):
    kind = rng.choice(["step64", "step32", "step32", "level_set", "momentum", "projection", "train"])
    if kind == "step64":
        preset = rng.choice(["default", "dam", "sloshing"])
        nx, ny, nz = (_log_size(rng, 20, 110) for _ in range(3))
        return {"kind": "step", "preset": preset, "nx": nx, "ny": ny, "nz": nz, "precision": 0, "net": 0, "tol": 1e-10}
    if kind == "step32":
        nx, ny, nz = _mg_sizes(rng, 6_000_000)
        net = 1 if rng.random() < 0.25 and not (nx % 8 or ny % 8 or nz % 8) else 0
        preset = rng.choice(["dam", "sloshing", "les"])
        return {"kind": "step", "preset": preset, "nx": nx, "ny": ny, "nz": nz, "precision": 1, "net": net,
                "tol": 1e-9 if preset == "les" else 1e-8}
    if kind == "projection":
        nx, ny, nz = _mg_sizes(rng, 4_200_000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": 1, "tol": 1e-8}
    if kind == "train":
        nx, ny, nz = (8 * rng.randint(2, 16) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    nx, ny, nz = (_log_size(rng, 12, 256) for _ in range(3))
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": rng.randint(0, 1)}
    if kind == "momentum":
        c["der"] = rng.randint(1, 2)
    if c["precision"]:   # precision 1 needs a grid the multigrid takes
        c["nx"], c["ny"], c["nz"] = _mg_sizes(rng, 6_000_000)
    return c


# ------------------------------------------------------------------------------- parameters
def _mixed(p, tol):
    """The mixed path as the benchmark sets it."""
    p.precision, p.cg_tol, p.inner_tol, p.refine_maxit = 1, tol, 1e-3, 40
    p.mg_omega, p.mg_alpha, p.mg_omega2 = 0.56, 1.8, 1.39
    return p


def _params(case):
    """Parameters of the case's workload, and its obstacle masks and inflow speed."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    preset = case.get("preset", "sloshing")
    masks, u_init = None, 0.0
    if preset == "default":
        p, _ = pkg.cases.reference_default(nx, ny, nz)
        u_init = 0.31
        p.cg_stop, p.cg_maxit = 1, 20000
        p.periodic_faces = 1   # the surface moves across the periodic x boundary
    elif preset == "dam":
        p, _ = pkg.cases.dam_break(nx, ny, nz)
    elif preset == "les":
        p, _, masks = pkg.cases.les_channel(nx, ny, nz)
        u_init = 1.0
    else:
        p, _ = pkg.cases.sloshing(nx, ny, nz, div_tol=1e-8)
    p.cg_tol = case.get("tol", 1e-8)
    p.der = case.get("der", p.der)
    if case["precision"] == 1:
        _mixed(p, p.cg_tol)
    return p, masks, u_init


# ------------------------------------------------------------------------------- inputs
# Arrays are torch tensors in the Fortran arrays' memory order: shape (n2, n1, n0).
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, lo, hi):
    return lo + (hi - lo) * float(torch.rand((), generator=g, device=DEV, dtype=F64))


def _noise(g, shape, sigma=3.0):
    """White noise smoothed by a Gaussian of `sigma` cells, unit variance."""
    f = torch.fft.rfftn(torch.randn(shape, generator=g, device=DEV, dtype=F64))
    freq = [torch.fft.fftfreq(shape[0], device=DEV, dtype=F64), torch.fft.fftfreq(shape[1], device=DEV, dtype=F64),
            torch.fft.rfftfreq(shape[2], device=DEV, dtype=F64)]
    k2 = freq[0][:, None, None] ** 2 + freq[1][None, :, None] ** 2 + freq[2][None, None, :] ** 2
    out = torch.fft.irfftn(f * torch.exp(-2.0 * (math.pi * sigma) ** 2 * k2), s=shape)
    return out / out.std()


def _level_set(p, g, preset):
    """Level set (positive in water) and the cell centres it was formed at."""
    n = (p.nx, p.ny, p.nz)
    h = (p.dx, p.dy, p.dz)
    ax = [(torch.arange(m, device=DEV, dtype=F64) + 0.5) * d for m, d in zip(n, h)]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    lx, ly, lz = (m * d for m, d in zip(n, h))
    if preset == "dam":
        a, top = lx * _uniform(g, 0.3, 0.5), lz * _uniform(g, 0.5, 0.7)
        inside = torch.minimum(a - X, top - Z) + 0 * Y
        out = -torch.sqrt((X - a).clamp(min=0) ** 2 + (Z - top).clamp(min=0) ** 2) + 0 * Y
        return torch.where(inside >= 0, inside, out).contiguous()
    depth = {"default": 0.5 / 0.9, "les": 2.0 / 3.0}.get(preset, 0.5) * lz
    amp = {"default": 0.01, "les": 0.01}.get(preset, 0.03) * lz * _uniform(g, 0.5, 1.0)
    kx, ky = (2 * math.pi if p.ccx0 == 0 else math.pi), (2 * math.pi if p.ccy0 == 0 else math.pi)
    ph = _uniform(g, 0, 2 * math.pi) if p.ccx0 == 0 else 0.0
    return (depth + amp * torch.cos(kx * X / lx + ph) * torch.cos(ky * Y / ly) - Z).contiguous()


def _velocity(p, g, scale, u_init):
    """A divergence-free velocity field with closed walls: the curl of a smooth random potential
    that vanishes on the walls, u_init added along x."""
    n = (p.nz, p.ny, p.nx)
    dim = {"x": 2, "y": 1, "z": 0}
    wall = {2: p.ccx0 != 0, 1: p.ccy0 != 0, 0: p.ccz0 != 0}

    def potential(along):
        a = _noise(g, [n[d] + (d != dim[along]) for d in range(3)], 4.0)
        for d in range(3):
            if d == dim[along]:
                continue
            if wall[d]:
                a.index_fill_(d, torch.tensor([0, n[d]], device=DEV), 0.0)
            else:
                a.narrow(d, n[d], 1).copy_(a.narrow(d, 0, 1))
        return a

    px, py, pz = potential("x"), potential("y"), potential("z")
    d = lambda a, axis, h: a.diff(dim=dim[axis]) / h
    u = d(pz, "y", p.dy) - d(py, "z", p.dz)
    v = d(px, "z", p.dz) - d(pz, "x", p.dx)
    w = d(py, "x", p.dx) - d(px, "y", p.dy)
    s = scale / float(torch.sqrt((u.square().mean() + v.square().mean() + w.square().mean()) / 3))
    out = {}
    for name, a, base in (("u", u, u_init), ("v", v, 0.0), ("w", w, 0.0)):
        full = torch.zeros(tuple(reversed(pkg.field_shape(p, name))), device=DEV, dtype=F64)
        full[1:1 + a.shape[0], 1:1 + a.shape[1], 1:1 + a.shape[2]] = s * a + base
        out[name] = full
    return out


def _pressure(p, ls):
    """Hydrostatic pressure of the level set, the start a running simulation has."""
    width = 1.5 * max(p.dx, p.dy, p.dz)
    H = (0.5 * (1 + ls / width)).clamp(0, 1)
    weight = (p.rho_f1 * (1 - H) + p.rho_f2 * H) * p.gz * p.dz
    q = weight.flip(0).cumsum(0).flip(0) - 0.5 * weight
    full = torch.zeros(tuple(reversed(pkg.field_shape(p, "prd1"))), device=DEV, dtype=F64)
    full[1:-1, 1:-1, 1:-1] = q
    return full


def _download(s, name, out):
    """Copy a field into a device tensor through the C-ABI (suli_download takes device memory)."""
    s._check(s.lib.suli_download(s._h, pkg.FIELD[name], ctypes.cast(ctypes.c_void_p(out.data_ptr()),
                                                                    ctypes.POINTER(ctypes.c_double))), name)
    return out


def _buffers(p, names):
    return {k: torch.empty(tuple(reversed(pkg.field_shape(p, k))), device=DEV, dtype=F64) for k in names}


STATE = ("u", "v", "w", "prd1", "ls")


def prepare(case, seed):
    g = _generator(seed)
    if case["kind"] == "train":
        return _prepare_train(case, g)
    p, masks, u_init = _params(case)
    s = pkg.Solver(p)
    preset = case.get("preset", "sloshing")
    if case["kind"] == "projection":
        ls, vel, _ = pkg.snapshots.SnapshotGenerator(s, int(seed)).draw()
        prd1 = torch.zeros(tuple(reversed(pkg.field_shape(p, "prd1"))), device=DEV, dtype=F64)
        return {"kind": case["kind"], "s": s, "in": {"ls": ls, "prd1": prd1, **vel},
                "out": _buffers(p, ("u", "v", "w", "prd1"))}
    if case["kind"] == "momentum":
        st = _momentum_inputs(p, g)
        for k, a in st.items():
            s.upload_device(k, a)
        return {"kind": case["kind"], "s": s, "out": _buffers(p, ("Fu", "Fv", "Fw"))}
    if masks is not None:
        s.set_obstacle(*masks)
    s.iniciais(u_init)
    ls = _level_set(p, g, preset)
    s.upload_device("ls", ls)
    s.level_set_ini()
    scale = (0.2 if case["kind"] == "level_set" else 0.01) * p.dx / p.dt   # the steps' own CFL 0.2-0.3 includes the wave speed
    st = {**_velocity(p, g, scale, u_init), "prd1": _pressure(p, ls), "ls": ls}
    if case["kind"] == "level_set":
        for k in ("u", "v", "w"):
            s.upload_device(k, st[k])
        return {"kind": case["kind"], "s": s, "ls": ls, "out": _buffers(p, ("ls", "rho", "kurv"))}
    if preset == "les":   # the seeded fluctuation of the inflow planes, zero inside the bump
        inflow = 1.0 + 0.05 * (2 * torch.rand(_plane(p, "bxx0"), generator=g, device=DEV, dtype=F64) - 1).cpu().numpy().T
        for name in ("bxx0", "bxx1"):
            plane = s.download(name)
            s.upload(name, np.where(plane == 0.0, 0.0, inflow[:, :, None]))
    net = None
    if case["net"]:
        net = pkg.learned.Net.load(p.nx, p.ny, p.nz)
        s.attach_nn(net)
    return {"kind": case["kind"], "s": s, "net": net, "in": st, "out": _buffers(p, STATE)}


def _plane(p, name):
    n0, n1, _ = pkg.field_shape(p, name)
    return n1, n0


# ------------------------------------------------------------------------------- one pass
def _centred(prd1):
    """The pressure of an all-Neumann problem is defined up to a constant: its mean removed."""
    q = prd1[1:-1, 1:-1, 1:-1]
    return q - q.mean()


def run(state):
    kind = state["kind"]
    if kind == "train":
        return state["net"].loss_grad(state["in3"], state["target"])
    s, out = state["s"], state["out"]
    if kind == "step":
        for k, a in state["in"].items():
            s.upload_device(k, a)
        s.contorno(1)
        s.step(1)
    elif kind == "level_set":
        s.upload_device("ls", state["ls"])
        s.level_set()
    elif kind == "momentum":
        s.visco()
        s.convdiff()
    else:
        for k, a in state["in"].items():
            s.upload_device(k, a)
        s.heaviside()
        s.graddin()
        s.posdin()
    for k, a in out.items():
        _download(s, k, a)
    if "prd1" not in out:
        return out
    return {**{k: a for k, a in out.items() if k != "prd1"}, "p": _centred(out["prd1"])}


# ------------------------------------------------------------------------------- work
def work(case):
    """Each input read once, each output written once; the operations of the stencils, and for
    the solves those of the operator applied once per stage."""
    n = float(case["nx"] * case["ny"] * case["nz"])
    kind = case["kind"]
    if kind == "train":
        # 14 convolutions forward, twice that backward; input and target in, parameters in and out
        conv = sum(2.0 * 27 * ci * co / 8 ** lv for ci, co, lv in pkg.learned.LAYERS) * n
        return {"bytes": 16.0 * n + 8.0 * pkg.learned.num_params(), "flops": 3.0 * conv}
    if kind == "level_set":   # three transport stages, S(phi0), three reinitialisation stages, normals, curvature
        return {"bytes": 8.0 * 7 * n, "flops": 9 * 600.0 * n}
    if kind == "momentum":
        return {"bytes": 8.0 * 12 * n, "flops": 400.0 * n}
    if kind == "projection":
        return {"bytes": 8.0 * 9 * n, "flops": 100.0 * n}
    stages = 2 if case["preset"] == "default" else 3
    return {"bytes": 8.0 * 10 * n, "flops": (9 * 600.0 + stages * 500.0) * n}


# ------------------------------------------------------------------------------- 64-bit values
def exact(case, seed):
    cells = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed) if cells <= 2_100_000 else None
    if kind in ("level_set", "momentum", "projection"):
        p, masks, u_init = _params(case)
        g = _generator(seed)
        if kind == "momentum":
            return _exact_momentum(p, _momentum_inputs(p, g))
        if kind == "level_set":
            ls = _level_set(p, g, case.get("preset", "sloshing"))
            return _exact_level_set(p, ls, _velocity(p, g, 0.2 * p.dx / p.dt, u_init))
        return _exact_projection(p, int(seed)) if cells <= 4_200_000 else None
    return None   # whole steps: converged to the residual test, no closed result


# --- level set
def _pencil(f, dim, rule):
    """Three ghosts on each side of axis `dim` by the reference's pencil rules (0 periodic with
    its offset, 1 and 2 extrapolation)."""
    n = f.shape[dim]
    at = lambda m: f.narrow(dim, m - 1, 1)   # 1-based
    if rule == 0:
        lo, hi = [at(n - 1), at(n - 2), at(n - 3)], [at(2), at(3), at(4)]
    else:
        def extend(a, b, c, low):
            ext = []
            for _ in range(3):
                q = (12. * a - 9. * b + 2. * c) / 5. if low else (18. * a - 9. * b + 2. * c) / 11.
                ext.append(q)
                a, b, c = q, a, b
            return ext
        lo, hi = extend(at(1), at(2), at(3), rule == 1), extend(at(n), at(n - 1), at(n - 2), False)
    return torch.cat([lo[2], lo[1], lo[0], f, *hi], dim)


def _weno(f, dim, rule, h):
    """Right- and left-biased fifth-order WENO derivatives of a cell field along an axis."""
    n = f.shape[dim]
    q = _pencil(f, dim, rule)
    D = [q.narrow(dim, m + 1, n) / h - q.narrow(dim, m, n) / h for m in range(6)]

    def side(a, b, c, d, e):
        beta = (13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
                13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
                13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2)
        al = [w / (1e-8 + s) ** 2 for w, s in zip((0.1, 0.6, 0.3), beta)]
        t = al[0] + al[1] + al[2]
        return (al[0] / t * (2 * a - 7 * b + 11 * c) + al[1] / t * (-b + 5 * c + 2 * d) +
                al[2] / t * (2 * c + 5 * d - e)) / 6
    return side(*D[5:0:-1]), side(*D[0:5])


def _gradients(p, f):
    rules = (0 if p.ccx0 == 0 else 2, 0 if p.ccy0 == 0 else 2, 0 if p.ccz0 == 0 else 1)
    return [_weno(f, 2 - a, rules[a], (p.dx, p.dy, p.dz)[a]) for a in range(3)]


def _heaviside(p, ls):
    w = p.alpha1 * max(p.dx, p.dy, p.dz)
    h = 0.5 * (1 + ls / w + torch.sin(math.pi * ls / w) / math.pi)
    return torch.where(ls < -w, torch.zeros_like(ls), torch.where(ls > w, torch.ones_like(ls), h))


def _exact_level_set(p, ls, vel):
    dx1 = max(p.dx, p.dy, p.dz)
    rk = ((1., 0., 1.), (3 / 4, 1 / 4, 1 / 4), (1 / 3, 2 / 3, 2 / 3))
    cells = (slice(1, p.nz + 1), slice(1, p.ny + 1), slice(1, p.nx + 1))
    centre = []
    for k, d in (("u", 2), ("v", 1), ("w", 0)):
        up = list(cells)
        up[d] = slice(cells[d].start + 1, cells[d].stop + 1)
        centre.append(0.5 * (vel[k][cells] + vel[k][tuple(up)]))

    def advect(f):
        return -sum(c.clamp(min=0) * dn + c.clamp(max=0) * dp for c, (dp, dn) in zip(centre, _gradients(p, f)))

    def size(f):
        tiny = torch.full_like(f, 1e-8)
        m = 0.
        for dp, dn in _gradients(p, f):
            a = torch.where(f > 0, torch.maximum(torch.maximum(dn, tiny), -torch.minimum(dp, tiny)),
                            torch.maximum(torch.maximum(dp, tiny), -torch.minimum(dn, tiny)))
            m = m + a * a
        return torch.sqrt(m)

    def stages(f, rate, dt):
        f0, before = f, f
        for a, b, c in rk:
            before, f = f, a * f0 + b * f + c * dt * rate(f)
        return f, before

    f, _ = stages(ls, advect, p.dt)
    sign = f / torch.sqrt(f * f + size(f) ** 2 * dx1 * dx1)
    for il in range(1, p.reinit_maxit + 1):
        f, before = stages(f, lambda q: sign * (1 - size(q)), p.dt1)
        band = f.abs() <= 2 * p.alpha1 * dx1
        if not float((f - before)[band].sum()) / max(1, int(band.sum())) > p.dt1 * dx1 * dx1:
            break
    larger = lambda q: torch.where(q[0].abs() > q[1].abs(), q[0], q[1])
    grad = [larger(q) for q in _gradients(p, f)]
    m = torch.sqrt(sum(q * q for q in grad))
    normal = [torch.where(m == 0, torch.zeros_like(m), q / m) for q in grad]
    rule = 0 if p.ccz0 == 0 else 1
    kurv = sum(larger(_weno(q, 2 - a, rule, (p.dx, p.dy, p.dz)[a])[::-1]) for a, q in enumerate(normal))
    H = _heaviside(p, f)
    return {"ls": f, "rho": p.rho_f1 * (1 - H) + p.rho_f2 * H, "kurv": kurv}


# --- momentum
def _momentum_inputs(p, g):
    ls = _level_set(p, g, "sloshing")
    st = {}
    for k in ("u", "v", "w"):
        st[k] = 0.1 * p.dx / p.dt * _noise(g, tuple(reversed(pkg.field_shape(p, k))))
    w = p.alpha1 * max(p.dx, p.dy, p.dz)
    H = _heaviside(p, ls)
    delta = torch.where(ls.abs() <= w, 0.5 * (1 + torch.cos(math.pi * ls / w)) / w, torch.zeros_like(ls))
    for k, d, h in (("hsx", 2, p.dx), ("hsy", 1, p.dy), ("hsz", 0, p.dz)):
        st[k] = (delta * torch.gradient(ls, spacing=h, dim=d)[0]).contiguous()
    st["kurv"] = _noise(g, tuple(ls.shape))
    st["rho"] = p.rho_f1 * (1 - H) + p.rho_f2 * H
    st["ls_nu"] = p.mi_f1 * (1 - H) + p.mi_f2 * H
    return st


def _exact_momentum(p, st):
    n, h = (p.nx, p.ny, p.nz), (p.dx, p.dy, p.dz)
    vel = (st["u"], st["v"], st["w"])

    def take(a, d, idx):   # 1-based positions idx along axis d of an array that starts at 1
        return a.index_select(2 - d, idx - 1)

    def to_face(a, d):     # cells 1..n -> faces 1..n+1, end faces copied
        f = torch.arange(1, a.shape[2 - d] + 2, device=DEV).clamp(2, a.shape[2 - d])
        return 0.5 * (take(a, d, f) + take(a, d, f - 1))

    def box(a, lo, cnt, off=(0, 0, 0)):   # a staggered array (starting at 0) on lo + off, cnt points
        return a[lo[2] + off[2]:lo[2] + off[2] + cnt[2], lo[1] + off[1]:lo[1] + off[1] + cnt[1],
                 lo[0] + off[0]:lo[0] + off[0] + cnt[0]]

    e = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    one, plus = (1, 1, 1), lambda a, b, s=1: tuple(x + s * y for x, y in zip(a, b))
    # Smagorinsky viscosity at the cells
    D = [[0.0] * 3 for _ in range(3)]   # D[c][d]: derivative of component c along d, face -> centre
    for c in range(3):
        for d in range(3):
            at = lambda o: box(vel[c], one, n, o)
            D[c][d] = 0.5 * sum((at(plus(o, e[d])) - at(plus(o, e[d], -1))) / (2 * h[d]) for o in ((0, 0, 0), e[c]))
    s = [D[c][c] + 0.5 * sum(D[c][d] + D[d][c] for d in range(3) if d != c) for c in range(3)]
    t = s[0] + s[1] + s[2]
    nut = (h[0] * h[1] * h[2]) ** (2 / 3) * p.csmag ** 2 * torch.sqrt(2 * t * t) * st["rho"]
    F = []
    for c in range(3):
        cnt = plus(n, e[c])
        face = to_face(st["ls_nu"], c) + to_face(nut, c)
        at = lambda o=(0, 0, 0), q=None: box(vel[c if q is None else q], one, cnt, o)
        a0 = at()
        adv = 0.0
        for d in range(3):
            up, dn = at(e[d]), at(plus((0, 0, 0), e[d], -1))
            if p.der == 1:
                if d == c:
                    speed = a0
                else:
                    back = plus((0, 0, 0), e[c], -1)
                    speed = 0.25 * (at((0, 0, 0), d) + at(back, d) + at(e[d], d) + at(plus(back, e[d]), d))
                adv = adv + speed.clamp(min=0) * (a0 - dn) / h[d] + speed.clamp(max=0) * (up - a0) / h[d]
            else:
                speed = a0 if d == c else to_face(0.5 * (box(vel[d], one, n) + box(vel[d], one, n, e[d])), c)
                adv = adv + speed * (up - dn) / (2 * h[d])
        visc = 0.0
        for d in range(3):
            up, dn = at(e[d]), at(plus((0, 0, 0), e[d], -1))
            if d == c:
                f = torch.arange(1, n[c] + 2, device=DEV)
                hi, lo = take(nut, c, f.clamp(1, n[c])), take(nut, c, (f - 1).clamp(1, n[c]))
                visc = visc + (2 * hi * (up - a0) - 2 * lo * (a0 - dn)) / h[c] ** 2
            else:
                edge = to_face(face, d)   # along d: positions 1..n+1, end copies
                f = torch.arange(1, n[d] + 1, device=DEV)
                hi, lo = take(edge, d, f + 1), take(edge, d, f)
                back = plus((0, 0, 0), e[c], -1)
                visc = visc + hi * ((up - a0) / h[d] + (at(e[d], d) - at(plus(back, e[d]), d)) / h[c]) / h[d]
                visc = visc - lo * ((a0 - dn) / h[d] + (at((0, 0, 0), d) - at(back, d)) / h[c]) / h[d]
        tension = to_face(st[("hsx", "hsy", "hsz")[c]] * st["kurv"] / st["rho"], c)
        body = (p.gx, 0.0, -p.gz)[c]
        F.append(-adv + visc / to_face(st["rho"], c) + body - p.sigma * tension)
    return {"Fu": F[0], "Fv": F[1], "Fw": F[2]}


# --- projection
def _exact_projection(p, seed):
    """The pressure problem of a closed tank solved to 1e-14 with a Jacobi-scaled CG in torch."""
    class Grid:   # what the snapshot generator reads of a solver
        params = p
    ls, vel, _ = pkg.snapshots.SnapshotGenerator(Grid, seed).draw()
    H = _heaviside(p, ls)
    rho = p.rho_f1 * (1 - H) + p.rho_f2 * H
    h = (p.dx, p.dy, p.dz)
    face = [p.dt / h[a] ** 2 / (0.5 * (rho.narrow(2 - a, 1, rho.shape[2 - a] - 1) +
                                        rho.narrow(2 - a, 0, rho.shape[2 - a] - 1))) for a in range(3)]

    def apply(q):
        out = torch.zeros_like(q)
        for a in range(3):
            m = q.shape[2 - a] - 1
            flow = face[a] * (q.narrow(2 - a, 1, m) - q.narrow(2 - a, 0, m))
            out.narrow(2 - a, 0, m).sub_(flow)
            out.narrow(2 - a, 1, m).add_(flow)
        return out

    diag = torch.zeros_like(rho)
    for a in range(3):
        m = rho.shape[2 - a] - 1
        diag.narrow(2 - a, 0, m).add_(face[a])
        diag.narrow(2 - a, 1, m).add_(face[a])
    cell = [slice(1, -1)] * 3
    inner = {}
    for k, a, extra in (("u", 0, p.nx + 1), ("v", 1, p.ny + 1), ("w", 2, p.nz + 1)):
        sl = [slice(1, p.nz + 1), slice(1, p.ny + 1), slice(1, p.nx + 1)]
        sl[2 - a] = slice(1, extra + 1)
        inner[k] = tuple(sl)
    b = -sum(vel[k][inner[k]].diff(dim=2 - a) / h[a] for k, a in (("u", 0), ("v", 1), ("w", 2)))
    q = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    d = z.clone()
    rz = (r * z).sum()
    stop = 1e-28 * rz
    for it in range(8000):
        Ad = apply(d)
        alpha = rz / (d * Ad).sum()
        q.add_(alpha * d)
        r.sub_(alpha * Ad)
        z = r / diag
        new = (r * z).sum()
        if it % 20 == 0 and bool(new < stop):
            break
        d = z + (new / rz) * d
        rz = new
    out = {}
    for k, a in (("u", 0), ("v", 1), ("w", 2)):
        f = vel[k].clone()
        m = q.shape[2 - a] - 1
        sl = list(inner[k])
        sl[2 - a] = slice(2, m + 2)
        f[tuple(sl)] -= face[a] * h[a] * (q.narrow(2 - a, 1, m) - q.narrow(2 - a, 0, m))
        out[k] = f
    return {**out, "p": q - q.mean()}


# --- training
def _prepare_train(case, g):
    """The shipped weights, and features and target with the distributions the solver records:
    scaled residual, Heaviside of a random tank, scaled previous pressure; scaled correction."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    in3, target = _train_inputs(case, g)
    return {"kind": "train", "net": pkg.learned.Net.load(nx, ny, nz), "in3": in3, "target": target}


def _train_inputs(case, g):
    shape = (case["nz"], case["ny"], case["nx"])
    level = 0.3 * case["nz"] * _uniform(g, 0.7, 2.0) + 3.0 * _noise(g, shape, 6.0)
    z = torch.arange(case["nz"], device=DEV, dtype=F64)[:, None, None]
    H = (0.5 + (level - z) / 3).clamp(0, 1)
    in3 = torch.stack([_noise(g, shape, 1.5), H, _noise(g, shape, 8.0)], dim=-1).float().reshape(-1, 3).contiguous()
    target = (0.1 * _noise(g, shape, 6.0)).float().reshape(-1).contiguous()
    return in3, target


def _exact_train(case, seed):
    in3, target = _train_inputs(case, _generator(seed))
    theta = torch.from_numpy(np.load(pkg.learned.WEIGHTS_PATH)).to(DEV, F64).requires_grad_(True)
    shape = (case["nz"], case["ny"], case["nx"])
    x = torch.zeros(16, *shape, device=DEV, dtype=F64)
    x[:3] = in3.to(F64).t().reshape(3, *shape)
    layers, o = [], 0
    for ci, co, _ in pkg.learned.LAYERS:
        layers.append((theta[o:o + 27 * co * ci].reshape(27, co, ci), theta[o + 27 * co * ci:o + 27 * co * ci + co]))
        o += 27 * co * ci + co

    class Conv(torch.autograd.Function):   # 3x3x3, zero padding, one matrix product a tap
        @staticmethod
        def forward(ctx, q, W):
            ctx.save_for_backward(q, W)
            s = q.shape[1:]
            pad = torch.nn.functional.pad(q, (1, 1, 1, 1, 1, 1))
            out = torch.zeros(W.shape[1], s[0] * s[1] * s[2], device=DEV, dtype=F64)
            for t in range(27):
                k, j, i = t // 9, (t // 3) % 3, t % 3
                out.addmm_(W[t], pad[:, k:k + s[0], j:j + s[1], i:i + s[2]].reshape(q.shape[0], -1))
            return out.reshape(-1, *s)

        @staticmethod
        def backward(ctx, gout):
            q, W = ctx.saved_tensors
            s = q.shape[1:]
            pad = torch.nn.functional.pad(q, (1, 1, 1, 1, 1, 1))
            gpad, gW, g2 = torch.zeros_like(pad), torch.empty_like(W), gout.reshape(gout.shape[0], -1)
            for t in range(27):
                sl = (slice(None), slice(t // 9, t // 9 + s[0]), slice((t // 3) % 3, (t // 3) % 3 + s[1]),
                      slice(t % 3, t % 3 + s[2]))
                gW[t] = g2 @ pad[sl].reshape(q.shape[0], -1).t()
                gpad[sl] += (W[t].t() @ g2).reshape(q.shape[0], *s)
            return gpad[:, 1:-1, 1:-1, 1:-1], gW

    conv = lambda l, q: torch.relu(Conv.apply(q, layers[l][0]) + layers[l][1][:, None, None, None])
    pool = lambda q: q.reshape(q.shape[0], q.shape[1] // 2, 2, q.shape[2] // 2, 2, q.shape[3] // 2, 2).mean((2, 4, 6))
    up = lambda q: q.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)
    skips = []
    for lv in range(4):
        x = conv(2 * lv + 1, conv(2 * lv, pool(x) if lv else x))
        skips.append(x)
    for l, lv in ((8, 2), (10, 1), (12, 0)):
        x = conv(l + 1, conv(l, torch.cat([up(x), skips[lv]])))
    y = (theta[o:o + 16] @ x.reshape(16, -1)) + theta[o + 16]
    loss = (y - target.to(F64)).square().mean()
    loss.backward()
    return float(loss.detach()), theta.grad
