"""Performance cases of the FDTD library: what its users run, through the Python
entry points (Solver, Batch), over the range of sizes the package is used at.

A case is a dict of plain values.  `kind` picks the work:

  run       a scene stepped `steps` times (fdtd_step, or its replayed form when
            `graph`), then the fields, the probe series and the far field read
            back -- the life of every simulation;
  batch     `count` uneven rough-surface instances stepped in lockstep;
  adjoint   objective and design gradient over `steps` steps, with checkpoints;
  farfield  the running DFTs of a run integrated to a whole far-field grid.

`prepare` builds the plan and uploads initial fields drawn from the seed; `run`
is one pass; `exact` restates the pass in FP64 with plain torch.  FP32 and
16-bit plans compute in FP32, so what they return as doubles (probe series,
spectra, objective, gradient) is compared as FP32 numbers.
"""
import ctypes as C
import math

import numpy as np
import torch

from gsvit_copy_b200 import abi, plan
from gsvit_copy_b200.solver import Batch, Solver

STORAGE = {"f32": abi.STORE_F32, "f16": abi.STORE_F16, "bf16": abi.STORE_BF16, "f64": abi.STORE_F64}
ESIZE = {"f32": 4, "f16": 2, "bf16": 2, "f64": 8}
PLANNED = 4000      # steps a plan is made for: length of its waveform and probe series


def _run(name, scene, x, y, z, depth, steps, graph, storage="f32"):
    return dict(name=name, kind="run", scene=scene, x=x, y=y, z=z, depth=depth, steps=steps, graph=graph, storage=storage)


def listed():
    return [
        # one small rough-surface instance stepped eagerly, as a script that looks at its probes now and
        # then does: launches and latency
        _run("rough_64_eager", "drude", 64, 64, 64, 8, 50, False),
        # the plain FP32 dielectric sphere, GSvit's usual first problem
        _run("sphere_100", "sphere", 100, 100, 100, 10, 100, True),
        # uneven extents, no row a multiple of 16 bytes: grids drawn by hand rather than by powers of two
        _run("lorentz_ragged", "lorentz", 150, 118, 131, 9, 40, True),
        # an ordinary production size
        _run("rough_256", "drude", 256, 256, 256, 16, 100, True),
        # the headline size of the package
        _run("rough_512", "drude", 512, 512, 512, 16, 64, True),
        # 16-bit field storage
        _run("rough_256_f16", "drude", 256, 256, 256, 16, 64, True, "f16"),
        _run("rough_192_bf16", "drude", 192, 192, 128, 12, 64, True, "bf16"),
        # reference precision, used to pin the others
        _run("sphere_128_f64", "sphere", 128, 128, 128, 10, 30, False, "f64"),
        # GSvit's self-test deck (voxel box, kappa 4, time-domain far field of one point), as the drop-in steps it
        _run("deck_200", "deck", 200, 200, 200, 10, 40, False),
        # independent realisations of uneven size in one batch
        dict(name="batch_12", kind="batch", count=12, steps=32),
        # inverse design: objective and gradient by the discrete adjoint
        dict(name="adjoint_128", kind="adjoint", x=128, y=128, z=96, depth=12, steps=60, checkpoint=20),
        # a finished run's whole far-field grid
        dict(name="farfield_192", kind="farfield", x=192, y=192, z=192, depth=16, theta=46, phi=91),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 8 + ["batch", "adjoint", "farfield"])
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(3, 12), steps=2 * rng.randint(6, 20))
    depth = rng.randint(8, 16)
    low = 2 * depth + 30     # room for the slabs, the boxes between them and the scatterer
    x, y, z = (_log(rng, low, 300) for _ in range(3))
    if kind == "adjoint":
        x, y, z = (_log(rng, low + 34, 180) for _ in range(3))
        steps = rng.randint(24, 60)
        return dict(kind="adjoint", x=x, y=y, z=z, depth=depth, steps=steps, checkpoint=rng.randint(8, steps))
    if kind == "farfield":
        return dict(kind="farfield", x=min(x, 200), y=min(y, 200), z=min(z, 200), depth=depth, theta=rng.randint(10, 46),
                    phi=rng.randint(19, 91))
    scene = rng.choice(["drude", "drude", "lorentz", "sphere"])
    storage = rng.choice(["f32"] * 7 + ["f16", "bf16", "f64"])
    if rng.random() < 0.6:   # most grids are chosen with even extents
        x, y, z = (max(low, v // 8 * 8) for v in (x, y, z))
    steps = max(16, min(100, int(6e8 / (x * y * z))))
    return dict(kind="run", scene=scene, x=x, y=y, z=z, depth=depth, steps=steps, graph=rng.random() < 0.6, storage=storage)


# ------------------------------------------------------------------ scenes

def _scene(case, seed):
    kind = case.get("scene", case["kind"])
    x, y, z, d = case["x"], case["y"], case["z"], case["depth"]
    if kind in ("drude", "lorentz", "farfield"):
        angles = (case["theta"], case["phi"]) if kind == "farfield" else (10, 19)
        s = plan.rough_surface_scene(res=x, yres=y, zres=z, nsteps=PLANNED, cpml_depth=d, seed=seed % (1 << 30),
                                     nfff_angles=angles, material="lorentz" if kind == "lorentz" else "drude")
    elif kind == "sphere":
        s = plan.sphere_scene(res=100, nsteps=PLANNED, cpml_depth=d)
        s.xres, s.yres, s.zres = x, y, z
        s.mat = np.zeros((x, y, z), dtype=np.int32)
        plan.sphere_map(s.mat, (x / 2, y / 2, z / 2), min(x, y, z) / 5, 1)
        lo = d + 5
        s.tsf["box"] = ((lo, lo, lo), (x - lo, y - lo, z - lo))
        s.probes = np.asarray([(x // 2, y // 2, 3 * z // 4), (x // 2, y // 2, d + 2), (x // 3, y // 2, z // 2)], dtype=np.int32)
    elif kind == "deck":
        s = plan.selftest_scene("31111", x, PLANNED)
        s.nfff["series"] = True
        s.probes = np.asarray([(x // 2, y // 2, z // 2)], dtype=np.int32)
    elif kind == "adjoint":
        s = plan.adjoint_scene(shape=(x, y, z), cpml_depth=d, nsteps=PLANNED, design_shape=(x // 4, y // 4, 8), seed=seed % (1 << 30),
                               glass_cells=8, pulse_delay=3e-16, pulse_width=1e-16)
    else:
        raise ValueError(kind)
    s.storage = STORAGE[case.get("storage", "f32")]
    return s


def _scenes(case, seed):
    if case["kind"] == "batch":
        return [_instance(p, seed) for p in plan.batch_params(case["count"])]
    return [_scene(case, seed)]


def _instance(p, seed):
    """One instance of plan.batch_scenes with a surface of its own for each seed."""
    x, y, z = p["shape"]
    return plan.rough_surface_scene(res=x, yres=y, zres=z, nsteps=PLANNED, cpml_depth=8, seed=(p["seed"] + seed) % (1 << 30),
                                    rms=p["rms"], corr_len=p["corr_len"], theta_deg=p["theta_deg"], tsf_margin=6,
                                    material=p["material"], nfff_angles=(10, 19))


def _noise(shape, seed):
    """Six field components on the GPU: smooth random waves a few cells long, E of order 1 and H of order
    1/377, as a field in the middle of a run."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for c in range(6):
        n = [max(2, v // 6) for v in shape]
        f = torch.randn([1, 1] + n, generator=g, device="cuda")
        f = torch.nn.functional.interpolate(f, size=list(shape), mode="trilinear", align_corners=False)[0, 0]
        out.append(f if c < 3 else f / 377.0)
    return out


_pinned = {}


def _host(shapes, dtype):
    """Pinned buffers (E, H) of each grid, kept from run to run as a program keeps them."""
    key = (tuple(tuple(s) for s in shapes), dtype)
    if key not in _pinned:
        _pinned.clear()
        _pinned[key] = [[torch.empty((3,) + tuple(s), dtype=dtype, pin_memory=True) for _ in range(2)] for s in shapes]
    return _pinned[key]


def _pointers(E, H, ctype):
    return (C.POINTER(ctype) * 6)(*[C.cast(f[c].data_ptr(), C.POINTER(ctype)) for f in (E, H) for c in range(3)])


def _upload(solver, seed):
    host = [f.cpu() for f in _noise(solver.shape, seed)]
    abi.check(solver.lib.fdtd_set_fields_f32(solver.h, abi.EH, _pointers(host[:3], host[3:], C.c_float)), "fdtd_set_fields_f32")
    solver.sync()


# ------------------------------------------------------------------ measured work

class State:
    def __init__(self, case):
        self.case = case
        self.solver = self.batch = self.obj = self.host = None

    def __del__(self):
        for h in (self.solver, self.batch):
            if h is not None:
                h.close()


def prepare(case, seed):
    st = State(case)
    scenes = _scenes(case, seed)
    if case["kind"] == "batch":
        st.batch = Batch(scenes)
        for q in range(len(scenes)):
            _upload(st.batch[q], seed + 7919 * (q + 1))
        st.host = _host([v.shape for v in st.batch.views], torch.float32)
        return st
    if case["kind"] == "adjoint":
        st.obj = plan.cone_objective(scenes[0])
    st.solver = Solver(scenes[0])
    _upload(st.solver, seed + 7919)
    if case["kind"] == "run":
        f64 = case["storage"] == "f64"
        st.host = _host([st.solver.shape], torch.float64 if f64 else torch.float32)
    if case["kind"] == "farfield":
        st.solver.step(24)
        st.solver.sync()
    return st


def _real(a, f64):
    return a if f64 else a.astype(np.complex64 if a.dtype.kind == "c" else np.float32)


def _read(g, host, f64=False):
    """Everything a finished run leaves: fields, probe series, far field."""
    if f64:
        abi.check(g.lib.fdtd_get_fields(g.h, abi.EH, _pointers(*host, C.c_double)), "fdtd_get_fields")
    else:
        abi.check(g.lib.fdtd_get_fields_f32(g.h, abi.EH, _pointers(*host, C.c_float)), "fdtd_get_fields_f32")
    out = dict(E=host[0], H=host[1], probes=_real(g.probes(), f64))
    if g.scene.nfff and g.scene.nfff.get("series"):
        out["series"] = _real(g.nfff_series(), f64)
    elif g.scene.nfff:
        out["spectrum"] = _real(g.nfff_spectrum(), f64)
    return out


def run(st):
    case, g = st.case, st.solver
    if case["kind"] == "batch":
        st.batch.step_graph(case["steps"])
        return [_read(v, h) for v, h in zip(st.batch.views, st.host)]
    if case["kind"] == "adjoint":
        J, grad = g.adjoint_gradient(st.obj, case["steps"], case["checkpoint"])
        return dict(J=np.float32(J), grad=_real(grad, False))
    if case["kind"] == "farfield":
        return dict(spectrum=_real(g.nfff_spectrum(), False))
    if case["graph"]:
        g.step_graph(case["steps"])
    else:
        g.step(case["steps"])
    return _read(g, st.host[0], case["storage"] == "f64")


def _step_work(x, y, z, d, es, dispersive, poles, nfreq, ns):
    """Bytes and operations of one time step: the six components read and written, one class byte a cell, the
    dispersive state, four psi values a CPML cell read and written, the surface samples and their running DFTs."""
    n = x * y * z
    psi = 2 * d * (x * y + y * z + x * z)
    st = 8 if es == 8 else 4
    b = n * (12 * es + 1) + dispersive * n * 3 * (2 * st + es + 4 * st * poles) + psi * 8 * es
    b += ns * (9 * es + nfreq * 6 * 32 / 8)
    f = n * 36 + dispersive * n * 3 * (9 + 14 * poles) + psi * 24 + ns * (6 + nfreq * 24)
    return b, f


def _surface(x, y, z, lo):
    a, b, c = x - 2 * lo, y - 2 * lo, z - 2 * lo
    return 2 * (a * b + b * c + a * c)


def work(case):
    if case["kind"] == "batch":
        b = f = 0
        for p in plan.batch_params(case["count"]):
            x, y, z = p["shape"]
            bb, ff = _step_work(x, y, z, 8, 4, 0.5, 1 if p["material"] == "lorentz" else 0, 3, _surface(x, y, z, 12))
            b, f = b + case["steps"] * bb + x * y * z * 24, f + case["steps"] * ff
        return {"bytes": b, "flops": f}
    x, y, z, d = case["x"], case["y"], case["z"], case["depth"]
    if case["kind"] == "farfield":
        ns, npt = _surface(x, y, z, d + 4), case["theta"] * case["phi"]
        return {"bytes": ns * (3 * 6 * 16 + 16) + npt * 3 * 3 * 16, "flops": ns * npt * (30 + 3 * 70)}
    if case["kind"] == "adjoint":
        # forward, recompute, and the transposed step: the adjoint state moves as the fields do
        b, f = _step_work(x, y, z, d, 4, 0, 0, 1, _surface(x, y, z, d + 2))
        box = (x // 4 + 1) * (y // 4 + 1) * 9
        return {"bytes": case["steps"] * (3 * b + box * 3 * 24), "flops": case["steps"] * 3 * f}
    es = ESIZE[case["storage"]]
    rough = case["scene"] in ("drude", "lorentz")
    b, f = _step_work(x, y, z, d, es, 0.5 if rough else 0, 1 if case["scene"] == "lorentz" else 0, 3 if rough else 0,
                      _surface(x, y, z, d + 4) if rough else 0)
    back = x * y * z * 6 * (8 if es == 8 else 4)
    return {"bytes": case["steps"] * b + back, "flops": case["steps"] * f}


# ------------------------------------------------------------------ the same work in FP64, plain torch

C0, MU0, EPS0 = 299792458.0, 1.256637061435917295e-6, 8.854187817620389850e-12


def _at(axis, s):
    i = [slice(None)] * 3
    i[axis] = s
    return tuple(i)


def _back(a, axis):
    """a at the cell one below along `axis` (the first plane: itself)."""
    return torch.cat([a[_at(axis, slice(0, 1))], a[_at(axis, slice(0, -1))]], axis)


def _fwd(a, axis):
    """a(+1) - a, with zero beyond the grid."""
    n = torch.zeros_like(a[_at(axis, slice(0, 1))])
    return torch.cat([a[_at(axis, slice(1, None))], n], axis) - a


def _diff(a, axis):
    """a - a(-1), zero in the first plane."""
    return a - _back(a, axis)


class Exact:
    """GSvit's time step (H, TSF, CPML; E with the dispersive branch, CPML, TSF) in FP64, whole-array torch, for
    scenes with CPML on all six faces.  `eps_design` (a tensor that may require a gradient) replaces the
    scene's design permittivities."""

    def __init__(self, s, fields, eps_design=None):
        self.s, self.n = s, 0
        dev = self.dev = fields[0].device
        self.R = (s.xres, s.yres, s.zres)
        dt, dx = s.dt, s.dx
        self.F = [f.double() for f in fields]
        full = s.matmode == abi.MATMODE_FULL
        vac, mu0 = (float(np.float32(EPS0)), float(np.float32(MU0))) if full else (EPS0, MU0)
        mats = s.mats or [None]
        mat = torch.zeros(self.R, dtype=torch.uint8, device=dev)
        if s.mat is not None:
            mat = torch.from_numpy(np.ascontiguousarray(s.mat.astype(np.uint8))).to(dev)
        eps = torch.tensor([vac] + [m.epsilon for m in mats[1:]], dtype=torch.float64, device=dev)[mat.long()]
        if s.epsilon is not None:
            eps = torch.from_numpy(s.epsilon).to(dev).double()
        ade = [q for q, m in enumerate(mats) if m is not None and m.type == abi.MAT_ADE]
        # interface cells average epsilon over the four cells of an edge
        rim = torch.zeros(self.R, dtype=torch.bool, device=dev)
        for ax in range(3):
            for q in (0, -1):
                rim[_at(ax, q)] = True
        lo = hi = eps
        if s.design:
            b = s.design["box"]
            box = (slice(b[0], b[1]), slice(b[2], b[3]), slice(b[4], b[5]))
            if eps_design is None:
                eps_design = torch.from_numpy(np.asarray(s.design["eps"], dtype=np.float64)).to(dev)
            eps = eps.clone()
            eps[box] = eps_design * EPS0
            lo = hi = eps.detach()
        for ax in range(3):
            lo = torch.minimum(lo, torch.minimum(_back(lo, ax), _back(lo.flip(ax), ax).flip(ax)))
            hi = torch.maximum(hi, torch.maximum(_back(hi, ax), _back(hi.flip(ax), ax).flip(ax)))
        rim |= lo != hi
        del lo, hi
        self.cb = []
        one = torch.ones(self.R, dtype=torch.float64, device=dev)
        for a in range(3):
            p, q = [ax for ax in range(3) if ax != a]
            tot, cnt = eps, one
            for axes in ((p,), (q,), (p, q)):
                sh, ok = eps, one
                for ax in axes:
                    sh = _back(sh, ax)
                    ok = ok.clone()
                    ok[_at(ax, 0)] = 0
                tot, cnt = tot + sh * ok, cnt + ok
            self.cb.append(dt / dx / torch.where(rim, tot / cnt, eps))
        del tot, cnt, one
        # H coefficient: mu of the material, the voxel value in vacuum
        self.db = torch.tensor([dt / mu0 / dx] + [dt / m.mu / dx for m in mats[1:]], dtype=torch.float64, device=dev)[mat.long()]
        self.own = None
        if ade:
            disp = mat == ade[0]
            self.own = []
            for a in range(3):
                p, q = [ax for ax in range(3) if ax != a]
                o = disp.clone()
                for axes in ((p,), (q,), (p, q)):
                    sh = disp
                    for ax in axes:
                        sh = _back(sh, ax).clone()
                        sh[_at(ax, 0)] = False
                    o |= sh
                self.own.append(o)
            self.branch = self.own[0] | self.own[1] | self.own[2]
            m = self.m = mats[ade[0]]
            self.cba = dt / m.epsilon / dx
            self.npoles = sum(1 for p in range(2) if m.cp_a[p] != 0)
            z = lambda: torch.zeros(self.R, dtype=torch.float64, device=dev)  # noqa: E731
            self.ep, self.P, self.Pm = [z() for _ in range(3)], [z() for _ in range(3)], [z() for _ in range(3)]
            self.p = [[z() for _ in range(self.npoles)] for _ in range(3)]
            self.pm = [[z() for _ in range(self.npoles)] for _ in range(3)]
        self._cpml()
        self._tsf(mat, eps.detach())
        if s.nfff:
            self._nfff()
        self.probes = np.zeros((len(s.probes), s.nsteps, 6))

    # CPML profiles (the grading of both field kinds) and psi
    def _cpml(self):
        s, dt = self.s, self.s.dt
        self.prof, self.psiE, self.psiH = {}, {}, {}
        self.ke = [torch.ones(n, dtype=torch.float64) for n in self.R]
        self.kh = [torch.ones(n, dtype=torch.float64) for n in self.R]
        for f in range(6):
            d, m, sig, kap, al = s.cpml[f]
            low, ax = f % 2 == 0, f // 2
            q = torch.arange(d, dtype=torch.float64)
            pos = q if low else d - q
            out = []
            for off in (0.0, -0.5 if low else 0.5):
                g = ((d - pos + off) / d) ** m
                sv, kv, av = sig * g, 1 + (kap - 1) * g, al * (pos + off) / d
                b = torch.exp(-(sv / kv + av) * dt / EPS0)
                c = torch.where(sv == 0, torch.zeros_like(sv), sv / (sv + kv * av) / kv * (b - 1))
                out += [b, c, kv]
            sl = slice(0, d) if low else slice(self.R[ax] - d, None)
            self.ke[ax][sl] = torch.maximum(self.ke[ax][sl], out[2])
            self.kh[ax][sl] = torch.maximum(self.kh[ax][sl], out[5])
            shape = [1, 1, 1]
            shape[ax] = d
            be, ce, bh, ch = (out[t].to(self.dev).reshape(shape) for t in (0, 1, 3, 4))
            base = 0 if low else self.R[ax] - d
            # E: positions 1 .. d-1, the other two indices >= 1; H: 0 .. d-2 (low) or 1 .. d-2, others off the rim
            e = [slice(1, None)] * 3
            e[ax] = slice(base + 1, base + d)
            h = [slice(1, n - 1) for n in self.R]
            h0, h1 = (0, d - 1) if low else (1, d - 1)
            h[ax] = slice(base + h0, base + h1)
            cut = lambda t, a, b: t[_at(ax, slice(a, b))]  # noqa: E731
            self.prof[f] = (tuple(e), cut(be, 1, d), cut(ce, 1, d) / s.dx, tuple(h), cut(bh, h0, h1), cut(ch, h0, h1) / s.dx)
            for psi, reg in ((self.psiE, e), (self.psiH, h)):
                sh = [len(range(*r.indices(n))) for r, n in zip(reg, self.R)]
                psi[f] = [torch.zeros(sh, dtype=torch.float64, device=self.dev) for _ in range(2)]
        for ax in range(3):
            shape = [1, 1, 1]
            shape[ax] = -1
            self.ke[ax] = self.ke[ax].to(self.dev).reshape(shape)
            self.kh[ax] = self.kh[ax].to(self.dev).reshape(shape)

    # the 1D grid of the plane wave and, per face of the TSF box, the interpolation weights
    def _tsf(self, mat, eps):
        s, t, dev = self.s, self.s.tsf, self.dev
        th, ph, ps = t["theta"], t["phi"], t["psi"]
        corr = 1 / math.sqrt(math.sin(th) ** 4 * (math.cos(ph) ** 4 + math.sin(ph) ** 4) + math.cos(th) ** 4)
        self.jn = int(math.sqrt(sum(n * n for n in self.R)) + 250)
        jdx = s.dx / corr
        self.je, self.jh, self.jb = np.zeros(self.jn + 4), np.zeros(self.jn + 4), np.zeros(8)
        self.jce, self.jch = s.dt / (EPS0 * jdx), s.dt / (MU0 * jdx)
        self.jl = (s.dt * C0 - jdx) / (s.dt * C0 + jdx)
        sp, cp, st, ct, sn, cs = math.sin(ps), math.cos(ps), math.sin(th), math.cos(th), math.sin(ph), math.cos(ph)
        ge = (cp * sn - sp * ct * cs, -cp * cs - sp * ct * sn, sp * st)
        gh = (sp * sn + cp * ct * cs, -sp * cs + cp * ct * sn, -cp * st)
        (lo, hi), skip, sd = t["box"], t.get("skip", [0] * 6), t.get("skipdepth", -1)
        oz = self.R[2] if th > math.pi / 2 else 0
        near = None
        if sd >= 0:      # cells within `skipdepth` of matter
            near = (eps / EPS0 - 1).abs() >= 0.001
            if s.mats:
                near = near | (mat > 0)
            for ax in range(3):
                acc = near.clone()
                for k in range(-sd, sd):
                    a, b = (slice(k, None), slice(0, -k)) if k > 0 else (slice(0, k), slice(-k, None)) if k < 0 else (slice(None),) * 2
                    acc[_at(ax, b)] |= near[_at(ax, a)]
                near = acc
        self.faces = []
        for f in range(6):
            ax, low = f // 2, f % 2 == 0
            p, q = [a for a in range(3) if a != ax]
            reg = [slice(lo[a], hi[a] + 1) for a in range(3)]
            pos = lo[ax] if low else hi[ax]
            reg[ax] = slice(pos, pos + 1)
            grid = torch.meshgrid(*[torch.arange(r.start, r.stop, dtype=torch.float64, device=dev) for r in reg], indexing="ij")
            on = torch.ones_like(grid[0]) * (0 if skip[f] else 1)
            if near is not None:
                on = on * (~near[tuple(reg)]).double()

            def taps(shift):
                g = list(grid)
                g[ax] = g[ax] - shift
                x = corr * (10.0 + st * cs * g[0] + st * sn * g[1] + ct * (g[2] - oz))
                i = x.floor()
                a = x - i
                w = [a + 1, a, 1 - a, 2 - a]
                w = [4 - 8 * v + 5 * v * v - v ** 3 if k in (0, 3) else 1 - 2 * v * v + v ** 3 for k, v in enumerate(w)]
                return i.long(), w

            # n x (value): signs of the two tangential components, zero on the last line across the component
            sg = 1.0 if low else -1.0
            keep = lambda a: (grid[a] < hi[a]).double() * on  # noqa: E731
            ce = s.dt / s.dx / eps[tuple(reg)]
            hc = s.dt / s.dx / MU0
            even = 1.0 if ax != 1 else -1.0
            hreg = list(reg)
            hreg[ax] = slice(pos - 1, pos) if low else reg[ax]
            self.faces.append(dict(
                e=tuple(reg), h=tuple(hreg), te=taps(1 if low else 0), th=taps(0),
                H=[(p, -sg * even * ge[q] * hc * keep(q)), (q, sg * even * ge[p] * hc * keep(p))],
                E=[(p, sg * even * gh[q] * ce * keep(p)), (q, -sg * even * gh[p] * ce * keep(q))]))

    def _line(self):
        e, h, b, r = self.je, self.jh, self.jb, self.jn
        e[1:r] += self.jce * (h[:r - 1] - h[1:r])
        e[0] = b[1] + self.jl * (e[1] - b[0])
        h[0] = b[3] + self.jl * (h[1] - b[2])
        e[r - 1] = b[5] + self.jl * (e[r - 2] - b[4])
        h[r - 1] = b[7] + self.jl * (h[r - 2] - b[6])
        b[:] = e[0], e[1], h[0], h[1], e[r - 1], e[r - 2], h[r - 1], h[r - 2]
        w = self.s.tsf["wave"]
        e[0] = w[self.n] if self.n < len(w) else 0.0
        h[:r - 1] += self.jch * (e[:r - 1] - e[1:r])
        self.le, self.lh = torch.from_numpy(e.copy()).to(self.dev), torch.from_numpy(h.copy()).to(self.dev)

    def _wave(self, line, taps):
        i, w = taps
        return sum(w[k] * line[i + k - 1] for k in range(4))

    def step(self):
        dx, E, H = self.s.dx, self.F[:3], self.F[3:]
        self._line()
        # H: hx += db (d_z ey - d_y ez) and cyclic, rows at the far rim of the other two axes untouched
        dif = {}
        N = []
        for a in range(3):
            p, q = (a + 1) % 3, (a + 2) % 3
            dqp, dpq = _fwd(E[p], q), _fwd(E[q], p)       # d_q E_p and d_p E_q
            dif[p, q], dif[q, p] = dqp, dpq
            new = H[a] + self.db * (dqp / self.kh[q] - dpq / self.kh[p])
            for ax in (p, q):
                new = torch.cat([new[_at(ax, slice(0, -1))], H[a][_at(ax, slice(-1, None))]], ax)
            N.append(new)
        for c in self.faces:
            ve = self._wave(self.le, c["th"])
            for a, w in c["H"]:
                N[a][c["h"]] += w * ve
        for f in range(6):
            ax = f // 2
            _, _, _, reg, b, c = self.prof[f]
            if min(self.psiH[f][0].shape) == 0:
                continue
            for k, (a, o) in enumerate(self._pairs(ax)):   # H_a corrected by d_ax E_o
                psi = b * self.psiH[f][k] + c * dif[o, ax][reg]
                self.psiH[f][k] = psi
                N[a][reg] += self._sign(a, ax) * (self.db[reg] * dx) * psi
        inner = [slice(1, n - 1) for n in self.R]
        for ax in range(3):
            reg = list(inner)
            reg[ax] = slice(self.R[ax] - 1, self.R[ax])
            for a in range(3):
                N[a][tuple(reg)] = 0
        H = self.F[3:] = N
        # E: curl with backward differences
        dif, N, drive = {}, [], []
        for a in range(3):
            p, q = (a + 1) % 3, (a + 2) % 3
            dpq, dqp = _diff(H[q], p), _diff(H[p], q)
            dif[q, p], dif[p, q] = dpq, dqp
            drive.append(dpq / self.ke[p] - dqp / self.ke[q])
        first = {}
        if self.own is not None:
            m = self.m
            for a in range(3):
                v = m.ade_c0 / dx * drive[a] + m.ade_c1 * (-m.ade_a0 * self.Pm[a] + (1 - m.ade_a1) * self.P[a])
                for k in range(self.npoles):
                    v = v + m.ade_c1 * (-m.ade_bp0[k] * self.pm[a][k] + (1 - m.ade_bp1[k]) * self.p[a][k])
                v = v + m.ade_c2 * self.ep[a] + m.ade_c3 * E[a]
                p, q = [x for x in range(3) if x != a]
                ok = torch.ones(self.R, dtype=torch.bool, device=self.dev)
                ok[_at(p, 0)] = False
                ok[_at(q, 0)] = False
                drive[a] = torch.where(self.own[a], torch.where(ok, v, E[a]), E[a] + self.cb[a] * drive[a])
            N = drive
            for f in range(6):   # CPML inside the dispersive branch: a first psi update
                ax, low = f // 2, f % 2 == 0
                reg, b, c = self.prof[f][:3]
                br = self.branch[reg]
                if low:
                    br = br.clone()
                    br[_at(ax, slice(0, 1))] = False
                for k, (a, o) in enumerate(self._pairs(ax)):
                    psi = torch.where(br, b * self.psiE[f][k] + c * dif[o, ax][reg], self.psiE[f][k])
                    self.psiE[f][k] = psi
                    if f != 0:      # scaled by zero on the first x face
                        N[a][reg] += torch.where(br & self.own[a][reg], -self._sign(a, ax) * dx * self.cba * psi, torch.zeros_like(psi))
            for a in range(3):
                e1 = N[a]
                o = self.own[a]
                new = m.ade_a0 * self.Pm[a] + m.ade_a1 * self.P[a] + m.ade_a2 * (self.ep[a] + 2 * E[a] + e1)
                self.Pm[a], self.P[a] = self.P[a], torch.where(o, new, self.P[a])
                for k in range(self.npoles):
                    new = m.ade_bp0[k] * self.pm[a][k] + m.ade_bp1[k] * self.p[a][k] + m.ade_bp2[k] * self.ep[a] + \
                        m.ade_bp3[k] * E[a] + m.ade_bp4[k] * e1
                    self.pm[a][k], self.p[a][k] = self.p[a][k], torch.where(o, new, self.p[a][k])
        else:
            N = [E[a] + self.cb[a] * drive[a] for a in range(3)]
        del drive
        for f in range(6):
            ax = f // 2
            reg, b, c = self.prof[f][:3]
            for k, (a, o) in enumerate(self._pairs(ax)):
                psi = b * self.psiE[f][k] + c * dif[o, ax][reg]
                self.psiE[f][k] = psi
                add = -self._sign(a, ax) * dx * self.cb[a][reg] * psi
                if self.own is not None:
                    gate = 2 if (f == 4 and a == 0) else a     # the first z face gates Ex by the z component
                    add = torch.where(self.own[gate][reg], torch.zeros_like(add), add)
                N[a][reg] += add
        for a in range(3):
            for ax in range(3):
                N[a][_at(ax, 0)] = 0
        for c in self.faces:
            vh = self._wave(self.lh, c["te"])
            for a, w in c["E"]:
                N[a][c["e"]] += w * vh
        if self.own is not None:
            self.ep = E
        self.F[:3] = N
        if self.s.nfff:
            self._sample()
        for q, (i, j, k) in enumerate(self.s.probes):
            self.probes[q, self.n] = [float(v.detach()[i, j, k]) for v in self.F]
        self.n += 1

    @staticmethod
    def _pairs(ax):
        """The two components a slab along `ax` corrects, each with the component whose d_ax drives it."""
        p, q = (ax + 1) % 3, (ax + 2) % 3
        return ((p, q), (q, p))

    @staticmethod
    def _sign(a, ax):
        """Sign of d_ax in the H curl of component a (E takes the opposite)."""
        return 1.0 if (ax - a) % 3 == 2 else -1.0

    # running DFTs of E and its normal derivative on the six faces of the box
    def _nfff(self):
        lo, hi = self.s.nfff["box"]
        w = torch.from_numpy(np.asarray(self.s.nfff["omega"], dtype=np.float64)).to(self.dev)
        self.om = w
        regs = []
        for f in range(6):
            ax = f // 2
            c = [slice(lo[a], hi[a]) for a in range(3)]
            pos = lo[ax] if f % 2 == 0 else hi[ax]
            three = []
            for o in (0, 1, -1):
                c[ax] = slice(pos + o, pos + o + 1)
                three.append(tuple(c))
            regs.append(three)
        self.surf = regs
        self.cells = torch.cat([torch.stack(torch.meshgrid(*[torch.arange(r.start, r.stop, dtype=torch.float64, device=self.dev)
                                                             for r in g[0]], indexing="ij"), -1).reshape(-1, 3) for g in regs])
        self.face = torch.cat([torch.full((len(range(*g[0][0].indices(1 << 30))) * len(range(*g[0][1].indices(1 << 30))) *
                                           len(range(*g[0][2].indices(1 << 30))),), f, device=self.dev) for f, g in enumerate(regs)])
        self.acc = torch.zeros((len(w), 2, 3, len(self.cells)), dtype=torch.complex128, device=self.dev)
        self.samples = []

    def _sample(self):
        v = [[torch.cat([self.F[a][g[k]].reshape(-1) for g in self.surf]) for a in range(3)] for k in range(3)]
        v = torch.stack([torch.stack(v[0]), (torch.stack(v[1]) - torch.stack(v[2])) / (2 * self.s.dx)])
        if self.s.nfff.get("series"):
            self.samples.append(v)
            return
        ph = torch.exp(-1j * self.om * (self.n * self.s.dt))
        self.acc = self.acc + ph[:, None, None, None] * v[None]

    def _geometry(self, point):
        """Weights of E (three taps), of dE/dn, and the retarded index of every surface cell for one far point."""
        dt, dx = self.s.dt, self.s.dx
        u = torch.tensor([float(v) for v in point], dtype=torch.float64, device=self.dev) - self.cells
        rc = (u * u).sum(1).sqrt()
        sg = (2 * (self.face % 2) - 1).double()
        cos = sg * u.gather(1, (self.face // 2).long()[:, None])[:, 0] / rc
        r = rc * dx
        a, b, c = 1 / (4 * math.pi * r), -cos / (4 * math.pi * r * r), -cos / (4 * math.pi * C0 * r) / (2 * dt)
        return sg * a * dx * dx, b * dx * dx, c * dx * dx, r / (C0 * dt)

    def spectrum(self, points=None):
        pts, ist = self.s.nfff["points"], self.s.nfff["istart"]
        dt = self.s.dt
        z1 = torch.exp(1j * self.om * dt)
        out = []
        for n in range(len(pts)) if points is None else points:
            a, b, c, t = self._geometry(pts[n])
            R = (1 + t).floor()
            row = []
            for f in range(len(self.om)):
                w = torch.polar(torch.ones_like(R), -self.om[f] * dt * (R - int(ist[n])))
                K = (b * z1[f] - c + c * z1[f] ** 2) * w
                L = a * z1[f] * w
                row.append((self.acc[f, 0] * K + self.acc[f, 1] * L).sum(-1))
            out.append(torch.stack(row))
        return torch.stack(out)

    def series(self):
        pts, ist = self.s.nfff["points"], self.s.nfff["istart"]
        nd = int(2000 + 2 * self.s.nsteps + math.sqrt(sum(n * n for n in self.R)) / (C0 * self.s.dt / self.s.dx))
        out = torch.zeros((len(pts), 3, nd), dtype=torch.float64, device=self.dev)
        for n in range(len(pts)):
            a, b, c, t = self._geometry(pts[n])
            for k, v in enumerate(self.samples):
                nn = ((k + 1) + t).floor().long() - int(ist[n])
                ok = (nn >= 3) & (nn < nd)
                i = nn[ok]
                for q in range(3):
                    for o, w in ((0, -c * v[0, q]), (1, a * v[1, q] + b * v[0, q]), (2, c * v[0, q])):
                        out[n, q].index_add_(0, i - o, w[ok])
        return out


def _results(x):
    """As _read."""
    E, H = (np.stack([v.cpu().numpy() for v in f]) for f in (x.F[:3], x.F[3:]))
    out = dict(E=E, H=H, probes=x.probes)
    if x.s.nfff and x.s.nfff.get("series"):
        out["series"] = x.series().cpu().numpy()
    elif x.s.nfff:
        out["spectrum"] = x.spectrum().cpu().numpy()
    return out


def exact(case, seed):
    scenes = _scenes(case, seed)
    if case["kind"] == "batch":
        outs = []
        with torch.no_grad():
            for q, s in enumerate(scenes):
                x = Exact(s, _noise((s.xres, s.yres, s.zres), seed + 7919 * (q + 1)))
                for _ in range(case["steps"]):
                    x.step()
                outs.append(_results(x))
        return outs
    s = scenes[0]
    if case["kind"] == "adjoint":
        return _exact_gradient(s, case, seed)
    with torch.no_grad():
        x = Exact(s, _noise((s.xres, s.yres, s.zres), seed + 7919))
        for _ in range(case.get("steps", 24)):
            x.step()
        if case["kind"] == "farfield":
            return dict(spectrum=x.spectrum().cpu().numpy())
        return _results(x)


def _exact_gradient(s, case, seed):
    """J and dJ/d eps_r by reverse-mode differentiation of the FP64 steps, segment by segment from checkpoints."""
    from torch.utils.checkpoint import checkpoint
    obj = plan.cone_objective(s)
    eps = torch.from_numpy(np.asarray(s.design["eps"], dtype=np.float64)).cuda().requires_grad_(True)
    x = Exact(s, _noise((s.xres, s.yres, s.zres), seed + 7919), eps)

    def segment(steps, acc, *state):
        x.F = list(state[:6])
        for f in range(6):
            x.psiE[f], x.psiH[f] = list(state[6 + 4 * f:8 + 4 * f]), list(state[8 + 4 * f:10 + 4 * f])
        x.acc, x.n, x.je, x.jh, x.jb = acc, steps[0], steps[1].copy(), steps[2].copy(), steps[3].copy()
        for _ in range(steps[4]):
            x.step()
        return (x.acc, *x.F, *[t for f in range(6) for t in x.psiE[f] + x.psiH[f]])

    state = (x.acc, *x.F, *[t for f in range(6) for t in x.psiE[f] + x.psiH[f]])
    done = 0
    while done < case["steps"]:
        n = min(8, case["steps"] - done)
        state = checkpoint(segment, (done, x.je.copy(), x.jh.copy(), x.jb.copy(), n), *state, use_reentrant=False)
        done += n
    x.acc = state[0]
    F = x.spectrum(obj["points"])[:, obj["freq"]]
    w = torch.from_numpy(np.asarray(obj["weights"])).cuda()
    J = (w[:, None] * (F.real ** 2 + F.imag ** 2)).sum()
    J.backward()
    return dict(J=float(J.detach()), grad=eps.grad.cpu().numpy())
