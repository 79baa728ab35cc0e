"""The workloads whose speed is tracked: mid-run states of the library's cases, advanced by some time steps.

One pass is what a program that keeps its fields in device memory does between two outputs: hand the
fields to a context (``ecg_upload_prim_device``), advance ``steps`` time steps with one ``ecg_step`` call,
and take the fields back (``ecg_download_prim_device``).  Batched cases go through ``ecg_batch_*``, whose
fields are host arrays (pinned here, as a program that cares about the copies keeps them).

The states are those of a run in progress, not of its first step: interfaces spread over a few cells, and
waves in pressure, velocity and density everywhere, so no part of the mesh is at rest.  Materials, lengths,
pressures, CFL numbers, limiters and relaxations are those of ``ecogen_b200.cases``.
"""
import math

import numpy as np
import torch

from ecogen_b200 import api, cases

# ---------------------------------------------------------------------------------------- the cases

# kind -> (model, phases, dimensions, limiter); the workload families of ecogen_b200.cases
KINDS = {
    "tube": ("kapila", 2, 1, None),          # water / air shock tube, first order
    "tube2": ("kapila", 2, 1, "vanleer"),    # the same, MUSCL
    "batch": ("kapila", 2, 1, "vanleer"),    # many independent tubes in one launch
    "bubble": ("kapila", 2, 2, "vanleer"),   # water shock over air bubbles
    "sharp": ("kapila", 2, 2, "minmod"),     # the same with THINC interfaces: run-time limiters, generic kernels
    "cavity": ("kapila", 3, 3, "minmod"),    # gas inclusions in a liquid under pressure
    "expansion": ("kapila", 2, 2, "vanleer"),  # liquid / vapour with p-T-mu relaxation
    "ptueq": ("ptueq", 2, 2, "vanleer"),     # one temperature and pressure, two phases
    "euler": ("euler", 1, 2, "vanleer"),     # single-phase blast
}


def listed():
    return [
        # the reference's CPU-sized tube: a handful of blocks, latency is all
        dict(name="tube1d_1000_first_order", kind="tube", nx=1000, ny=1, nz=1, steps=100),
        # a finer tube in MUSCL, ragged against every tile
        dict(name="tube1d_4093_muscl", kind="tube2", nx=4093, ny=1, nz=1, steps=40),
        # a parameter study: few tubes, and the full batch of the benchmark
        dict(name="batch_64_tubes", kind="batch", nx=64, ny=1, nz=1, steps=40),
        dict(name="batch_4096_tubes", kind="batch", nx=4096, ny=1, nz=1, steps=40),
        # 2D shock-bubble: a coarse odd mesh while a case is being set up, and the benchmark's
        dict(name="bubble2d_191x103", kind="bubble", nx=191, ny=103, nz=1, steps=20),
        dict(name="bubble2d_2048x2048", kind="bubble", nx=2048, ny=2048, nz=1, steps=6),
        # sharpened interfaces (volume-fraction limiter THINC): the kernels without compiled-in limiters
        dict(name="sharp2d_1000x601", kind="sharp", nx=1000, ny=601, nz=1, steps=6),
        # 3D three-phase cavity collapse: a ragged box and the benchmark's
        dict(name="cavity3d_67x53x61", kind="cavity", nx=67, ny=53, nz=61, steps=10),
        dict(name="cavity3d_256", kind="cavity", nx=256, ny=256, nz=256, steps=4),
        # phase change
        dict(name="expansion2d_1024x1024", kind="expansion", nx=1024, ny=1024, nz=1, steps=6),
        # the two other models
        dict(name="ptueq2d_2048x2048", kind="ptueq", nx=2048, ny=2048, nz=1, steps=6),
        dict(name="euler2d_2048x2048", kind="euler", nx=2048, ny=2048, nz=1, steps=8),
    ]


def draw(rng):
    """A case of the same families, its sizes spread over the ranges the listed ones mark out."""
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n | 1 if rng.random() < 0.5 else n

    kind = rng.choice(sorted(KINDS))
    dim = KINDS[kind][2]
    if kind == "batch":
        return dict(kind=kind, nx=size(8, 4000), ny=1, nz=1, steps=rng.randint(10, 40))
    if dim == 1:
        return dict(kind=kind, nx=size(200, 20000), ny=1, nz=1, steps=rng.randint(20, 100))
    if kind == "cavity":
        return dict(kind=kind, nx=size(24, 240), ny=size(24, 240), nz=size(24, 240), steps=rng.randint(2, 4))
    if kind in ("ptueq", "euler") and rng.random() < 0.3:  # these models in 3D
        return dict(kind=kind, nx=size(24, 160), ny=size(24, 160), nz=size(24, 160), steps=rng.randint(2, 6))
    return dict(kind=kind, nx=size(64, 2000), ny=size(64, 2000), nz=1, steps=rng.randint(2, 6))


def dim_of(case):
    return 1 + (case["ny"] > 1) + (case["nz"] > 1)


def batch_sizes(ncases):
    """Cells of each tube of a batch: log-uniform in [200, 8000], as cases.batch_shock_tubes draws them."""
    r = np.random.default_rng(ncases)
    return np.exp(r.uniform(math.log(200), math.log(8000), ncases)).round().astype(np.int64)


def cells_of(case):
    return int(batch_sizes(case["nx"]).sum()) if case["kind"] == "batch" else case["nx"] * case["ny"] * case["nz"]


def spec_of(case):
    """The ecogen_b200.cases description of the case (materials, limiter, CFL, relaxation, lengths)."""
    kind, cells = case["kind"], (case["nx"], case["ny"], case["nz"])
    if kind in ("tube", "tube2"):
        return cases.shock_tube_1d(ncells=cells[0], iterations=1, order=KINDS[kind][3])
    if kind == "expansion":
        s = cases.expansion_tube_2d(n=64, iterations=1)
    elif kind == "cavity":
        s = cases.cavity_collapse_3d(n=64, iterations=1, ninclusions=1)
    elif kind == "ptueq":
        s = cases.ptueq_bubble_2d(n=64, iterations=1, nz=cells[2])
    elif kind == "euler":
        s = cases.euler_blast_2d(n=64, iterations=1, nz=cells[2])
    else:
        s = cases.shock_bubble_2d(n=64, iterations=1)
    if kind == "sharp":
        s.second_order, s.interface_limiter, s.vf_limiter, s.interface_vf_limiter = "minmod", "superbee", "vanleer", "THINC"
    s.cells = cells
    # square or cubic cells of the family's size along x
    h = s.lengths[0] / cells[0]
    s.lengths = tuple(h * n if n > 1 else s.lengths[i] for i, n in enumerate(cells))
    return s


def batch_specs(case):
    return [cases.shock_tube_1d(ncells=int(n), iterations=1, order="vanleer") for n in batch_sizes(case["nx"])]


def work(case):
    """Bytes: one read and one write of the state that defines a step, per cell and step (alpha_k, rho_k, p,
    u, E; what the other models store), and the fields in and out once.  Operations: additions,
    multiplications, comparisons, divisions, roots and powers of the scheme, each counted as one, per face
    (two reconstructed sides, closure, HLLC) and per cell (update, closure, one Newton evaluation)."""
    model, np_, _, lim = KINDS[case["kind"]]
    dim, n, passes = dim_of(case), cells_of(case), 2 if lim else 1
    state = {"kapila": 2 * np_ + 2 + dim, "euler": 3 + dim, "ptueq": 5 + dim}[model]
    face = {"kapila": 63 * np_ + 60 + 4 * dim, "euler": 90 + 4 * dim, "ptueq": 120 + 4 * dim}[model]
    limited = {"kapila": 3 * np_ + dim, "euler": 2 + dim, "ptueq": 4 + dim}[model] * (16 if lim else 0)
    cell = {"kapila": 75 * np_ + 20 * dim, "euler": 12 + 12 * dim, "ptueq": 70 + 12 * dim}[model]
    if case["kind"] == "expansion":
        cell += 500  # pure-phase tests and saturation Newton
    flops = n * passes * (dim * (face + limited + 6 * np_) + cell)
    return {"bytes": 16.0 * state * n * (case["steps"] + 1), "flops": float(flops) * case["steps"]}


# ------------------------------------------------------------------------------------ initial states


def _modes(gen, coords, count=4, kmax=6):
    """A smooth field in [-1, 1]: a few sine waves with drawn wave vectors and phases."""
    out = torch.zeros_like(sum(coords))
    for _ in range(count):
        arg = 2 * math.pi * torch.rand((), generator=gen, dtype=torch.float64).item()
        for x in coords:
            arg = arg + 2 * math.pi * int(torch.randint(1, kmax + 1, (), generator=gen)) * x
        out = out + torch.sin(arg)
    return out / count


def _eos_e(q, rho, p):
    return (p + q.gamma * q.pinf) / (q.gamma - 1.) / rho + q.eref


def _total_energy(eos, a, r, p, u):
    rho = sum(ai * ri for ai, ri in zip(a, r))
    return sum(ai * ri / rho * _eos_e(q, ri, p) for q, ai, ri in zip(eos, a, r)) + 0.5 * sum(v * v for v in u)


def _cell_centres(case, dev):
    """Cell centres along the used axes, in units of the x length, on the (z, y, x) grid."""
    n = (case["nx"], case["ny"], case["nz"])
    out = []
    for ax in range(dim_of(case)):
        x = (torch.arange(n[ax], device=dev, dtype=torch.float64) + 0.5) / n[0]
        shape = [1, 1, 1]
        shape[2 - ax] = n[ax]
        out.append(x.reshape(shape).expand(n[2], n[1], n[0]))
    return out


def _step_up(d, width):
    """0 -> 1 over a few `width` around d = 0."""
    return 0.5 * (1. + torch.tanh(d / width))


def initial_fields(case, seed, dev):
    """Fields in the ABI's order, as torch tensors of the grid's shape."""
    gen = torch.Generator().manual_seed(int(seed))
    rnd = lambda lo, hi: lo + (hi - lo) * torch.rand((), generator=gen, dtype=torch.float64).item()  # noqa: E731
    spec, kind, dim = spec_of(case), case["kind"], dim_of(case)
    X = _cell_centres(case, dev)
    h = 1.0 / case["nx"]
    ext = [case["nx"] * h, case["ny"] * h, case["nz"] * h]
    mode = lambda: _modes(gen, X)  # noqa: E731
    zero = torch.zeros_like(X[0] + 0.)
    floor = 1e-6

    def blobs(count, rlo, rhi):
        m = zero.clone()
        for _ in range(count):
            r = rnd(rlo, rhi)
            d2 = sum((x - rnd(0.1, 0.9) * ext[i]) ** 2 for i, x in enumerate(X))
            m = torch.maximum(m, _step_up(r - torch.sqrt(d2), 1.5 * h))
        return m

    if kind in ("tube", "tube2"):
        water = _step_up(rnd(0.3, 0.7) - X[0], 1.5 * h)
        a0 = floor + (1 - 2 * floor) * water
        a, r = [a0, 1. - a0], [1000. * (1 + 0.01 * mode()), 50. * (1 + 0.05 * mode())]
        p = 1e5 + math.exp(rnd(math.log(1e7), math.log(1e9))) * water * (1 + 0.05 * mode())
        u = [20. * mode()]
    elif kind in ("bubble", "sharp"):
        gas = blobs(3, 0.04, 0.12)
        a1 = floor + (1 - 2 * floor) * gas
        shocked = _step_up(rnd(0.1, 0.3) - X[0], 1.5 * h) * (1 - gas)
        rho1, u1 = cases.sg_hugoniot_post_shock(spec.eos[0], 1000.0, 1.0e5, 1.0e9)
        a = [1. - a1, a1]
        r = [(1000. + (rho1 - 1000.) * shocked) * (1 + 0.002 * mode()), 1.2 * (1 + 0.1 * mode())]
        p = (1e5 + (1e9 - 1e5) * shocked) * (1 + 0.1 * mode())
        u = [u1 * shocked + 5. * mode(), 5. * mode()]
    elif kind == "cavity":
        b, c = blobs(8, 0.03, 0.1), blobs(8, 0.03, 0.1)
        c = c * (1 - b)
        a1, a2 = floor + (1 - 3 * floor) * b, floor + (1 - 3 * floor) * c
        a = [1. - a1 - a2, a1, a2]
        r = [1000. * (1 + 0.002 * mode()), 1.2 * (1 + 0.1 * mode()), 0.16 * (1 + 0.1 * mode())]
        p = (1e5 + (5e7 - 1e5) * (1 - b - c)) * (1 + 0.1 * mode())
        u = [5. * mode() for _ in range(3)]
    elif kind == "expansion":
        av = 1e-2 * (1 + 0.3 * mode())
        a, p, T = [1. - av, av], 1e5 * (1 + 0.02 * mode()), 355. + zero
        r = [(p + q.pinf) / ((q.gamma - 1.) * q.cv * T) for q in spec.eos]
        mid, strip = 0.5 * ext[0], _step_up(0.25 * ext[1] - (X[1] - 0.5 * ext[1]).abs(), 2 * h)
        u = [rnd(200., 500.) * strip * (2 * _step_up(X[0] - mid, 2 * h) - 1) + 2. * mode(), 2. * mode()]
    elif kind == "ptueq":
        gas = blobs(3, 0.05, 0.2)
        a0 = floor + (1 - 2 * floor) * gas
        hp = _step_up(rnd(0.1, 0.3) - X[0], 1.5 * h) * (1 - gas)
        a = [a0, 1. - a0]
        p, T = (1e5 + (1e8 - 1e5) * hp) * (1 + 0.1 * mode()), (300. + 20. * hp) * (1 + 0.02 * mode())
        r = [(p + q.pinf) / ((q.gamma - 1.) * q.cv * T) for q in spec.eos]
        u = [50. * hp + 5. * mode()] + [5. * mode() for _ in range(dim - 1)]
    else:  # euler
        hot = blobs(2, 0.1, 0.2)
        a, r = [1. + zero], [(1. + 4. * hot) * (1 + 0.1 * mode())]
        p = (1e5 + 9e5 * hot) * (1 + 0.1 * mode())
        u = [40. * mode() for _ in range(dim)]
    E = _total_energy(spec.eos, a, r, p, u)
    u = u + [zero] * (3 - len(u))
    if kind == "euler":
        out = [r[0], p, *u, E]
    elif kind == "ptueq":
        out = [*a, *r, p, *u, E, T]
    else:
        out = [*a, *r, p, *u, E]
    return [f.contiguous().clone() for f in out]


def batch_fields(case, seed, dev):
    """The tubes' fields one after another, (alpha_0, alpha_1, rho_0, rho_1, p, u, E)."""
    sizes = batch_sizes(case["nx"])
    r = np.random.default_rng(int(seed))
    rep = torch.from_numpy(sizes).to(dev)
    per = lambda v: torch.repeat_interleave(torch.from_numpy(np.asarray(v, dtype=np.float64)).to(dev), rep)  # noqa: E731
    nc, total = len(sizes), int(sizes.sum())
    off = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    n = per(sizes)
    x = (torch.arange(total, device=dev, dtype=torch.float64) - per(off) + 0.5) / n

    def mode():
        return torch.sin(2 * math.pi * (per(r.integers(1, 7, nc)) * x + per(r.uniform(0, 1, nc))))

    water = _step_up(per(r.uniform(0.3, 0.7, nc)) - x, 1.5 / n)
    a0 = 1e-6 + (1 - 2e-6) * water
    a, rho = [a0, 1. - a0], [1000. * (1 + 0.01 * mode()), 50. * (1 + 0.05 * mode())]
    p = 1e5 + per(np.exp(r.uniform(math.log(1e6), math.log(1e9), nc))) * water * (1 + 0.05 * mode())
    u = 20. * mode()
    E = _total_energy([cases.WATER_SG, cases.AIR_IG], a, rho, p, [u])
    return [*a, *rho, p, u, E]


def _sound_speed(model, eos, a, r, p):
    rho = sum(ai * ri for ai, ri in zip(a, r))
    return torch.sqrt(sum(ai * ri / rho * q.gamma * (p + q.pinf) / ri for q, ai, ri in zip(eos, a, r)))


def _split(model, np_, f):
    """(a, r, p, u) of fields in the ABI's order."""
    if model == "euler":
        return [torch.ones_like(f[0])], [f[0]], f[1], f[2:5]
    return f[:np_], f[np_:2 * np_], f[2 * np_], f[2 * np_ + 1:2 * np_ + 4]


def first_dt(case, f):
    """The time step the run was taking: cfl lCFL / max(|u| + c)."""
    spec = spec_of(case)
    model, np_ = KINDS[case["kind"]][:2]
    a, r, p, u = _split(model, np_, f)
    c = _sound_speed(model, spec.eos, a, r, p)
    s = max((v.abs() + c).max().item() for v in u)
    h = spec.lengths[0] / spec.cells[0]
    return spec.cfl * h * (0.6 if dim_of(case) > 1 else 1.0) / s


# ------------------------------------------------------------------------------------------ one pass


def _ptrs(fields):
    p = (api.C.POINTER(api.C.c_double) * len(fields))()
    for i, f in enumerate(fields):
        p[i] = api.C.cast(f.data_ptr(), api.C.POINTER(api.C.c_double))
    return p


def prepare(case, seed):
    dev = torch.device("cuda")
    if case["kind"] == "batch":
        f = batch_fields(case, seed, dev)
        zero = torch.zeros_like(f[0])
        f = [*f[:6], zero, zero, f[6]]  # the ABI's two other velocity components
        host = [x.cpu().pin_memory() for x in f]
        out = [torch.empty_like(x).pin_memory() for x in host]
        specs = batch_specs(case)
        recs = (api.Case * len(specs))(*[api.case_from_spec(s) for s in specs])
        h = api.C.c_void_p()
        api.check(api.lib().ecg_batch_create(recs, len(specs), api.C.byref(h)), "ecg_batch_create")
        api.check(api.lib().ecg_batch_set_shape(h, 256, 256), "ecg_batch_set_shape")
        dt = np.array([s.cfl / s.cells[0] / 2000. for s in specs])
        return _Batch(h, case, host, out, dt)
    f = initial_fields(case, seed, dev)
    ctx = api.Context(api.case_from_spec(spec_of(case)))
    out = [torch.empty_like(x) for x in f]
    dt = first_dt(case, f)
    torch.cuda.synchronize()
    return _Single(ctx, case, f, out, dt)


class _Single:
    def __init__(self, ctx, case, fields, out, dt):
        self.ctx, self.case, self.fields, self.out, self.dt0 = ctx, case, fields, out, dt
        self.inp, self.outp = _ptrs(fields), _ptrs(out)

    def run(self):
        c = self.ctx
        api.check(api.lib().ecg_upload_prim_device(c.h, self.inp, c.n), "ecg_upload_prim_device")
        c.dt.value, c.t.value = self.dt0, 0.0
        c.step(self.case["steps"])
        api.check(api.lib().ecg_download_prim_device(c.h, self.outp, c.n), "ecg_download_prim_device")
        return {"fields": self.out, "dt": c.dt.value, "t": c.t.value}


class _Batch:
    def __init__(self, h, case, host, out, dt):
        self.h, self.case, self.host, self.out, self.dt0 = h, case, host, out, dt
        self.total = int(api.lib().ecg_batch_total_cells(h))
        self.inp, self.outp = _ptrs(host), _ptrs(out)

    def run(self):
        dp = api.C.POINTER(api.C.c_double)
        dt, t, st = self.dt0.copy(), np.zeros(len(self.dt0)), api.StepStats()
        L = api.lib()
        api.check(L.ecg_batch_upload_prim(self.h, self.inp, self.total), "ecg_batch_upload_prim")
        api.check(L.ecg_batch_step(self.h, self.case["steps"], dt.ctypes.data_as(dp), t.ctypes.data_as(dp),
                                   api.C.byref(st)), "ecg_batch_step")
        api.check(L.ecg_batch_download_prim(self.h, self.outp, self.total), "ecg_batch_download_prim")
        return {"fields": self.out, "dt": dt, "t": t}

    def __del__(self):
        api.lib().ecg_batch_destroy(self.h)


def run(state):
    return state.run()


# --------------------------------------------------------------------- the same in plain torch, 64 bits


def _limit(kind, s1, s2):
    prod, zero = s1 * s2, torch.zeros_like(s1)
    kind = (kind or "none").lower()
    if kind in ("minmod", "thinc"):
        return torch.where(prod > 1e-9, torch.sign(s1) * torch.minimum(s1.abs(), s2.abs()), zero)
    if kind == "vanleer":
        s = s1 + s2
        return torch.where((s.abs() > 1e-6) & (prod > 1e-6), 2. * prod / s, zero)
    if kind == "superbee":
        m = torch.maximum(torch.minimum(2 * s1.abs(), s2.abs()), torch.minimum(s1.abs(), 2 * s2.abs()))
        return torch.where(prod > 1e-6, torch.sign(s1) * m, zero)
    raise ValueError(kind)


class _Exact:
    """The scheme on whole grids: HLLC, first order or MUSCL-Hancock, the three models' closures."""

    def __init__(self, case):
        spec = spec_of(case) if case["kind"] != "batch" else cases.shock_tube_1d(order="vanleer", iterations=1)
        self.eos, self.cfl = spec.eos, spec.cfl
        self.model, self.np, _, _ = KINDS[case["kind"]]
        self.dim = dim_of(case)
        self.null = bool(spec.alpha_null)
        self.ptmu = spec.ptmu is not None
        self.second = spec.second_order is not None
        g = spec.second_order
        il = spec.interface_limiter or g
        self.lim = (g, il, spec.vf_limiter or g, spec.interface_vf_limiter or il)
        dev = torch.device("cuda")
        if case["kind"] == "batch":
            sizes = batch_sizes(case["nx"])
            self.owner = torch.repeat_interleave(torch.arange(len(sizes), device=dev),
                                                 torch.from_numpy(sizes).to(dev))
            self.h = (1.0 / torch.from_numpy(sizes.astype(np.float64)).to(dev))
            off = np.concatenate([[0], np.cumsum(sizes)[:-1]])
            self.first, self.last = torch.from_numpy(off).to(dev), torch.from_numpy(off + sizes - 1).to(dev)
            self.link = self.owner[1:] == self.owner[:-1]
            self.hc = self.h[self.owner].reshape(1, 1, -1)
            self.ncases = len(sizes)
        else:
            self.owner = self.link = None
            self.hc = spec.lengths[0] / spec.cells[0]
            self.h = torch.tensor([self.hc], device=dev, dtype=torch.float64)
            self.ncases = 1
        self.lcfl = self.h * (0.6 if self.dim > 1 else 1.0)

    # -- closures
    def fix_p(self, k, p):
        q = self.eos[k]
        return torch.clamp(p, min=1e-8 if q.kind == "IG" else -(1. - 1e-15) * q.pinf + 1e-15)

    def fix_ar(self, a, r):
        if self.null:
            return a.clamp(0., 1.), r.clamp(min=1e-15)
        a = torch.where(a < 1e-15, 1e-14, torch.where(a > 1. - 1e-15, 1. - 1e-14, a))
        return a, torch.where(r < 1e-15, 1e-14, r)

    def rho_pT(self, k, p, T):
        q = self.eos[k]
        return (p + q.pinf) / ((q.gamma - 1.) * q.cv * T)

    def side(self, a, r, pk, u):
        rho = sum(x * y for x, y in zip(a, r))
        Y = [x * y / rho for x, y in zip(a, r)]
        c2 = [q.gamma * (p + q.pinf) / y for q, p, y in zip(self.eos, pk, r)]
        e = [_eos_e(q, y, p) for q, y, p in zip(self.eos, r, pk)]
        return dict(a=a, r=r, pk=pk, u=u, rho=rho, p=sum(x * p for x, p in zip(a, pk)),
                    c=torch.sqrt(sum(y * c for y, c in zip(Y, c2))), e=sum(y * x for y, x in zip(Y, e)), ek=e)

    # -- fluxes through the faces between sides L and R (normal axis ax): masses, volume fractions,
    #    phase energies, momentum, total energy, contact speed, interface speed, fastest wave
    def hllc(self, L, R, ax):
        uL, uR = L["u"][ax], R["u"][ax]
        sL, sR = torch.minimum(uL - L["c"], uR - R["c"]), torch.maximum(uR + R["c"], uL + L["c"])
        mL, mR = L["rho"] * (sL - uL), R["rho"] * (sR - uR)
        sM = (R["p"] - L["p"] + mL * uL - mR * uR) / (mL - mR)
        sM = torch.where(sM.abs() < 1e-8, 0., sM)
        left = (sL >= 0.) | ((sR > 0.) & (sM >= 0.))
        plain = (sL >= 0.) | (sR <= 0.)
        S = lambda key: torch.where(left, L[key], R[key])  # noqa: E731
        SL = lambda key: [torch.where(left, x, y) for x, y in zip(L[key], R[key])]  # noqa: E731
        a, r, pk, ek, u = SL("a"), SL("r"), SL("pk"), SL("ek"), SL("u")
        rho, p, e = S("rho"), S("p"), S("e")
        sK, mK, un = torch.where(left, sL, sR), torch.where(left, mL, mR), u[ax]
        Et = e + 0.5 * sum(x * x for x in u)
        f = torch.where(plain, 1., (sK - un) / (sK - sM))
        v = torch.where(plain, un, sM)
        P = torch.where(plain, p, mK * (sM - un) + p)
        E = torch.where(plain, Et, Et + (sM - un) * (sM + p / mK))
        rs = rho * f
        rk = [x * f for x in r]
        mass = [x * y * v for x, y in zip(a, rk)]
        mom = [rs * v * x for x in u]
        mom[ax] = rs * v * v + P
        out = dict(mass=mass, mom=mom, E=(rs * E + P) * v, speed=torch.maximum(sL.abs(), sR.abs()))
        if self.model == "kapila":
            ps = [(x + q.pinf) * f ** q.gamma - q.pinf for q, x in zip(self.eos, pk)]
            es = [torch.where(plain, x, _eos_e(q, y, z)) for q, x, y, z in zip(self.eos, ek, rk, ps)]
            out.update(al=[x * sM for x in a], en=[x * y for x, y in zip(mass, es)], sM=sM, us=v)
        return out

    def outward(self, S, ax, sign):
        """Flux out of a cell through a non-reflecting side."""
        un = sign * S["u"][ax]
        sM = torch.where(un.abs() < 1e-8, 0., un)
        mass = [x * y * sM for x, y in zip(S["a"], S["r"])]
        mom = [S["rho"] * sM * x for x in S["u"]]
        mom[ax] = sign * (S["rho"] * sM * sM + S["p"])
        Et = S["e"] + 0.5 * sum(x * x for x in S["u"])
        out = dict(mass=mass, mom=mom, E=(S["rho"] * Et + S["p"]) * sM, speed=un.abs() + S["c"])
        if self.model == "kapila":
            out.update(al=[x * sM for x in S["a"]], en=[x * y for x, y in zip(mass, S["ek"])], sM=sM, us=sM)
        return out

    def prim(self, q):
        """Primitive fields of a stored state that are reconstructed, by group."""
        if self.model == "ptueq":
            return q["a"] + [q["p"], q["T"]] + q["u"]
        if self.model == "euler":
            return [q["r"][0], q["p"]] + q["u"]
        return q["a"] + q["r"] + [self.fix_p(k, q["p"]) for k in range(self.np)] + q["u"]

    def side_of(self, w):
        """A side from reconstructed primitives."""
        n = self.np
        if self.model == "ptueq":
            a, p, T, u = w[:2], w[2], w[3], w[4:]
            return self.side(a, [self.rho_pT(k, p, T) for k in range(2)], [p, p], u)
        if self.model == "euler":
            return self.side([torch.ones_like(w[0])], [w[0]], [w[1]], w[2:])
        return self.side(w[:n], w[n:2 * n], w[2 * n:3 * n], w[3 * n:])

    def clamp_side(self, w):
        n = self.np
        if self.model == "euler":
            return [w[0].clamp(min=1e-10), self.fix_p(0, w[1])] + w[2:]
        if self.model == "ptueq":
            return w
        ar = [self.fix_ar(w[k], w[n + k]) for k in range(n)]
        return [x for x, _ in ar] + [y for _, y in ar] + [self.fix_p(k, w[2 * n + k]) for k in range(n)] + w[3 * n:]

    def residual(self, q, sn, speed):
        """-div F (with the non-conservative terms) of state q; speed: fastest wave per case so far."""
        w = self.prim(q)
        acc = {}
        a0 = sn["a"][0] if self.model != "euler" else None
        an = sn["a"]
        pn = [self.fix_p(k, sn["p"]) for k in range(self.np)] if self.model == "kapila" else None

        def put(key, i, lo, ln, dim, val):
            t = acc.setdefault((key, i), torch.zeros_like(q["p"]))
            t.narrow(dim, lo, ln).add_(val)

        for ax in range(self.dim):
            dim = 2 - ax
            m = q["p"].shape[dim]
            lo = lambda x: x.narrow(dim, 0, m - 1)  # noqa: E731
            hi = lambda x: x.narrow(dim, 1, m - 1)  # noqa: E731
            if self.second:
                hf = lo(self.hc) if self.link is not None else self.hc
                s = [(hi(x) - lo(x)) / hf for x in w]
                if self.link is not None:
                    s = [x * self.link for x in s]
                edge = torch.zeros_like(s[0].narrow(dim, 0, 1))
                prev = lambda x: torch.cat([edge, x.narrow(dim, 0, m - 2)], dim)  # noqa: E731
                nxt = lambda x: torch.cat([x.narrow(dim, 1, m - 2), edge], dim)  # noqa: E731
                sides = []
                for sgn, cell, other, opp in ((1., lo, hi, prev), (-1., hi, lo, nxt)):
                    iface = None
                    mixed = self.lim[1] != self.lim[0] or self.lim[3] != self.lim[2]
                    if self.model != "euler" and mixed:
                        # the neighbour beyond the cell, at time n (0 where there is none)
                        far = prev(lo(a0)) if sgn > 0 else nxt(hi(a0))
                        near, across = cell(q["a"][0]), other(q["a"][0])
                        iface = (near >= 1e-4) & (near <= 1 - 1e-4) & ((across - near) * (near - far) >= 1e-8)
                    x = []
                    for i, wi in enumerate(w):
                        vf = self.model == "kapila" and i < self.np
                        g, f = (self.lim[2], self.lim[3]) if vf else (self.lim[0], self.lim[1])
                        sl = _limit(g, s[i], opp(s[i]))
                        if iface is not None and f != g:
                            sl = torch.where(iface, _limit(f, s[i], opp(s[i])), sl)
                        x.append(cell(wi) + sgn * sl * (0.5 * hf))
                    x = self.clamp_side(x)
                    if iface is not None and "THINC" in self.lim:
                        x = self.thinc(x, iface, sgn, near, across, far)
                    sides.append(self.side_of(x))
                    del x
                L, R = sides
            else:
                L, R = self.side_of([lo(x) for x in w]), self.side_of([hi(x) for x in w])
            F = self.hllc(L, R, ax)
            del L, R
            sp = F.pop("speed")
            if self.link is None:
                speed = torch.maximum(speed, sp.max().reshape(1))
            else:
                speed = speed.scatter_reduce(0, self.owner[:-1], (sp * self.link).reshape(-1), "amax")
            cell = self.side_of(w)
            # the two sides of the domain (of every case): outward fluxes
            out = []
            for sgn in (-1., 1.):
                idx = (torch.tensor([0 if sgn < 0 else m - 1], device=q["p"].device) if self.link is None
                       else (self.first if sgn < 0 else self.last))
                pick = lambda x: x.index_select(dim, idx)  # noqa: E731
                S = {k: ([pick(y) for y in v] if isinstance(v, list) else pick(v)) for k, v in cell.items()}
                B = self.outward(S, ax, sgn)
                sp = B.pop("speed")
                if self.link is None:
                    speed = torch.maximum(speed, sp.max().reshape(1))
                else:
                    speed = torch.maximum(speed, sp.reshape(-1))
                out.append((idx, B))
            del cell
            noncons = {"al": [-x for x in an], "en": [x * y for x, y in zip(an, pn)]} if pn else {}
            for key, val in F.items():
                if key in ("sM", "us"):
                    continue
                for i, f in enumerate(val if isinstance(val, list) else [val]):
                    if self.link is not None:
                        f = f * self.link
                    fl, fr = f, f
                    if key in noncons:
                        v = F["sM" if key == "al" else "us"]
                        v = v if self.link is None else v * self.link
                        fr = f + hi(noncons[key][i]) * v  # seen by the right cell
                        fl = f + lo(noncons[key][i]) * v  # seen by the left cell
                    put(key, i, 1, m - 1, dim, fr / (hi(self.hc) if self.link is not None else self.hc))
                    put(key, i, 0, m - 1, dim, -fl / (lo(self.hc) if self.link is not None else self.hc))
            for idx, B in out:
                for key, val in B.items():
                    if key in ("sM", "us"):
                        continue
                    for i, f in enumerate(val if isinstance(val, list) else [val]):
                        if key in noncons:
                            f = f + noncons[key][i].index_select(dim, idx) * B["sM" if key == "al" else "us"]
                        hb = self.hc.index_select(dim, idx) if self.link is not None else self.hc
                        acc[(key, i)].index_add_(dim, idx, -f / hb)
        return acc, speed

    def thinc(self, w, iface, sgn, near, across, far):
        up, down = (across, far) if sgn > 0 else (far, across)  # the neighbours on the far and near x side
        sg = torch.where(up - down > 0., 1., -1.).to(torch.float64)
        lo = torch.minimum(up, down)
        rng = torch.maximum(up, down) - lo
        beta, th = 1.6, math.tanh(1.6)
        C = (near - lo + 1e-20) / (rng + 1e-20)
        A = (torch.exp(sg * beta * (2. * C - 1.)) / math.cosh(beta) - 1.) / th
        v = (1. + sg * (th + A) / (1. + A * th)) if sgn > 0 else (1. + sg * A)
        na = (lo + 0.5 * rng * v).clamp(1e-4, 1. - 1e-4)
        return [torch.where(iface, na, w[0]), torch.where(iface, 1. - na, w[1])] + w[2:]

    # -- update of a cell from its accumulated fluxes
    def update(self, sn, acc, scale):
        n = self.np
        a, u = sn["a"], sn["u"]
        if self.model == "ptueq":
            r = [self.rho_pT(k, sn["p"], sn["T"]) for k in range(2)]
        else:
            r = sn["r"]
        rho = sum(x * y for x, y in zip(a, r))
        m = [x * y + scale * acc[("mass", k)] for k, (x, y) in enumerate(zip(a, r))]
        tot = sum(m)
        un = [(rho * x + scale * acc[("mom", d)]) / tot for d, x in enumerate(u)]
        un = [torch.where(x.abs() < 1e-8, 0., x) for x in un]
        E = (rho * sn["E"] + scale * acc[("E", 0)]) / tot
        ie = E - 0.5 * sum(x * x for x in un)
        if self.model == "euler":
            q = self.eos[0]
            return dict(a=[torch.ones_like(tot)], r=[tot], p=(q.gamma - 1.) * tot * (ie - q.eref) - q.gamma * q.pinf,
                        u=un, E=E)
        if self.model == "ptueq":
            Y = [x / tot for x in m]
            Z = [y * (q.gamma - 1.) * q.cv for y, q in zip(Y, self.eos)]
            cv = sum(y * q.cv for y, q in zip(Y, self.eos))
            ref = sum(y * q.eref for y, q in zip(Y, self.eos))
            A = [z / cv * (tot * (ie - ref) - q.pinf) for z, q in zip(Z, self.eos)]
            pi = [q.pinf for q in self.eos]
            p = 0.5 * (A[0] + A[1] - (pi[0] + pi[1])) + torch.sqrt(
                0.25 * (A[1] - A[0] - (pi[1] - pi[0])) ** 2 + A[0] * A[1])
            T = 1. / (tot * sum(z / (p + x) for z, x in zip(Z, pi)))
            return dict(a=[x / self.rho_pT(k, p, T) for k, x in enumerate(m)], p=p, T=T, u=un, E=E)
        ae = [x * y * _eos_e(q, y, self.fix_p(k, sn["p"])) + scale * acc[("en", k)]
              for k, (q, x, y) in enumerate(zip(self.eos, a, r))]
        al = [x + scale * acc[("al", k)] for k, x in enumerate(a)]
        al = [x.clamp(0., 1.) if self.null else x.clamp(1e-15, 1. - 1e-15) for x in al]
        s = sum(al)
        a, r, p = [x / s for x in al], [], []
        for k, q in enumerate(self.eos):
            rk = m[k] / (a[k].clamp(min=1e-15) if self.null else a[k])
            ek = ae[k] / (m[k].clamp(min=1e-15) if self.null else m[k])
            pk = (q.gamma - 1.) * rk * (ek - q.eref) - q.gamma * q.pinf
            a[k], rk = self.fix_ar(a[k], rk)
            r.append(rk)
            p.append(self.fix_p(k, pk))
        rho = sum(x * y for x, y in zip(a, r))
        e = sum(x * y / rho * _eos_e(q, y, z) for q, x, y, z in zip(self.eos, a, r, p))
        a, r, p = self.relax_p(a, r, p)
        if self.ptmu:
            a, r, p = self.relax_ptmu(a, r, p, rho, e)
            rho = sum(x * y for x, y in zip(a, r))
        num, den = rho * ie, 0.
        for q, x, y in zip(self.eos, a, r):
            num = num - x * (q.gamma * q.pinf / (q.gamma - 1.) + y * q.eref)
            den = den + x / (q.gamma - 1.)
        ar = [self.fix_ar(x, y) for x, y in zip(a, r)]
        return dict(a=[x for x, _ in ar], r=[y for _, y in ar], p=num / den, u=un, E=E)

    def relax_p(self, a, r, p):
        """Pressure equilibrium: sum_k alpha_k rho_k / rho_k*(p*) = 1 along the phases' relaxation paths."""
        on = torch.ones_like(a[0], dtype=torch.bool)
        if self.null:
            for x in a:
                on &= x <= 1. - 1e-5
        ps = sum(x * y for x, y in zip(a, p))
        act = on.clone()
        aS, rS = [x.clone() for x in a], [x.clone() for x in r]
        for _ in range(100):
            for k in range(self.np):
                ps = torch.where(act, self.fix_p(k, ps), ps)
            f, df = -1., 0.
            for k, q in enumerate(self.eos):
                num = q.gamma * (ps + q.pinf)
                den = num + p[k] - ps
                rk = r[k] * num / den
                dr = r[k] * q.gamma * (p[k] + q.pinf) / (den * den)
                rS[k] = torch.where(act, rk, rS[k])
                aS[k] = torch.where(act, a[k] * r[k] / rk, aS[k])
                f = f + a[k] * r[k] / rk
                df = df - a[k] * r[k] * dr / (rk * rk)
            act = act & (f.abs() > 1e-10)
            if not bool(act.any()):
                break
            ps = torch.where(act, ps - f / df, ps)
        return aS, rS, [torch.where(on, ps, x) for x in p]

    def t_sat(self, p):
        Lq, Vq = self.eos
        den = (Vq.gamma - 1.) * Vq.cv
        A = (Lq.gamma * Lq.cv - Vq.gamma * Vq.cv + Vq.sref - Lq.sref) / den
        B, C = (Lq.eref - Vq.eref) / den, (Vq.gamma * Vq.cv - Lq.gamma * Lq.cv) / den
        D = (Lq.gamma - 1.) * Lq.cv / den
        const = A - torch.log(p + Vq.pinf) + D * torch.log(p + Lq.pinf)
        T = torch.full_like(p, 0.1 * B / C)
        for _ in range(50):
            f, df = const + B / T + C * torch.log(T), C / T - B / (T * T)
            act = f.abs() > 1e-10
            if not bool(act.any()):
                break
            T = torch.where(act, T - f / df, T)
        return T, (1. / (p + Vq.pinf) - D / (p + Lq.pinf)) / df

    def relax_ptmu(self, a, r, p, rho, e):
        """Saturation state of two phases at (rho, e), or a single phase where that is stable."""
        Lq, Vq = self.eos
        pc = (Lq.pinf * (Vq.gamma - 1.) * Vq.cv - Vq.pinf * (Lq.gamma - 1.) * Lq.cv) / (
            (Lq.gamma - 1.) * Lq.cv - (Vq.gamma - 1.) * Vq.cv)
        ps = sum(x * y for x, y in zip(a, p))
        todo = ps <= pc
        one = torch.ones_like(ps)
        alone = []
        for q, hot in ((Vq, True), (Lq, False)):
            pp = (q.gamma - 1.) * rho * (e - q.eref) - q.gamma * q.pinf
            T = (pp + q.pinf) / (q.gamma - 1.) / rho / q.cv
            Ts, _ = self.t_sat(torch.where(pp > 0., pp, 1e5 * one))
            alone.append((todo & (pp > 0.) & ((T >= Ts) if hot else (T <= Ts)), pp))
            todo = todo & ~alone[-1][0]
        act, both = todo.clone(), todo.clone()
        sol = [x.clone() for x in (a[0], r[0], r[1], ps)]
        ps = torch.where(act, ps, 1e5 * one)
        for _ in range(50):
            for k in range(2):
                ps = self.fix_p(k, ps)
            Ts, dT = self.t_sat(ps)
            v = []
            for q in (Lq, Vq):
                g = (q.gamma - 1.) * q.cv
                rs = (ps + q.pinf) / (g * Ts)
                dr = (g * Ts - (ps + q.pinf) * g * dT) / (g * Ts) ** 2
                v.append((rs, dr, (ps + q.gamma * q.pinf) / (q.gamma - 1.) + rs * q.eref, 1. / (q.gamma - 1.) + dr * q.eref))
            (rl, dl, el, del_), (rv, dv, ev, dev_) = v
            al = (rho - rv) / (rl - rv)
            dal = (-dv * (rl - rv) - (rho - rv) * (dl - dv)) / (rl - rv) ** 2
            f = (rho * e - al * el - (1. - al) * ev) / (rho * e)
            df = -(dal * el + al * del_ - dal * ev + (1. - al) * dev_) / (rho * e)
            sol = [torch.where(act, x, y) for x, y in zip((al, rl, rv, ps), sol)]
            act = act & (f.abs() > 1e-10)
            if not bool(act.any()):
                break
            ps = torch.where(act, ps - f / df, ps)
        al, rl, rv, ps = sol
        a = [torch.where(both, al, a[0]), torch.where(both, 1. - al, a[1])]
        r = [torch.where(both, rl, r[0]), torch.where(both, rv, r[1])]
        p = [torch.where(both, ps, x) for x in p]
        for (m, pp), k in zip(alone, (1, 0)):
            a[k], a[1 - k] = torch.where(m, 1., a[k]), torch.where(m, 0., a[1 - k])
            r[k], p[k] = torch.where(m, rho, r[k]), torch.where(m, pp, p[k])
        return a, r, p

    def steps(self, s, dt, count):
        t = torch.zeros_like(dt)
        for _ in range(count):
            scale = dt[self.owner].reshape(1, 1, -1) if self.owner is not None else dt.item()
            speed = torch.zeros(self.ncases, device=dt.device, dtype=torch.float64)
            q = s
            if self.second:
                acc, speed = self.residual(s, s, speed)
                q = self.update(s, acc, 0.5 * scale)
            acc, speed = self.residual(q, s, speed)
            s = self.update(s, acc, scale)
            t, dt = t + dt, self.cfl * self.lcfl / speed
        return s, dt, t


def exact(case, seed):
    dev = torch.device("cuda")
    x = _Exact(case)
    if case["kind"] == "batch":
        f = [v.reshape(1, 1, -1) for v in batch_fields(case, seed, dev)]
        dt = x.cfl * x.h / 2000.
        s = dict(a=f[:2], r=f[2:4], p=f[4], u=[f[5]], E=f[6])
    else:
        f = initial_fields(case, seed, dev)
        dt = torch.tensor([first_dt(case, f)], device=dev, dtype=torch.float64)
        a, r, p, u = _split(x.model, x.np, f)
        s = dict(a=a, r=r, p=p, u=u[:x.dim], E=f[8] if x.model == "ptueq" else f[-1])
        if x.model == "ptueq":
            s["T"] = f[9]
    s, dt, t = x.steps(s, dt, case["steps"])
    zero = torch.zeros_like(s["p"])
    u = s["u"] + [zero] * (3 - x.dim)
    if x.model == "euler":
        out = [s["r"][0], s["p"], *u, s["E"]]
    elif x.model == "ptueq":
        out = [*s["a"], *[x.rho_pT(k, s["p"], s["T"]) for k in range(2)], s["p"], *u, s["E"], s["T"]]
    else:  # the mixture pressure sum_k alpha_k p_k
        out = [*s["a"], *s["r"], sum(y * x.fix_p(k, s["p"]) for k, y in enumerate(s["a"])), *u, s["E"]]
    if case["kind"] == "batch":
        return {"fields": [v.reshape(-1).cpu() for v in out], "dt": dt.cpu().numpy(), "t": t.cpu().numpy()}
    return {"fields": out, "dt": dt.item(), "t": t.item()}
