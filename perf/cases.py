"""Performance cases of nuosc_b200: whole solves, batches of uneven solves and
single right-hand sides, over the sizes, precisions and options a user runs.

Three kinds of pass, each through the public entry points:

  solve  one handle: seeded initial data (fillInitValue), `steps` RK4 steps
         with the analysis record read every `every` of them, then the state
         read back into page-locked host memory (nuosc_get_state) -- what one
         point of a parameter scan costs a program that keeps its handle.
  batch  the same for `n` uneven solves stepped together (Batch.step_stream
         with streamed records and the device-side stop test every 10 steps,
         as the server runs them).
  rhs    one right-hand side on the caller's own device buffers
         (nuosc_calrhs_noalloc), the call a program with its own time stepper
         makes.

Cell spacing 0.125 (a power of two, so every box is an exact number of cells),
CFL 0.4, KO 0.1.  Solves in FP32 that run more than a few tens of steps use
the 4th-difference KO: the 6th-difference form amplifies grid-scale modes
(as the reference does), single-precision rounding among them.  `pmo` 0.1 is
the class's default vacuum term, 0 the production recipe's.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import nuosc_b200 as nb
from nuosc_b200._lib import check

DX, CFL, KO = 0.125, 0.4, 0.1
FIELDS = nb.FIELDS[:8]
# the diagnostics that are well-conditioned numbers; max||P|-1|, its averages
# and ELNe are residues of cancellation at these amplitudes (last bits only)
DIAGS = ("phy_time", "surv", "survb", "aM0", "Lex")
HALT_EVERY = 10


# ------------------------------------------------------------------ the cases
def listed():
    solve = dict(kind="solve", precision="f64", ko_order=6, pmo=0.0, every=10)
    return [
        # the smallest solve of the mixed workload: latency and launches
        dict(solve, name="solve_32x32x42_f64", nx=32, nz=32, nn=2, steps=100),
        # the reference's own configuration: 100 steps, diagnostics every 10
        dict(solve, name="solve_64x64x162_f64", nx=64, nz=64, nn=4, steps=100),
        # the parity grid of the production run with its velocity sphere
        dict(solve, name="solve_128x128x642_f64", nx=128, nz=128, nn=8, steps=60, every=20),
        # the production path at memory-bound size (several GB per register)
        dict(solve, name="solve_512x256x642_f64", nx=512, nz=256, nn=8, steps=40, every=20),
        # the mixed-precision run, 4th-difference KO (long FP32 solves)
        dict(solve, name="solve_256x256x642_f32", nx=256, nz=256, nn=8, precision="f32", ko_order=4, steps=100,
             every=50),
        # FP32 on the default KO, mid size, vacuum term on (class default)
        dict(solve, name="solve_192x128x162_f32", nx=192, nz=128, nn=4, precision="f32", pmo=0.1, steps=40, every=20),
        # ragged grids: a box that is not a multiple of any tile
        dict(solve, name="solve_100x90x162_f64", nx=100, nz=90, nn=4, pmo=0.1, steps=100),
        dict(solve, name="solve_75x150x642_f32", nx=75, nz=150, nn=8, precision="f32", ko_order=4, steps=80, every=20),
        # uneven solves served together
        dict(name="batch_16_f64", kind="batch", precision="f64", ko_order=6, n=16, shapes=4, steps=30, every=10),
        dict(name="batch_16_f32", kind="batch", precision="f32", ko_order=4, n=16, shapes=4, steps=60, every=20),
        # one right-hand side for a caller's own time stepper
        dict(name="rhs_128x128x642_f64", kind="rhs", precision="f64", ko_order=6, pmo=0.0, nx=128, nz=128, nn=8),
        dict(name="rhs_250x130x162_f32", kind="rhs", precision="f32", ko_order=4, pmo=0.1, nx=250, nz=130, nn=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Half of the sizes are powers of two (the mixed workload's), half any number."""
    if rng.random() < 0.5:
        return 2 ** rng.randint(int(math.log2(lo)), int(math.log2(hi)))
    return _log_int(rng, lo, hi)


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["batch", "rhs"])
    precision = rng.choice(["f64", "f32"])
    if kind == "batch":
        n = rng.randint(3, 12)
        return dict(kind=kind, precision=precision, ko_order=6 if precision == "f64" else rng.choice([4, 6]), n=n,
                    shapes=rng.randrange(1 << 20), steps=20, every=rng.choice([5, 10, 20]))
    if kind == "rhs":
        while True:
            nx, nz, nn = _size(rng, 16, 512), _size(rng, 16, 512), rng.choice([1, 2, 3, 4, 6, 8])
            if nx * nz <= 65536 and nx * nz * (10 * nn * nn + 2) <= 3e7:
                break
        return dict(kind=kind, precision=precision, ko_order=rng.choice([4, 6]), pmo=rng.choice([0.0, 0.1]), nx=nx,
                    nz=nz, nn=nn)
    while True:
        nx, nz, nn = _size(rng, 24, 512), _size(rng, 24, 512), rng.choice([1, 2, 3, 4, 4, 8, 8])
        points = nx * nz * (10 * nn * nn + 2)
        if points <= 2e7:
            break
    steps = max(20, min(100, int(1.2e9 / points)))
    if precision == "f32":  # FP32 on the 6th-difference KO: few steps
        ko_order = rng.choice([4, 6])
        steps = min(steps, 40) if ko_order == 6 else steps
    else:
        ko_order = rng.choice([6, 6, 4])
    every = rng.choice([10, 20])
    return dict(kind=kind, precision=precision, ko_order=ko_order, pmo=rng.choice([0.0, 0.1]), nx=nx, nz=nz, nn=nn,
                steps=steps // every * every, every=every)


# ------------------------------------------------------------------ inputs
def _physics(case, seed):
    """Parameters of one solve: the production recipe, the cells' draw from the seed."""
    return dict(nx=case["nx"], nz=case["nz"], nn=case["nn"], mu=1.0, pmo=case["pmo"], alpha=0.9, eps0=1e-6, lnue=0.6,
                lnueb=0.5, seed=seed + 1)


def _members(case, seed):
    """The members of a batch: shapes from the case, physics from the seed
    (the mixed workload: nx, nz of {32, 64, 128, 256}, nv of {42, 162, 642})."""
    shapes, phys = random.Random(case["shapes"]), random.Random(seed)
    out = []
    for k in range(case["n"]):
        out.append(dict(nx=shapes.choice((32, 64, 128, 256)), nz=shapes.choice((32, 64, 128, 256)),
                        nn=shapes.choice((2, 4, 8)), mu=phys.uniform(0.5, 2.0), pmo=0.0, alpha=phys.uniform(0.7, 1.3),
                        eps0=10 ** phys.uniform(-7, -3), lnue=phys.uniform(0.4, 0.8), lnueb=phys.uniform(0.3, 0.7),
                        seed=phys.randrange(1, 1 << 62)))
    return out


def _solver(p, case):
    ghost = 3 if case["ko_order"] == 6 else 2
    lx, lz = p["nx"] * DX / 2, p["nz"] * DX / 2
    s = nb.NuOsc(1, 1, p["nn"], 0, ghost, ghost, -lx, lx, -lz, lz, DX, DX, CFL, KO,
                 precision=nb.FP64 if case["precision"] == "f64" else nb.FP32)
    assert (s.grid.nx, s.grid.nz) == (p["nx"], p["nz"])
    s.set_mu(p["mu"])
    s.set_pmo(p["pmo"])
    return s


class _Host:
    """Where a solve's state is read back to: 8 page-locked double arrays
    (the C ABI's element type), and for FP32 solves their float copies."""

    def __init__(self, s, f32):
        shape = (8, s.grid.nx, s.grid.nz, s.grid.nv)
        self.wide = torch.empty(shape, dtype=torch.float64, pin_memory=True)
        self.ptr = [C.cast(self.wide[f].data_ptr(), C.POINTER(C.c_double)) for f in range(8)]
        self.out = torch.empty(shape, dtype=torch.float32) if f32 else self.wide

    def read(self, s):
        for f in range(8):
            check(nb.lib().nuosc_get_state(s.handle, nb.REG_STAT, f, self.ptr[f], nb.LAYOUT_COMPACT))
        if self.out is not self.wide:
            self.out.copy_(self.wide)
        return self.out


class _RhsDesc(C.Structure):
    """nuosc_rhs_desc of include/nuosc_b200.h."""
    _fields_ = [("nx", C.c_int), ("nz", C.c_int), ("nv", C.c_int), ("nv_stride", C.c_int),
                ("precision", C.c_int), ("ko_order", C.c_int),
                ("dx", C.c_double), ("dz", C.c_double), ("ko", C.c_double), ("mu", C.c_double),
                ("pmo", C.c_double),
                ("vx", C.c_void_p), ("vy", C.c_void_p), ("vz", C.c_void_p), ("vw", C.c_void_p)]


def _rhs_state(case, seed, quad, nvs, dtype):
    """A state on its way: polarisation vectors a little off the flavour axis
    in every cell and direction, spectra as in the production recipe."""
    nv = len(quad[0])
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    vz, vw = (torch.tensor(a, device=dev) for a in (quad[2], quad[3]))
    st = torch.zeros((8, case["nx"], case["nz"], nvs), dtype=torch.float64, device=dev)
    for h, (amp, width) in enumerate(((1.0, 0.6), (0.9, 0.5))):
        g = torch.exp(-(vz - 1.0) ** 2 / (2 * width * width))
        g *= amp / (g * vw).sum()
        p = 1e-3 * torch.randn((2, case["nx"], case["nz"], nv), dtype=torch.float64, device=dev, generator=gen)
        p3 = torch.sqrt(1.0 - p[0] ** 2 - p[1] ** 2)
        st[4 * h + 0, ..., :nv] = 0.5 * g * (1.0 + p3)
        st[4 * h + 1, ..., :nv] = 0.5 * g * (1.0 - p3)
        st[4 * h + 2, ..., :nv] = 0.5 * g * p[0]
        st[4 * h + 3, ..., :nv] = 0.5 * g * p[1]
    return st.to(dtype)


def _pad(n, case):
    align = 2 if case["precision"] == "f64" else 4  # rows of whole 16-byte units
    return (n + align - 1) // align * align


def prepare(case, seed):
    f32 = case["precision"] == "f32"
    if case["kind"] == "solve":
        p = _physics(case, seed)
        s = _solver(p, case)
        return dict(case=case, p=p, s=s, host=_Host(s, f32))
    if case["kind"] == "batch":
        ps = _members(case, seed)
        ss = [_solver(p, case) for p in ps]
        b = nb.Batch(ss)
        b.set_halt(HALT_EVERY)
        return dict(case=case, ps=ps, ss=ss, b=b, hosts=[_Host(s, f32) for s in ss])
    quad = icosahedron(case["nn"])
    nv = len(quad[0])
    nvs = _pad(nv, case)
    dev = torch.device("cuda")
    dtype = torch.float32 if f32 else torch.float64
    d_quad = []
    for a in quad:
        t = torch.zeros(nvs, dtype=torch.float64, device=dev)
        t[:nv] = torch.tensor(a)
        d_quad.append(t)
    desc = _RhsDesc(nx=case["nx"], nz=case["nz"], nv=nv, nv_stride=nvs, precision=nb.FP32 if f32 else nb.FP64,
                    ko_order=case["ko_order"], dx=DX, dz=DX, ko=KO, mu=1.0, pmo=case["pmo"],
                    vx=d_quad[0].data_ptr(), vy=d_quad[1].data_ptr(), vz=d_quad[2].data_ptr(), vw=d_quad[3].data_ptr())
    fn = nb.lib().nuosc_calrhs_noalloc
    fn.argtypes = [C.POINTER(_RhsDesc), C.c_void_p, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    src = _rhs_state(case, seed, quad, nvs, dtype)
    return dict(case=case, fn=fn, desc=desc, quad=d_quad, src=src, dst=torch.empty_like(src))


# ------------------------------------------------------------------ one pass
def _fill(s, p):
    s.fillInitValue(1, p["alpha"], p["eps0"], 1.0, p["lnue"], p["lnueb"], seed=p["seed"])


def _solve_out(state, diags, case):
    dtype = np.float32 if case["precision"] == "f32" else np.float64
    out = {name: state[f] for f, name in enumerate(FIELDS)}
    out["diag"] = np.array([[d[k] for k in DIAGS] for d in diags], dtype=dtype)
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "solve":
        s = state["s"]
        _fill(s, state["p"])
        diags = []
        for _ in range(case["steps"] // case["every"]):
            s.step_rk4(case["every"])
            diags.append(s.analysis())
        return _solve_out(state["host"].read(s), diags, case)
    if case["kind"] == "batch":
        for s, p in zip(state["ss"], state["ps"]):
            _fill(s, p)
        b = state["b"]
        records = b.step_stream(case["steps"], case["every"])
        b.synchronize()
        diags = [[] for _ in state["ss"]]
        for member, _step, d in b.collect(records):
            diags[member].append(d)
        dtype = np.float32 if case["precision"] == "f32" else np.float64
        return {"state": [h.read(s) for h, s in zip(state["hosts"], state["ss"])],
                "diag": [np.array([[d[k] for k in DIAGS] for d in m], dtype=dtype) for m in diags]}
    rc = state["fn"](C.byref(state["desc"]), state["src"].data_ptr(), state["dst"].data_ptr(),
                     torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(nb.lib().nuosc_last_error())
    return state["dst"]


# ------------------------------------------------------------------ the work
def _step_work(p, case):
    """One RK4 step: the state in and out; per point and stage 4 fields x 2
    flavours of a 13- (KO6) or 9-point stencil, commutator, update, moments."""
    points = p["nx"] * p["nz"] * (10 * p["nn"] ** 2 + 2)
    e = 8 if case["precision"] == "f64" else 4
    per_stage = 8 * (2 * 13 if case["ko_order"] == 6 else 2 * 9) + 8 * 2 + 70
    return points * 16 * e, points * 4 * per_stage, points * 8 * e


def work(case):
    if case["kind"] == "rhs":
        b, f, _ = _step_work(case, case)
        return {"bytes": b, "flops": f / 4}
    ps = [_physics(case, 0)] if case["kind"] == "solve" else _members(case, 0)
    n_bytes = flops = 0
    for p in ps:
        b, f, state = _step_work(p, case)
        # initial data written, every step, every analysis, the read-back
        n_bytes += state + case["steps"] * b + (case["steps"] // case["every"]) * state + state
        flops += case["steps"] * f
    return {"bytes": n_bytes, "flops": flops}


# ------------------------------------------------------------------ 64-bit reference
def icosahedron(nn):
    """Velocity sphere: the subdivided icosahedron, each of 10 rhombic patches
    refined bilinearly into nn x nn cells and projected, weights from the
    flat triangles' circumcentre areas.  Returns vx, vy, vz, vw."""
    lam = 1.10714871779409
    base = np.zeros((12, 3))
    for i in range(1, 6):
        for k, ang in ((i, 2 * i * math.pi / 5), (i + 5, (2 * i + 1) * math.pi / 5)):
            base[k] = math.cos(ang) * math.sin(lam), math.sin(ang) * math.sin(lam), math.cos(lam) * (1 if k < 6 else -1)
    base[0], base[11] = (0, 0, 1), (0, 0, -1)
    patch = [(1, 0, 2, 6), (6, 2, 7, 11), (2, 0, 3, 7), (7, 3, 8, 11), (3, 0, 4, 8),
             (8, 4, 9, 11), (4, 0, 5, 9), (9, 5, 10, 11), (5, 0, 1, 10), (10, 1, 6, 11)]
    lattice = np.zeros((10, nn + 1, nn + 1, 3))
    for p, corners in enumerate(patch):
        a, b, c, d = (base[k] for k in corners)
        for i in range(nn + 1):
            for j in range(nn + 1):
                q = i * (j * c + (nn - j) * d) + (nn - i) * (j * b + (nn - j) * a)
                lattice[p, i, j] = q / np.linalg.norm(q)
    pts = np.concatenate([base[:1], lattice[:, :nn, :nn].reshape(-1, 3), base[11:]])
    # a patch's edges belong to its neighbours: every lattice point's owner is the nearest point
    owner = np.argmin(((lattice.reshape(-1, 1, 3) - pts) ** 2).sum(-1), axis=1).reshape(10, nn + 1, nn + 1)
    w = np.zeros(len(pts))
    area = lambda u, v: 0.25 * np.linalg.norm(np.cross(u, v))  # noqa: E731
    for p in range(10):
        for i in range(nn):
            for j in range(nn):
                for mid in (owner[p, i, j + 1], owner[p, i + 1, j]):
                    ids = owner[p, i, j], mid, owner[p, i + 1, j + 1]
                    a, b, c = pts[ids[0]], pts[ids[1]], pts[ids[2]]
                    n = np.cross(b - a, c - a)
                    o = a + 0.5 / n.dot(n) * np.cross(n, (c - a).dot(c - a) * (b - a) - (b - a).dot(b - a) * (c - a))
                    ab, bc, ca = area(o - a, b - a), area(o - b, c - b), area(o - c, a - c)
                    w[ids[0]] += ab + ca
                    w[ids[1]] += bc + ab
                    w[ids[2]] += ca + bc
    return pts[:, 0].copy(), pts[:, 1].copy(), pts[:, 2].copy(), w


def _uniform(seed, nx, nz):
    """U[0, 1) per (x, z) cell: splitmix64 of (seed, i, j)."""
    def mix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))
    i, j = np.meshgrid(np.arange(nx, dtype=np.uint64), np.arange(nz, dtype=np.uint64), indexing="ij")
    with np.errstate(over="ignore"):
        bits = mix(mix(np.full((nx, nz), seed, dtype=np.uint64)) ^ ((i << np.uint64(32)) | j))
    return (bits >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


class _Exact:
    """calRHS, the RK4 step and the diagnostics in plain 64-bit torch."""

    def __init__(self, quad, ko_order, mu, pmo):
        self.dev = torch.device("cuda")
        self.vx, self.vy, self.vz, self.vw = (torch.tensor(a, dtype=torch.float64, device=self.dev) for a in quad)
        self.r = 3 if ko_order == 6 else 2
        self.mu, self.pmo = mu, pmo
        eps = -KO / DX / (64 if ko_order == 6 else 16)
        ko = {3: 1.0, 2: -6.0, 1: 15.0} if ko_order == 6 else {2: 1.0, 1: -4.0}
        adv = {-2: 1.0, -1: -8.0, 1: 8.0, 2: -1.0}
        self.taps = []  # (axis, offset, weight per velocity)
        for axis, v in ((0, self.vx), (1, self.vz)):
            for o in range(-self.r, self.r + 1):
                if o:
                    self.taps.append((axis, o, eps * ko[abs(o)] - v / (12 * DX) * adv.get(o, 0.0)))
        self.centre = 2 * eps * (-20.0 if ko_order == 6 else 6.0)
        self.w4 = torch.stack([self.vw, self.vw * self.vx, self.vw * self.vy, self.vw * self.vz], 1)
        self.n4 = torch.stack([torch.ones_like(self.vx), -self.vx, -self.vy, -self.vz], 0)

    def rhs(self, s):
        r, nx, nz = self.r, s.shape[1], s.shape[2]
        a, b, e = (d @ self.w4 @ self.n4 for d in (s[6] - s[2], s[7] + s[3], s[4] - s[5] - s[0] + s[1]))
        th = 37 * math.pi / 180
        ct, st = math.cos(2 * th), math.sin(2 * th)
        out = torch.empty_like(s)
        for h in (0, 4):
            ee, mm, er, ei = s[h], s[h + 1], s[h + 2], s[h + 3]
            iee = 2 * self.mu * (ei * a + er * b) - 2 * self.pmo * st * ei
            out[h], out[h + 1] = iee, -iee
            out[h + 2] = -self.mu * ((ee - mm) * b + e * ei) - 2 * self.pmo * ct * ei
            out[h + 3] = self.mu * ((mm - ee) * a + e * er) + self.pmo * (2 * ct * er + st * (ee - mm))
        for f in range(8):
            x = torch.cat([s[f, -r:], s[f], s[f, :r]], 0)
            z = torch.cat([s[f, :, -r:], s[f], s[f, :, :r]], 1)
            out[f].add_(s[f], alpha=self.centre)
            for axis, o, w in self.taps:
                out[f].addcmul_(x[r + o:r + o + nx] if axis == 0 else z[:, r + o:r + o + nz], w)
        return out

    def step(self, u, dt):
        k = self.rhs(u)
        acc = u + dt / 6 * k
        k = self.rhs(u + dt / 2 * k)
        acc.add_(k, alpha=dt / 3)
        k = self.rhs(u + dt / 2 * k)
        acc.add_(k, alpha=dt / 3)
        k = self.rhs(u + dt * k)
        return acc.add_(k, alpha=dt / 6)

    def initial(self, p):
        t = torch.tensor(p["eps0"] * (2.0 * _uniform(p["seed"], p["nx"], p["nz"]) - 1.0), device=self.dev)[..., None]
        p3 = torch.sqrt(1.0 - t * t)
        s = torch.zeros((8, p["nx"], p["nz"], len(self.vx)), dtype=torch.float64, device=self.dev)
        self.g = []
        for h, (amp, width) in enumerate(((1.0, p["lnue"]), (p["alpha"], p["lnueb"]))):
            g = torch.exp(-(self.vz - 1.0) ** 2 / (2.0 * width * width))
            g = amp * g / (g * self.vw).sum()
            self.g.append(g)
            s[4 * h], s[4 * h + 1], s[4 * h + 2] = 0.5 * g * (1.0 + p3), 0.5 * g * (1.0 - p3), 0.5 * g * t
        return s

    def diag(self, s, time):
        cells = s.shape[1] * s.shape[2]
        m = [float((s[f].sum((0, 1)) * self.vw).sum()) for f in range(8)]
        g, gb = (float((x * self.vw).sum()) * cells for x in self.g)
        lz = 0.5 * (m[0] - m[1] - m[4] + m[5])
        return [time, m[0] / g, m[4] / gb, math.sqrt((m[2] - m[6]) ** 2 + (m[3] + m[7]) ** 2 + lz * lz) / cells,
                lz / cells]


def _exact_solve(p, case):
    ref = _Exact(icosahedron(p["nn"]), case["ko_order"], p["mu"], p["pmo"])
    s = ref.initial(p)
    dt, diags = DX * CFL, []
    for k in range(1, case["steps"] + 1):
        s = ref.step(s, dt)
        if k % case["every"] == 0:
            diags.append(ref.diag(s, k * dt))
    return s, np.array(diags)


def exact(case, seed):
    if case["kind"] == "rhs":
        quad = icosahedron(case["nn"])
        nv = len(quad[0])
        nvs = _pad(nv, case)
        dtype = torch.float32 if case["precision"] == "f32" else torch.float64
        s = _rhs_state(case, seed, quad, nvs, dtype)[..., :nv].double()
        out = torch.zeros(s.shape[:3] + (nvs,), dtype=torch.float64, device=s.device)
        out[..., :nv] = _Exact(quad, case["ko_order"], 1.0, case["pmo"]).rhs(s)
        return out
    ps = [_physics(case, seed)] if case["kind"] == "solve" else _members(case, seed)
    if sum(p["nx"] * p["nz"] * (10 * p["nn"] ** 2 + 2) for p in ps) * case["steps"] > 5e9:
        return None  # over about 20 seconds
    got = [_exact_solve(p, case) for p in ps]
    if case["kind"] == "solve":
        state, diag = got[0]
        return dict({name: state[f] for f, name in enumerate(FIELDS)}, diag=diag)
    return {"state": [g[0].cpu() for g in got], "diag": [g[1] for g in got]}
