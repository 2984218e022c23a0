"""The calls this library is used for, as cases that can be timed and compared.

A pass is what a solver's time loop does between two outputs: one time step
(every Runge-Kutta stage with its pressure solve) through the public entry
points, then the fields the program reads back.  The cases cover both
execution forms and the contracted FP64 build, single grids to the 4096-grid
tiling, cubic and ragged grids, walls with an LES model, a grid hierarchy with
the ghost-cell immersed boundary, scalars, and the adjoint.

exact() restates the periodic cases (uniform spacing, one level) in torch in
64 bits: fluxes, the low-storage Runge-Kutta update, and the SIP solver with
its lagged halos at the same iteration counts.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "mglet-base_gb300"))

from mglet_gb300 import abi, cases, channel, gpu  # noqa: E402

# Taylor-Green at the Reynolds number of the library's benchmark
NU = 1.0 / 1600
NOUTER, NINNER = 9, 5
PRANDTL, GRAVITY, BETA = 0.71, -9.81, 3e-3
FORMS = {"plain": abi.FORM_PLAIN, "plain_fma": abi.FORM_PLAIN_FMA, "mixed": abi.FORM_MIXED}
STAGES = {"williamson": 3, "bernardini": 5, "berland": 6}


def _flow(name, form, nx, ny, nz, ni, nj, nk, rk="williamson"):
    return {"name": name, "kind": "flow", "form": form, "nx": nx, "ny": ny, "nz": nz, "ni": ni,
            "nj": nj, "nk": nk, "rk": rk}


def listed():
    return [
        # the first thing a user runs: one 32^3 Taylor-Green box in the
        # bit-exact form; every launch is small, so latency counts
        _flow("plain-1x32", "plain", 1, 1, 1, 32, 32, 32),
        # a validation run in the bit-exact form on an ordinary tiling
        _flow("plain-64x24", "plain", 4, 4, 4, 24, 24, 24),
        # an FP64 production run: the contracted build on 7.1 M cells
        _flow("fma-512x24", "plain_fma", 8, 8, 8, 24, 24, 24),
        # the mixed form where a node is shared: a handful of grids
        _flow("mixed-8x24", "mixed", 2, 2, 2, 24, 24, 24),
        # the mixed form on a mid-size production tiling
        _flow("mixed-512x24", "mixed", 8, 8, 8, 24, 24, 24),
        # the benchmark tiling, 56.6 M cells
        _flow("mixed-4096x24", "mixed", 16, 16, 16, 24, 24, 24),
        # grids whose edges divide nothing, with the five-stage scheme
        _flow("mixed-ragged", "mixed", 5, 6, 7, 21, 26, 19, "bernardini"),
        # wall-resolved turbulent channel: graded walls, WALE model, driven by
        # a pressure gradient
        {"name": "channel-les", "kind": "channel", "form": "mixed", "nx": 6, "ny": 4, "nz": 6,
         "n": 24},
        # flow past a sphere: three levels, ghost-cell immersed boundary
        {"name": "sphere-ib", "kind": "sphere", "form": "mixed", "nx": 8, "ny": 4, "nz": 4, "n": 16},
        # heated flow: scalar transport with buoyancy in the bit-exact form
        {"name": "scalar-216x20", "kind": "scalar", "form": "plain", "nx": 6, "ny": 6, "nz": 6,
         "ni": 20, "nj": 20, "nk": 20, "rk": "williamson"},
        # optimal control: the kinetic energy's gradient through two steps
        {"name": "adjoint-27x24", "kind": "adjoint", "form": "plain", "nx": 3, "ny": 3, "nz": 3,
         "ni": 24, "nj": 24, "nk": 24, "rk": "williamson"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tiles(rng, lo, hi):
    """Tile counts of about lo..hi grids, spread over the logarithm."""
    total = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = total ** (1.0 / 3.0)
    t = [max(1, int(side * rng.uniform(0.7, 1.4))) for _ in range(3)]
    while t[0] * t[1] * t[2] > hi:
        t[t.index(max(t))] -= 1
    return t


def draw(rng):
    kind = rng.choice(["plain", "plain_fma", "mixed", "mixed", "mixed", "ragged", "channel", "sphere",
                       "scalar", "adjoint"])
    if kind in ("plain", "plain_fma"):
        n = rng.choice([16, 20, 24, 28, 32])
        nx, ny, nz = _tiles(rng, 1, int(512 * (24 / n) ** 3))
        return {k: v for k, v in _flow("", kind, nx, ny, nz, n, n, n).items() if k != "name"}
    if kind == "mixed":
        n = rng.choice([16, 20, 24, 28, 32])
        nx, ny, nz = _tiles(rng, 1, int(3000 * (24 / n) ** 3))
        return {k: v for k, v in _flow("", kind, nx, ny, nz, n, n, n).items() if k != "name"}
    if kind == "ragged":
        form = rng.choice(["plain", "plain_fma", "mixed", "mixed"])
        ni, nj, nk = rng.randint(9, 30), rng.randint(9, 30), 2 * rng.randint(4, 14) + 1
        nx, ny, nz = _tiles(rng, 1, 300)
        rk = rng.choice(["williamson", "bernardini", "berland"])
        return {k: v for k, v in _flow("", form, nx, ny, nz, ni, nj, nk, rk).items() if k != "name"}
    if kind == "channel":
        return {"kind": "channel", "form": rng.choice(["mixed", "plain"]), "nx": rng.randint(2, 6),
                "ny": rng.randint(2, 4), "nz": rng.randint(2, 6), "n": rng.choice([16, 20, 24])}
    if kind == "sphere":
        return {"kind": "sphere", "form": rng.choice(["mixed", "plain"]), "nx": 8, "ny": 4,
                "nz": rng.choice([4, 6]), "n": rng.choice([8, 12])}
    if kind == "scalar":
        nx, ny, nz = _tiles(rng, 8, 216)
        n = [rng.randint(9, 24) for _ in range(3)]
        return {"kind": "scalar", "form": rng.choice(["plain", "plain_fma"]), "nx": nx, "ny": ny,
                "nz": nz, "ni": n[0], "nj": n[1], "nk": n[2], "rk": "williamson"}
    nx, ny, nz = _tiles(rng, 2, 64)
    n = rng.choice([8, 12, 16, 20, 24])
    return {"kind": "adjoint", "form": "plain", "nx": nx, "ny": ny, "nz": nz, "ni": n, "nj": n,
            "nk": n, "rk": "williamson"}


# -- grids -------------------------------------------------------------------

_spheres = {}


def _sphere(c):
    """The blocking and the stencil lists of a body are a program's mesh: they
    depend on no flow state, so a process builds them once."""
    key = (c["nx"], c["ny"], c["nz"], c["n"])
    if key not in _spheres:
        _spheres.clear()
        sc = channel.SphereChannel(tiles=key[:3], n=c["n"], grid_size=0.5, diameter=0.5,
                                   refine_radii=(0.5, 0.5), samples=4)
        sc.lists
        _spheres[key] = sc
    return _spheres[key]


def _graded(box, nz, n):
    """Grid lines of a box of height 2 along z, drawn towards both walls."""
    edges = 1.0 + np.tanh(2.0 * (np.arange(-2, nz * n + 3) / (nz * n) * 2 - 1)) / np.tanh(2.0)
    edges[:2] = 2 * edges[2] - edges[4:2:-1]
    edges[-2:] = 2 * edges[-3] - edges[-4:-6:-1]
    w = edges[1:] - edges[:-1]
    x = 0.5 * (edges[1:] + edges[:-1])
    d = np.append(x[1:] - x[:-1], w[-1])
    pick = lambda a: np.concatenate([a[g * n:g * n + n + 4] for g in box.gridpos[:, 2]])
    box.z, box.dz, box.ddz = pick(x), pick(d), pick(w)
    return box


def _box(c):
    if c["kind"] == "channel":
        box = cases.periodic_box(c["nx"], c["ny"], c["nz"], n=c["n"], length=(4.0, 2.0, 2.0),
                                 walls={5: abi.BC_NOS, 6: abi.BC_NOS})
        return _graded(box, c["nz"], c["n"])
    return cases.periodic_box(c["nx"], c["ny"], c["nz"], n=c["ni"], nj=c["nj"], nk=c["nk"])


def _dt(c, box):
    if c["kind"] == "sphere":
        return 0.1 * float(box.ddx.min())
    return 0.1 * min(float(box.ddx.min()), float(box.ddy.min()), float(box.ddz.min()))


def _params(c, box):
    kw = dict(gmol=NU, epcorr=1e-10, nouter=NOUTER, ninner=NINNER, form=FORMS[c["form"]])
    if c["kind"] == "channel":
        kw.update(gmol=2e-4, gradp=(-1e-2, 0.0, 0.0))
    if c["kind"] == "adjoint":
        kw.update(gmol=5e-3, epcorr=0.0, nouter=12, nouter_min=12)
    return abi.make_flow_params(**kw)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _start_fields(c, box, seed):
    """U, V, W, P (and T1, or the body force) over the flat layout
    [ngrid, ii, jj, kk]: a shifted Taylor-Green vortex, or a channel profile,
    with noise on the interior."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    phase = random.Random(seed).uniform(0, 2 * math.pi)
    t = lambda a, shape: torch.from_numpy(np.ascontiguousarray(a)).to(dev).reshape(shape)
    g, ii, jj, kk = box.ngrid, box.ii, box.jj, box.kk
    x, y, z = t(box.x, (g, ii, 1, 1)), t(box.y, (g, 1, jj, 1)), t(box.z, (g, 1, 1, kk))
    xs, ys = x + 0.5 * t(box.dx, (g, ii, 1, 1)), y + 0.5 * t(box.dy, (g, 1, jj, 1))
    full = (g, ii, jj, kk)

    def noise(f, amplitude):
        f = f.expand(full).clone()
        r = torch.rand((g, ii - 4, jj - 4, kk - 4), generator=gen, device=dev, dtype=torch.float64)
        f[:, 2:-2, 2:-2, 2:-2] += amplitude * (2 * r - 1)
        return f

    if c["kind"] == "channel":
        out = {"U": noise(1.5 * (1 - (z - 1) ** 2).clamp(min=0.0), 0.1),
               "V": noise(torch.zeros_like(x), 0.1), "W": noise(torch.zeros_like(x), 0.1),
               "P": torch.zeros(full, device=dev, dtype=torch.float64)}
    else:
        x, xs = x + phase, xs + phase
        out = {"U": noise(torch.sin(xs) * torch.cos(y) * torch.cos(z), 1e-2),
               "V": noise(-torch.cos(x) * torch.sin(ys) * torch.cos(z), 1e-2),
               "W": noise(torch.zeros_like(x), 1e-2),
               "P": noise((torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2) / 16, 0.0)}
    if c["kind"] == "scalar":
        out["T1"] = noise(torch.sin(z).expand(full), 0.1)
    if c["kind"] == "adjoint":
        for n in ("FX", "FY", "FZ"):
            out[n] = 0.1 * noise(torch.zeros_like(x), 1.0)
    return out


class _State:
    """A solver with its case loaded, and pinned buffers for what is read back."""

    def __init__(self, c, seed):
        self.c = c
        sc = _sphere(c) if c["kind"] == "sphere" else None
        self.box = box = sc.case if sc else _box(c)
        self.dt = _dt(c, box)
        self.rk = gpu.rk_scheme(c.get("rk", "williamson"))
        self.nrk = self.rk.nrk
        if sc:
            prm = sc.flow_params(FORMS[c["form"]], epcorr=1e-10, nouter=NOUTER, ninner=NINNER)
        else:
            prm = _params(c, box)
        self.s = s = gpu.Solver(box, prm)
        names = {"scalar": ["U", "V", "W", "P", "T1"], "channel": ["U", "V", "W", "P", "G"],
                 "adjoint": ["GFX", "GFY", "GFZ", "U", "V", "W"]}.get(c["kind"], ["U", "V", "W", "P"])
        self.out = {n: torch.empty(box.idim3d, dtype=torch.float64,
                                   pin_memory=torch.cuda.is_available()).numpy() for n in names}
        self.it = 0
        if sc:
            sc.setup(s)
            self._perturb(seed)
            return
        stage = self.out[names[0]]
        fields = _start_fields(c, box, seed)
        if c["kind"] == "scalar":
            s.set_scalars([PRANDTL])
            s.set_buoyancy([0.0, 0.0, GRAVITY], BETA)
        for n in ("U", "V", "W", "P", "T1"):
            if n in fields:
                torch.from_numpy(stage).copy_(fields[n].reshape(-1))
                s.set(n, stage)
        if c["kind"] == "adjoint":
            s.set_body_force(*(fields[n].reshape(-1).cpu().numpy() for n in ("FX", "FY", "FZ")))
        s.connect(0, 2, "U", "V", "W", "P", corners=True)
        if c["kind"] == "scalar":
            s.connect(0, 2, s1="T1", corners=True)
        if c["kind"] == "channel":
            s.bound_flow(0)
            s.set_lesmodel(2)

    def _perturb(self, seed):
        """Inflow turbulence of the sphere's start: noise on the fluid cells
        of the coarse and fine grids alike, then the reference's start-up."""
        s, box = self.s, self.box
        gen = torch.Generator().manual_seed(seed)
        bp = _sphere(self.c).geo["bp"]
        for n in ("U", "V", "W"):
            a = s.get(n)
            r = torch.rand(box.idim3d, generator=gen, dtype=torch.float64).numpy()
            box.interior(a)[...] += box.interior(2e-2 * (2 * r - 1) * bp)
            s.set(n, a)
        lo, hi = int(box.level.min()), int(box.level.max())
        for lv in range(lo, hi + 1):
            s.connect(lv, 2, v1="U", v2="V", v3="W", s1="P", corners=True)
        for lv in range(hi, lo, -1):
            s.ftoc_multiple(lv, v=("U", "V", "W"), s=("P",))
        for lv in range(lo, hi + 1):
            s.connect(lv, 1, v1="U", v2="V", v3="W", normal=True, forward=1)
            s.parent(lv, v=("U", "V", "W"), s=("P",))
            s.bound_flow(lv)
        s.setpointvalues(True)


def prepare(case, seed):
    return _State(case, seed)


def run(st):
    s, c = st.s, st.c
    st.it += 1
    if c["kind"] == "adjoint":
        energy, _ = st.s.energy_gradient(2, 1, st.dt, st.rk)
        return {"energy": energy, **{n: s.get(n, out=a) for n, a in st.out.items()}}
    for irk in range(1, st.nrk + 1):
        if c["kind"] == "scalar":
            s.timeintegrate_scalar(st.dt, irk, st.rk)
        s.timeintegrate_flow(st.it, st.it, 0.0, st.dt, irk, st.rk)
    return {n: s.get(n, out=a) for n, a in st.out.items()}


def _shape(c):
    """Points with ghosts, interior cells."""
    if c["kind"] == "sphere":
        box = _sphere(c).case
        return box.idim3d, box.ncells
    n = [c["n"]] * 3 if "n" in c else [c["ni"], c["nj"], c["nk"]]
    g = c["nx"] * c["ny"] * c["nz"]
    return g * (n[0] + 4) * (n[1] + 4) * (n[2] + 4), g * n[0] * n[1] * n[2]


def work(case):
    """Bytes: the state read once and the returned fields written once, at 8
    bytes.  Operations: per stage the momentum terms (three components, about
    60 each with every face flux taken once) and the update, the divergence and
    the projection, and per inner iteration the 7-point operator and the two
    triangular sweeps of the SIP solver, per outer iteration the residual."""
    points, cells = _shape(case)
    stages = STAGES[case.get("rk", "williamson")]
    nouter = 12 if case["kind"] == "adjoint" else NOUTER
    per_stage = 3 * 64 + 8 + 14 + nouter * (NINNER * (13 + 8 + 7) + 16)
    fields = {"scalar": 11, "channel": 9, "adjoint": 13}.get(case["kind"], 8)
    if case["kind"] == "scalar":
        per_stage += 40
    if case["kind"] == "channel":
        per_stage += 70
    # two steps forward, recomputed, and their transpose
    passes = 6 if case["kind"] == "adjoint" else 1
    return {"bytes": 8.0 * fields * points, "flops": float(passes * stages * per_stage * cells)}


# -- the same numbers in plain torch, 64 bits ---------------------------------

_RK = {
    "williamson": ([0.0, -5 / 9, -153 / 128], [1 / 3, 15 / 16, 8 / 15]),
    "bernardini": ([0.0, -1.0, -1.55798 - 3.88856487394645e-7, -1.0, -0.45031 - 3.88856487394645e-7],
                   [0.2, 0.83204 - 3.88856487394645e-7, 0.6, 0.35394 - 3.88856487394645e-7, 0.2]),
    "berland": ([0.0, -0.737101392796, -1.634740794341, -0.744739003780, -1.469897351522,
                 -2.813971388035],
                [0.032918605146, 0.823256998200, 0.381530948900, 0.200092213184, 1.718581042715,
                 0.27]),
}


class _Blocks:
    """The SIP solver of a periodic tiling of equal blocks with equal spacing.
    A block's points (with one ghost layer) are the rows of a matrix, its
    columns the blocks, so that a hyperplane of all blocks is a set of rows."""

    def __init__(self, c, h, dev):
        self.n, self.t = (c["ni"], c["nj"], c["nk"]), (c["nx"], c["ny"], c["nz"])
        ni, nj, nk = self.n
        self.st = ((nj + 2) * (nk + 2), nk + 2, 1)
        self.rows = (ni + 2) * (nj + 2) * (nk + 2)
        self.dev = dev
        i, j, k = np.meshgrid(*(np.arange(1, m + 1) for m in self.n), indexing="ij")
        row = i * self.st[0] + j * self.st[1] + k * self.st[2]
        self.inner = torch.from_numpy(row.ravel()).to(dev)
        m = (i + j + k).ravel()
        self.planes = [torch.from_numpy(row.ravel()[m == q]).to(dev) for q in range(3, sum(self.n) + 1)]
        # columns of the neighbours, and the rows of the four layers of each axis
        col = np.arange(self.t[0] * self.t[1] * self.t[2]).reshape(self.t)
        cells = (i, j, k)
        self.faces = []
        for d in range(3):
            low, high = row[cells[d] == 1], row[cells[d] == self.n[d]]
            self.faces.append(tuple(torch.from_numpy(a).to(dev) for a in (
                low - self.st[d], low, high, high + self.st[d], np.roll(col, 1, d).ravel(),
                np.roll(col, -1, d).ravel())))
        self.a = [1.0 / (q * q) for q in h]
        self.ap = -sum(2.0 / (q * q) for q in h)
        self._factors()

    def _factors(self):
        z = lambda: torch.zeros(self.rows, dtype=torch.float64, device=self.dev)
        lw, ls, lb, lpr, ue, un, ut = (z() for _ in range(7))
        alfa, tiny = float(np.float32(0.92)), float(np.float32(1e-20))
        sx, sy, sz = self.st
        ax, ay, az = self.a
        for p in self.planes:
            im, jm, km = p - sx, p - sy, p - sz
            w = ax / (1 + alfa * (un[im] + ut[im]))
            s = ay / (1 + alfa * (ue[jm] + ut[jm]))
            b = az / (1 + alfa * (un[km] + ue[km]))
            p1 = alfa * (b * ue[km] + s * ue[jm])
            p2 = alfa * (b * un[km] + w * un[im])
            p3 = alfa * (w * ut[im] + s * ut[jm])
            r = 1 / (self.ap + p1 + p2 + p3 - b * ut[km] - w * ue[im] - s * un[jm] + tiny)
            lw[p], ls[p], lb[p], lpr[p] = w * r, s * r, b * r, r
            ue[p], un[p], ut[p] = (ax - p1) * r, (ay - p2) * r, (az - p3) * r
        # per hyperplane: its rows and coefficients as columns
        self.lpr = lpr[self.inner][:, None]
        self.fwd = [(p, lw[p][:, None], ls[p][:, None], lb[p][:, None]) for p in self.planes]
        self.bwd = [(p, ue[p][:, None], un[p][:, None], ut[p][:, None]) for p in reversed(self.planes)]

    def split(self, f):
        """A global field as the matrix of blocks, ghost rows zero."""
        (ni, nj, nk), (tx, ty, tz) = self.n, self.t
        b = f.reshape(tx, ni, ty, nj, tz, nk).permute(1, 3, 5, 0, 2, 4).reshape(ni * nj * nk, -1)
        m = torch.zeros(self.rows, b.shape[1], dtype=torch.float64, device=self.dev)
        m[self.inner] = b
        return m

    def join(self, m):
        (ni, nj, nk), (tx, ty, tz) = self.n, self.t
        b = m[self.inner].reshape(ni, nj, nk, tx, ty, tz).permute(3, 0, 4, 1, 5, 2)
        return b.reshape(tx * ni, ty * nj, tz * nk)

    def exchange(self, m, low=True):
        for g0, low_in, high_in, g1, before, after in self.faces:
            high = m[low_in][:, after]
            if low:
                m[g0] = m[high_in][:, before]
            m[g1] = high

    def laplacian(self, m):
        p, a = self.inner, self.a
        s = sum(-a[d] * (m[p - self.st[d]] + m[p + self.st[d]]) for d in range(3))
        return s - self.ap * m[p]

    def solve(self, rhs, prefak):
        """The outer defect-correction loop around NINNER SIP iterations; a
        block's low residual ghosts lag one iteration, as the code exchanges
        them."""
        sx, sy, sz = self.st
        p = self.inner
        rhs = self.split(rhs)[p]
        dp = torch.zeros(self.rows, rhs.shape[1], dtype=torch.float64, device=self.dev)
        res = torch.zeros_like(dp)
        for _ in range(NOUTER):
            h = torch.zeros_like(dp)
            for il in range(1, NINNER + 1):
                res[p] = (rhs + self.laplacian(h)) * self.lpr
                for q, lw, ls, lb in self.fwd:
                    res[q] = res[q] - lb * res[q - sz] - ls * res[q - sy] - lw * res[q - sx]
                self.exchange(res, low=il < NINNER)
                for q, ue, un, ut in self.bwd:
                    res[q] = res[q] - ut * res[q + sz] - un * res[q + sy] - ue * res[q + sx]
                h[p] += res[p]
                self.exchange(h)
            rhs = rhs + self.laplacian(h)
            dp += h
            if float(rhs.abs().max()) / prefak < 1e-10:
                break
        return self.join(dp)


def _momentum(u, v, w, p, h):
    """-div(u u) + nu lap(u) - grad p at the staggered points of a periodic
    uniform box; u sits half a cell after the cell centre along its axis."""
    vel = (u, v, w)
    up = lambda a, d: torch.roll(a, -1, d)
    down = lambda a, d: torch.roll(a, 1, d)
    out = []
    for c in range(3):
        q = vel[c]
        r = torch.zeros_like(q)
        for d in range(3):
            if d == c:   # through the cell centre after the point
                adv = 0.5 * (q + up(q, d))
            else:        # the transporting component averaged along c
                adv = 0.5 * (vel[d] + up(vel[d], c))
            flux = adv * 0.5 * (q + up(q, d)) - NU * (up(q, d) - q) / h[d]
            r -= (flux - down(flux, d)) / h[d]
        out.append(r - (up(p, c) - p) / h[c])
    return out


def _scalar_rate(t, vel, h):
    r = torch.zeros_like(t)
    for d in range(3):
        nxt = torch.roll(t, -1, d)
        flux = vel[d] * 0.5 * (t + nxt) - NU / PRANDTL * (nxt - t) / h[d]
        r -= (flux - torch.roll(flux, 1, d)) / h[d]
    return r


def exact(case, seed):
    c = case
    if c["kind"] not in ("flow", "scalar"):
        return None   # walls, hierarchies, bodies and the adjoint are not restated
    if STAGES[c["rk"]] * (c["ni"] + c["nj"] + c["nk"]) * _shape(c)[1] > 3 * 72 * 1.2e7:
        return None   # too slow
    dev = _device()
    box = _box(c)
    dt, h = _dt(c, box), (float(box.dx[0]), float(box.dy[0]), float(box.dz[0]))
    tx, ty, tz = c["nx"], c["ny"], c["nz"]
    ni, nj, nk = c["ni"], c["nj"], c["nk"]

    def gather(f):   # [ngrid (x fastest), ii, jj, kk] -> the global box
        f = f[:, 2:-2, 2:-2, 2:-2].reshape(tz, ty, tx, ni, nj, nk)
        return f.permute(2, 3, 1, 4, 0, 5).reshape(tx * ni, ty * nj, tz * nk)

    def scatter(f):  # the global box -> every grid with its periodic ghosts
        ax = [torch.arange(-2, n + 2, device=dev) for n in (ni, nj, nk)]
        out = []
        for g in range(tx * ty * tz):
            gx, gy, gz = (int(q) for q in box.gridpos[g])
            i, j, k = (ax[0] + gx * ni) % (tx * ni), (ax[1] + gy * nj) % (ty * nj), (ax[2] + gz * nk) % (tz * nk)
            out.append(f[i][:, j][:, :, k])
        return torch.stack(out).reshape(-1)

    f = {n: gather(a) for n, a in _start_fields(c, box, seed).items()}
    blocks = _Blocks(c, h, dev)
    a, b = _RK[c["rk"]]
    nst = len(a)
    at = [0.0]
    for i in range(1, nst):   # stage times of the low-storage scheme
        s, q = 0.0, 1.0
        for j in range(1, i + 1):
            q = 1.0
            for k in range(2, j + 1):
                q = a[k - 1] * q + 1.0
            s += b[j - 1] * q
        at.append(s)
    vel = [f["U"], f["V"], f["W"]]
    p, t = f["P"], f.get("T1")
    reg = [torch.zeros_like(p) for _ in range(4)]
    for i in range(nst):
        told = t
        if t is not None:
            reg[3] = a[i] * reg[3] + _scalar_rate(t, vel, h)
            t = t + dt * b[i] * reg[3]
        rate = _momentum(*vel, p, h)
        if told is not None:
            rate[2] = rate[2] - GRAVITY * BETA * 0.5 * (told + torch.roll(told, -1, 2))
        for d in range(3):
            reg[d] = a[i] * reg[d] + rate[d]
            vel[d] = vel[d] + dt * b[i] * reg[d]
        dts = dt * (at[i + 1] if i + 1 < nst else 1.0)
        div = sum((vel[d] - torch.roll(vel[d], 1, d)) / h[d] for d in range(3)) / dts
        dp = blocks.solve(div, 1.0 / dts)
        p = p + dp
        for d in range(3):
            vel[d] = vel[d] + dts * (dp - torch.roll(dp, -1, d)) / h[d]
    out = {"U": vel[0], "V": vel[1], "W": vel[2], "P": p}
    if t is not None:
        out["T1"] = t
    return {n: scatter(q) for n, q in out.items()}
