"""The work that is timed: what programs have this package do, through its public entry points.

kinds
  steps    a resident box takes `steps` time steps (Context.simulate) and its slot array comes back
  stages   a staged run with rescales and thermo samples (Context.run_stages), then energies per atom
  cascade  a box is set up, one atom is kicked, `steps` steps at the variable timestep (collision_step)
  batch    several cascades advanced together (Batch.run)
  host     one step from and to the caller's page-locked slot array (Context.step_host)
  hooks    the three accelerator hooks on the caller's slot array (eam_rho_calc, eam_df_calc, eam_force_calc)

Boxes are BCC crystals of Fe (n_ele 1) or dilute Fe-Cu-Ni (n_ele 3) with thermal displacements and Maxwell
velocities from the seed. The potential is a setfl table of 5000 knots with a 5.6 A cutoff: a Morse pair
term with a screened-Coulomb core, an exponential density, a square-root embedding function.
"""
import ctypes
import importlib.util
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEV = "cuda" if torch.cuda.is_available() else "cpu"

A0, CUTOFF = 2.855, 5.6
RCF = CUTOFF / A0
GHOST = 3                                   # ceil(cutoff / a0) + 1 unit cells on every side
MASS = (55.845, 63.546, 58.6934)
NUMBER = (26, 29, 28)
BOLTZ, MVV2E = 8.617343e-5, 1.0364269e-4
NR = NRHO = 5000
RHO_MAX = 200.0
TEMPERATURE, SPREAD = 320.0, 0.06           # K, and the displacements' standard deviation in A
DX_MAX, DT_MIN, DT_MAX = 0.01, 1e-5, 1e-3   # variable timestep of the cascades (A, ps)
DT = 0.001


# ---- the cases --------------------------------------------------------------------------------------
def _case(name, kind, precision, cells, n_ele, steps, energy=0.0, replicas=1):
    c = {"kind": kind, "precision": precision, "nx": cells[0], "ny": cells[1], "nz": cells[2], "n_ele": n_ele,
         "steps": steps, "energy": energy, "replicas": replicas}
    return dict({"name": name}, **c) if name else c


def listed():
    return [
        _case("steps_20c_fp64", "steps", "fp64", (20, 20, 20), 1, 100),
        _case("steps_20c_mixed", "steps", "mixed", (20, 20, 20), 1, 100),
        _case("steps_53x47x61_fp64", "steps", "fp64", (53, 47, 61), 3, 20),
        _case("steps_75x61x49_mixed", "steps", "mixed", (75, 61, 49), 3, 64),
        _case("steps_100c_fp64", "steps", "fp64", (100, 100, 100), 1, 8),
        _case("steps_100c_mixed", "steps", "mixed", (100, 100, 100), 1, 64),
        _case("steps_200c_mixed", "steps", "mixed", (200, 200, 200), 3, 32),
        _case("stages_32c_fp64", "stages", "fp64", (32, 32, 32), 3, 40),
        _case("cascade_40c_mixed", "cascade", "mixed", (40, 40, 40), 3, 120, 2000.0),
        _case("batch_6x30c_mixed", "batch", "mixed", (30, 30, 30), 3, 60, 1000.0, 6),
        _case("host_100c_mixed", "host", "mixed", (100, 100, 100), 3, 1),
        _case("hooks_50c_fp64", "hooks", "fp64", (50, 50, 50), 1, 1),
    ]


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "stages", "cascade", "batch", "host", "hooks"])
    precision = rng.choice(["fp64", "mixed"])
    n_ele = rng.choice([1, 3])
    edge = {"steps": (8, 200) if precision == "mixed" else (8, 110), "stages": (10, 60), "cascade": (20, 70),
            "batch": (14, 40), "host": (16, 150), "hooks": (8, 90)}[kind]
    n = math.exp(rng.uniform(math.log(edge[0]), math.log(edge[1])))
    cells = [max(6, min(edge[1], round(n * math.exp(rng.uniform(-0.2, 0.2))))) for _ in range(3)]
    atoms = 2 * cells[0] * cells[1] * cells[2]
    steps, energy, replicas = 1, 0.0, 1
    if kind == "steps":
        most = 4e8 if precision == "mixed" else 1.6e7
        steps = int(max(1, min(100, most / atoms)) * rng.uniform(0.5, 1.0)) + 1
    elif kind == "stages":
        steps = 10 * rng.randint(1, 4)
    elif kind in ("cascade", "batch"):
        steps = rng.randint(30, 120) if precision == "mixed" else rng.randint(10, 30)
        energy = round(rng.uniform(200.0, 1000.0 if n < 30 else 5000.0), 1)
        replicas = rng.randint(2, 6) if kind == "batch" else 1
    return _case(None, kind, precision, cells, n_ele, steps, energy, replicas)


# ---- the potential ----------------------------------------------------------------------------------
def _step5(t):
    t = np.clip(t, 0.0, 1.0)
    return t**3 * (10.0 - 15.0 * t + 6.0 * t * t)


def tables(n_ele):
    """F[e], rho[e], r*phi[pair i >= j] on their knots, drho, dr."""
    dr, drho = CUTOFF / (NR - 1), RHO_MAX / (NRHO - 1)
    r, q = np.arange(NR) * dr, np.arange(NRHO) * drho
    cut = 1.0 - _step5((r - 5.0) / 0.6)
    # per element: Morse depth, exponent, minimum; density decay
    par = [(0.40, 1.40, 2.65, 1.50)] if n_ele == 1 else [(0.40, 1.40, 2.62, 1.50), (0.37, 1.45, 2.66, 1.43),
                                                         (0.42, 1.37, 2.60, 1.56)]
    F = [-np.sqrt(q) for _ in par]
    rho = [np.exp(-b * (r - 2.5)) * cut for _, _, _, b in par]
    pairs = []
    for i in range(n_ele):
        for j in range(i + 1):
            d, a, m = (math.sqrt(par[i][k] * par[j][k]) for k in range(3))
            morse = r * d * (np.exp(-2 * a * (r - m)) - 2 * np.exp(-a * (r - m))) * cut
            # screened Coulomb core (Ziegler, Biersack and Littmark, 1985), joined on [1, 2] A
            s = r * (NUMBER[i] ** 0.23 + NUMBER[j] ** 0.23) / 0.46850
            core = 14.399645 * NUMBER[i] * NUMBER[j] * (0.18175 * np.exp(-3.19980 * s) + 0.50986 * np.exp(-0.94229 * s) +
                                                        0.28022 * np.exp(-0.40290 * s) + 0.02817 * np.exp(-0.20162 * s))
            w = _step5(r - 1.0)
            pairs.append((1.0 - w) * core + w * morse)
    return F, rho, pairs, drho, dr


_files = {}


def potential_file(n_ele):
    if n_ele not in _files:
        F, rho, pairs, drho, dr = tables(n_ele)
        path = os.path.join(tempfile.mkdtemp(prefix="setfl_"), "%d.setfl" % n_ele)
        symbols = ("Fe", "Cu", "Ni")[:n_ele]
        with open(path, "w") as f:
            f.write("Morse pair, exponential density, square-root embedding\n\n\n%d %s\n" % (n_ele, " ".join(symbols)))
            f.write("%d %.17g %d %.17g %.17g\n" % (NRHO, drho, NR, dr, CUTOFF))
            for e in range(n_ele):
                f.write("%d %.17g %.17g bcc\n" % (NUMBER[e], MASS[e], A0))
                f.writelines("%.17g\n" % v for v in np.concatenate([F[e], rho[e]]))
            for p in pairs:
                f.writelines("%.17g\n" % v for v in p)
        _files[n_ele] = path
    return _files[n_ele]


# ---- the boxes --------------------------------------------------------------------------------------
def package():
    """The package, by the loader that its own entry script uses."""
    if "misa_md_gb300" not in sys.modules:
        where = os.path.join(ROOT, "misa-md_gb300")
        spec = importlib.util.spec_from_file_location("misa_md_gb300", os.path.join(where, "__init__.py"),
                                                      submodule_search_locations=[where])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["misa_md_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["misa_md_gb300"]


def crystal(cells, n_ele, seed):
    """Types [N], positions, velocities and sites [N, 3] of the box's atoms in k, j, i order."""
    nx, ny, nz = cells
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + 17 * nx + 5 * ny + nz)
    i = torch.arange(2 * nx, device=DEV, dtype=torch.float64).view(1, 1, -1)
    j = torch.arange(ny, device=DEV, dtype=torch.float64).view(1, -1, 1)
    k = torch.arange(nz, device=DEV, dtype=torch.float64).view(-1, 1, 1)
    half = (i % 2) * 0.5
    shape = (nz, ny, 2 * nx)
    site = torch.stack([(i * 0.5 * A0).expand(shape), ((j + half) * A0).expand(shape), ((k + half) * A0).expand(shape)], -1)
    site = site.reshape(-1, 3)
    n = site.shape[0]
    kind = torch.zeros(n, dtype=torch.int32, device=DEV)
    if n_ele == 3:
        u = torch.rand(n, generator=g, device=DEV)
        kind[u < 0.025] = 1
        kind[u < 0.010] = 2
    mass = torch.tensor(MASS, dtype=torch.float64, device=DEV)[kind.long()].unsqueeze(1)
    x = site + SPREAD * torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64).clamp(-3.5, 3.5)
    v = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64) * torch.sqrt(BOLTZ * TEMPERATURE / (mass * MVV2E))
    v -= (v * mass).mean(0, keepdim=True) / mass
    return kind, x, v, site


def records(cells, kind, x, v, dtype):
    """The ghost-extended slot array that a caller uploads (ghost slots vacant)."""
    nx, ny, nz = cells
    full = (nz + 2 * GHOST, ny + 2 * GHOST, 2 * (nx + 2 * GHOST))
    rec = torch.zeros(full + (13,), dtype=torch.int64, device=DEV)  # id, type, x, v, f, rho, df: 13 words
    rec[..., 1] = 0xFFFFFFFF
    box = rec[GHOST:GHOST + nz, GHOST:GHOST + ny, 2 * GHOST:2 * (GHOST + nx)]
    n = kind.numel()
    box[..., 0] = torch.arange(1, n + 1, device=DEV).view(box.shape[:-1])
    box[..., 1] = kind.long().view(box.shape[:-1])
    box[..., 2:5] = x.view(torch.int64).view(box.shape[:-1] + (3,))
    box[..., 5:8] = v.contiguous().view(torch.int64).view(box.shape[:-1] + (3,))
    host = np.empty(rec.numel() // 13, dtype=dtype)
    torch.from_numpy(host.view(np.int64)).copy_(rec.view(-1))
    return host


class Box:
    """A context with its potential and state, and the slot arrays that come back from it."""

    def __init__(self, case, cells, seed, pinned=True):
        pkg = package()
        self.pkg, self.cells, self.pinned = pkg, cells, False
        self.ctx = pkg.Context(cells, A0, RCF, precision=case["precision"])
        self.ctx.pot_init_setfl(potential_file(case["n_ele"]))
        self.ctx.set_timestep(DT)
        kind, x, v, _ = crystal(cells, case["n_ele"], seed)
        self.atoms = records(cells, kind, x, v, pkg.ATOM_DTYPE)
        self.inter = np.zeros(4096, dtype=pkg.ATOM_DTYPE)
        if pinned:
            pkg.host_register(self.atoms)
            self.pinned = True

    def __del__(self):
        if getattr(self, "pinned", False):
            self.pkg.host_unregister(self.atoms)
        if getattr(self, "ctx", None) is not None:
            self.ctx.close()

    def start(self):
        self.ctx.upload(self.atoms)
        self.ctx.prepare()

    def fetch(self, into):
        """mg_download into an array that the program keeps."""
        n = ctypes.c_int64()
        c = self.ctx
        c._check(c.lib.mg_download(c.h, into.ctypes.data, into.size, self.inter.ctypes.data, self.inter.size, ctypes.byref(n)))
        return dict(self.fields(into), n_inter=n.value)

    def fields(self, atoms):
        nx, ny, nz = self.cells
        box = atoms.reshape(nz + 2 * GHOST, ny + 2 * GHOST, 2 * (nx + 2 * GHOST))
        box = box[GHOST:GHOST + nz, GHOST:GHOST + ny, 2 * GHOST:2 * (GHOST + nx)]
        out = {f: box[f] for f in ("type", "x", "v", "f", "rho", "df")}
        out["id"] = box["id"].view(np.int64)
        return out


def _cells(case):
    return (case["nx"], case["ny"], case["nz"])


def _direction(seed):
    d = np.random.default_rng(seed).standard_normal(3)
    return d / np.linalg.norm(d)


def prepare(case, seed):
    kind, cells = case["kind"], _cells(case)
    s = {"case": case}
    if kind in ("steps", "stages", "host", "hooks"):
        b = s["box"] = Box(case, cells, seed, pinned=kind != "hooks")
        b.start()
        if kind in ("host", "hooks"):
            b.fetch(b.atoms)  # ghosts, densities and forces as after a step
        if kind == "host":
            s["n_inter"] = 0
    else:
        s["boxes"] = [Box(case, cells, seed + 100 * r) for r in range(case["replicas"])]
        s["back"] = [np.empty_like(b.atoms) for b in s["boxes"]]
        for b, a in zip(s["boxes"], s["back"]):
            b.start()
            b.fetch(a)
            b.ctx.set_variable_timestep(DX_MAX, DT_MIN, DT_MAX)
        s["dir"] = [_direction(seed + 100 * r) for r in range(case["replicas"])]
        if kind == "batch":
            s["batch"] = package().Batch([b.ctx for b in s["boxes"]], steps_per_launch=10)
    return s


def run(s):
    case = s["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "steps":
        b = s["box"]
        b.ctx.simulate(steps)
        return b.fetch(b.atoms)
    if kind == "stages":
        b = s["box"]
        n = 2 * case["nx"] * case["ny"] * case["nz"]
        stage = {"steps": steps, "step_length": DT, "rescale_t": TEMPERATURE, "rescale_every": 5}
        got = b.ctx.run_stages([stage], steps, DT, n, thermo_interval=5)
        t = b.ctx.thermo(with_energy=True)
        e, _ = b.ctx.energies()
        out = b.fetch(b.atoms)
        nx, ny, nz = b.cells
        out["e"] = e.reshape(nz + 2 * GHOST, ny + 2 * GHOST, -1)[GHOST:-GHOST, GHOST:-GHOST, 2 * GHOST:-2 * GHOST]
        out["mvv"] = np.array([g["mvv"] for g in got])
        out["potential"] = np.array([t["potential_energy"]])
        return out
    if kind == "host":
        b = s["box"]
        s["n_inter"] = b.ctx.step_host(b.atoms, b.inter, s["n_inter"], 1)
        return dict(b.fields(b.atoms), n_inter=s["n_inter"])
    if kind == "hooks":
        b = s["box"]
        b.ctx.eam_rho_calc(b.atoms)
        b.ctx.eam_df_calc(b.atoms)
        b.ctx.eam_force_calc(b.atoms)
        return b.fields(b.atoms)
    nx, ny, nz = _cells(case)
    for b, d in zip(s["boxes"], s["dir"]):
        b.start()
        b.ctx.collision_step([nx // 2, ny // 2, nz // 2, 0], d, case["energy"])
    if kind == "batch":
        s["batch"].run(steps)
    else:
        s["boxes"][0].ctx.simulate(steps)
    out = {"boxes": [b.fetch(a) for b, a in zip(s["boxes"], s["back"])]}
    out["inter"] = {f: np.stack([b.inter[f] for b in s["boxes"]]) for f in ("type", "x", "v", "f", "rho", "df")}
    return out


# ---- what a pass cannot do without ------------------------------------------------------------------
PAIRS = 58                 # neighbours inside the cutoff
RECORD = 104               # bytes of a slot record
STEP_BYTES = 138           # positions, types, dF, velocities read; positions, velocities, dF written
STEP_FLOPS = PAIRS * (8 + 3 + 6 + 2 + 8 + 7 + 9 + 6) + 40  # distance twice, splines, the pair force, the sums; Verlet


def work(case):
    nx, ny, nz = _cells(case)
    atoms = 2 * nx * ny * nz * case["replicas"]
    slots = 2 * (nx + 2 * GHOST) * (ny + 2 * GHOST) * (nz + 2 * GHOST) * case["replicas"]
    passes = case["steps"] + {"steps": 0, "stages": 1, "cascade": 2, "batch": 2, "host": 0, "hooks": 0}[case["kind"]]
    copies = {"steps": 1, "stages": 1, "cascade": 2, "batch": 2, "host": 2, "hooks": 1}[case["kind"]]
    more = {"stages": 8 * slots, "hooks": 25 * slots + 40 * atoms}.get(case["kind"], 0)
    return {"bytes": float(STEP_BYTES * atoms * passes + RECORD * slots * copies + more),
            "flops": float(STEP_FLOPS * atoms * passes)}


# ---- the same in 64 bits ----------------------------------------------------------------------------
def _spline(f):
    """Cubic per knot interval from 5-point slopes: c0..c3 (in the interval's own coordinate)."""
    s = np.empty_like(f)
    s[0], s[1], s[-2], s[-1] = f[1] - f[0], 0.5 * (f[2] - f[0]), 0.5 * (f[-1] - f[-3]), f[-1] - f[-2]
    s[2:-2] = ((f[:-4] - f[4:]) + 8.0 * (f[3:-1] - f[1:-3])) / 12.0
    c = np.zeros((f.size, 4))
    c[:, 0], c[:, 1] = f, s
    rise = f[1:] - f[:-1]
    c[:-1, 2] = 3.0 * rise - 2.0 * s[:-1] - s[1:]
    c[:-1, 3] = s[:-1] + s[1:] - 2.0 * rise
    return torch.from_numpy(c).to(DEV)


class Crystal64:
    """The same crystal stepped by plain tensors: the two sublattices, whole-box shifts for neighbours."""

    def __init__(self, case, seed):
        cells = _cells(case)
        self.shape = (cells[2], cells[1], cells[0])
        kind, x, v, site = crystal(cells, case["n_ele"], seed)
        split = lambda a, w: [a.view(self.shape + (2,) + w)[:, :, :, p] for p in (0, 1)]  # noqa: E731
        self.kind = [t.long().contiguous() for t in split(kind, ())]
        self.site = split(site, (3,))
        self.u = [(a - b).contiguous() for a, b in zip(split(x, (3,)), self.site)]
        self.v = [a.clone() for a in split(v, (3,))]
        F, rho, pairs, self.drho, self.dr = tables(case["n_ele"])
        self.n = case["n_ele"]
        self.F = torch.stack([_spline(f) for f in F]).view(-1, 4)
        self.rho_t = torch.stack([_spline(f) for f in rho]).view(-1, 4)
        order = [[max(a, b) * (max(a, b) + 1) // 2 + min(a, b) for b in range(self.n)] for a in range(self.n)]
        self.z = torch.stack([_spline(pairs[order[a][b]]) for a in range(self.n) for b in range(self.n)]).view(-1, 4)
        self.mass = torch.tensor(MASS, dtype=torch.float64, device=DEV)
        # half of the neighbour vectors in units of a0 / 2: all even (same sublattice) or all odd
        lim = 2 * (RCF + 0.4)
        r = range(-5, 6)
        self.vec = [(a, b, c) for a in r for b in r for c in r
                    if a % 2 == b % 2 == c % 2 and (c, b, a) > (0, 0, 0) and a * a + b * b + c * c < lim * lim]

    def pairs(self):
        """Per sublattice and vector: the in-range pair's distance vector, r, knot and fraction."""
        for p in (0, 1):
            for a, b, c in self.vec:
                q = p ^ (a & 1)
                if a & 1:  # from corner to centre the centre's own index is half a cell less
                    e = -1 if p == 0 else 1
                    sh = ((c + e) // 2, (b + e) // 2, (a + e) // 2)
                else:
                    sh = (c // 2, b // 2, a // 2)
                back = tuple(-t for t in sh)
                step = torch.tensor((a, b, c), dtype=torch.float64, device=DEV) * (0.5 * A0)
                d = (self.u[p] - torch.roll(self.u[q], back, (0, 1, 2))) - step
                r2 = (d * d).sum(-1)
                near = r2 < CUTOFF * CUTOFF
                if not bool(near.any()):
                    continue
                r = torch.sqrt(torch.where(near, r2, CUTOFF * CUTOFF * torch.ones_like(r2)))
                x = r / self.dr
                m = x.long().clamp_(0, NR - 2)
                yield p, q, sh, back, d, r, m, (x - m).clamp_(max=1.0), near

    def value(self, tab, i, t):
        c = tab[i.view(-1)].view(i.shape + (4,))
        return ((c[..., 3] * t + c[..., 2]) * t + c[..., 1]) * t + c[..., 0]

    def slope(self, tab, i, t, delta):
        c = tab[i.view(-1)].view(i.shape + (4,))
        return ((3.0 * c[..., 3] * t + 2.0 * c[..., 2]) * t + c[..., 1]) / delta

    def eam(self, energy=False):
        self.rho = [torch.zeros(self.shape, dtype=torch.float64, device=DEV) for _ in (0, 1)]
        for p, q, sh, back, d, r, m, t, near in self.pairs():
            tj = torch.roll(self.kind[q], back, (0, 1, 2))
            self.rho[p] += torch.where(near, self.value(self.rho_t, tj * NR + m, t), 0.0)
            self.rho[q] += torch.roll(torch.where(near, self.value(self.rho_t, self.kind[p] * NR + m, t), 0.0), sh, (0, 1, 2))
        knot = [(a / self.drho).long().clamp_(0, NRHO - 2) for a in self.rho]
        frac = [(a / self.drho - m).clamp_(max=1.0) for a, m in zip(self.rho, knot)]
        at = [k * NRHO + m for k, m in zip(self.kind, knot)]
        self.df = [self.slope(self.F, i, t, self.drho) for i, t in zip(at, frac)]
        self.f = [torch.zeros(self.shape + (3,), dtype=torch.float64, device=DEV) for _ in (0, 1)]
        self.e = [self.value(self.F, i, t) for i, t in zip(at, frac)]
        for p, q, sh, back, d, r, m, t, near in self.pairs():
            tj = torch.roll(self.kind[q], back, (0, 1, 2))
            zi = (self.kind[p] * self.n + tj) * NR + m
            zv, zp = self.value(self.z, zi, t), self.slope(self.z, zi, t, self.dr)
            dj = torch.roll(self.df[q], back, (0, 1, 2))
            s = (self.df[p] * self.slope(self.rho_t, tj * NR + m, t, self.dr) +
                 dj * self.slope(self.rho_t, self.kind[p] * NR + m, t, self.dr) + (zp - zv / r) / r)
            f = torch.where(near, -s / r, 0.0).unsqueeze(-1) * d
            self.f[p] += f
            self.f[q] -= torch.roll(f, sh, (0, 1, 2))
            if energy:
                h = torch.where(near, 0.5 * zv / r, 0.0)
                self.e[p] += h
                self.e[q] += torch.roll(h, sh, (0, 1, 2))

    def kick(self, dt):
        for p in (0, 1):
            self.v[p] += self.f[p] * (0.5 * dt / (self.mass[self.kind[p]] * MVV2E)).unsqueeze(-1)

    def step(self, dt):
        self.kick(dt)
        for p in (0, 1):
            self.u[p] = self.u[p] + dt * self.v[p]
        self.eam()
        self.kick(dt)

    def mvv(self):
        return sum((self.mass[k] * (v * v).sum(-1)).sum() for k, v in zip(self.kind, self.v))

    def together(self, a):
        return torch.stack(list(a), 3).reshape(self.shape[0], self.shape[1], -1, *a[0].shape[3:])

    def out(self):
        return {"type": None, "x": self.together([a + b for a, b in zip(self.u, self.site)]), "v": self.together(self.v),
                "f": self.together(self.f), "rho": self.together(self.rho), "df": self.together(self.df), "id": None}


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    atoms = 2 * case["nx"] * case["ny"] * case["nz"]
    if kind in ("cascade", "batch") or (steps + 1) * max(0.035, 1.2e-7 * atoms) > 18.0:
        return None
    c = Crystal64(case, seed)
    c.eam()
    if kind == "stages":
        mvv, dof = [], 3 * atoms - 3
        for k in range(steps):
            if k % 5 == 0:
                f = torch.sqrt(TEMPERATURE / (c.mvv() * MVV2E / (dof * BOLTZ)))
                c.v = [v * f for v in c.v]
            c.step(DT)
            if (k + 1) % 5 == 0:
                mvv.append(c.mvv())
        c.eam(energy=True)
        out = c.out()
        out["e"] = c.together(c.e)
        out["mvv"] = torch.stack(mvv)
        out["potential"] = out["e"].sum().view(1)
        return out
    if kind != "hooks":
        for _ in range(steps):
            c.step(DT)
    return c.out()
