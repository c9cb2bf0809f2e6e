"""The FP64 form's fixed-point pair arithmetic on the CPU: every function of a pair against the setfl spline
evaluated with 50 digits, at knots, between them, near the cutoff and at large coordinates."""
import ctypes
import os
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
A0 = 2.855
CUTOFF = 5.6
RCF = CUTOFF / A0


@pytest.fixture(scope="module")
def lib(tmp_path_factory, pkg):
    so = str(tmp_path_factory.mktemp("fix") / "libfix.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(pkg.build.nvcc())), "include")
    src = os.path.join(ROOT, "misa-md_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-pthread", "-I", cuda, "-I", src,
                    "-o", so, os.path.join(ROOT, "tests", "fixed_point_support.cpp"), os.path.join(src, "mg_fixed.cpp"),
                    os.path.join(src, "mg_potential.cpp")], check=True)
    return ctypes.CDLL(so)


def _open(lib, path, a0=A0, rcf=RCF):
    return lib.fix_open(os.fsencode(path), ctypes.c_double(a0), ctypes.c_double(rcf), 116)


def _pairs(lib, xi, xj, ti, tj):
    n = len(ti)
    cls, out = np.zeros(n, dtype=np.int32), np.zeros((n, 6))
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    lib.fix_pairs(n, p(np.ascontiguousarray(xi)), p(np.ascontiguousarray(xj)), p(np.asarray(ti, dtype=np.int32)),
                  p(np.asarray(tj, dtype=np.int32)), p(cls), p(out))
    return cls, out


class Spline:
    """The table's cubic per interval, coefficients in doubles as the library builds them."""

    def __init__(self, f, dr):
        n = len(f)
        s = np.empty(n)
        s[0], s[1], s[-2], s[-1] = f[1] - f[0], 0.5 * (f[2] - f[0]), 0.5 * (f[-1] - f[-3]), f[-1] - f[-2]
        for m in range(2, n - 2):
            s[m] = ((f[m - 2] - f[m + 2]) + 8.0 * (f[m + 1] - f[m - 1])) / 12.0
        rise = f[1:] - f[:-1]
        self.c = np.zeros((n, 4))
        self.c[:, 0], self.c[:, 1] = f, s
        self.c[:-1, 2] = 3.0 * rise - 2.0 * s[:-1] - s[1:]
        self.c[:-1, 3] = s[:-1] + s[1:] - 2.0 * rise
        self.inv = 1.0 / dr
        self.n = n

    def at(self, r, side=0):
        """Value and derivative at a Decimal distance; side -1 / +1: by the cubic of the interval beside it."""
        x = r * Decimal(self.inv)
        m = max(0, min(int(x) + side, self.n - 2))
        p = x - m
        c = [Decimal(float(v)) for v in self.c[m]]
        d = [Decimal(float(v)) for v in (self.c[m, 1] * self.inv, 2.0 * self.c[m, 2] * self.inv, 3.0 * self.c[m, 3] * self.inv)]
        return c[0] + p * (c[1] + p * (c[2] + p * c[3])), d[0] + p * (d[1] + p * d[2])


def _r2(a, b):
    return sum((Decimal(float(u)) - Decimal(float(v))) ** 2 for u, v in zip(a, b))


@pytest.mark.parametrize("n_ele,nr", [(1, 5000), (3, 5000), (1, 9001)])
def test_pair_functions_against_50_digits(lib, wl, tmp_path, n_ele, nr):
    getcontext().prec = 50
    spec = wl.PotentialSpec(n_ele=n_ele, seed=5, nr=nr)
    assert _open(lib, wl.write_setfl(str(tmp_path / "p.setfl"), spec)) == 1
    F, rho, rphi, drho, dr = wl.potential_tables(spec)
    rng = np.random.default_rng(nr + n_ele)
    n = 1500
    r = rng.uniform(2.2, CUTOFF, n)
    r[:300] = np.round(r[:300] / dr) * dr                       # knots
    r[300:500] = np.round(r[300:500] / dr) * dr * (1 + rng.uniform(-1e-6, 1e-6, 200))
    r[500:520] = CUTOFF - rng.uniform(0, 1e-12, 20)
    d = rng.standard_normal((n, 3))
    d[520:600] = np.eye(3)[rng.integers(0, 3, 80)]              # along the axes
    d /= np.linalg.norm(d, axis=1)[:, None]
    xi = rng.uniform(-10.0, 600.0, (n, 3))
    xi[600:700] *= 1e-3
    xj = xi - d * r[:, None]
    ti, tj = rng.integers(0, n_ele, n), rng.integers(0, n_ele, n)
    cls, out = _pairs(lib, xi, xj, ti, tj)
    sr = [Spline(rho[e], dr) for e in range(n_ele)]
    sz = {}
    k = 0
    for a in range(n_ele):
        for b in range(a + 1):
            sz[a, b] = sz[b, a] = Spline(rphi[k], dr)
            k += 1
    rc2 = Decimal(A0 * RCF) ** 2
    got, want = [], []
    for q in range(n):
        r2 = _r2(xi[q], xj[q])
        got_r2 = Decimal(float(out[q, 4])) + Decimal(float(out[q, 5]))
        assert abs(got_r2 - r2) <= Decimal(2.0 ** -52)   # 4 units of r^2: the coordinates' rounding and the products'
        if abs(r2 - rc2) < Decimal(1e-14):
            continue
        assert (cls[q] != 0) == (r2 < rc2)
        if cls[q] != 1:
            continue
        R = r2.sqrt()
        # within 1e-6 of a knot either interval's cubic is the spline: they differ by their coefficients' rounding
        off = R * Decimal(sr[0].inv) % 1
        sides = [0] + ([-1] if off < Decimal(1e-6) else [1] if off > 1 - Decimal(1e-6) else [])
        values = []
        for side in sides:
            rv, rd = sr[tj[q]].at(R, side)
            zv, zd = sz[ti[q], tj[q]].at(R, side)
            values.append([rv, rd / R, (zd - zv / R) / (R * R), zv / R])
        got.append(out[q, :4])
        want.append([min((v[k] for v in values), key=lambda v: abs(v - Decimal(float(out[q, k])))) for k in range(4)])
    assert len(got) > 1300
    got = np.array(got)
    for k in range(4):
        w = [x[k] for x in want]
        top = max(abs(v) for v in w)
        for g, v in zip(got[:, k], w):
            # the bound every record is built to (2^-49), and the conversion of the result to a double
            assert abs(Decimal(float(g)) - v) <= Decimal(2.0 ** -48) * max(abs(v), top / 32)


def test_vacant_slots_and_far_coordinates_stay_outside(lib, wl, tmp_path):
    """Coordinates half a period away from a site of the full table are outside the cutoff, whatever the
    displacements; so are all atoms beyond the cutoff up to the largest candidate distance."""
    assert _open(lib, wl.write_setfl(str(tmp_path / "p.setfl"), wl.PotentialSpec(n_ele=1))) == 1
    rng = np.random.default_rng(1)
    n = 4000
    site = rng.integers(-6, 7, (n, 3)) * (0.5 * A0)
    site = site[np.linalg.norm(site, axis=1) < (RCF + 1) * A0]
    xi = 300.0 + rng.uniform(-0.6, 0.6, site.shape) * A0
    z = np.zeros(len(site), dtype=np.int32)
    cls, _ = _pairs(lib, xi, 300.0 + site + 16.0, z, z)  # 2^4 A: half of the period 2^5 A at this lattice constant
    assert (cls == 0).all()
    xj = 300.0 + site + rng.uniform(-0.6, 0.6, site.shape) * A0
    cls, out = _pairs(lib, xi, xj, z, z)
    r = np.linalg.norm(xi - xj, axis=1)
    assert ((cls != 0) == (r < A0 * RCF)).all()


@pytest.mark.parametrize("nr,scale", [(80, 1.0), (5000, 1e6)])
def test_tables_that_do_not_suit_it_are_refused(lib, wl, tmp_path, nr, scale):
    """Coarse tables (no accurate quartic per interval) and densities far from the scale of F'."""
    F, rho, rphi, drho, dr = wl.potential_tables(wl.PotentialSpec(n_ele=1, nr=nr))
    path = tmp_path / "p.setfl"
    body = np.concatenate([F[0], rho[0] * scale, rphi[0]])
    path.write_text(f"\n\n\n1 Fe\n{len(F[0])} {drho!r} {nr} {dr!r} {CUTOFF!r}\n26 55.845 {A0} bcc\n" +
                    "\n".join(repr(float(v)) for v in body) + "\n")
    assert _open(lib, str(path)) == 0
