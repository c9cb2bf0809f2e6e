"""Whatever potential the fixed-point tables are made for, the forces they give are no further from the exact ones than the
FP64 loops', and the atoms of a crystal do not fall back to those: on the CPU, over density units, embedding and
pair strengths, knots, and crystals of each element."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory, pkg):
    so = str(tmp_path_factory.mktemp("fixerr") / "libfixerr.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(pkg.build.nvcc())), "include")
    src = os.path.join(ROOT, "misa-md_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-pthread", "-I", cuda, "-I", src,
                    "-o", so, os.path.join(ROOT, "tests", "fixed_point_error_support.cpp"), os.path.join(src, "mg_fixed.cpp"),
                    os.path.join(src, "mg_potential.cpp")], check=True)
    return ctypes.CDLL(so)


def _write(wl, path, n_ele, nr, density, embed, pair, second=1.0):
    """The density, with its unit, times `density`; the embedding and pair energies times the others; the second element's
    density alone times `second`."""
    F, rho, rphi, drho, dr = wl.potential_tables(wl.PotentialSpec(n_ele=n_ele, seed=5, nr=nr))
    lines = ["", "", "", "%d %s" % (n_ele, " ".join(("Fe", "Cu", "Ni")[:n_ele])), "%d %.17g %d %.17g 5.6" % (len(F[0]), drho * density, nr, dr)]
    for e, z in zip(range(n_ele), (26, 29, 28)):
        lines.append("%d 55.845 2.855 bcc" % z)
        lines += ["%.17g" % v for v in np.concatenate([np.asarray(F[e]) * embed, np.asarray(rho[e]) * density * (second if e == 1 else 1.0)])]
    for p in rphi:
        lines += ["%.17g" % v for v in np.asarray(p) * pair]
    path.write_text("\n".join(lines) + "\n")
    return str(path)


@pytest.mark.parametrize("n_ele,nr,density,embed,pair,fixed", [
    (1, 5000, 1.0, 1.0, 1.0, True), (3, 5000, 1.0, 1.0, 1.0, True), (1, 4500, 1.0, 1.0, 1.0, True), (1, 20000, 1.0, 1.0, 1.0, True),
    (1, 5000, 0.2, 1.0, 1.0, True), (3, 5000, 0.3, 1.0, 1.0, True), (1, 5000, 4.0, 1.0, 1.0, None), (1, 5000, 10.0, 1.0, 1.0, None),
    (3, 5000, 8.0, 1.0, 1.0, None), (1, 5000, 1.0, 0.1, 1.0, None), (1, 5000, 1.0, 6.0, 1.0, None), (1, 5000, 1.0, 1.0, 0.1, None),
    (1, 5000, 1.0, 1.0, 0.3, None), (1, 5000, 1.0, 1.0, 3.0, None),
    (1, 5000, 1.0, 10.0, 1.0, False)])  # F' of 1.2 at the crystal's density
def test_forces_are_no_less_exact_than_the_fp64_loops(lib, wl, tmp_path, n_ele, nr, density, embed, pair, fixed):
    path = _write(wl, tmp_path / "p.setfl", n_ele, nr, density, embed, pair)
    for spread in (0.02, 0.08):
        for pure in ((-1, 0, 1, 2) if n_ele == 3 else (-1,)):
            out = (ctypes.c_double * 6)()
            st = lib.force_errors(os.fsencode(path), ctypes.c_double(spread), pure, out)
            assert st >= 0 and fixed in (None, bool(st))
            if st:
                assert out[2] == 0
                assert out[1] <= out[0], (spread, pure, out[0], out[1], out[3])
                assert out[5] <= out[4], (spread, pure, out[4], out[5])


@pytest.mark.parametrize("second,embed,pair", [(0.3, 1.0, 1.0), (0.1, 0.3, 4.0), (0.03, 0.3, 4.0), (0.01, 0.1, 4.0), (3.0, 1.0, 1.0),
                                               (10.0, 1.0, 4.0)])
def test_elements_of_unlike_densities(lib, wl, tmp_path, second, embed, pair):
    """The sums of all elements have one unit, set by the largest density; crystals of the element with a smaller one."""
    path = _write(wl, tmp_path / "p.setfl", 3, 5000, 1.0, embed, pair, second)
    for pure in (-1, 0, 1, 2):
        out = (ctypes.c_double * 6)()
        st = lib.force_errors(os.fsencode(path), ctypes.c_double(0.06), pure, out)
        assert st >= 0
        if st:
            assert out[1] <= out[0] and out[5] <= out[4], (pure, list(out))
