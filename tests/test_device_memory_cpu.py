"""Boxes near the device's memory, on a fake device: the FP64 form's fixed-point arrays (72 bytes a slot) are taken only
beside what a call needs, and given back for a later call that needs their room."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
A0, RCF = 2.855, 5.6 / 2.855
CELLS = (40, 40, 40)
RECORD, FIX = 104, 72  # bytes a slot: the slot array's records, and the fixed-point arrays
SLACK = 4 << 20        # the tables and more


@pytest.fixture(scope="module")
def lib(tmp_path_factory, pkg):
    d = tmp_path_factory.mktemp("fake")
    cuda = os.path.join(os.path.dirname(os.path.dirname(pkg.build.nvcc())), "include")
    src = os.path.join(ROOT, "misa-md_gb300", "csrc")
    gxx = ["g++", "-O1", "-std=c++17", "-fPIC", "-pthread", "-I", cuda, "-I", src]
    objs = []
    for f in [os.path.join(ROOT, "tests", "fake_device_support.cpp")] + [
            os.path.join(src, n) for n in ("mg_api.cpp", "mg_fixed.cpp", "mg_potential.cpp", "mg_dump.cpp")]:
        objs.append(str(d / (os.path.basename(f) + ".o")))
        subprocess.run(gxx + ["-c", "-o", objs[-1], f], check=True)
    names = subprocess.run(["nm", "-u"] + objs, capture_output=True, text=True, check=True).stdout
    have = set(re.findall(r" [TW] (\w+)", subprocess.run(["nm"] + objs, capture_output=True, text=True, check=True).stdout))
    want = {n for n in re.findall(r" U (\w+)", names) if n not in have and (n.startswith("cuda") or "2mg" in n)}
    stubs = d / "stubs.c"
    stubs.write_text("".join(f"long {n}(void) {{ return 0; }}\n" for n in sorted(want)))
    subprocess.run(["gcc", "-fPIC", "-c", "-o", str(d / "stubs.o"), str(stubs)], check=True)
    so = str(d / "libfake.so")
    subprocess.run(["g++", "-shared", "-pthread", "-Wl,--no-undefined", "-o", so, str(d / "stubs.o")] + objs, check=True)
    lib = ctypes.CDLL(so)
    lib.fake_used.restype = ctypes.c_size_t
    lib.fake_limit.argtypes = [ctypes.c_size_t]
    lib.fake_largest.argtypes = [ctypes.c_size_t]
    lib.mg_last_error.restype = ctypes.c_char_p
    yield lib
    lib.fake_limit(2**63)


class Ctx:
    def __init__(self, lib, wl, pot, limit):
        self.lib, self.h = lib, ctypes.c_void_p()
        Sx, Sy, Sz = wl.grid(CELLS, RCF)[:3]
        self.n = Sx * Sy * Sz
        lib.fake_limit(2**63)
        self.start = lib.fake_used()
        box = (ctypes.c_int64 * 3)(*CELLS)
        assert lib.mg_create(box, ctypes.c_double(A0), ctypes.c_double(RCF), 0, ctypes.c_int64(256), ctypes.byref(self.h)) == 0
        assert lib.mg_pot_init_setfl(self.h, os.fsencode(pot)) == 0
        self.atoms = np.zeros(self.n * RECORD, dtype=np.uint8)
        self.base = lib.fake_used()
        lib.fake_limit(self.base + limit(self.n))

    def call(self, name, *args):
        return getattr(self.lib, name)(self.h, *args)

    def upload(self):
        return self.call("mg_upload", self.atoms.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(self.n), None, ctypes.c_int64(0))

    def step_host(self):
        n = ctypes.c_int64(0)
        return self.call("mg_step_host", self.atoms.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(self.n), None,
                         ctypes.c_int64(0), ctypes.byref(n), ctypes.c_int64(1))

    def taken(self):
        return self.lib.fake_used() - self.base

    def close(self):
        assert self.call("mg_destroy") == 0
        assert self.lib.fake_used() == self.start


@pytest.mark.parametrize("room,fixed", [(RECORD, False), (RECORD + 40, False), (RECORD + FIX, True)])
def test_upload_needs_no_more_than_the_slot_array(lib, wl, potentials, room, fixed):
    c = Ctx(lib, wl, potentials["fe"], lambda n: n * room + SLACK)
    assert c.upload() == 0, c.call("mg_last_error")
    assert (c.taken() > c.n * RECORD + c.n * FIX) == fixed
    c.close()


def test_host_step_takes_the_fixed_point_arrays_room(lib, wl, potentials):
    """The overlapped host step keeps its input: a second slot array."""
    c = Ctx(lib, wl, potentials["fe"], lambda n: n * 2 * RECORD + SLACK)
    assert c.upload() == 0
    assert c.taken() > c.n * RECORD + c.n * FIX
    assert c.call("mg_set_host_pipeline", 8) == 0
    for _ in range(2):
        assert c.step_host() == 0, c.call("mg_last_error")
    assert 2 * RECORD * c.n <= c.taken() < 2 * RECORD * c.n + SLACK
    c.close()


def test_dump_takes_the_fixed_point_arrays_room(lib, wl, potentials, tmp_path):
    c = Ctx(lib, wl, potentials["fe"], lambda n: n * RECORD + n * FIX + SLACK)
    assert c.upload() == 0
    assert c.taken() > c.n * RECORD + c.n * FIX
    lib.fake_limit(c.base + c.taken() + c.n * 30)  # of two frames' 64 bytes or more an atom
    d = ctypes.c_void_p()
    assert c.call("mg_dump_open", os.fsencode(str(tmp_path / "d.bin")), 0, ctypes.c_int64(0), ctypes.byref(d)) == 0
    assert lib.mg_dump_close(d) == 0
    c.close()


@pytest.mark.parametrize("largest", [1000, 50000, 300000])  # bytes; the tables and what they are made from take more
def test_no_host_memory_for_the_tables(lib, wl, potentials, largest):
    c = Ctx(lib, wl, potentials["fe"], lambda n: n * (RECORD + FIX) + SLACK)
    lib.fake_largest(largest)
    st = c.upload()
    lib.fake_largest(2**63)
    assert st == 0, c.call("mg_last_error")
    assert c.taken() < RECORD * c.n + SLACK
    c.close()
