"""The parts of a step that mg_kernel_times reports, on a fake device."""
import ctypes

import pytest

from test_device_memory_cpu import Ctx, lib  # noqa: F401  (the fixture)

PARTS = ["firststep", "inter_firststep", "inter_manage", "ghost_copy", "lat_rho", "inter_rho", "lat_df", "ghost_df", "lat_force",
         "inter_force", "secondstep"]


@pytest.mark.parametrize("cap", [32, 5, 0])
def test_parts_of_a_step(lib, wl, potentials, cap):  # noqa: F811
    c = Ctx(lib, wl, potentials["fe"], lambda n: 2**40)
    assert c.upload() == 0 and c.call("mg_prepare") == 0
    for timed in (False, True):
        if timed:
            assert c.call("mg_enable_timing", 1) == 0 and c.call("mg_simulate", ctypes.c_int64(3), 1) == 0
        n, ms, names = ctypes.c_int32(), (ctypes.c_double * 32)(*[-1.0] * 32), (ctypes.c_char_p * 32)()
        assert c.call("mg_kernel_times", ms, cap, ctypes.byref(n), names) == 0
        assert n.value == 11
        assert [s.decode() for s in names[:min(cap, 11)]] == PARTS[:cap]
        assert list(ms[:min(cap, 11)]) == [0.0] * min(cap, 11) and names[min(cap, 11)] is None
    c.close()
