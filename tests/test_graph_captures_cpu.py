"""Programs that switch between the fixed and the variable timestep rule capture each rule's steps once, alone and in a
batch; a change that voids captured steps voids those of both rules. On a fake device that counts the graphs."""
import ctypes

import numpy as np
import pytest

from test_device_memory_cpu import Ctx, lib  # noqa: F401  (the fixture)

pytestmark = pytest.mark.usefixtures("lib")


def _ctx(lib, wl, pot):  # noqa: F811
    c = Ctx(lib, wl, pot, lambda n: 2**40)
    assert c.upload() == 0 and c.call("mg_prepare") == 0
    return c


def _rule(c, variable):
    if variable:
        return c.call("mg_set_variable_timestep", *(ctypes.c_double(v) for v in (0.01, 1e-5, 1e-3)))
    return c.call("mg_set_timestep", ctypes.c_double(0.001))


@pytest.mark.parametrize("steps", [1, 80])
def test_simulate_captures_each_rule_once(lib, wl, potentials, steps):  # noqa: F811
    c = _ctx(lib, wl, potentials["fe"])
    graphs = 1 if steps == 1 else 2  # one body, and several
    start = lib.fake_graphs_made()
    made = []
    for k in range(6):
        assert _rule(c, k % 2) == 0
        assert c.call("mg_simulate", ctypes.c_int64(steps), 1) == 0
        made.append(lib.fake_graphs_made() - start)
    assert made == [graphs] + [2 * graphs] * 5
    assert c.call("mg_set_neighbour_skin", ctypes.c_double(0.1)) == 0
    for k in range(4):
        assert _rule(c, k % 2) == 0
        assert c.call("mg_simulate", ctypes.c_int64(steps), 1) == 0
    assert lib.fake_graphs_made() - start == 4 * graphs
    c.close()
    assert lib.fake_graphs_alive() == 0


def test_batch_captures_each_set_of_rules_once(lib, wl, potentials):  # noqa: F811
    cs = [_ctx(lib, wl, potentials["fe"]) for _ in range(2)]
    b = ctypes.c_void_p()
    start = lib.fake_graphs_made()
    assert lib.mg_batch_create((ctypes.c_void_p * 2)(*(c.h for c in cs)), 2, 4, ctypes.byref(b)) == 0
    made = []
    for rules in ((0, 0), (1, 1), (0, 0), (1, 1), (1, 0), (1, 1), (0, 0)):
        for c, r in zip(cs, rules):
            assert _rule(c, r) == 0
        assert lib.mg_batch_run(b, ctypes.c_int64(9), 1) == 0
        made.append((lib.fake_graphs_made() - start) // 2)  # four bodies, and one
    assert made == [1, 2, 2, 2, 3, 3, 4]                      # the last two sets are kept
    assert cs[0].call("mg_set_neighbour_skin", ctypes.c_double(0.1)) == 0
    for rules in ((0, 0), (1, 1)):
        for c, r in zip(cs, rules):
            assert _rule(c, r) == 0
        assert lib.mg_batch_run(b, ctypes.c_int64(9), 1) == 0
    assert (lib.fake_graphs_made() - start) // 2 == 6
    assert lib.mg_batch_destroy(b) == 0
    assert lib.fake_graphs_alive() == 0
    for c in reversed(cs):
        assert c.call("mg_destroy") == 0
