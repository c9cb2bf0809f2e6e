"""The overlapped host step with atoms farther from their site than the FP64 form's fixed-point records allow, and with
ghost records that nothing has brought up to date: bit for bit the unpipelined path, and so are the steps after it."""
import numpy as np
import pytest

from test_step_host import A0, RCF, _ctx, _prepared_state

pytestmark = pytest.mark.gpu
CELLS = (8, 8, 40)


def _both(pkg, pot, precision, a0, chunks):
    out = []
    for c in (chunks, 0):
        ctx = _ctx(pkg, CELLS, pot, precision, c)
        a, inter = a0.copy(), np.zeros(64, dtype=pkg.ATOM_DTYPE)
        n = ctx.step_host(a, inter, 0, 1)
        parts = [a.tobytes(), n, inter[:n].tobytes()]
        ctx.simulate(3)
        a, left = ctx.download()
        parts += [a.tobytes(), left.tobytes()]
        n = ctx.step_host(a, inter, 0, 1) if left.size == 0 else 0
        out.append(parts + [a.tobytes(), n])
        ctx.close()
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("plane", [6, 21, 37])
@pytest.mark.parametrize("d", [(0.7, 0.0, 0.0), (0.0, -0.7, 0.65), (5.6, 0.0, 0.0)])
def test_an_atom_far_from_its_site_voids_the_overlapped_step(pkg, wl, potentials, gpu_lib, precision, plane, d):
    """0.7 a0 is past the records' 0.6 a0; 5.6 a0 is half the period of their coordinates, where a vacancy's are (one is
    put there, and one elsewhere)."""
    a0, _ = _prepared_state(pkg, wl, CELLS, potentials["fecuni"], precision)
    loc = wl.local_slot_indices(CELLS, RCF)
    nxy = 2 * CELLS[0] * CELLS[1]
    for k in (plane * nxy + 77 + 10, plane * nxy + 40):
        a0["type"][loc[k]] = -1
        a0["v"][loc[k]] = 0.0
    a0["x"][loc[plane * nxy + 77]] += A0 * np.asarray(d)
    got, want = _both(pkg, potentials["fecuni"], precision, a0, 8)
    assert want[1] == 1
    assert got == want


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_stale_ghost_records_leave_the_overlapped_step_alone(pkg, wl, potentials, gpu_lib, precision):
    a0, _ = _prepared_state(pkg, wl, CELLS, potentials["fecuni"], precision)
    ghost = np.setdiff1d(np.arange(a0.size), wl.local_slot_indices(CELLS, RCF))
    late = ghost[ghost > a0.size // 2][::7]
    a0["type"][late] = 0
    a0["x"][late] = 1000.0
    got, want = _both(pkg, potentials["fecuni"], precision, a0, 8)
    assert want[1] == 0
    assert got == want
