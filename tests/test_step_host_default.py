"""Host steps with the number of chunks left to the box's size (none, the staged form's two and four, the overlapped form's
six and eight) against the unpipelined path, bit for bit."""
import numpy as np
import pytest

from test_step_host import A0, RCF

pytestmark = pytest.mark.gpu


# slots of 104 bytes: 12, 20, 63, 137 and 245 MB
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cells", [(33, 31, 32), (40, 40, 40), (64, 63, 60), (60, 60, 146), (98, 101, 99)])
def test_default_chunks_are_bit_identical(pkg, wl, potentials, gpu_lib, precision, cells):
    a0 = wl.build_state(cells, A0, RCF, temperature=400.0, seed=3, cu_frac=0.05)
    out = []
    for default in (True, False):
        ctx = pkg.Context(cells, A0, RCF, precision=precision, inter_capacity=1024)
        ctx.pot_init_setfl(potentials["fecuni"])
        ctx.set_timestep(0.001)
        if not default:
            ctx.set_host_pipeline(0)
        a, inter, n = a0.copy(), np.zeros(16, dtype=pkg.ATOM_DTYPE), 0
        for _ in range(2):
            n = ctx.step_host(a, inter, n, 1)
        assert n == 0
        out.append(a)
        ctx.close()
    assert out[0].tobytes() == out[1].tobytes()
