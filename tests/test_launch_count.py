"""The kernels of a step that mg_launches_per_step states: before a capture of the timestep rule in use as after it."""
import pytest

from test_gpu_parity import A0, RCF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_launches_per_step_by_rule(pkg, wl, potentials, gpu_lib, prec):
    cells = (7, 6, 8)
    for rules in (("fixed", "variable"), ("variable", "fixed")):
        ctx = pkg.Context(cells, A0, RCF, precision=prec)
        ctx.pot_init_setfl(potentials["fe"])
        ctx.upload(wl.build_state(cells, A0, RCF, temperature=300.0, seed=1))
        ctx.prepare()
        for rule in rules:
            if rule == "fixed":
                ctx.set_timestep(0.001)
            else:
                ctx.set_variable_timestep(0.01, 1e-5, 1e-3)
            stated = ctx.launches_per_step()
            ctx.simulate(1)
            assert stated == ctx.launches_per_step() == (8 if rule == "fixed" else 9)
        ctx.close()
