"""A step's kernels differ by the timestep rule (variable: a step head before firststep; fixed: the list manager keeps
the clock), and several steps share a graph launch. Switching the rule, by a call or by a stage, and cutting a run into
launches of any length leave the clock, the dt history and the trajectory what single steps give."""
import numpy as np
import pytest

from test_gpu_parity import A0, RCF

pytestmark = pytest.mark.gpu
RULE = (0.01, 1e-5, 1e-3)


def _ctx(pkg, pot, cells, atoms, prec, single):
    ctx = pkg.Context(cells, A0, RCF, precision=prec)
    ctx.pot_init_setfl(pot)
    if single:
        ctx.set_step_fusion(0)
    ctx.upload(atoms)
    ctx.prepare()
    return ctx


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("run", [1, 3, 41])
def test_rule_switches_and_launch_lengths(pkg, wl, potentials, gpu_lib, prec, run):
    cells = (8, 9, 7)
    n = 2 * 8 * 9 * 7
    atoms = wl.build_state(cells, A0, RCF, temperature=600.0, seed=3)
    out = []
    for single in (False, True):
        ctx = _ctx(pkg, potentials["fe"], cells, atoms, prec, single)
        steps = 0
        for rule in ("fixed", "variable", "stages", "variable", "fixed"):
            if rule == "fixed":
                ctx.set_timestep(0.0007)
            elif rule == "variable":
                ctx.set_variable_timestep(*RULE)
            if rule == "stages":
                ctx.run_stages([{"steps": run, "step_length": 0.0005}], run, 0.001, n)
            elif single:
                for _ in range(run):
                    ctx.simulate(1)
            else:
                ctx.simulate(run)
            steps += run
            hist = ctx.dt_history()
            assert ctx.clock()[0] == steps == len(hist)
            if rule != "variable":
                assert np.all(hist[-run:] == (0.0007 if rule == "fixed" else 0.0005))
        a, _ = ctx.download()
        out.append((a.tobytes(), np.asarray(hist).tobytes(), ctx.clock()))
        ctx.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("temperature,kick,dt", [(1800.0, None, 0.001), (600.0, 300.0, 0.0002), (600.0, None, 0.001)])
def test_fp64_fused_bodies_give_the_bits_of_single_steps(pkg, wl, potentials, gpu_lib, temperature, kick, dt):
    """Hot crystals put pairs below the range of the tables (their distances come from the records, since a fused pass
    changes the positions in place); a kicked atom makes inter atoms come and go, which bodies are not fused with."""
    cells = (9, 8, 10)
    atoms = wl.build_state(cells, A0, RCF, temperature=temperature, seed=12, cu_frac=0.05)
    out = []
    for single in (False, True):
        ctx = _ctx(pkg, potentials["fecuni"], cells, atoms, "fp64", single)
        ctx.set_timestep(dt)
        if kick:
            ctx.collision_step([4, 4, 5, 0], np.array([1.0, 3.0, 5.0]) / 35**0.5, kick)
        for run in (40, 23, 1):
            ctx.simulate(run)
        a, inter = ctx.download()
        out.append((a.tobytes(), inter.tobytes(), ctx.clock()))
        ctx.close()
    assert out[0] == out[1]
