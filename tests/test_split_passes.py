"""The lattice passes of small boxes split a 32-site group's candidates over the warps of a block (8, 4, 2 or none,
by the groups in flight). The split changes the schedule, not the sums: the FP64 form adds integers and the mixed
form adds the same terms in the same order, so every split gives the same bits. A batch counts a
member's groups once for each member, so the same box runs with fewer warps in a larger batch."""
import numpy as np
import pytest

from test_gpu_parity import A0, RCF

pytestmark = pytest.mark.gpu

FIELDS = ("id", "type", "x", "v", "f", "rho", "df")


def _ctx(pkg, pot, cells, atoms, prec, kick=None):
    ctx = pkg.Context(cells, A0, RCF, precision=prec, inter_capacity=2048)
    ctx.pot_init_setfl(pot)
    ctx.set_timestep(0.001)
    ctx.upload(atoms)
    ctx.prepare()
    if kick:
        ctx.set_variable_timestep(0.01, 1e-5, 1e-3)
        ctx.collision_step([c // 2 for c in cells] + [0], np.array([1.0, 3.0, 5.0]) / 35**0.5, kick)
    return ctx


# 13x17x31: 430 groups of 32 sites, the last of each parity a short one; 9x10x14: 80; 24x25x27: 1014. On 152 SMs the
# members make them run with every number of split warps and with none.
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("cells,members,kick", [((9, 10, 14), (10,), None), ((13, 17, 31), (2, 4, 10, 24), None),
                                                ((13, 17, 31), (4, 10, 24), 400.0), ((24, 25, 27), (2, 5, 7), 800.0)])
def test_every_split_gives_the_same_bits(pkg, wl, potentials, gpu_lib, prec, cells, members, kick):
    pot = potentials["fecuni"]
    atoms = wl.build_state(cells, A0, RCF, temperature=600.0, seed=31, cu_frac=0.06, ni_frac=0.04)
    alone = _ctx(pkg, pot, cells, atoms, prec, kick)
    alone.simulate(25)
    want, inter = alone.download()
    clock = alone.clock()
    alone.close()
    for n in members:
        ctxs = [_ctx(pkg, pot, cells, atoms, prec, kick)]
        few = wl.build_state((6, 6, 6), A0, RCF, temperature=600.0, seed=5)
        ctxs += [_ctx(pkg, pot, (6, 6, 6), few, prec) for _ in range(n - 1)]
        batch = pkg.Batch(ctxs, steps_per_launch=5)
        batch.run(25)
        got, gi = ctxs[0].download()
        for f in FIELDS:
            assert np.array_equal(got[f], want[f]), (n, f)
        assert gi.size == inter.size and np.array_equal(gi["x"], inter["x"])
        assert ctxs[0].clock() == clock
        batch.close()
        for c in ctxs:
            c.close()


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("mixed", 1e-4)])
@pytest.mark.parametrize("cells", [(6, 6, 6), (7, 9, 11), (13, 17, 31), (24, 25, 27), (31, 33, 35)])
def test_split_passes_follow_the_oracle(pkg, orc, wl, potentials, gpu_lib, cells, prec, tol):
    # the tolerances of the parity tests on the force (eV/A) after a few steps
    atoms = wl.build_state(cells, A0, RCF, temperature=600.0, seed=8)
    ref = orc.OracleSim(cells, A0, RCF, potentials["fe"], dt=0.001)
    ref.set_atoms(atoms)
    ref.prepare()
    ref.simulate(3)
    want = ref.get_atoms()
    ctx = _ctx(pkg, potentials["fe"], cells, atoms, prec)
    ctx.simulate(3)
    got, _ = ctx.download()
    ctx.close()
    local = wl.local_slot_indices(cells, RCF)
    assert np.abs(got["f"][local] - want["f"][local]).max() <= tol
    assert np.array_equal(got["type"][local], want["type"][local])
