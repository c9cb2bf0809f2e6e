"""The FP64 form at other lattice constants and cutoffs than the rest of the tests', whose scales the fixed-point tables
follow: a few steps against the oracle, in split and whole-group passes."""
import numpy as np
import pytest

from test_gpu_parity import F64_TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a0,cutoff,cells", [(2.855, 4.2, (7, 8, 9)), (3.165, 5.4, (9, 8, 8)), (3.3, 6.4, (8, 9, 7)),
                                             (2.2, 4.3, (9, 9, 9)), (4.3, 8.4, (8, 8, 9)), (3.165, 5.4, (50, 53, 51))])
def test_other_lattices_follow_the_oracle(pkg, orc, wl, gpu_lib, tmp_path, a0, cutoff, cells):
    rcf = cutoff / a0
    spec = wl.PotentialSpec(n_ele=1, cutoff=cutoff, r_on=cutoff - 0.6, lattice_const=a0,
                            params=[wl.EamParams(r0=2.65 / 2.855 * a0)])
    pot = wl.write_setfl(str(tmp_path / "p.setfl"), spec)
    atoms = wl.build_state(cells, a0, rcf, temperature=300.0, seed=13)
    steps = 3 if cells[0] < 20 else 1
    ref = orc.OracleSim(cells, a0, rcf, pot, dt=0.001)
    ref.set_atoms(atoms)
    ref.prepare()
    ref.simulate(steps)
    want = ref.get_atoms()
    ctx = pkg.Context(cells, a0, rcf)
    ctx.pot_init_setfl(pot)
    ctx.set_timestep(0.001)
    ctx.upload(atoms)
    ctx.prepare()
    ctx.simulate(steps)
    got, inter = ctx.download()
    ctx.close()
    loc = wl.local_slot_indices(cells, rcf)
    assert inter.size == ref.get_inter().size
    assert np.array_equal(got["type"][loc], want["type"][loc])
    assert np.abs(got["f"][loc] - want["f"][loc]).max() < F64_TOL
    assert np.abs(got["x"][loc] - want["x"][loc]).max() < 1e-12
