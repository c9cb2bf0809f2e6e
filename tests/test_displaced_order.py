"""firststep appends displaced atoms to a list in any order; the list manager puts them in scan order, by counting up
to 1024 of them and by ranges of local indices above."""
import numpy as np
import pytest

from test_gpu_parity import A0, RCF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 33, 1023, 1024, 1025, 4000])
def test_displaced_atoms_join_the_list_in_scan_order(pkg, orc, wl, potentials, gpu_lib, count):
    cells = (14, 13, 15)
    atoms = wl.build_state(cells, A0, RCF, temperature=100.0, seed=count)
    loc = wl.local_slot_indices(cells, RCF)
    rng = np.random.default_rng(count)
    moved = loc[rng.choice(loc.size, count, replace=False)]
    # past the middle between two sites along x: nearest a site that is occupied unless its atom moved as well
    atoms["x"][moved, 0] += 0.55 * A0
    ref = orc.OracleSim(cells, A0, RCF, potentials["fe"], dt=0.001)
    ref.set_atoms(atoms)
    ref.decide()
    ctx = pkg.Context(cells, A0, RCF)
    ctx.pot_init_setfl(potentials["fe"])
    ctx.upload(atoms)
    ctx.phase(1)
    got, inter = ctx.download()
    ctx.close()
    want, wi = ref.get_atoms(), ref.get_inter()
    assert inter.size == wi.size > 0
    assert np.array_equal(inter["id"], wi["id"]) and np.array_equal(inter["x"], wi["x"])
    assert np.array_equal(got["id"][loc], want["id"][loc]) and np.array_equal(got["type"][loc], want["type"][loc])
