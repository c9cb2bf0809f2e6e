"""Short inter-atom lists take paths of their own in the list manager: up to 32 entries, one warp finds what the border
exchange sends and ranks the bucket index; when the entries pass 32 from one dimension to the next, the block carries on.
The lists against the oracle's bit for bit, and the forces from the index."""
import numpy as np
import pytest

from test_gpu_parity import A0, F64_TOL, RCF, assert_records_equal

pytestmark = pytest.mark.gpu
CELLS = (10, 9, 11)


def _picks(low, high, face, middle):
    """Corner sites of cells at the low corner (three images in every direction: seven of each atom), the high one, a face
    (one image) and the middle (none)."""
    c = [(x, y, z) for z in range(3) for y in range(3) for x in range(3)]
    m = [(4 + x, 4 + y, 4 + z) for z in range(3) for y in range(2) for x in range(3)] + [(5, 4, 3), (4, 4, 3), (6, 4, 3)]
    f = [(0, 4, z) for z in range(3, 8)] + [(0, 5, z) for z in range(3, 8)]
    return c[:low] + [tuple(n - 1 - v for n, v in zip(CELLS, s)) for s in c[:high]] + f[:face] + m[:middle]


# entries before each dimension's exchange, and in the index: (4) 4 8 16 32; (5) 5 10 20 40; (8) 8 16 32 64; (9) 9 18 36;
# (16) 16 32 64; (17) 17 34; 11 with faces; and lists of 31, 32 and 33
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("low,high,face,middle", [(0, 0, 0, 1), (1, 0, 0, 0), (4, 0, 0, 0), (3, 1, 0, 0), (5, 0, 0, 0), (8, 0, 0, 0),
                                                  (4, 5, 0, 0), (9, 0, 0, 2), (16, 0, 0, 0), (9, 8, 0, 0), (3, 0, 8, 0), (1, 1, 10, 10),
                                                  (20, 11, 0, 0), (20, 2, 10, 0), (20, 3, 10, 0)])
def test_border_and_index_of_short_lists(pkg, orc, wl, potentials, gpu_lib, prec, low, high, face, middle):
    atoms = wl.build_state(CELLS, A0, RCF, temperature=50.0, seed=low + 31 * high)
    loc = wl.local_slot_indices(CELLS, RCF)
    picks = _picks(low, high, face, middle)
    for x, y, z in picks:  # nearest the occupied centre of its cell
        atoms["x"][loc[(z * CELLS[1] + y) * 2 * CELLS[0] + 2 * x]] += 0.3 * A0
    ref = orc.OracleSim(CELLS, A0, RCF, potentials["fe"], dt=0.001)
    ref.set_atoms(atoms)
    ctx = pkg.Context(CELLS, A0, RCF, precision=prec)
    ctx.pot_init_setfl(potentials["fe"])
    ctx.upload(atoms)
    fields = ("id", "type", "x", "v", "f", "rho")
    for phase, fn in ((1, ref.decide), (2, ref.exchange_inter), (3, ref.border_inter)):
        ctx.phase(phase)
        fn()
        got, inter = ctx.download()
        assert_records_equal(got[loc], ref.get_atoms()[loc], fields)
        assert_records_equal(inter, ref.get_inter(), fields)
    assert inter.size == len(picks)
    gi, wi = ctx.download_ghost_inter(), ref.get_ghost_inter()
    assert gi.size == wi.size
    assert np.array_equal(gi["type"], wi["type"]) and np.array_equal(gi["x"], wi["x"])
    ctx.phase(4)
    ref.exchange_atom_first()  # fixes the ghosts that the exchange brings up to date
    ctx.phase(5)
    ref.clear_force()
    ref.compute_eam()
    got, inter = ctx.download()
    want, winter = ref.get_atoms(), ref.get_inter()
    tol = F64_TOL if prec == "fp64" else 50 * 1e-4  # those of the parity tests with inter atoms
    assert np.abs(got["f"][loc] - want["f"][loc]).max() < tol
    assert np.abs(inter["f"] - winter["f"]).max() < tol
    ctx.close()
