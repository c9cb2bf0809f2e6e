"""The FP64 form's fixed-point lattice passes at their edges, against the oracle: pairs closer than the tables
reach (a few, and more than a thread keeps), F'(rho) outside its fixed-point range, atoms too far from
their sites for the wrapped coordinates, vacancies, tables that the fixed-point form refuses; and bit for
bit across launch shapes and candidate lists, since the sums do not depend on their order."""
import numpy as np
import pytest

from test_gpu_parity import A0, RCF, local, make_pair

pytestmark = pytest.mark.gpu

CELLS = (8, 9, 10)


def _eam(pkg, orc, wl, pot, atoms, cells=CELLS):
    ctx, ref = make_pair(pkg, orc, wl, pot, cells, atoms)
    ctx.prepare()
    ref.prepare()
    got, _ = ctx.download()
    want = ref.get_atoms()
    ctx.close()
    loc = local(wl, cells)
    return got[loc], want[loc]


def _close(got, want):
    """The oracle's tiers (rho 1e-13, forces 1e-9 eV/A), the forces relative where close pairs make them large."""
    assert np.array_equal(got["type"], want["type"])
    live = want["type"] >= 0
    assert np.allclose(got["rho"][live], want["rho"][live], rtol=1e-13, atol=0)
    assert np.allclose(got["df"][live], want["df"][live], rtol=1e-12, atol=1e-15)
    big = np.maximum(1.0, np.abs(want["f"][live]).max(axis=1))[:, None]
    assert (np.abs(got["f"][live] - want["f"][live]) <= 1e-9 * big).all()


def _index(wl, cells, x, y, z):
    return (z * cells[1] + y) * 2 * cells[0] + x


@pytest.mark.parametrize("pot", ["fe", "fecuni"])
@pytest.mark.parametrize("gap", [0.3, 1.2, 1.9, 2.02, 2.06, 2.2])
def test_close_pairs(pkg, orc, wl, potentials, gpu_lib, pot, gap):
    """Corner and centre of one cell moved to a distance `gap` of each other, several cells at once."""
    atoms = wl.build_state(CELLS, A0, RCF, temperature=300.0, seed=3, cu_frac=0.2 if pot == "fecuni" else 0.0)
    loc = local(wl, CELLS)
    nn = np.sqrt(0.75) * A0
    for x, y, z in ((0, 0, 0), (6, 4, 5), (15, 8, 9), (8, 2, 1)):
        a = loc[_index(wl, CELLS, x - x % 2, y, z)]
        b = loc[_index(wl, CELLS, x - x % 2 + 1, y, z)]
        move = 0.5 * (nn - gap) / nn * 0.5 * A0 * np.ones(3)
        atoms["x"][a] += move
        atoms["x"][b] -= move
    _close(*_eam(pkg, orc, wl, potentials[pot], atoms))


@pytest.mark.parametrize("count", [4, 5, 8])
def test_many_close_pairs_of_one_atom(pkg, orc, wl, potentials, gpu_lib, count):
    """`count` of an atom's eight nearest neighbours drawn in to 1.9 A: a thread keeps four."""
    cells = CELLS
    atoms = wl.build_state(cells, A0, RCF, temperature=0.0, seed=3)
    loc = local(wl, cells)
    c = loc[_index(wl, cells, 9, 4, 5)]  # a body centre; its cube's corners
    corners = [loc[_index(wl, cells, 8 + 2 * i, 4 + j, 5 + k)] for i in (0, 1) for j in (0, 1) for k in (0, 1)]
    for s in corners[:count]:
        d = atoms["x"][s] - atoms["x"][c]
        atoms["x"][s] = atoms["x"][c] + d * (1.9 / np.linalg.norm(d))
    _close(*_eam(pkg, orc, wl, potentials["fe"], atoms))


def test_steep_embedding_of_few_neighbours(pkg, orc, wl, potentials, gpu_lib):
    """Atoms with one or two distant neighbours: rho far below the crystal's, F' outside its range."""
    atoms = wl.build_state(CELLS, A0, RCF, temperature=0.0, seed=3)
    loc = local(wl, CELLS)
    keep = {_index(wl, CELLS, *s) for s in ((4, 4, 5), (8, 4, 5), (9, 7, 8), (0, 0, 0), (15, 8, 9))}
    for k in range(loc.size):
        if k not in keep:
            atoms["type"][loc[k]] = -1
    rng = np.random.default_rng(5)
    atoms["x"][loc] += rng.uniform(-0.1, 0.1, (loc.size, 3))
    got, want = _eam(pkg, orc, wl, potentials["fe"], atoms)
    _close(got, want)
    assert np.abs(want["df"][want["type"] >= 0]).max() > 1.0


@pytest.mark.parametrize("shift", [0.61, 0.93, 32.0 / A0])
def test_atoms_far_from_their_sites(pkg, orc, wl, potentials, gpu_lib, shift):
    """An uploaded state before its first decide: an atom `shift` lattice constants from its site (32 A is
    the period of the wrapped coordinates)."""
    atoms = wl.build_state(CELLS, A0, RCF, temperature=300.0, seed=3)
    loc = local(wl, CELLS)
    atoms["x"][loc[_index(wl, CELLS, 7, 4, 5)], 0] += shift * A0
    atoms["type"][loc[_index(wl, CELLS, 2, 2, 2)]] = -1
    _close(*_eam(pkg, orc, wl, potentials["fe"], atoms))


@pytest.mark.parametrize("nr", [80, 600])
def test_coarse_tables(pkg, orc, wl, gpu_lib, tmp_path, nr):
    pot = wl.write_setfl(str(tmp_path / "p.setfl"), wl.PotentialSpec(n_ele=1, nr=nr))
    atoms = wl.build_state(CELLS, A0, RCF, temperature=300.0, seed=3)
    loc = local(wl, CELLS)
    atoms["x"][loc] += np.random.default_rng(2).uniform(-0.1, 0.1, (loc.size, 3))
    _close(*_eam(pkg, orc, wl, pot, atoms))


def test_lists_and_launch_shapes_give_the_same_bits(pkg, wl, potentials, gpu_lib):
    """Candidate lists, no lists (skin 0 rebuilds them, several sites per thread walk every candidate) and
    thread orders, over steps with rebuilds, vacancies and recombinations."""
    cells = (11, 9, 13)
    atoms = wl.build_state(cells, A0, RCF, temperature=900.0, seed=31, cu_frac=0.1, ni_frac=0.05)
    loc = local(wl, cells)
    atoms["type"][loc[7::211]] = -1
    atoms["x"][loc[100]] += 0.3 * A0 * np.array([1.0, 0.2, 0.1])
    states = []
    for skin, tune in ((None, None), (0.0, None), (0.4, (1, 128, 0, 256)), (None, (0, 512, 1, 128, 2, 4)),
                       (None, (1, 256, 1, 512))):
        ctx = pkg.Context(cells, A0, RCF, precision="fp64", inter_capacity=1024)
        ctx.pot_init_setfl(potentials["fecuni"])
        ctx.set_timestep(0.001)
        if skin is not None:
            ctx.set_neighbour_skin(skin)
        if tune:
            ctx.set_tuning(*tune)
        ctx.upload(atoms)
        ctx.prepare()
        ctx.simulate(40)
        states.append([a.tobytes() for a in ctx.download()])
        ctx.close()
    assert all(s == states[0] for s in states)
