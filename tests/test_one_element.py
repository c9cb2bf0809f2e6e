"""The force passes leave the types out where every type has the same tables (a potential of one
element). A potential with that element's tables under three names takes the general passes; iron alone gives the
same operations in both, so the same bits."""
import numpy as np
import pytest

from test_gpu_parity import A0, RCF

pytestmark = pytest.mark.gpu


def _three_names(path, out):
    lines = open(path).read().split("\n")
    nrho, _, nr, _, _ = lines[4].split()
    header, numbers, rest = lines[5], " ".join(lines[6:]).split(), int(nrho) + int(nr)
    block, pair = "\n".join(numbers[:rest]), "\n".join(numbers[rest:rest + int(nr)])
    text = lines[:3] + ["3 Fe Cu Ni", lines[4]]
    for z in (26, 29, 28):
        text += [" ".join([str(z)] + header.split()[1:]), block]
    out.write_text("\n".join(text + [pair] * 6) + "\n")
    return str(out)


# 8116 groups with short last ones, and 62500 of 32 sites (the mixed form's wider blocks); 18, 430, 1014 and 3906 groups
# for the split passes
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("cells,steps", [((53, 50, 49), 21), ((100, 100, 100), 3), ((6, 6, 8), 21), ((13, 17, 31), 21),
                                         ((24, 25, 27), 21), ((40, 39, 40), 21)])
def test_one_element_gives_the_same_bits(pkg, wl, potentials, gpu_lib, tmp_path, prec, cells, steps):
    atoms = wl.build_state(cells, A0, RCF, temperature=900.0, seed=12)
    got = []
    for pot in (potentials["fe"], _three_names(potentials["fe"], tmp_path / "three.setfl")):
        ctx = pkg.Context(cells, A0, RCF, precision=prec)
        ctx.pot_init_setfl(pot)
        ctx.set_timestep(0.001)
        ctx.upload(atoms)
        ctx.prepare()
        ctx.simulate(steps)
        got.append(ctx.download()[0])
        ctx.close()
    for f in ("type", "x", "v", "f", "rho", "df"):
        assert np.array_equal(got[0][f], got[1][f]), f
    assert np.abs(got[0]["f"]).max() > 0.1
