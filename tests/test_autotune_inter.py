"""Autotuning times passes on the resident state; with inter atoms in the box it leaves their shares of the lattice
atoms' densities and forces in place."""
import numpy as np
import pytest

from test_gpu_parity import A0, RCF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("cells", [(12, 11, 13), (52, 50, 51)])
def test_autotune_with_inter_atoms(pkg, wl, potentials, gpu_lib, prec, cells):
    atoms = wl.build_state(cells, A0, RCF, temperature=300.0, seed=23, ni_frac=0.03)
    loc = wl.local_slot_indices(cells, RCF)
    for k in (17, 400, 901):  # to an octahedral interstice
        atoms["x"][loc[k]] += A0 * np.array([0.5, 0.5, 0.0])
    out = []
    for tuned in (False, True):
        ctx = pkg.Context(cells, A0, RCF, precision=prec)
        ctx.pot_init_setfl(potentials["fecuni"])
        ctx.set_timestep(0.0002)
        ctx.upload(atoms)
        ctx.prepare()
        ctx.simulate(2)
        if tuned:
            ctx.autotune(reps=1)
        a, inter = ctx.download()
        parts = [a[f].tobytes() for f in ("x", "v", "f", "rho", "df")] + [inter.tobytes()]
        ctx.simulate(3)
        a, inter = ctx.download()
        assert inter.size > 0
        out.append(parts + [a[f].tobytes() for f in ("x", "v", "f", "rho", "df")] + [inter.tobytes()])
        ctx.close()
    assert out[0] == out[1]
