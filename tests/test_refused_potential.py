"""A potential that is refused leaves the one in use as it was."""
import numpy as np
import pytest

from test_gpu_parity import A0, RCF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("cells", [(7, 9, 8), (52, 50, 51)])  # split and whole-group passes
def test_refused_potential_changes_nothing(pkg, wl, potentials, gpu_lib, tmp_path, prec, cells):
    atoms = wl.build_state(cells, A0, RCF, temperature=300.0, seed=2, cu_frac=0.1, ni_frac=0.1)
    short = wl.write_setfl(str(tmp_path / "short.setfl"), wl.PotentialSpec(n_ele=1, cutoff=5.2, r_on=4.6))
    got = []
    for refused in (False, True):
        ctx = pkg.Context(cells, A0, RCF, precision=prec)
        ctx.pot_init_setfl(potentials["fecuni"])
        if refused:
            with pytest.raises(pkg.MgError):
                ctx.pot_init_setfl(short)
        ctx.upload(atoms)
        ctx.prepare()
        ctx.simulate(3)
        got.append(ctx.download()[0])
        ctx.close()
    for f in ("type", "x", "v", "f", "rho", "df"):
        assert np.array_equal(got[0][f], got[1][f]), f
