"""Autotuning leaves the steps their group candidate lists, in boxes of split passes and of whole-group ones, on the
first call and from the cache, and changes no bits."""
import numpy as np
import pytest

from test_gpu_parity import A0, RCF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("cells", [(20, 20, 20), (52, 50, 51)])  # 500 and 8288 groups of 32 sites
def test_steps_after_autotune_use_the_lists(pkg, wl, potentials, gpu_lib, prec, cells):
    atoms = wl.build_state(cells, A0, RCF, temperature=300.0, seed=17, cu_frac=0.03)
    out = []
    for tuned in (False, True, True):
        ctx = pkg.Context(cells, A0, RCF, precision=prec)
        ctx.pot_init_setfl(potentials["fecuni"])
        ctx.upload(atoms)
        ctx.prepare()
        if tuned:
            t = ctx.autotune(reps=1)
            assert t["rho_apt"] == t["force_apt"] == 1
        before = ctx.skin_stats()[0]
        ctx.simulate(6)
        assert ctx.skin_stats()[0] == before + 6
        out.append(ctx.download()[0])
        ctx.close()
    for got in out[1:]:
        for f in ("x", "v", "f", "rho", "df"):
            assert np.array_equal(got[f], out[0][f]), f


@pytest.mark.parametrize("pot,cells", [("fe", (99, 100, 101)), ("fecuni", (99, 100, 101)), ("fe", (70, 70, 70))])  # 512, 256, 256
def test_default_blocks_keep_the_bits(pkg, wl, potentials, gpu_lib, pot, cells):
    """The mixed force pass's default block follows from the box and the potential, and changes no bits."""
    atoms = wl.build_state(cells, A0, RCF, temperature=300.0, seed=6)
    out = []
    for tune in (None, (1, 512, 1, 256), (1, 512, 1, 512)):
        ctx = pkg.Context(cells, A0, RCF, precision="mixed")
        if tune:
            ctx.set_tuning(*tune)
        ctx.pot_init_setfl(potentials[pot])
        ctx.upload(atoms)
        ctx.prepare()
        ctx.simulate(2)
        out.append(ctx.download()[0]["f"])
        ctx.close()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
