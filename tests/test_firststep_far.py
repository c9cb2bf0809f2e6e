"""firststep as a phase of its own need not be followed by decide: an atom it takes far from its site is then still the
atom it is to the passes, wherever its coordinates would wrap to in the FP64 form's fixed-point records."""
import numpy as np
import pytest

from test_gpu_parity import A0, F64_TOL, RCF

pytestmark = pytest.mark.gpu


def _sums(ctx, slots, loc, df=None):
    """rho, or (with df) the force, of the local slots over their candidates, by the potential's splines in numpy."""
    rho, z, sx = ctx.pot_spline(1, 0), ctx.pot_spline(2, 0, 0), ctx.grid[0]
    inv = rho[1, 4] / rho[1, 1]
    out = np.zeros((loc.size, 3) if df is not None else loc.size)
    for par in (0, 1):
        mine = np.flatnonzero((loc % sx) % 2 == par)
        i = loc[mine]
        j = i[:, None] + ctx.nei_offsets(4 + par)
        d = slots["x"][i][:, None] - slots["x"][j]
        r = np.sqrt((d * d).sum(axis=2))
        use = (r < A0 * RCF) & (slots["type"][j] >= 0)
        r = np.where(use, r, 3.0)
        m = np.clip((r * inv).astype(int), 0, len(rho) - 2)
        p = r * inv - m
        cubic = lambda t: t[m, 0] + p * (t[m, 1] + p * (t[m, 2] + p * t[m, 3]))  # noqa: E731
        slope = lambda t: t[m, 4] + p * (t[m, 5] + p * t[m, 6])  # noqa: E731
        if df is None:
            out[mine] = np.where(use, cubic(rho), 0.0).sum(axis=1)
            continue
        f = (df[i][:, None] + df[j]) * slope(rho) + (slope(z) - cubic(z) / r) / r
        out[mine] = -(np.where(use, f / r, 0.0)[:, :, None] * d).sum(axis=1)
    return out


@pytest.mark.parametrize("way", [3.0, 31.9, 32.0, 33.5])  # A; the records' coordinates repeat after 32 A
def test_passes_after_a_firststep_without_decide(pkg, wl, potentials, gpu_lib, way):
    cells = (14, 7, 8)
    a = wl.build_state(cells, A0, RCF, temperature=100.0, seed=4)
    loc = wl.local_slot_indices(cells, RCF)
    k = loc[3 * 2 * 14 * 7 + 3 * 2 * 14 + 1]  # a corner site near the lower end along x
    ctx = pkg.Context(cells, A0, RCF)
    ctx.pot_init_setfl(potentials["fe"])
    ctx.set_timestep(0.001)
    a["v"][:], a["f"][:] = 0.0, 0.0
    a["v"][k, 0] = way / 0.001
    ctx.upload(a)
    for phase in (0, 4, 5):
        ctx.phase(phase)
    got = ctx.download()[0]
    rho, f = _sums(ctx, got, loc), _sums(ctx, got, loc, got["df"])
    ctx.close()
    if way > 20.0:
        assert got["rho"][k] == 0.0 and not got["f"][k].any()
    # both evaluate r / dr (up to 5000) to 2^-53, so a pair's terms agree to 1e-12 of the largest
    assert np.abs(got["rho"][loc] - rho).max() < F64_TOL + 1e-11 * np.abs(rho).max()
    assert np.abs(got["f"][loc] - f).max() < F64_TOL + 1e-11 * np.abs(f).max()
