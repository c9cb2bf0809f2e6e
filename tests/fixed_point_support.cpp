// Host access to the fixed-point pair arithmetic (mg_fixed.h) for the CPU tests: the tables of a setfl
// file, and the functions of single pairs evaluated by the same integer operations as the kernels'.
#include <cmath>

#include "mg_internal.h"

using namespace mg;

static FixParams g_fp;
static FixTables g_tab;

extern "C" int fix_open(const char *path, double a0, double rcf, int n_part) {
    HostPotential hp;
    std::string err;
    if (!read_setfl(path, hp, err)) return -1;
    int ele[3];
    for (int t = 0; t < 3; t++) ele[t] = std::max(0, hp.ele(type_key(t)));
    return build_fixed(hp, ele, a0, rcf, n_part, g_fp, g_tab) ? 1 : 0;
}

// Per pair: positions xi, xj (3 doubles each), types. out[6 p ..]: rho_tj, rho_tj'/r, phi'/r, phi and r^2 (as
// the sum of two doubles).
// Returned class: 0 outside the cutoff, 1 inside the tables' range, 2 closer than it.
extern "C" void fix_pairs(int n, const double *xi, const double *xj, const int *ti, const int *tj, int *cls, double *out) {
    const FixParams &p = g_fp;
    for (int k = 0; k < n; k++) {
        i64 d[3];
        for (int q = 0; q < 3; q++)
            d[q] = (i64) ((uint64_t) fix_coord(xi[3 * k + q], p.kx) + (uint64_t) kFixBias - (uint64_t) fix_coord(xj[3 * k + q], p.kx));
        const i64 r2 = fix_r2(fix_delta(d[0], d[1], d[2]), p.b0);
        out[6 * k + 4] = std::ldexp((double) ((r2 - p.b0) >> 32), 96 - 2 * p.kx);
        out[6 * k + 5] = std::ldexp((double) ((r2 - p.b0) & 0xffffffff), 64 - 2 * p.kx);
        cls[k] = (uint64_t) r2 >= (uint64_t) p.rc2 ? 0 : (uint64_t) r2 < (uint64_t) p.lo ? 2 : 1;
        if (cls[k] != 1) continue;
        int m;
        const FixCoord t = fix_locate(p, r2, m);
        const FixPoly *zg = &g_tab.zg[2 * ((size_t) (ti[k] * 3 + tj[k]) * p.nr1 + m)];
        // units of the factors: the force unit is 2^-(kx + kf - 64), kf = kd + kg - 64
        const int kf = -(int) std::lround(std::log2(p.f_unit)) + 64 - p.kx, kg = kf - p.kd + 64;
        out[6 * k + 0] = (double) fix_poly(g_tab.rho[(size_t) tj[k] * p.nr1 + m], t, p.e3_rho) * p.rho_unit;
        out[6 * k + 1] = std::ldexp((double) (fix_poly(zg[0], t, p.e3_g) - kFixBias), -kg);
        out[6 * k + 2] = std::ldexp((double) (fix_poly(zg[1], t, p.e3_h) - kFixBias), -kf);
        out[6 * k + 3] = (double) fix_poly(g_tab.phi[(size_t) (ti[k] * 3 + tj[k]) * p.nr1 + m], t, p.e3_phi) * p.e_unit;
    }
}
