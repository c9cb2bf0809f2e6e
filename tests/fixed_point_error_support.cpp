// Forces on the atoms of a thermal BCC crystal by the fixed-point pair arithmetic and by the FP64 loops' operations, against
// long double, for the CPU tests.
#include <cmath>
#include <random>

#include "mg_internal.h"

using namespace mg;
typedef long double ld;

struct Atom {
    double x[3];
    int type;
};
struct Pair {
    int j;
    double x[3];  // of the periodic image
};
template <class T>
static T value(const HostSpline &s, int m, T p) {
    return std::fma(std::fma(std::fma((T) s.c3[m], p, (T) s.c2[m]), p, (T) s.c1[m]), p, (T) s.c0[m]);
}
template <class T>
static T slope(const HostSpline &s, int m, T p) {
    return std::fma(std::fma((T) s.d2[m], p, (T) s.d1[m]), p, (T) s.d0[m]);
}
template <class T>
static int knot(T x, double inv, int n, T &p) {
    const int m = std::max(0, std::min((int) (x * (T) inv), n - 2));
    p = std::min(x * (T) inv - m, (T) 1);
    return m;
}

// spread: standard deviation of the displacements (A); pure: every atom's type (or -1: 80 / 10 / 10 %). Returns 0 where
// the tables are refused. out: rms errors of the force components by the FP64 operations and in fixed point; atoms whose
// F' is past the fixed-point bound; the force sums' unit; rms errors of the densities, relative, by both.
extern "C" int force_errors(const char *path, double spread, int pure, double *out) {
    HostPotential P;
    std::string err;
    if (!read_setfl(path, P, err)) return -1;
    const double a0 = 2.855, rc = 5.6, rc2 = rc * rc;
    const int cells = 5;
    FixParams fp;
    FixTables tab;
    int ele[3];
    for (int t = 0; t < 3; t++) ele[t] = std::max(0, P.ele(type_key(t)));
    if (!build_fixed(P, ele, a0, rc / a0, 116, fp, tab, false)) return 0;
    std::mt19937_64 g(5);
    auto uniform = [&] { return (double) (g() >> 11) * 0x1p-53; };
    std::vector<Atom> at;
    for (int k = 0; k < cells; k++)
        for (int j = 0; j < cells; j++)
            for (int i = 0; i < 2 * cells; i++) {
                Atom a;
                const double h = (i & 1) * 0.5, site[3] = {0.5 * i, j + h, k + h};
                for (int d = 0; d < 3; d++) {  // the sum of twelve: close to normal
                    double s = -6.0;
                    for (int q = 0; q < 12; q++) s += uniform();
                    a.x[d] = site[d] * a0 + spread * s;
                }
                const double t = uniform();
                a.type = P.n_ele == 1 ? 0 : pure >= 0 ? pure : t < 0.8 ? 0 : t < 0.9 ? 1 : 2;
                at.push_back(a);
            }
    const int n = (int) at.size();
    std::vector<std::vector<Pair>> near(n);
    for (int i = 0; i < n; i++)
        for (int j = 0; j < n; j++)
            for (int s = 0; s < 27; s++) {
                const int sh[3] = {s % 3 - 1, s / 3 % 3 - 1, s / 9 - 1};
                Pair p{j, {}};
                double r2 = 0.0;
                for (int d = 0; d < 3; d++) {
                    p.x[d] = sh[d] ? at[j].x[d] + sh[d] * (cells * a0) : at[j].x[d];
                    r2 += (at[i].x[d] - p.x[d]) * (at[i].x[d] - p.x[d]);
                }
                if ((j != i || s != 13) && r2 < 1.01 * rc2) near[i].push_back(p);
            }
    const double inv = P.rho[0].inv_delta;
    auto fixed_r2 = [&](const Atom &a, const Pair &b, FixDelta &d) {
        i64 v[3];
        for (int q = 0; q < 3; q++)
            v[q] = (i64) ((uint64_t) fix_coord(a.x[q], fp.kx) + (uint64_t) kFixBias - (uint64_t) fix_coord(b.x[q], fp.kx));
        d = fix_delta(v[0], v[1], v[2]);
        return fix_r2(d, fp.b0);
    };
    auto r2_of = [](const Atom &a, const Pair &b, auto *d) {
        for (int q = 0; q < 3; q++) d[q] = std::remove_reference_t<decltype(*d)>(a.x[q]) - b.x[q];
        return std::fma(d[2], d[2], std::fma(d[1], d[1], d[0] * d[0]));
    };
    std::vector<double> df(n), dfx(n);
    std::vector<ld> dfl(n);
    int past = 0;
    ld r64 = 0.0L, rfx = 0.0L, rr = 0.0L;
    for (int i = 0; i < n; i++) {
        double rho = 0.0, close = 0.0, d[3], p;
        ld rhol = 0.0L, dl[3], pl;
        i64 sum = 0;
        for (const Pair &b : near[i]) {
            const HostSpline &s = P.rho[ele[at[b.j].type]];
            const double r2 = r2_of(at[i], b, d);
            const int m = knot(r2 * (1.0 / std::sqrt(r2)), inv, P.nr, p);
            if (r2 < rc2) rho += value(s, m, p);
            const ld r2l = r2_of(at[i], b, dl);
            const int ml = knot(std::sqrt(r2l), inv, P.nr, pl);
            if (r2l < (ld) rc2) rhol += value(s, ml, pl);
            FixDelta fd;
            const i64 f2 = fixed_r2(at[i], b, fd);
            int mf;
            if ((uint64_t) (f2 - fp.lo) < (uint64_t) (fp.rc2 - fp.lo)) {
                const FixCoord t = fix_locate(fp, f2, mf);
                sum += fix_poly(tab.rho[(size_t) at[b.j].type * fp.nr1 + mf], t, fp.e3_rho);
            } else if ((uint64_t) f2 < (uint64_t) fp.lo) {
                close += value(s, m, p);
            }
        }
        const HostSpline &F = P.F[ele[at[i].type]];
        int m = knot(rho, F.inv_delta, P.nrho, p);
        df[i] = slope(F, m, p);
        const double rhox = (double) sum * fp.rho_unit + close;
        r64 += ((ld) rho - rhol) * ((ld) rho - rhol);
        rfx += ((ld) rhox - rhol) * ((ld) rhox - rhol);
        rr += rhol * rhol;
        m = knot(rhox, F.inv_delta, P.nrho, p);
        dfx[i] = slope(F, m, p);
        m = knot(rhol, F.inv_delta, P.nrho, pl);
        dfl[i] = slope(F, m, pl);
        past += fix_df(fp, dfx[i]) == kFixBadDf;
    }
    ld e64 = 0.0L, efx = 0.0L;
    for (int i = 0; i < n; i++) {
        const int ti = at[i].type;
        double f[3] = {0.0, 0.0, 0.0}, close[3] = {0.0, 0.0, 0.0}, d[3], p;
        ld fl[3] = {0.0L, 0.0L, 0.0L}, dl[3], pl;
        i64 sum[3] = {0, 0, 0};
        const i64 dfb = fix_df(fp, dfx[i]) + kFixBias;
        for (const Pair &b : near[i]) {
            const int tj = at[b.j].type;
            const HostSpline &z = P.z2[HostPotential::pair_index(ele[ti], ele[tj])], &si = P.rho[ele[ti]], &sj = P.rho[ele[tj]];
            const double r2 = r2_of(at[i], b, d), ri = 1.0 / std::sqrt(r2);
            const int m = knot(r2 * ri, inv, P.nr, p);
            const double phi = value(z, m, p) * ri, phip = slope(z, m, p) * ri - phi * ri;
            auto pair = [&](double di, double dj) { return -(di * slope(sj, m, p) + dj * slope(si, m, p) + phip) * ri; };
            if (r2 < rc2)
                for (int q = 0; q < 3; q++) f[q] = std::fma(d[q], pair(df[i], df[b.j]), f[q]);
            const ld r2l = r2_of(at[i], b, dl), rl = std::sqrt(r2l);
            const int ml = knot(rl, inv, P.nr, pl);
            const ld pairl = -(dfl[i] * slope(sj, ml, pl) + dfl[b.j] * slope(si, ml, pl) + (slope(z, ml, pl) - value(z, ml, pl) / rl) / rl) / rl;
            if (r2l < (ld) rc2)
                for (int q = 0; q < 3; q++) fl[q] += dl[q] * pairl;
            FixDelta fd;
            const i64 f2 = fixed_r2(at[i], b, fd);
            if ((uint64_t) (f2 - fp.lo) < (uint64_t) (fp.rc2 - fp.lo)) {
                int mf;
                const FixCoord t = fix_locate(fp, f2, mf);
                const FixPoly *rec = &tab.zg[2 * ((size_t) (ti * 3 + tj) * fp.nr1 + mf)];
                const i64 gj = fix_poly(rec[0], t, fp.e3_g), dfj = fix_df(fp, dfx[b.j]), both = dfb + dfj, djb = dfj + kFixBias;
                i64 v = fix_poly(rec[1], t, fp.e3_h);
                if (tj == ti) {
                    v = fix_mul_add(fix_hi(both), fix_lo(both), fix_hi(gj), fix_lo(gj), v);
                } else {
                    const i64 gi = fix_poly(tab.zg[2 * ((size_t) (tj * 3 + ti) * fp.nr1 + mf)], t, fp.e3_g);
                    v = fix_mul_add(fix_hi(dfb), fix_lo(dfb), fix_hi(gj), fix_lo(gj), v);
                    v = fix_mul_add(fix_hi(djb), fix_lo(djb), fix_hi(gi), fix_lo(gi), v);
                }
                sum[0] = fix_mul_add(fd.xh, fd.xl, fix_hi(v), fix_lo(v), sum[0]);
                sum[1] = fix_mul_add(fd.yh, fd.yl, fix_hi(v), fix_lo(v), sum[1]);
                sum[2] = fix_mul_add(fd.zh, fd.zl, fix_hi(v), fix_lo(v), sum[2]);
            } else if ((uint64_t) f2 < (uint64_t) fp.lo) {
                for (int q = 0; q < 3; q++) close[q] = std::fma(d[q], pair(dfx[i], dfx[b.j]), close[q]);
            }
        }
        for (int q = 0; q < 3; q++) {
            const ld a = (ld) f[q] - fl[q], c = (ld) (-(double) sum[q] * fp.f_unit + close[q]) - fl[q];
            e64 += a * a;
            efx += c * c;
        }
    }
    out[0] = (double) std::sqrt(e64 / (3 * n));
    out[1] = (double) std::sqrt(efx / (3 * n));
    out[2] = past;
    out[3] = fp.f_unit;
    out[4] = (double) std::sqrt(r64 / rr);
    out[5] = (double) std::sqrt(rfx / rr);
    return 1;
}
