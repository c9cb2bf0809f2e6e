// Tables of the fixed-point pair arithmetic (mg_fixed.h): for every knot interval of the potential's r
// tables, the interval's own cubic as a polynomial in s = r^2 about the interval's centre.
//
// On interval m the spline is a cubic in p = r / dr - m, and r = r_c sqrt(1 + y) with y = (s - s_c) / s_c,
// |y| <= about 1 / (2 m). Composing the binomial series of sqrt(1 + y), (1 + y)^(-1/2) and their powers
// with the cubic gives the polynomial to y^5, and its last term is spread over the lower ones by the
// Chebyshev polynomial T5, which leaves a sixteenth of it as the error (2e-18 of the value at the
// nearest-neighbour distance for 5000 knots). The value at the centre is found in double-double arithmetic
// (T. J. Dekker, "A floating-point technique for extending the available precision", Numer. Math. 18,
// 1971) where it decides the value, so a coefficient is rounded once, to its integer. Coarse or rough tables
// do not meet the error bound that every record is checked against, and the FP64 loops stay in use for them.

#include <algorithm>
#include <array>
#include <cmath>
#include <future>

#include "mg_internal.h"

namespace mg {

namespace {

struct dd {
    double h, l;
    dd(double a = 0.0) : h(a), l(0.0) {}
    dd(double a, double b) : h(a), l(b) {}
};
dd quick(double a, double b) {
    const double s = a + b;
    return dd(s, b - (s - a));
}
dd operator+(dd a, dd b) {
    const double s = a.h + b.h, v = s - a.h;
    const double e = (a.h - (s - v)) + (b.h - v);
    return quick(s, e + (a.l + b.l));
}
dd operator-(dd a) { return dd(-a.h, -a.l); }
dd operator-(dd a, dd b) { return a + (-b); }
dd operator*(dd a, dd b) {
    const double p = a.h * b.h;
    return quick(p, std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
dd operator/(dd a, dd b) {
    const double q = a.h / b.h;
    const dd r = a - b * dd(q);
    const double q2 = r.h / b.h;
    const dd r2 = r - b * dd(q2);
    return quick(q, q2) + dd(r2.h / b.h);
}
dd root(dd a) {
    const double s = std::sqrt(a.h);
    const dd r = a - dd(s) * dd(s);
    return quick(s, r.h / (2.0 * s));
}
dd scaled(dd a, int k) { return dd(std::ldexp(a.h, k), std::ldexp(a.l, k)); }
// nearest integer; false when it does not fit
bool to_i64(dd a, i64 &out) {
    if (!(std::fabs(a.h) < 4.5e18)) return false;
    const double whole = std::nearbyint(a.h);
    out = (i64) whole + (i64) std::nearbyint((a.h - whole) + a.l);
    return true;
}

constexpr int kTerms = 6;  // powers 0..5 of y
struct Series {
    double c[kTerms];
};
Series mul(const Series &a, const Series &b) {
    Series r{};
    for (int i = 0; i < kTerms; i++)
        for (int j = 0; i + j < kTerms; j++) r.c[i + j] += a.c[i] * b.c[j];
    return r;
}
Series times(const Series &a, double f) {
    Series r;
    for (int i = 0; i < kTerms; i++) r.c[i] = a.c[i] * f;
    return r;
}
// (1 + y)^(e/2)
Series power(int e) {
    Series r;
    double c = 1.0;
    for (int i = 0; i < kTerms; i++) {
        r.c[i] = c;
        c = c * (e - 2.0 * i) / (2.0 * (i + 1));
    }
    return r;
}
// c0 + p (c1 + p (c2 + p c3)) of a series p, given its square and cube
Series cubic(const Series &p, const Series &p2, const Series &p3, double c0, double c1, double c2, double c3) {
    Series r;
    for (int i = 0; i < kTerms; i++) r.c[i] = c1 * p.c[i] + (c2 * p2.c[i] + c3 * p3.c[i]);
    r.c[0] += c0;
    return r;
}
dd cubic_at(dd p, double c0, double c1, double c2, double c3) { return dd(c0) + p * (dd(c1) + p * (dd(c2) + p * dd(c3))); }

// a distance on interval m, for the functions' values in closed form
struct Place {
    dd p, ir;  // the interval's coordinate and 1 / r
};
Place place(dd r, double inv_dr, int m) { return Place{r * dd(inv_dr) - dd((double) m), dd(1.0) / r}; }

enum { FN_RHO, FN_G, FN_H, FN_PHI };
// s: the density's spline (rho, rho'/r) or r phi's (phi'/r, phi)
dd value_at(const HostSpline &s, int m, int fn, const Place &q) {
    if (fn == FN_RHO) return cubic_at(q.p, s.c0[m], s.c1[m], s.c2[m], s.c3[m]);
    if (fn == FN_G) return cubic_at(q.p, s.d0[m], s.d1[m], s.d2[m], 0.0) * q.ir;
    const dd phi = cubic_at(q.p, s.c0[m], s.c1[m], s.c2[m], s.c3[m]) * q.ir;
    if (fn == FN_PHI) return phi;
    return (cubic_at(q.p, s.d0[m], s.d1[m], s.d2[m], 0.0) - phi) * (q.ir * q.ir);
}
// One interval: what every function's expansion about its centre shares.
struct Interval {
    int m;             // of the spline (the last one for the records past it)
    i64 sc;            // centre, in units of r^2
    Place at;          // centre
    double unit;       // y per unit of the interval coordinate
    double xm;         // half width in that coordinate
    Series p, p2, p3;  // the spline's coordinate and its powers, in y
    i64 check;         // a point to check the records at: its interval coordinate t and place
    Place check_at;
};
Series expanded(const HostSpline &s, int fn, const Interval &v) {
    static const Series inv1 = power(-1), inv2 = power(-2), inv3 = power(-3);
    const double ir = v.at.ir.h;
    const int m = v.m;
    if (fn == FN_G) return times(mul(cubic(v.p, v.p2, v.p3, s.d0[m], s.d1[m], s.d2[m], 0.0), inv1), ir);
    const Series c = cubic(v.p, v.p2, v.p3, s.c0[m], s.c1[m], s.c2[m], s.c3[m]);
    if (fn == FN_RHO) return c;
    if (fn == FN_PHI) return times(mul(c, inv1), ir);
    Series h = times(mul(cubic(v.p, v.p2, v.p3, s.d0[m], s.d1[m], s.d2[m], 0.0), inv2), ir * ir);
    const Series z = times(mul(c, inv3), ir * ir * ir);
    for (int i = 0; i < kTerms; i++) h.c[i] -= z.c[i];
    return h;
}

// largest exponent e with bound * 2^e <= 2^bits
int exponent_for(double bound, int bits) {
    int e;
    std::frexp(bound, &e);  // bound < 2^e
    return bits - e;
}

// the largest values of the functions from a knot on to the cutoff, over elements and pairs
struct Largest {
    double rho, g, h, phi, rg, rh;
};
// at[m]: from knot m on (m_from <= m <= nr - 2); one pass serves every inner end that is tried
std::vector<Largest> largest_from(const HostPotential &hp, int m_from) {
    std::vector<Largest> at(hp.nr - 1, Largest{});
    Largest v{};
    for (int m = hp.nr - 2; m >= m_from; m--) {
        const double r = m * hp.dr;
        for (int a = 0; a < hp.n_ele; a++) {
            const double g = std::fabs(hp.rho[a].d0[m]) / r;
            v.rho = std::max(v.rho, std::fabs(hp.rho[a].c0[m]));
            v.g = std::max(v.g, g);
            v.rg = std::max(v.rg, r * g);
            for (int b = 0; b <= a; b++) {
                const HostSpline &z = hp.z2[HostPotential::pair_index(a, b)];
                const double phi = z.c0[m] / r, h = std::fabs((z.d0[m] - phi) / (r * r));
                v.phi = std::max(v.phi, std::fabs(phi));
                v.h = std::max(v.h, h);
                v.rh = std::max(v.rh, r * h);
            }
        }
        at[m] = v;
    }
    return at;
}
int first_knot(double r_lo, double dr) { return std::max(1, (int) (r_lo / dr) - 1); }

}  // namespace

// A perfect crystal's neighbours of a site in the order the loops visit them (in half lattice constants, BCC: all even or
// all odd), and over the elements: the least density of crystals of one of them, and the least and the largest |F'(rho)|
// of an element on a site whose neighbours are of one.
struct Crystal {
    std::vector<std::array<int, 3>> near;
    double rho_least = HUGE_VAL, df_least = HUGE_VAL, df_most = 0.0;
};
static double distance_of(const std::array<int, 3> &n, double a0) {
    return 0.5 * a0 * std::sqrt((double) (n[0] * n[0] + n[1] * n[1] + n[2] * n[2]));
}
static double crystal_rho(const HostPotential &hp, const Crystal &c, double a0, int b) {
    const HostSpline &s = hp.rho[b];
    double rho = 0.0;
    for (const auto &n : c.near) {
        const double x = distance_of(n, a0) * s.inv_delta;
        const int m = std::min((int) x, hp.nr - 2);
        rho += cubic_at(dd(x - m), s.c0[m], s.c1[m], s.c2[m], s.c3[m]).h;
    }
    return rho;
}
static double embedding_df(const HostPotential &hp, int a, double rho) {
    const HostSpline &F = hp.F[a];
    const int m = std::max(0, std::min((int) (rho * F.inv_delta), hp.nrho - 2));
    return cubic_at(dd(std::min(rho * F.inv_delta - m, 1.0)), F.d0[m], F.d1[m], F.d2[m], 0.0).h;
}
static Crystal crystal_of(const HostPotential &hp, double a0, double rc) {
    Crystal c;
    const int n = 2 * ((int) (rc / a0) + 1);
    for (int k = -n; k <= n; k++)
        for (int j = -n; j <= n; j++)
            for (int i = -n; i <= n; i++)
                if (!(((i ^ j) | (j ^ k)) & 1) && (i || j || k) && distance_of({i, j, k}, a0) < rc) c.near.push_back({i, j, k});
    for (int b = 0; b < hp.n_ele; b++) {
        const double rho = crystal_rho(hp, c, a0, b);
        c.rho_least = std::min(c.rho_least, rho);
        if (!(rho <= (hp.nrho - 1) * hp.drho)) continue;  // past the embedding tables: no crystal to judge by
        for (int a = 0; a < hp.n_ele; a++) {
            const double df = std::fabs(embedding_df(hp, a, rho));
            c.df_least = std::min(c.df_least, df);
            c.df_most = std::max(c.df_most, df);
        }
    }
    return c;
}
// The FP64 loops' rms error in a component of the force on an atom: what each pair's roundings make of its force, near
// its crystal distance, against double-double arithmetic, and the roundings of the sum. The least over crystals of one
// element.
static double fp64_error(const HostPotential &hp, const Crystal &c, double a0, double rc) {
    const double dir[3] = {0.48, 0.6, 0.64}, inv = hp.rho[0].inv_delta;
    double least = HUGE_VAL;
    for (int a = 0; a < hp.n_ele; a++) {
        const HostSpline &s = hp.rho[a], &z = hp.z2[HostPotential::pair_index(a, a)];
        const double df2 = 2.0 * embedding_df(hp, a, crystal_rho(hp, c, a0, a));
        double sum = 0.0, part[3] = {0.0, 0.0, 0.0};
        int at = 0;
        for (const auto &n : c.near) {
            // distances within 2% of the crystal's, another for each neighbour
            const double r0 = distance_of(n, a0), want = r0 * (1.0 + 0.04 * (std::fmod(0.618034 * ++at, 1.0) - 0.5));
            const double x = want * dir[0], y = want * dir[1], w = want * dir[2];
            const double r2 = std::fma(w, w, std::fma(y, y, x * x));
            if (r2 >= rc * rc) continue;
            const double ri = 1.0 / std::sqrt(r2), r = r2 * ri;
            const int m = std::min((int) (r * inv), hp.nr - 2);
            const double p = r * inv - m;
            const double rhop = std::fma(std::fma(s.d2[m], p, s.d1[m]), p, s.d0[m]);
            const double phi = std::fma(std::fma(std::fma(z.c3[m], p, z.c2[m]), p, z.c1[m]), p, z.c0[m]) * ri;
            const double phip = std::fma(std::fma(z.d2[m], p, z.d1[m]), p, z.d0[m]) * ri - phi * ri;
            const double f = (df2 * rhop + phip) * ri;
            const Place q = place(root(dd(x) * dd(x) + dd(y) * dd(y) + dd(w) * dd(w)), inv, m);
            const double err = (dd(f) - (dd(df2) * value_at(s, m, FN_G, q) + value_at(z, m, FN_H, q))).h * r;
            sum += err * err;
            for (int d = 0; d < 3; d++) {
                part[d] += 0.5 * a0 * n[d] * f;
                const double unit = part[d] != 0.0 ? std::ldexp(1.0, std::ilogb(part[d]) - 52) : 0.0;
                sum += unit * unit / 12.0;
            }
        }
        least = std::min(least, std::sqrt(sum / 3.0));
    }
    return least;
}

// build_fixed for one inner end r_lo of the tables' range and F'(rho) in units of 2^-kd; exact: the FP64 loops' error in a
// force.
// depth: the scales only, whether the innermost intervals (where the quartics are at their worst) meet the bound, or
// everything into tab
enum Depth { SCALES, INNERMOST, TABLES };
static bool build_from(const HostPotential &hp, const int ele_of_type[3], double a0, double rcf, int n_part, double r_lo, int kd,
                       double exact, const Crystal &crystal, const std::vector<Largest> &largest, FixParams &fp, FixTables *tab,
                       bool want_phi, Depth depth) {
    fp = FixParams{};
    const double rc = a0 * rcf, dr = hp.dr;
    const int nr = hp.nr;
    if (nr < 64 || nr > 20000) return false;
    // Coordinates wrap at 2^63 units. Candidate sites lie within (rcf + 1) a0 and an atom within 0.6 a0 of
    // its site, so no difference wraps; a vacancy's coordinates are moved by half the period, after which
    // every component of its distance is above rc / sqrt(3).
    const double half = std::max((rcf + 2.2) * a0, (rcf + 1.6) * a0 + 0.6 * rc);
    fp.kx = exponent_for(half, 63);
    if (fp.kx < 1 || fp.kx > 110) return false;
    const int kr = 2 * fp.kx - 64;  // r^2 in units of 2^-kr
    fp.nr1 = nr + 1;
    // interval centres: ((2m + 1) dr / 2)^2, as (2m + 1)^2 << ks times a 31-bit constant
    const double kreal = std::ldexp(0.25 * dr * dr, kr);
    fp.ks = std::max(0, -exponent_for(kreal, 31));
    const double kc = std::nearbyint(std::ldexp(kreal, -fp.ks));
    const double last = 2.0 * nr + 1;
    if (!(kc >= 1048576.0) || kc >= 2147483647.0 || std::ldexp(last * last, fp.ks) >= 2147483647.0) return false;
    fp.k = (int) kc;
    // t of the widest interval, with room for a knot found from the single-precision root
    fp.sh = exponent_for(2.0 * kreal * last * 1.02, 63);
    if (fp.sh < 1 || fp.sh > 31) return false;
    fp.b0 = 1LL << (31 - fp.sh);
    if (!to_i64(scaled(dd(rc * rc), kr), fp.rc2)) return false;
    fp.rc2 += fp.b0;
    fp.to_knot = (float) (std::ldexp(1.0, 48 - fp.kx) / dr);
    fp.quarter = (float) std::ldexp(kc, fp.ks + fp.sh - 32);

    // the range of the tables: pairs closer than r_lo take the FP64 loops
    const int m_lo = first_knot(r_lo, dr);
    const int m_hi = nr - 2;
    if (m_lo + 8 > m_hi || !((m_lo + 1) * dr < rc)) return false;
    const double inv_dr = hp.rho[0].inv_delta;
    const Largest &top = largest[m_lo];
    const double rho_max = top.rho, g_max = top.g, h_max = top.h, phi_max = top.phi, rg_max = top.rg, rh_max = top.rh;
    if (!(rho_max > 0) || !(g_max > 0) || !(h_max > 0) || !std::isfinite(rho_max + g_max + h_max + phi_max))
        return false;
    const double room = 1.01;  // values between the knots
    // F'(rho) below 2^(60 - kd): |F' g| at the bound is the pair force of a bond at full embedding, so the
    // product's unit follows from both
    fp.kd = kd;
    const int kg = exponent_for(g_max * room, 62);
    const int kf = fp.kd + kg - 64;                 // pair factor (F'_i + F'_j) g + h
    const int kF = fp.kx + kf - 64;                 // force sums
    const double df2 = std::ldexp(2.0, 60 - fp.kd);  // bound of |F'_i| + |F'_j|
    const int krho = exponent_for(n_part * rho_max * room, 62);
    const int kphi = exponent_for(n_part * phi_max * room, 62);
    if ((df2 * g_max + h_max) * room >= std::ldexp(1.0, 62 - kf)) return false;
    if (n_part * (df2 * rg_max + rh_max) * room >= std::ldexp(1.0, 63 - kF)) return false;
    // The sums are to be no less exact than the FP64 loops'. Rms errors in thermal crystals: forces 2.3 to 2.5 units, densities
    // (all elements' in one unit, which the largest sets) 5.5 units against the loops' 2.1e-16 to 2.8e-16 of the density.
    if (2.5 * std::ldexp(1.0, -kF) > exact || 5.5 * std::ldexp(1.0, -krho) > 2.1e-16 * crystal.rho_least) return false;
    fp.rho_unit = std::ldexp(1.0, -krho);
    fp.e_unit = std::ldexp(1.0, -kphi);
    fp.f_unit = std::ldexp(1.0, -kF);
    fp.lo = (i64) (std::ldexp((m_lo + 1) * dr * (m_lo + 1) * dr, kr - 32) + 1.0) << 32;

    if (depth == SCALES) return true;
    const int m_end = depth == INNERMOST ? std::min(m_lo + 16, fp.nr1) : fp.nr1;

    // the intervals; the records past the last one (a cutoff at the table's end, found a knot too far)
    // continue its cubic
    auto distance = [&](i64 v) {
        return root(scaled(dd((double) (v >> 31)) * dd(2147483648.0) + dd((double) (v & 0x7fffffff)), -kr));
    };
    const Series sq = power(1);
    std::vector<Interval> iv(m_end);
    for (int m = m_lo; m < m_end; m++) {
        Interval &v = iv[m];
        v.m = std::min(m, m_hi);
        v.sc = -fix_centre_sub(fp, m, 0);
        const dd r = distance(v.sc);
        v.at = place(r, inv_dr, v.m);
        v.unit = std::ldexp(1.0 / (r.h * r.h), 63 - fp.sh - kr);
        v.xm = std::ldexp(kreal * (2.0 * m + 1) * 2.0, fp.sh - 63);
        v.p = times(sq, r.h * inv_dr);
        v.p.c[0] = v.at.p.h;
        v.p2 = mul(v.p, v.p);
        v.p3 = mul(v.p2, v.p);
        v.check = (i64) (kreal * (2.0 * m + 1) * 1.6) * (m % 2 ? 1 : -1);  // 0.8 of the half width
        v.check_at = place(distance(v.sc + v.check), inv_dr, v.m);
    }
    // The tables: one per element (rho, rho'/r) or element pair (phi'/r, phi), filled side by side. Only c0
    // needs more than double precision: the others are below 2^-9 of it.
    struct Table {
        int fn, kv;
        bool factor;       // the value is a factor of a product: c0 biased
        double fmax;
        const HostSpline *s;
        std::vector<FixPoly> out;
        std::vector<Series> w;
        double w3 = 0, w4 = 0;
        bool ok = false;
    };
    const int n_pair = hp.n_ele * (hp.n_ele + 1) / 2;
    std::vector<Table> tables;
    auto add = [&](int fn, int kv, bool factor, double fmax) {
        const bool pairs = fn == FN_H || fn == FN_PHI;
        for (int at = 0; at < (pairs ? n_pair : hp.n_ele); at++) {
            Table t;
            t.fn = fn; t.kv = kv; t.factor = factor; t.fmax = fmax;
            t.s = pairs ? &hp.z2[at] : &hp.rho[at];
            tables.push_back(std::move(t));
        }
        return (int) tables.size() - (pairs ? n_pair : hp.n_ele);
    };
    const int first[4] = {add(FN_RHO, krho, false, rho_max), add(FN_G, kg, true, g_max), add(FN_H, kf, true, h_max),
                          want_phi ? add(FN_PHI, kphi, false, phi_max) : 0};
    auto expand = [&](Table &t) {
        t.w.resize(m_end);
        t.out.assign(m_end, FixPoly{});
        for (int m = m_lo; m < m_end; m++) {
            const Interval &v = iv[m];
            Series &w = t.w[m] = expanded(*t.s, t.fn, v);
            double f = 1.0;
            for (int i = 0; i < kTerms; i++) {
                w.c[i] *= f;
                f *= v.unit;
            }
            // x^5 = xm^5 (T5(x / xm) + 20 (x / xm)^3 - 5 (x / xm)) / 16 on [-xm, xm]
            const double x2 = v.xm * v.xm;
            w.c[3] += w.c[5] * (1.25 * x2);
            w.c[1] -= w.c[5] * (0.3125 * x2 * x2);
            t.w3 = std::max(t.w3, std::fabs(w.c[3]));
            t.w4 = std::max(t.w4, std::fabs(w.c[4]));
        }
    };
    auto round_all = [&](Table &t, int e3) {
        for (int m = m_lo; m < m_end; m++) {
            const Interval &v = iv[m];
            // What the coarse units of c4 and c3 leave over goes to the lower coefficients, as T4 and T3 put it:
            // x^4 = xm^2 x^2 - xm^4 / 8 and x^3 = (3/4) xm^2 x, to xm^4 / 8 and xm^3 / 4.
            double *w = t.w[m].c;
            const double x2 = v.xm * v.xm, u4 = std::ldexp(1.0, -(t.kv + 4 - e3)), u3 = std::ldexp(1.0, -(t.kv + 3 - e3));
            i64 c[5];
            c[4] = (i64) std::nearbyint(w[4] / u4);
            const double left4 = w[4] - (double) c[4] * u4;
            c[3] = (i64) std::nearbyint(w[3] / u3);
            const double left3 = w[3] - (double) c[3] * u3;
            if (!to_i64(dd(std::ldexp(w[2] + left4 * x2, t.kv + 2)), c[2]) ||
                !to_i64(dd(std::ldexp(w[1] + left3 * 0.75 * x2, t.kv + 1)), c[1]) ||
                !to_i64(scaled(value_at(*t.s, v.m, t.fn, v.at) - dd(left4 * 0.125 * x2 * x2), t.kv), c[0]))
                return;
            FixPoly &o = t.out[m];
            o.c0 = c[0] + (t.factor ? kFixBias : 0);
            o.c1 = c[1] + kFixBias;
            o.c2 = c[2] + kFixBias;
            o.c3 = (int) c[3];
            o.c4 = (int) c[4];
            // against the spline itself: 2^-49 of the value or of 1/32 of the largest (an FP64 evaluation is
            // off by 2^-50 through its rounded r / dr alone)
            const i64 tb = (i64) ((uint64_t) (v.check + fp.b0) << fp.sh);
            const i64 got = fix_poly(o, fix_coord_of(tb), e3) - (t.factor ? kFixBias : 0);
            const dd want = scaled(value_at(*t.s, v.m, t.fn, v.check_at), t.kv);
            i64 near;
            if (!to_i64(want, near)) return;
            const double err = std::fabs((double) (got - near));
            if (err > std::max(4.0, std::ldexp(std::max(std::fabs(want.h), std::ldexp(t.fmax, t.kv - 5)), -49))) return;
        }
        t.ok = true;
    };
    auto side_by_side = [&](auto &&work) {
        if (depth == INNERMOST) {
            for (Table &t : tables) work(t);
            return;
        }
        std::vector<std::future<void>> f;
        for (Table &t : tables) f.push_back(std::async([&work, &t] { work(t); }));  // (in turn where no thread can be had)
        for (auto &x : f) x.get();
    };
    side_by_side(expand);
    // the finest unit of c3 and c4 that every table of a kind fits
    int e3[4];
    for (int k = 0; k < 4; k++) {
        double top = 0;
        for (const Table &t : tables)
            if (t.fn == k) top = std::max(top, std::ldexp(t.w3, t.kv + 3) + std::ldexp(t.w4, t.kv + 4));
        e3[k] = std::max(1, -exponent_for(top * 1.0001 + 4.0, 31));
        if (!(top < 1e30) || e3[k] > 24) return false;
    }
    side_by_side([&](Table &t) { round_all(t, e3[t.fn]); });
    for (const Table &t : tables)
        if (!t.ok) return false;
    if (depth == INNERMOST) return true;
    fp.e3_rho = e3[FN_RHO];
    fp.e3_g = e3[FN_G];
    fp.e3_h = e3[FN_H];
    fp.e3_phi = e3[FN_PHI];
    tab->rho.assign((size_t) 3 * fp.nr1, FixPoly{});
    tab->zg.assign((size_t) 18 * fp.nr1, FixPoly{});
    tab->phi.assign(want_phi ? (size_t) 9 * fp.nr1 : 0, FixPoly{});
    for (int a = 0; a < 3; a++) {
        std::copy_n(tables[first[FN_RHO] + ele_of_type[a]].out.data(), fp.nr1, &tab->rho[(size_t) a * fp.nr1]);
        for (int b = 0; b < 3; b++) {
            const int pi = HostPotential::pair_index(ele_of_type[a], ele_of_type[b]);
            if (want_phi) std::copy_n(tables[first[FN_PHI] + pi].out.data(), fp.nr1, &tab->phi[(size_t) (a * 3 + b) * fp.nr1]);
            const FixPoly *pg = tables[first[FN_G] + ele_of_type[b]].out.data(), *ph = tables[first[FN_H] + pi].out.data();
            for (int m = 0; m < fp.nr1; m++) {
                FixPoly *r = &tab->zg[2 * ((size_t) (a * 3 + b) * fp.nr1 + m)];
                r[0] = pg[m];
                r[1] = ph[m];
            }
        }
    }
    fp.on = 1;
    return true;
}

// see mg_internal.h. The inner end of the range: where no sum can overflow, and the force sums' unit is the
// finest that any end up to 0.86 of the nearest-neighbour distance allows, as close as the tables' error
// bound admits. The closer it is, the fewer pairs of a hot crystal take the FP64 terms; at 320 K about one
// pair in 1e5 is closer than 0.82.
// F' stays below 1 in most tables (in eV; others scale with the density's unit). An atom above the bound takes the FP64
// loop after its fixed-point one, and so does every neighbour, so where every perfect crystal is at it already, the
// tables are refused. Where the bound of 1 leaves the force sums' unit too coarse, a lower one serves if it is five
// quarters of a crystal's F' or more (next to a vacancy F' grows by a tenth).
bool build_fixed(const HostPotential &hp, const int ele_of_type[3], double a0, double rcf, int n_part, FixParams &fp,
                 FixTables &tab, bool want_phi) {
    fp = FixParams{};
    if (hp.nr < 64 || hp.nr > 20000) return false;
    const double nn = 0.5 * std::sqrt(3.0) * a0, percent = 0.01 * nn;
    const int m_from = std::min(first_knot(70 * percent, hp.dr), hp.nr - 1);
    const std::vector<Largest> largest = largest_from(hp, m_from);
    const Crystal crystal = crystal_of(hp, a0, a0 * rcf);
    if (!(1.05 * crystal.df_least < 1.0)) return false;
    const double exact = fp64_error(hp, crystal, a0, a0 * rcf);
    if (!std::isfinite(exact)) return false;  // no crystal of one element to hold the sums against
    int kd = 60;
    auto from = [&](int f, Depth depth) {
        return build_from(hp, ele_of_type, a0, rcf, n_part, f * percent, kd, exact, crystal, largest, fp, &tab, want_phi, depth);
    };
    double finest = 0.0;
    for (int k = 60; k <= 80 && finest == 0.0 && (k == 60 || std::ldexp(1.25 * crystal.df_most, k - 60) <= 1.0); k++) {
        kd = k;
        for (int f = 70; f <= 86; f += 2)
            if (from(f, SCALES) && (finest == 0.0 || fp.f_unit < finest)) finest = fp.f_unit;
    }
    for (int f = 70; f <= 86 && finest > 0.0; f += 2)
        if (from(f, SCALES) && fp.f_unit == finest && from(f, INNERMOST) && from(f, TABLES)) return true;
    fp = FixParams{};
    return false;
}

}  // namespace mg
