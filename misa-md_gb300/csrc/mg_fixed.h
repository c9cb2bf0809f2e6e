// Fixed-point pair arithmetic of the FP64 form's lattice passes, shared by the kernels and by the host
// code that builds and checks the tables.
//
// GB300 issues two FP64 operations per clock and SM and 64 32x32+64-bit integer multiply-adds, so the
// FP64 form's pair sums are carried in 64-bit integers: coordinates as multiples of 2^-kx A (differences
// are exact), r^2 as a 64-bit integer, and rho, rho'/r, phi'/r and phi as degree-4 polynomials in r^2
// on each knot interval of the potential's own tables. Products keep the high 64 of 128 bits, rounded.
// Sums of integers do not depend on their order.
//
// A 64-bit factor is read as hi * 2^32 + lo with lo signed. Adding 2^31 to the number beforehand (the
// "biased" form) makes its upper word that hi, and flipping the top bit of its lower word gives lo.
#pragma once

#include <math.h>
#include <stdint.h>

#include <cmath>

#ifdef __CUDACC__
#define MG_FIX __host__ __device__ __forceinline__
#else
#define MG_FIX inline
#endif

namespace mg {

typedef long long i64;
constexpr i64 kFixBias = 0x80000000LL;

// polynomial of one knot interval: c1 and c2 biased; c0 biased where the value is a factor of a product
struct alignas(32) FixPoly {
    i64 c0, c1, c2;
    int c3, c4;
};

MG_FIX i64 fix_mad(int a, int b, i64 c) {
#ifdef __CUDA_ARCH__
    i64 r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
#else
    return (i64) ((uint64_t) ((i64) a * b) + (uint64_t) c);
#endif
}
MG_FIX int fix_hi(i64 v) { return (int) ((uint64_t) v >> 32); }
MG_FIX int fix_lo(i64 biased) { return (int) ((uint32_t) (uint64_t) biased ^ 0x80000000u); }

// c + (high 64 bits of (ah:al) * (bh:bl), rounded); the factors' low words signed
MG_FIX i64 fix_mul_add(int ah, int al, int bh, int bl, i64 c) {
    i64 x = fix_mad(ah, bl, kFixBias);
    x = fix_mad(al, bh, x);
    return fix_mad(fix_hi(x), 1, fix_mad(ah, bh, c));
}

// Interval coordinate t 2^sh in units of 2^-63: upper and (signed) lower word, and its square's upper word.
struct FixCoord {
    int h, l, h2;
};
// The polynomial at t. A level's unit is half the one's below it, but that of c3 and c4 is 2^e3 times larger,
// so that they fit 32 bits (e3 >= 1).
MG_FIX i64 fix_poly(const FixPoly &p, const FixCoord &t, int e3) {
    const i64 q = fix_mad(t.h2, p.c4, fix_mad(t.h, p.c3, 0));
    const i64 b = fix_mad(fix_hi(q), 1 << e3, p.c2) + (i64) ((uint32_t) (uint64_t) q >> (32 - e3));
    const i64 c = fix_mul_add(t.h, t.l, fix_hi(b), fix_lo(b), p.c1);
    return fix_mul_add(t.h, t.l, fix_hi(c), fix_lo(c), p.c0);
}
MG_FIX FixCoord fix_coord_of(i64 t) {
    const int h = fix_hi(t);
    return FixCoord{h, fix_lo(t), fix_hi(fix_mad(h, h, kFixBias))};
}

// r^2 of a biased difference vector, in units of 2^-(2 kx - 64) A^2, plus b0
struct FixDelta {
    int xh, xl, yh, yl, zh, zl;
};
MG_FIX FixDelta fix_delta(i64 dx, i64 dy, i64 dz) {
    return FixDelta{fix_hi(dx), fix_lo(dx), fix_hi(dy), fix_lo(dy), fix_hi(dz), fix_lo(dz)};
}
MG_FIX i64 fix_r2(const FixDelta &d, i64 b0) {
    i64 s = fix_mad(d.xh, d.xh, b0);
    s = fix_mad(d.yh, d.yh, s);
    s = fix_mad(d.zh, d.zh, s);
    i64 c = fix_mad(d.xh, d.xl, kFixBias);
    c = fix_mad(d.yh, d.yl, c);
    c = fix_mad(d.zh, d.zl, c);
    return fix_mad(fix_hi(c), 2, s);
}

// x modulo 2^64 in units of 2^-k, rounded to nearest (0 for infinities and NaN)
MG_FIX i64 fix_coord(double x, int k) {
    union { double d; uint64_t u; } v;
    v.d = x;
    const int e = (int) ((v.u >> 52) & 0x7ff);
    if (e == 0 || e == 0x7ff) return 0;
    const uint64_t m = (v.u & 0xfffffffffffffull) | 0x10000000000000ull;
    const int sh = e - 1075 + k;
    uint64_t r;
    if (sh >= 0) r = sh < 64 ? m << sh : 0;
    else r = sh > -55 ? (m + (1ull << (-sh - 1))) >> -sh : 0;
    return (i64) ((v.u >> 63) ? 0 - r : r);
}

// A slot's coordinates and type (-1: vacant, the coordinates half a period away from the site).
struct alignas(32) FixRec {
    i64 x, y, z, type;
};

// Scales and tables of one context and potential (a kernel parameter).
struct FixParams {
    int on;                 // 0: the tables do not suit the fixed-point form; the passes run in FP64
    int kx;                 // coordinates in units of 2^-kx A
    int nr1;                // records per table (knots + 1)
    int sh;                 // t = r^2 - centre is scaled by 2^sh
    int ks, k;              // centre of interval m: ((2m + 1)^2 << ks) * k
    int kd;                 // F'(rho) in units of 2^-kd
    int e3_rho, e3_g, e3_h, e3_phi;  // fix_poly's e3 of each table
    float to_knot;          // sqrt(upper word of r^2) * to_knot = r / dr
    float quarter;          // the upper word of t runs from -(4m + 1) to (4m + 3) quarters on interval m
    i64 b0;                 // bias of r^2
    i64 lo, rc2;            // r^2 (biased) of the tables' inner end and of the cutoff
    double rho_unit, f_unit, e_unit;  // the sums' units
    const FixPoly *rho;     // [3][nr1]       rho of a type
    const FixPoly *zg;      // [9][nr1][2]    rho'/r of type tj, phi'/r of pair (ti, tj)
    const FixPoly *phi;     // [9][nr1]       phi of pair (ti, tj)
};
constexpr i64 kFixBadDf = 3LL << 60;   // F'(rho) outside the range; no valid sum of two reaches 2^61
constexpr int kFixBadHi = 1 << 29;     // upper word of 2^61

// centre of interval m
MG_FIX i64 fix_centre_sub(const FixParams &p, int m, i64 r2) {
    const int n = 2 * m + 1;
    return fix_mad(n * (n << p.ks), -p.k, r2);
}

// Interval coordinate of r2 (biased): the interval m, found from the single-precision root, may be one off
// next to a knot, where the root's rounding (about 1e-3 of a knot) decides; the coordinate itself then tells,
// to 1e-7 of a knot. Closer than that the neighbour's cubic may serve: value and slope are continuous there.
MG_FIX FixCoord fix_locate(const FixParams &p, i64 r2, int &m) {
    const float rf = (float) fix_hi(r2);
#ifdef __CUDA_ARCH__
    float sq;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(sq) : "f"(rf));
    const float fm = __fmaf_rz(sq, p.to_knot, 8388608.0f);  // 2^23 + floor(r / dr)
    m = __float_as_int(fm) - 0x4b000000;
    const float mf = fm - 8388608.0f;
#else
    m = (int) (std::sqrt(rf) * p.to_knot);
    const float mf = (float) m;
#endif
    i64 t = (i64) ((uint64_t) fix_centre_sub(p, m, r2) << p.sh);
    // |th - quarter| <= (4m + 2) quarters inside the interval
    const float off = (float) fix_hi(t) - p.quarter;
    if (fabsf(off) > p.quarter * (4.0f * mf + 2.0f)) {
        m += off > 0.0f ? 1 : -1;
        t = (i64) ((uint64_t) fix_centre_sub(p, m, r2) << p.sh);
    }
    return fix_coord_of(t);
}

// F'(rho) as a factor (unbiased)
MG_FIX i64 fix_df(const FixParams &p, double df) {
    union { double d; uint64_t u; } v;
    v.d = df;
    // |df| < 2^(60 - kd)
    const int e = (int) ((v.u >> 52) & 0x7ff);
    if (e >= 1023 + 60 - p.kd) return kFixBadDf;
    return fix_coord(df, p.kd);
}

}  // namespace mg
