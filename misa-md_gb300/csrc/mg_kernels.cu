// GB300 (sm_103a) kernels for MISA-MD's per-step EAM hot path.
//
// Layout: structure-of-arrays over the reference's ghost-extended slot grid (doubled x), one thread
// per local slot. The lattice density and force passes are full-neighbour gathers over the offset
// table pruned to sites that can lie inside the cutoff (no Newton-3 scatter, no reverse fold, no
// atomics); inter atoms (few) keep the reference's structure for their own sums, and the lattice
// owners they touch gather their Newton-3 shares in a fixed order. The periodic ghost copy replaces
// the MPI halo exchange.
//
// Exact-rounding intrinsics (__dadd_rn / __dmul_rn / __ddiv_rn) are used wherever the reference's
// result must be reproduced bit for bit: velocity-Verlet, the decide distance test, the
// Wigner-Seitz mapping, ghost shifts and setv.

#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdio>

#include "mg_internal.h"

namespace mg {

// ------------------------------------------------------------------------------------------------
// constant tables
// ------------------------------------------------------------------------------------------------
__constant__ double c_mass[3];

void configure_manage_kernel();
void set_mass_table(cudaStream_t stream) {
    configure_manage_kernel();
    const double mass[3] = {atom_mass(0), atom_mass(1), atom_mass(2)};
    cudaMemcpyToSymbolAsync(c_mass, mass, sizeof(mass), 0, cudaMemcpyHostToDevice, stream);
    cudaStreamSynchronize(stream);
}

// the fixed-point form's parameters of a launch (off when the context has none)
inline FixParams fix_params(const LaunchCtx &lc) { return lc.fp ? *lc.fp : FixParams{}; }

// ------------------------------------------------------------------------------------------------
// index helpers
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ int lin(const Geom &g, int x, int y, int z) { return (z * g.Sy + y) * g.Sx + x; }
// parity-split index of a slot (x even and odd sites in two halves) for the mixed form's gather arrays
__device__ __forceinline__ int sidx(const Geom &g, int s) { return (s & 1) * g.half + (s >> 1); }
// Thread order of the gathers. Warps always cover one site parity, so the candidate loop reads
// warp-uniform offsets. Order 0: all even local sites (k, j, i order), then all odd ones. Order 1:
// each run of 64 threads covers 32 consecutive even sites (first warp) and the 32 odd sites beside
// them (second warp), so both halves of each output sector are written close in time. The
// autotuner picks per kernel. Returns -1 past the end.
__device__ __forceinline__ int gather_site(const Geom &g, int t, int order, int &par, int &u) {
    if (order) {
        par = (t >> 5) & 1;
        u = ((t >> 6) << 5) | (t & 31);  // index among the sites of this parity
    } else {
        par = t >= g.n_local_half ? 1 : 0;
        u = par ? t - g.n_local_half : t;
    }
    if (u >= g.n_local_half) return -1;
    const int ih = u % g.nxh;
    const int r = u / g.nxh;
    return lin(g, 2 * ih + par + g.gx, r % g.by + g.gy, r / g.by + g.gz);
}
__device__ __forceinline__ int gather_slot(const Geom &g, int t, int order, int &par) {
    int u;
    return gather_site(g, t, order, par, u);
}
// threads to launch for the gathers
inline int gather_threads(const Geom &g, int order) {
    return order ? ((g.n_local_half + 31) / 32) * 64 : 2 * g.n_local_half;
}

__device__ __forceinline__ int local_slot(const Geom &g, int t, int &i, int &j, int &k) {
    i = t % g.bx;
    const int r = t / g.bx;
    j = r % g.by;
    k = r / g.by;
    return lin(g, i + g.gx, j + g.gy, k + g.gz);
}

// The slot a ghost (or local) slot mirrors under the periodic self-exchange, with the per-dimension
// shift the exchange adds (src/pack/lat_particle_packer.cpp:22-32: +L when sent LOWER, -L HIGHER).
__device__ __forceinline__ int wrap_axis(int c, int g, int b, int &sgn) {
    if (c < g) { sgn = -1; return c + b; }
    if (c >= g + b) { sgn = 1; return c - b; }
    sgn = 0;
    return c;
}
__device__ __forceinline__ int owner_slot(const Geom &g, int s) {
    const int X = s % g.Sx, r = s / g.Sx, Y = r % g.Sy, Z = r / g.Sy;
    int a, b, c;
    return lin(g, wrap_axis(X, g.gx, g.bx, a), wrap_axis(Y, g.gy, g.by, b), wrap_axis(Z, g.gz, g.bz, c));
}

// ------------------------------------------------------------------------------------------------
// Wigner-Seitz mapping (src/lattice/ws_utils.cpp:66-189), one rank: sub-box low corner at 0.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void voronoy_exact(double X, double Y, double Z, double lc, long long &cx, long long &cy,
                                              long long &cz) {
    const double qx = __ddiv_rn(X, lc), qy = __ddiv_rn(Y, lc), qz = __ddiv_rn(Z, lc);
    cx = llround(qx);
    cy = llround(qy);
    cz = llround(qz);
    const double dx = __dsub_rn(qx, (double) cx);
    const double dy = __dsub_rn(qy, (double) cy);
    const double dz = __dsub_rn(qz, (double) cz);
    const bool bx = dx > 0, by = dy > 0, bz = dz > 0;
    cx = 2 * cx;
    const double plane = __dadd_rn(__dadd_rn(__dadd_rn(bx ? dx : -dx, by ? dy : -dy), bz ? dz : -dz), -0.75);
    if (plane >= 0.0) {
        cx += bx ? 1 : -1;
        cy += by ? 0 : -1;
        cz += bz ? 0 : -1;
    }
}
// The integers above depend on the quotient q = RN(X / lc) only through three decisions per axis
// (the nearest integer, the sign of q minus it) and the sign of the bisector-plane sum. The quotient
// is first estimated as RN(X * RN(1 / lc)), within 3 * 2^-53 |q| of RN(X / lc), i.e. below 4e-10 for
// |q| < 2^20. Where every decision clears its boundary by kWsMargin, far above that error, the
// estimate makes the same decisions (the plane sum is the same monotone chain of rounded additions
// on inputs that moved by less than the margin), so the integers are the exact search's. Sites,
// half-way points, bisector planes, NaN and huge coordinates take the exact divisions. On this
// part an FP64 division costs several times a multiply, and the list manager runs these searches
// in a single block, so their latency is its own.
constexpr double kWsMargin = 1e-9;
__device__ __forceinline__ void voronoy(double X, double Y, double Z, const Geom &g, long long &cx, long long &cy,
                                        long long &cz) {
    const double qx = __dmul_rn(X, g.inv_a0), qy = __dmul_rn(Y, g.inv_a0), qz = __dmul_rn(Z, g.inv_a0);
    const double rx = rint(qx), ry = rint(qy), rz = rint(qz);
    const double dx = __dsub_rn(qx, rx), dy = __dsub_rn(qy, ry), dz = __dsub_rn(qz, rz);
    const double ax = fabs(dx), ay = fabs(dy), az = fabs(dz);
    const double plane = __dadd_rn(__dadd_rn(__dadd_rn(ax, ay), az), -0.75);
    const double amax = fmax(ax, fmax(ay, az)), amin = fmin(ax, fmin(ay, az));
    const double qmax = fmax(fabs(qx), fmax(fabs(qy), fabs(qz)));
    const bool clear = amin > kWsMargin && amax < 0.5 - kWsMargin && fabs(plane) > kWsMargin && qmax < 1048576.0;
    if (!clear) {
        voronoy_exact(X, Y, Z, g.a0, cx, cy, cz);
        return;
    }
    cx = 2 * (long long) rx;
    cy = (long long) ry;
    cz = (long long) rz;
    if (plane >= 0.0) {
        cx += dx > 0 ? 1 : -1;
        cy += dy > 0 ? 0 : -1;
        cz += dz > 0 ? 0 : -1;
    }
}
__device__ __forceinline__ uint32_t is_out_box(const Geom &g, double x, double y, double z) {
    long long cx, cy, cz;
    voronoy(x, y, z, g, cx, cy, cz);
    uint32_t f = kInBox;
    if (cx < 0) f |= kXLow; else if (cx >= g.bx) f |= kXHigh;
    if (cy < 0) f |= kYLow; else if (cy >= g.by) f |= kYHigh;
    if (cz < 0) f |= kZLow; else if (cz >= g.bz) f |= kZHigh;
    return f;
}
// ghost-extended coordinates of the nearest site (ws::getNearLatCoord)
__device__ __forceinline__ void near_lat_coord(const Geom &g, double x, double y, double z, long long c[3]) {
    voronoy(x, y, z, g, c[0], c[1], c[2]);
    c[0] += g.gx;
    c[1] += g.gy;
    c[2] += g.gz;
}
// ws::findNearLatIndexInSubBox: -1 outside the sub-box
__device__ __forceinline__ int near_index_in_sub_box(const Geom &g, double x, double y, double z) {
    long long cx, cy, cz;
    voronoy(x, y, z, g, cx, cy, cz);
    if (cx < 0 || cy < 0 || cz < 0 || cx >= g.bx || cy >= g.by || cz >= g.bz) return -1;
    return lin(g, (int) cx + g.gx, (int) cy + g.gy, (int) cz + g.gz);
}
// lattice site of a slot in global coordinates (decide's formula, src/atom.cpp:34-38, extended to
// ghost slots)
__device__ __forceinline__ void site_of(const Geom &g, int X, int Y, int Z, double &xs, double &ys, double &zs) {
    const int i = X - g.gx, j = Y - g.gy, k = Z - g.gz;
    const double half = (X & 1) ? 0.5 : 0.0;
    xs = __dmul_rn((double) i * 0.5, g.a0);
    ys = __dmul_rn((double) j + half, g.a0);
    zs = __dmul_rn((double) k + half, g.a0);
}
__device__ __forceinline__ float4 make_u4(const Geom &g, double x, double y, double z, double xs, double ys,
                                          double zs, int type) {
    return make_float4(__double2float_rn(__dmul_rn(__dsub_rn(x, xs), g.inv_h)),
                       __double2float_rn(__dmul_rn(__dsub_rn(y, ys), g.inv_h)),
                       __double2float_rn(__dmul_rn(__dsub_rn(z, zs), g.inv_h)), __int_as_float(type));
}

// u4 of a vacant slot: NaN coordinates, so every distance test against it fails without a type
// check in the candidate loops; w = INVALID
__device__ __forceinline__ float4 vacant_u4() {
    const float nan = __int_as_float(0x7fffffff);
    return make_float4(nan, nan, nan, __int_as_float(kInvalid));
}
// one 32-byte read-only load (sm_100 and later): a force record of the mixed form
__device__ __forceinline__ void ld_nc_v8(const float *p, float (&v)[8]) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
}
// Pairs of floats in one 64-bit register pair: sm_100 and later execute add/sub/mul/fma .f32x2 as
// one instruction, each lane rounded exactly as the scalar operation.
struct f2 {
    unsigned long long v;
};
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2 a, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ double dt_inv_m_of(const StepParams *p, int type) {
    return type == 0 ? p->dt_inv_m[0] : (type == 1 ? p->dt_inv_m[1] : p->dt_inv_m[2]);
}
// |v|^2 in the order the oracle computes it ((vx^2 + vy^2) + vz^2, each operation rounded)
__device__ __forceinline__ double speed2(double vx, double vy, double vz) {
    return __dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz));
}
// The max-|v|^2 words feed only the variable-timestep rule; the kicks of a fixed-dt run skip them, and
// the host recomputes them (k_vmax_full) before the first step after the rule is switched on.
__device__ __forceinline__ bool variable_dt(const StepParams *sp) { return sp->dx_max > 0.0; }
// Max of v2 over the lanes that call this together, then one atomicMax per such group into a word
// picked by the warp's index, so the words see few atomics each. Non-negative doubles order like
// their bit patterns, so the max is taken on the 64-bit patterns, high word first.
__device__ __forceinline__ void note_vmax2(StepParams *sp, double v2) {
    const unsigned mask = __activemask();
    const unsigned long long b = (unsigned long long) __double_as_longlong(v2);
    const unsigned hi = (unsigned) (b >> 32), lo = (unsigned) b;
    const unsigned mhi = __reduce_max_sync(mask, hi);
    const unsigned mlo = __reduce_max_sync(mask, hi == mhi ? lo : 0u);
    if ((threadIdx.x & 31) == (unsigned) (__ffs(mask) - 1)) {
        const int w = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) & (kVmaxSlots - 1);
        atomicMax(&sp->vmax2[w], ((unsigned long long) mhi << 32) | mlo);
    }
}
__device__ __forceinline__ void set_error(Inter &in, uint32_t bit) { atomicOr((unsigned *) &in.cnt[CNT_ERRORS], bit); }
// Lattice passes can fuse df / the half-kick only when no other kernel adds density or force to
// lattice slots afterwards, i.e. when there are no inter atoms.
__device__ __forceinline__ bool lattice_only(const Inter &in) { return in.cnt[CNT_INTER] == 0; }
// Whether the lattice force pass may take the second half-kick of slot sl itself: always without inter
// atoms; with them, for every atom the density pass's inter-atom sweep did not list (no inter atom
// within the cutoff, so no inter-atom force is added later). The listed owners are kicked by the
// inter-atom force pass's owner gather once their force is complete.
// The same holds for F'(rho) in the density pass: the inter-atom density pass runs before it and lists
// the owners, whose gather adds their inter-atom terms and takes their F' afterwards.
__device__ __forceinline__ bool untouched(const Inter &in, int sl) {
    return lattice_only(in) || !((in.touch_bits[sl >> 5] >> (sl & 31)) & 1u);
}
// FP64 displacement test of atom::decide (src/atom.cpp:34-42) for a local slot
__device__ __forceinline__ bool displaced_fp64(const Geom &g, const Slots &s, int sl) {
    const int X = sl % g.Sx, r = sl / g.Sx, Y = r % g.Sy, Z = r / g.Sy;
    double xs, ys, zs;
    site_of(g, X, Y, Z, xs, ys, zs);
    const double ex = __dsub_rn(s.x[sl], xs), ey = __dsub_rn(s.y[sl], ys), ez = __dsub_rn(s.z[sl], zs);
    double dist = __dmul_rn(ex, ex);
    dist = __dadd_rn(dist, __dmul_rn(ey, ey));
    dist = __dadd_rn(dist, __dmul_rn(ez, ez));
    return dist > g.thr;
}

// ------------------------------------------------------------------------------------------------
// spline evaluation
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void locate_d(double x, double inv, int n, int &m, double &p) {
    p = x * inv;
    m = (int) p;
    m = max(0, min(m, n - 2));
    p -= m;
    p = fmin(p, 1.0);
}
__device__ __forceinline__ double val_d(const Knot64 *t, int m, double p) {
    const double2 *q = reinterpret_cast<const double2 *>(t + m);
    const double2 lo = __ldg(q), hi = __ldg(q + 1);  // {c0, c1}, {c2, c3}
    return fma(fma(fma(hi.y, p, hi.x), p, lo.y), p, lo.x);
}
__device__ __forceinline__ double der_d(const Knot64 *t, int m, double p) {
    const double2 *q = reinterpret_cast<const double2 *>(t + m);
    const double2 lo = __ldg(q), hi = __ldg(q + 1);  // {d0, d1}, {d2, 0}
    return fma(fma(hi.x, p, lo.y), p, lo.x);
}
__device__ __forceinline__ void locate_f(float x, float inv, int n, int &m, float &p) {
    p = x * inv;
    m = (int) p;
    m = max(0, min(m, n - 2));
    p -= (float) m;
    p = fminf(p, 1.0f);
}
// Knot record number and fraction of a pair distance in the FP32 gathers (0 < r < rc <= (nr - 1) dr), and
// 1 / r (half-lattice units). The passes are bound by instruction issue, and conversions between floats
// and integers go through a quarter-rate pipe: adding 2^23 rounded toward zero leaves floor(x) in the low
// bits of the sum, and subtracting 2^23 gives it back as a float, the same numbers at full rate. m keeps
// the bits of the sum, kKnotBias above the knot; the minimum guards rounding at r ~ rc (it keeps m on the
// last knot, whose record exists, for a NaN as well). r^2 is never subnormal: the site vector has a
// component of at least one unit. 16M atoms, with the pair terms' roundings spelled out and 3 c3 tabled:
// force pass 3.87 -> 3.75 ms, density pass 1.86 -> 1.78 ms.
constexpr int kKnotBias = 0x4b000000;
struct PairKnot {
    float rinv, p;
    int m;
};
__device__ __forceinline__ PairKnot pair_knot(const PotTables &pt, float r2) {
    PairKnot k;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(k.rinv) : "f"(r2));
    const float x = __fmul_rn(__fmul_rn(r2, k.rinv), pt.h_inv_dr_f);
    const float b = fminf(__fadd_rz(x, 8388608.0f), pt.knot_max_f);
    k.m = __float_as_int(b);
    k.p = __fsub_rn(x, __fsub_rn(b, 8388608.0f));
    return k;
}
__device__ __forceinline__ float val_f(const float4 *t, int m, float p) {
    const float4 c = __ldg(t + m);
    return fmaf(fmaf(fmaf(c.w, p, c.z), p, c.y), p, c.x);
}
__device__ __forceinline__ float der_f(const float4 *t, int m, float p) {
    const float4 c = __ldg(t + m);
    return fmaf(fmaf(c.z, p, c.y), p, c.x);
}
__device__ __forceinline__ void kahan(float &sum, float &comp, float term) {
    const float y = term - comp;
    const float t = sum + y;
    comp = (t - sum) - y;
    sum = t;
}

// ------------------------------------------------------------------------------------------------
// Fixed-point records of the FP64 form (mg_fixed.h), kept beside the positions where s.kx is set: whoever changes a
// position writes its slot's record. A candidate then costs one 32-byte load instead of three 8-byte loads and three
// conversions per pair, and no pass over the slots makes the records (35 us of a step of 2.0 ms at 2M atoms, 4 us of
// 55 at 16k).
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void fix_store(FixRec *to, i64 x, i64 y, i64 z, i64 type) {
    longlong2 *o = reinterpret_cast<longlong2 *>(to);
    o[0] = make_longlong2(x, y);
    o[1] = make_longlong2(z, type);
}
__device__ __forceinline__ void fix_put(FixRec *to, int kx, double x, double y, double z, int type) {
    fix_store(to, fix_coord(x, kx), fix_coord(y, kx), fix_coord(z, kx), type);
}
// a vacant slot's: half a period away from its site
__device__ __forceinline__ void fix_put_vacant(const Geom &g, FixRec *to, int kx, int sl) {
    const int X = sl % g.Sx, q = sl / g.Sx, Y = q % g.Sy, Z = q / g.Sy;
    double xs, ys, zs;
    site_of(g, X, Y, Z, xs, ys, zs);
    const unsigned long long away = 1ull << 63;
    fix_store(to, (i64) ((unsigned long long) fix_coord(xs, kx) ^ away), (i64) ((unsigned long long) fix_coord(ys, kx) ^ away),
              (i64) ((unsigned long long) fix_coord(zs, kx) ^ away), kInvalid);
}
// too far from its site for the wrapped coordinates: 1.2 half-lattice units (recombined atoms sit up to
// sqrt(5) / 2 of them from their site)
__device__ __forceinline__ bool fix_wild(float4 u) {
    return !(fmaxf(fmaxf(fabsf(u.x), fabsf(u.y)), fabsf(u.z)) <= 1.2f) || u.x != u.x || u.y != u.y || u.z != u.z;
}
// with the FP64 form's records (off when the launch's form keeps none)
inline Slots with_records(const LaunchCtx &lc, Slots s) {
    s.kx = lc.fp ? lc.fp->kx : 0;
    s.spec = lc.spec;
    return s;
}
// whether a pass takes every atom in FP64: the same in every thread of its grid, since nothing writes the word while a
// pass that reads it runs (the overlapped host step, whose passes run beside later chunks, leaves it at 0)
__device__ __forceinline__ bool pass_wild(const Slots &s) { return s.skin->wild != 0; }

// ------------------------------------------------------------------------------------------------
// AoS <-> SoA (the reference's AtomElement array crosses the boundary as raw records)
// ------------------------------------------------------------------------------------------------
__global__ void k_unpack_aos(Geom g, const mg_atom_element *aos, Slots s, Inter in, int types_ok_mask, bool mixed, int s0,
                             int s1, FixParams fp) {
    const int t = s0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= s1) return;
    mg_atom_element a = aos[t];
    if (a.type < -1 || a.type > 2 || (a.type >= 0 && !((types_ok_mask >> a.type) & 1))) {
        set_error(in, MG_DEVERR_BAD_TYPE);
        a.type = kInvalid;
    }
    s.x[t] = a.x[0]; s.y[t] = a.x[1]; s.z[t] = a.x[2];
    s.vx[t] = a.v[0]; s.vy[t] = a.v[1]; s.vz[t] = a.v[2];
    s.fx[t] = a.f[0]; s.fy[t] = a.f[1]; s.fz[t] = a.f[2];
    s.rho[t] = a.rho; s.df[t] = a.df;
    s.type[t] = (int8_t) a.type;
    s.id[t] = a.id;
    {  // u4 in both precisions: the gathers' FP32 candidate test reads it
        const int X = t % g.Sx, r = t / g.Sx, Y = r % g.Sy, Z = r / g.Sy;
        double xs, ys, zs;
        site_of(g, X, Y, Z, xs, ys, zs);
        const float4 u = a.type < 0 ? vacant_u4() : make_u4(g, a.x[0], a.x[1], a.x[2], xs, ys, zs, a.type);
        const int si = sidx(g, t);
        s.u4[si] = u;
        if (s.kx && a.type < 0) fix_put_vacant(g, s.fix + si, s.kx, t);
        else if (s.kx) {
            fix_put(s.fix + si, s.kx, a.x[0], a.x[1], a.x[2], a.type);
            if (fix_wild(u) && !s.spec) s.skin->wild = 1;
        }
    }
    if (mixed) s.df32[sidx(g, t)] = (float) a.df;
    else if (fp.on) s.dfq[sidx(g, t)] = fix_df(fp, a.df);
}

__global__ void k_pack_aos(Geom g, mg_atom_element *aos, Slots s, int fields, bool mixed, int s0, int s1) {
    const int t = s0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= s1) return;
    mg_atom_element &a = aos[t];
    const double df = mixed ? (double) s.df32[sidx(g, t)] : s.df[t];
    if (fields == PACK_ALL) {
        mg_atom_element b;
        b.id = s.id[t];
        b.type = s.type[t];
        b.pad_ = 0;
        b.x[0] = s.x[t]; b.x[1] = s.y[t]; b.x[2] = s.z[t];
        b.v[0] = s.vx[t]; b.v[1] = s.vy[t]; b.v[2] = s.vz[t];
        b.f[0] = s.fx[t]; b.f[1] = s.fy[t]; b.f[2] = s.fz[t];
        b.rho = s.rho[t];
        b.df = df;
        a = b;
        return;
    }
    if (fields & PACK_RHO) a.rho = s.rho[t];
    if (fields & PACK_DF) a.df = df;
    if (fields & PACK_F) { a.f[0] = s.fx[t]; a.f[1] = s.fy[t]; a.f[2] = s.fz[t]; }
}

void launch_unpack_aos(const LaunchCtx &lc, const Geom &g, const mg_atom_element *aos, Slots s, Inter in,
                       int types_ok_mask, bool mixed, int s0, int s1) {
    if (s1 < 0) s1 = g.n_slots;
    if (s1 <= s0) return;
    const int b = 256;
    if (lc.fp && s0 == 0) cudaMemsetAsync(&s.skin->wild, 0, 2 * sizeof(int), lc.stream);  // a state's first part
    k_unpack_aos<<<(s1 - s0 + b - 1) / b, b, 0, lc.stream>>>(g, aos, with_records(lc, s), in, types_ok_mask, mixed, s0, s1, fix_params(lc));
    launch_skin_dirty(lc, s);
}
__global__ void k_set_counts(Inter in, int n_inter) {
    in.cnt[CNT_INTER] = n_inter;
    in.cnt[CNT_GHOST] = 0;
    in.cnt[CNT_DISPLACED] = 0;
    *in.n_bucket = 0;
}
void launch_set_counts(const LaunchCtx &lc, Inter in, int n_inter) { k_set_counts<<<1, 1, 0, lc.stream>>>(in, n_inter); }
void launch_pack_aos(const LaunchCtx &lc, const Geom &g, mg_atom_element *aos, Slots s, int fields, bool mixed, int s0,
                     int s1) {
    if (s1 < 0) s1 = g.n_slots;
    if (s1 <= s0) return;
    const int b = 256;
    k_pack_aos<<<(s1 - s0 + b - 1) / b, b, 0, lc.stream>>>(g, aos, s, fields, mixed, s0, s1);
}

// ------------------------------------------------------------------------------------------------
// velocity-Verlet first half + drift (src/newton_motion.cpp:30-44) fused with the displacement test
// of atom::decide (src/atom.cpp:27-53). Displaced slots are collected unordered; the list kernel
// sorts them into the reference's k, j, i scan order.
// ------------------------------------------------------------------------------------------------
__global__ void k_site_table(double a0, int n, double *out) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < n) out[m] = __dmul_rn((double) m * 0.5, a0);  // site_of: (i * 0.5) * a0, (j + half) * a0
}
void launch_site_table(const LaunchCtx &lc, const Geom &g, double *site_half) {
    k_site_table<<<(g.n_site_half + 255) / 256, 256, 0, lc.stream>>>(g.a0, g.n_site_half, site_half);
}

// decide's distance test (src/atom.cpp:34-42) with each operation rounded on its own; a displaced atom
// appends its local index to the displaced list, in any order (the list manager sorts it into the
// reference's k, j, i scan order)
__device__ __noinline__ void note_displaced(double ex, double ey, double ez, double thr, int t, int *count, int *list, int cap) {
    double dist = __dmul_rn(ex, ex);
    dist = __dadd_rn(dist, __dmul_rn(ey, ey));
    dist = __dadd_rn(dist, __dmul_rn(ez, ez));
    if (dist > thr) {
        const int q = atomicAdd(count, 1);
        if (q < cap) list[q] = t;
    }
}

// the step's largest change of a displacement record: one reduction per group of converged lanes and
// one atomic max per group, spread over kSkinSlots words (squares of non-negative floats order like
// their bit patterns; a NaN orders above every number, so it forces a rebuild)
__device__ __forceinline__ void skin_note(const Slots &s, float d2) {
    const unsigned m = __activemask();
    const unsigned v = __reduce_max_sync(m, __float_as_uint(d2));
    if ((int) (threadIdx.x & 31) == __ffs(m) - 1) atomicMax(&s.skin->step_max2[blockIdx.x & (kSkinSlots - 1)], v);
}

// NewtonMotion::firststep for one lattice atom (src/newton_motion.cpp:30-55) and decide's displacement
// test (src/atom.cpp:34-42): v += c f, x += dt v (each operation rounded as the reference rounds it),
// the displacement record u4 (written to u4_out, parity-split index) and, where displaced, local index t
// into the displaced list. MOVE = false: the test alone, on the current positions. u4_prev holds the record the last
// density pass read (for the skin's displacement bound). PART: may be a launch of the overlapped host step (the force passes,
// which take the next firststep in fused bodies, are not, and have no register to spare for it).
template <bool MOVE, bool DECIDE, bool PART = false>
__device__ __forceinline__ void first_half(const Geom &g, const Slots &s, const Inter &in, const StepParams *__restrict__ p,
                                           int sl, int t, int i, int j, int k, int ty, double vx, double vy, double vz,
                                           double fx, double fy, double fz, float4 *u4_out, const float4 *u4_prev, FixRec *fix_out) {
    double x = s.x[sl], y = s.y[sl], z = s.z[sl];
    if (MOVE) {
        const double c = dt_inv_m_of(p, ty);
        vx = __dadd_rn(vx, __dmul_rn(c, fx));
        vy = __dadd_rn(vy, __dmul_rn(c, fy));
        vz = __dadd_rn(vz, __dmul_rn(c, fz));
        const double dt = p->dt;
        x = __dadd_rn(x, __dmul_rn(dt, vx));
        y = __dadd_rn(y, __dmul_rn(dt, vy));
        z = __dadd_rn(z, __dmul_rn(dt, vz));
        s.vx[sl] = vx; s.vy[sl] = vy; s.vz[sl] = vz;
        s.x[sl] = x; s.y[sl] = y; s.z[sl] = z;
    }
    // the site from the table (the same rounded values site_of computes; gx is even, so the x parity
    // of the slot is i & 1)
    const int par = i & 1;
    const double xs = g.site_half[i], ys = g.site_half[2 * j + par], zs = g.site_half[2 * k + par];
    const double ex = __dsub_rn(x, xs), ey = __dsub_rn(y, ys), ez = __dsub_rn(z, zs);
    const float exf = __double2float_rn(ex), eyf = __double2float_rn(ey), ezf = __double2float_rn(ez);
    if (MOVE) {
        const float ih = g.inv_h_f;
        const float4 nu = make_float4(exf * ih, eyf * ih, ezf * ih, __int_as_float(ty));
        const int si = sidx(g, sl);
        if (g.skin_h > 0.f) {  // read before the store: in place, u4_prev is u4_out
            const float4 o = u4_prev[si];
            const float dx = nu.x - o.x, dy = nu.y - o.y, dz = nu.z - o.z;
            skin_note(s, dx * dx + dy * dy + dz * dz);
        }
        u4_out[si] = nu;
        if (s.kx) {
            fix_put(fix_out + si, s.kx, x, y, z, ty);
            if (fix_wild(nu)) {
                if (!PART || !s.spec) {
                    s.skin->wild_next = 1;
                    if (!DECIDE) s.skin->wild = 1;  // firststep as a phase of its own: no decide need follow
                } else {  // its wrapped coordinates could meet a vacancy's
                    in.cnt[CNT_SPEC_VOID] = 1;
                    u4_out[si] = vacant_u4();
                    fix_put_vacant(g, fix_out + si, s.kx, sl);
                }
            }
        }
    }
    if (DECIDE) {
        // the exact FP64 test of decide runs only where the FP32 distance is not clearly below it
        // (a call, so the rare path stays a branch instead of being evaluated for every atom)
        if (!(exf * exf + eyf * eyf + ezf * ezf < g.thr_lo_f))
            note_displaced(ex, ey, ez, g.thr, t, &in.cnt[CNT_DISPLACED], in.displaced, in.dcap);
    }
}

__device__ void mark_far_neighbourhoods(const NeighTables &nt, const Geom &g, const Inter &in, int a0, int a1, int8_t v, int t0,
                                        int stride) {
    const int per = nt.nfull + 1;
    const int total = (a1 - a0) * per;
    for (int e = t0; e < total; e += stride) {
        const int sl = in.far_list[a0 + e / per];
        const int q = e % per;
        const int par = (sl % g.Sx) & 1;
        const int sj = q == nt.nfull ? sl : sl + nt.lat[par][q];
        in.far_flag[owner_slot(g, sj)] = v;
    }
}

// NewtonMotion::firststep for the inter atoms
__device__ __forceinline__ void inter_firststep(const Inter &in, const StepParams *__restrict__ p, int t0, int stride) {
    const int n = in.cnt[CNT_INTER];
    const double dt = p->dt;
    for (int a = t0; a < n; a += stride) {
        const double c = dt_inv_m_of(p, in.type[a]);
        double vx = __dadd_rn(in.vx[a], __dmul_rn(c, in.fx[a]));
        double vy = __dadd_rn(in.vy[a], __dmul_rn(c, in.fy[a]));
        double vz = __dadd_rn(in.vz[a], __dmul_rn(c, in.fz[a]));
        in.vx[a] = vx; in.vy[a] = vy; in.vz[a] = vz;
        in.x[a] = __dadd_rn(in.x[a], __dmul_rn(dt, vx));
        in.y[a] = __dadd_rn(in.y[a], __dmul_rn(dt, vy));
        in.z[a] = __dadd_rn(in.z[a], __dmul_rn(dt, vz));
    }
}

// fused: the previous step's force pass already took this firststep for every local slot and wrote
// its displacement records into this step's u4 buffer, and the FP64 form's records into this step's fix buffer
// (when no inter atoms exist; else the work is done here). Every local slot's u4 is written, vacancies included, so the two buffers a fused graph
// alternates between are always complete.
// alt: inside a graph whose bodies alternate their u4 buffers, where the previous body's records are
// in s.u4n
// whole: the step's only firststep launch (not one of several over parts of the box). It takes the inter
// atoms' firststep too and (deciding) clears the previous far list's neighbourhood marks, which nothing
// reads between the previous force pass and the marks decide makes: a small box's step is a chain of
// short kernels at 1 to 2 us each, whatever they do.
// A grid-stride loop over a grid of a few blocks per SM: a fused body's launch, which returns at once,
// then costs one small launch instead of a grid over every slot.
template <bool MOVE, bool DECIDE>
__global__ void __launch_bounds__(kFirstThreads) k_firststep(const NeighTables *nt, Geom g, Slots s, Inter in,
                                                             const StepParams *__restrict__ p, int t0, int t1, bool fused, bool alt,
                                                             bool whole) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (MOVE && whole) {
        inter_firststep(in, p, tid, stride);
        if (DECIDE) mark_far_neighbourhoods(*nt, g, in, 0, min(in.cnt[CNT_FAR], in.fcap), 0, tid, stride);
    }
    if (fused && lattice_only(in) && !(s.kx && s.skin->wild)) return;  // wild: as the force pass saw it
    for (int t = t0 + tid; t < t1; t += stride) {
        int i, j, k;
        const int sl = local_slot(g, t, i, j, k);
        const int ty = s.type[sl];
        if (ty < 0) {
            if (MOVE) s.u4[sidx(g, sl)] = vacant_u4();
            if (MOVE && s.kx) fix_put_vacant(g, s.fix + sidx(g, sl), s.kx, sl);
            continue;
        }
        if (MOVE)
            first_half<true, DECIDE, true>(g, s, in, p, sl, t, i, j, k, ty, s.vx[sl], s.vy[sl], s.vz[sl], s.fx[sl], s.fy[sl],
                                           s.fz[sl], s.u4, alt ? s.u4n : s.u4, s.fix);
        else
            first_half<false, DECIDE>(g, s, in, p, sl, t, i, j, k, ty, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, s.u4, s.u4, s.fix);
    }
}

// one block: counts a[0..n) -> base + exclusive offsets (in place); returns base + the total (every
// thread). Each thread takes one contiguous chunk: a pass summing it, one block scan of the chunk
// sums, and a pass writing the chunk's offsets (one scan instead of one per blockDim.x counts).
__device__ int block_scan_counts(int *a, int n, int base) {
    __shared__ int warp_tot[32];
    const int per = (n + (int) blockDim.x - 1) / (int) blockDim.x;
    const int b0 = min(n, (int) threadIdx.x * per), b1 = min(n, b0 + per);
    int v = 0;
#pragma unroll 4
    for (int b = b0; b < b1; b++) v += a[b];
    int x = v;  // inclusive warp scan of the chunk sums
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) >= o) x += y;
    }
    if ((threadIdx.x & 31) == 31) warp_tot[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
        int w = threadIdx.x < (blockDim.x >> 5) ? warp_tot[threadIdx.x] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (threadIdx.x >= o) w += y;
        }
        warp_tot[threadIdx.x] = w;  // inclusive over warps
    }
    __syncthreads();
    int run = base + ((threadIdx.x >> 5) ? warp_tot[(threadIdx.x >> 5) - 1] : 0) + x - v;
    for (int b = b0; b < b1; b++) {
        const int c = a[b];
        a[b] = run;
        run += c;
    }
    const int total = base + warp_tot[(blockDim.x >> 5) - 1];
    __syncthreads();  // warp_tot is free again for a later call
    return total;
}

void launch_firststep(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, const StepParams *p, bool decide, int t0,
                      int t1, bool fused, bool alt) {
    const bool whole = t1 < 0;
    if (whole) t1 = g.n_local;
    if (t1 <= t0) return;
    const int b = kFirstThreads, n = std::min((t1 - t0 + b - 1) / b, lc.num_sms * 8);
    s = with_records(lc, s);
    if (decide) k_firststep<true, true><<<n, b, 0, lc.stream>>>(lc.ntd, g, s, in, p, t0, t1, fused, alt, whole);
    else k_firststep<true, false><<<n, b, 0, lc.stream>>>(lc.ntd, g, s, in, p, t0, t1, fused, alt, whole);
}
void launch_decide_scan(const LaunchCtx &lc, const Geom &g, Slots s, Inter in) {
    const int b = kFirstThreads, n = std::min((g.n_local + b - 1) / b, lc.num_sms * 8);
    cudaMemsetAsync(&in.cnt[CNT_DISPLACED], 0, sizeof(int), lc.stream);
    k_firststep<false, true><<<n, b, 0, lc.stream>>>(lc.ntd, g, s, in, nullptr, 0, g.n_local, false, false, false);
}
__global__ void k_inter_firststep(Inter in, const StepParams *__restrict__ p) {
    inter_firststep(in, p, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
void launch_inter_firststep(const LaunchCtx &lc, Inter in, const StepParams *p) {
    k_inter_firststep<<<lc.num_sms, 256, 0, lc.stream>>>(in, p);
}

// ------------------------------------------------------------------------------------------------
// periodic ghost copy (replaces AtomList::exchangeAtom + LatPacker, src/atom/atom_list.cpp:51-57):
// ghost slot <- (type, x with per-dimension +-L) of its owner. One hop reproduces the reference's
// x -> y -> z phases exactly: each coordinate receives at most one shift.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ int ghost_slot(const Geom &g, int t) {
    const int nz = 2 * g.gz * g.Sy * g.Sx;
    const int ny = 2 * g.gy * g.bz * g.Sx;
    int X, Y, Z;
    if (t < nz) {
        const int plane = g.Sy * g.Sx;
        int zz = t / plane;
        const int r = t % plane;
        Z = zz < g.gz ? zz : zz + g.bz;
        Y = r / g.Sx;
        X = r % g.Sx;
    } else if (t < nz + ny) {
        const int u = t - nz;
        const int row = g.Sx;
        const int yy = u / (g.bz * row);
        const int r = u % (g.bz * row);
        Y = yy < g.gy ? yy : yy + g.by;
        Z = g.gz + r / row;
        X = r % row;
    } else {
        const int u = t - nz - ny;
        const int xx = u % (2 * g.gx);
        const int r = u / (2 * g.gx);
        X = xx < g.gx ? xx : xx + g.bx;
        Y = g.gy + r % g.by;
        Z = g.gz + r / g.by;
    }
    return lin(g, X, Y, Z);
}

// the coordinate of a periodic image (sgn: the side it lies on)
__device__ __forceinline__ double shifted(double x, int sgn, double L) { return sgn ? __dadd_rn(x, sgn > 0 ? L : -L) : x; }
__device__ __forceinline__ void ghost_copy_one(const Geom &g, const Slots &s, int gs) {
    const int X = gs % g.Sx, r = gs / g.Sx, Y = r % g.Sy, Z = r / g.Sy;
    int sx, sy, sz;
    const int os = lin(g, wrap_axis(X, g.gx, g.bx, sx), wrap_axis(Y, g.gy, g.by, sy), wrap_axis(Z, g.gz, g.bz, sz));
    const int type = s.type[os];
    const double x = shifted(s.x[os], sx, g.L[0]), y = shifted(s.y[os], sy, g.L[1]), z = shifted(s.z[os], sz, g.L[2]);
    s.type[gs] = (int8_t) type;
    s.x[gs] = x;
    s.y[gs] = y;
    s.z[gs] = z;
    const int si = sidx(g, gs);
    s.u4[si] = s.u4[sidx(g, os)];
    if (s.kx && type < 0) fix_put_vacant(g, s.fix + si, s.kx, gs);
    else if (s.kx) fix_put(s.fix + si, s.kx, x, y, z, type);
}
// The ghost slots inside the local planes [k0, k1) (y-ghost rows, then x-ghost columns of each plane;
// their owners lie in the same plane), or (k0 < 0) the ghost planes below and above the box, whose
// owners are the top and bottom local planes. Together the calls cover every ghost slot once.
__global__ void k_ghost_copy_planes(Geom g, Slots s, int k0, int k1) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (k0 < 0) {
        if (t < 2 * g.gz * g.Sy * g.Sx) ghost_copy_one(g, s, ghost_slot(g, t));  // the z-ghost planes come first
        return;
    }
    const int rows = 2 * g.gy * g.Sx, per = rows + 2 * g.gx * g.by;
    if (t >= (k1 - k0) * per) return;
    const int Z = g.gz + k0 + t / per, v = t % per;
    int X, Y;
    if (v < rows) {
        const int yy = v / g.Sx;
        Y = yy < g.gy ? yy : yy + g.by;
        X = v % g.Sx;
    } else {
        const int w = v - rows, xx = w % (2 * g.gx);
        X = xx < g.gx ? xx : xx + g.bx;
        Y = g.gy + w / (2 * g.gx);
    }
    ghost_copy_one(g, s, lin(g, X, Y, Z));
}
void launch_ghost_copy_planes(const LaunchCtx &lc, const Geom &g, Slots s, int k0, int k1) {
    const int b = 256;
    const int work = k0 < 0 ? 2 * g.gz * g.Sy * g.Sx : (k1 - k0) * (2 * g.gy * g.Sx + 2 * g.gx * g.by);
    if (work <= 0) return;
    k_ghost_copy_planes<<<(work + b - 1) / b, b, 0, lc.stream>>>(g, with_records(lc, s), k0, k1);
}

// forward df (DfEmbedPacker, src/pack/df_embed_packer.cpp): lattice ghosts and ghost inter atoms
template <bool MIXED>
__device__ __forceinline__ void ghost_df_one(const Geom &g, const Slots &s, int gs, int os) {
    if (MIXED) {
        s.df32[sidx(g, gs)] = s.df32[sidx(g, os)];
    } else {
        s.df[gs] = s.df[os];
        if (s.dfq) s.dfq[sidx(g, gs)] = s.dfq[sidx(g, os)];
    }
}
// The step's maximum change of a displacement record into the skin's sum, or a restart after a rebuild. One warp.
__device__ __forceinline__ void skin_advance(SkinState *k) {
    static_assert(kSkinSlots == 64, "two words per lane");
    const int lane = threadIdx.x & 31;
    const unsigned m = __reduce_max_sync(0xffffffffu, max(k->step_max2[lane], k->step_max2[lane + 32]));
    k->step_max2[lane] = 0u;
    k->step_max2[lane + 32] = 0u;
    if (lane != 0) return;
    if (k->rebuilt) {  // built on this step's records: the sum restarts
        k->acc = 0.f;
        k->dirty = 0;
        k->rebuilt = 0;
        k->rebuilds++;
    } else {
        k->acc += sqrtf(__uint_as_float(m));  // a NaN or infinity forces the next pass to rebuild
    }
    k->passes++;
}
// the same copy for the ghost slots inside the local planes [k0, k1) (y-ghost rows, then x-ghost
// columns of each plane; their owners lie in the same plane), or (k0 < 0) for the ghost planes below
// and above the box together with the ghost inter atoms
template <bool MIXED>
__global__ void k_ghost_df_planes(Geom g, Slots s, Inter in, int k0, int k1) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (k0 < 0) {
        if (t < 2 * g.gz * g.Sy * g.Sx) {
            const int gs = ghost_slot(g, t);  // the z-ghost planes come first in the ghost enumeration
            const int os = owner_slot(g, gs);
            ghost_df_one<MIXED>(g, s, gs, os);
        }
        const int ng = in.cnt[CNT_GHOST];
        for (int q = t; q < ng; q += gridDim.x * blockDim.x) in.gdf[q] = in.df[in.groot[q]];
        return;
    }
    const int rows = 2 * g.gy * g.Sx, per = rows + 2 * g.gx * g.by;
    if (t >= (k1 - k0) * per) return;
    const int Z = g.gz + k0 + t / per, v = t % per;
    int X, Y;
    if (v < rows) {
        const int yy = v / g.Sx;
        Y = yy < g.gy ? yy : yy + g.by;
        X = v % g.Sx;
    } else {
        const int w = v - rows, xx = w % (2 * g.gx);
        X = xx < g.gx ? xx : xx + g.bx;
        Y = g.gy + w / (2 * g.gx);
    }
    const int gs = lin(g, X, Y, Z);
    const int os = owner_slot(g, gs);
    ghost_df_one<MIXED>(g, s, gs, os);
}
void launch_ghost_df_planes(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, bool mixed, int k0, int k1) {
    const int b = 256;
    const int work = k0 < 0 ? 2 * g.gz * g.Sy * g.Sx : (k1 - k0) * (2 * g.gy * g.Sx + 2 * g.gx * g.by);
    if (work <= 0) return;
    const int n = (work + b - 1) / b;
    if (mixed) k_ghost_df_planes<true><<<n, b, 0, lc.stream>>>(g, s, in, k0, k1);
    else k_ghost_df_planes<false><<<n, b, 0, lc.stream>>>(g, s, in, k0, k1);
}

// ------------------------------------------------------------------------------------------------
// lattice density pass (atom::latRho, src/atom.cpp:151-192, as a full gather) with dF/drho fused
// when no inter or far atom adds density afterwards (atom::latDf, src/atom.cpp:286-309).
// Warps are parity-uniform (gather_slot), so the candidate loop reads warp-uniform constants; far
// atoms continue over the entries beyond the pruned set.
// ------------------------------------------------------------------------------------------------
// FP32 candidate test of the FP64 gathers: r^2 from the u4 displacements, against rc^2 (1 + 1e-4).
// Its error is below 1e-6 of rc^2, so every pair the exact FP64 test accepts passes it; vacancies
// (NaN) never do. Only candidates that pass load their FP64 positions.
__device__ __forceinline__ bool near_f32(const Geom &g, f2 uixy, float uiz, float4 D, float4 uj) {
    const f2 dxy = f2_sub(f2_sub(uixy, f2_pack(uj.x, uj.y)), f2_pack(D.x, D.y));
    const float dz = (uiz - uj.z) - D.z;
    float dx, dy;
    f2_unpack(dxy, dx, dy);
    return dx * dx + dy * dy + dz * dz < g.rc2_pre;
}

// rho_tj(r) of one pair inside the cutoff
__device__ __forceinline__ double rho_term_fp64(const PotTables &pt, double r2, int tj) {
    const double r = r2 * rsqrt(r2);
    int m; double p;
    locate_d(r, pt.inv_dr, pt.nr, m, p);
    return val_d(pt.rho_v + tj * pt.nr, m, p);
}
template <int PAR>
__device__ __forceinline__ double rho_sum_fp64(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt, int sl,
                                               int si, float4 ui, double xi, double yi, double zi, int q0, int q1) {
    double acc = 0.0;
    const f2 uixy = f2_pack(ui.x, ui.y);
#pragma unroll 4
    for (int q = q0; q < q1; q++) {
        const float4 D = nt.cand[PAR][q];
        const float4 uj = __ldg(s.u4 + si + __float_as_int(D.w));
        if (!near_f32(g, uixy, ui.z, D, uj)) continue;
        const int sj = sl + nt.lat[PAR][q];
        const int tj = __float_as_int(uj.w);
        const double dx = xi - s.x[sj], dy = yi - s.y[sj], dz = zi - s.z[sj];
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 < g.rc2) acc += rho_term_fp64(pt, r2, tj);
    }
    return acc;
}
// the density of one atom, all in FP64
__device__ __forceinline__ double rho_atom_fp64(const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                                const PotTables &pt, int sl, int par) {
    const double xi = s.x[sl], yi = s.y[sl], zi = s.z[sl];
    const int si = sidx(g, sl);
    const float4 ui = s.u4[si];
    const int np = nt.npruned;
    double acc = par ? rho_sum_fp64<1>(nt, g, s, pt, sl, si, ui, xi, yi, zi, 0, np)
                     : rho_sum_fp64<0>(nt, g, s, pt, sl, si, ui, xi, yi, zi, 0, np);
    if (in.far_flag[sl]) {
        const int nf = nt.nfull;
        acc += par ? rho_sum_fp64<1>(nt, g, s, pt, sl, si, ui, xi, yi, zi, np, nf)
                   : rho_sum_fp64<0>(nt, g, s, pt, sl, si, ui, xi, yi, zi, np, nf);
    }
    return acc;
}

__device__ __forceinline__ void k_lat_rho_fp64_site(int t, const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in, const PotTables &pt, bool hook, int order) {
    int par;
    const int sl = gather_slot(g, t, order, par);
    if (sl < 0) return;
    const int ti = s.type[sl];
    if (ti < 0) { s.rho[sl] = 0.0; return; }
    const double acc = rho_atom_fp64(nt, g, s, in, pt, sl, par);
    s.rho[sl] = acc;
    if (!hook && untouched(in, sl)) {
        int m; double p;
        locate_d(acc, pt.inv_drho, pt.nrho, m, p);
        s.df[sl] = der_d(pt.F_d + ti * pt.nrho, m, p);
    }
}
template <bool LOOP>  // LOOP: several sites per thread, one grid stride apart
__global__ void __launch_bounds__(512) k_lat_rho_fp64(const __grid_constant__ NeighTables nt, Geom g, Slots s, Inter in, PotTables pt, bool hook, int order, int tbase,
                                                       int nthreads) {
    const int t0 = tbase + blockIdx.x * blockDim.x + threadIdx.x;  // threads [tbase, nthreads)
    if (!LOOP) {
        if (t0 < nthreads) k_lat_rho_fp64_site(t0, nt, g, s, in, pt, hook, order);
        return;
    }
    for (int t = t0; t < nthreads; t += gridDim.x * blockDim.x) k_lat_rho_fp64_site(t, nt, g, s, in, pt, hook, order);
}

// r^2 of a candidate pair in half-lattice units (and the pair vector), each operation rounded as
// written: the density and force passes both compute it and must agree bit for bit on which pairs
// lie inside the cutoff (the force pass skips the tail candidates no site of a group had inside)
__device__ __forceinline__ float pair_r2(f2 uixy, float uiz, float4 D, float4 uj, f2 &dxy, float &dz) {
    dxy = f2_sub(f2_sub(uixy, f2_pack(uj.x, uj.y)), f2_pack(D.x, D.y));
    dz = __fsub_rn(__fsub_rn(uiz, uj.z), D.z);
    float dx, dy;
    f2_unpack(dxy, dx, dy);
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}
// one density term (in range): rho_tj(r)
__device__ __forceinline__ float rho_term_mixed(const PotTables &pt, float r2, int tj) {
    const PairKnot k = pair_knot(pt, r2);
    return val_f(pt.rho_vf, tj * pt.nr + k.m - kKnotBias, k.p);
}
__device__ __forceinline__ void rho_pair(const PotTables &pt, float r2, float4 uj, float &sum, float &comp) {
    kahan(sum, comp, rho_term_mixed(pt, r2, __float_as_int(uj.w)));
}
template <int PAR>
__device__ __forceinline__ void rho_sum_mixed(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt, int si, float4 ui,
                                              int q0, int q1, float &sum, float &comp) {
    const float rc2 = g.rc2_h;
    const f2 uixy = f2_pack(ui.x, ui.y);
#pragma unroll 2  // 1, 4 and 8 measured slower
    for (int q = q0; q < q1; q++) {
        const float4 D = nt.cand[PAR][q];
        const float4 uj = __ldg(s.u4 + si + __float_as_int(D.w));
        f2 dxy; float dz;
        const float r2 = pair_r2(uixy, ui.z, D, uj, dxy, dz);
        if (r2 < rc2) rho_pair(pt, r2, uj, sum, comp);  // false for vacancies (NaN coordinates)
    }
}
// The pruned candidates [q0, q1), q1 - q0 <= 32, noting which this site has within rc + skin (bit j:
// candidate q0 + j; rcs2_h >= rc2_h). FULL: q1 - q0 is 32, known at compile time (the full chunks; a
// runtime count there costs registers).
template <int PAR, bool FULL>
__device__ __forceinline__ unsigned rho_sum_noted(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt,
                                                  int si, float4 ui, int q0, int q1, float &sum, float &comp) {
    const float rc2 = g.rc2_h;
    const f2 uixy = f2_pack(ui.x, ui.y);
    unsigned nb = 0;
#pragma unroll 2
    for (int j = 0; j < (FULL ? 32 : q1 - q0); j++) {
        const float4 D = nt.cand[PAR][q0 + j];
        const float4 uj = __ldg(s.u4 + si + __float_as_int(D.w));
        f2 dxy; float dz;
        const float r2 = pair_r2(uixy, ui.z, D, uj, dxy, dz);
        if (r2 < g.rcs2_h) {
            nb |= 1u << j;
            if (r2 < rc2) rho_pair(pt, r2, uj, sum, comp);
        }
    }
    return nb;
}
// the candidates q0 + j of the set bits j of `word` (a word of the group's list), in increasing order,
// so the in-range pairs are summed in the same order as by the full loop
template <int PAR>
__device__ __forceinline__ void rho_sum_listed(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt,
                                               int si, float4 ui, int q0, unsigned word, float &sum, float &comp) {
    const float rc2 = g.rc2_h;
    const f2 uixy = f2_pack(ui.x, ui.y);
    for (unsigned w = word; w; w &= w - 1) {
        const int j = __ffs(w) - 1;
        const float4 D = nt.cand[PAR][q0 + j];
        const float4 uj = __ldg(s.u4 + si + __float_as_int(D.w));
        f2 dxy; float dz;
        const float r2 = pair_r2(uixy, ui.z, D, uj, dxy, dz);
        if (r2 < rc2) rho_pair(pt, r2, uj, sum, comp);
    }
}
// Whether this density pass rebuilds the group lists: the same answer in every thread of the grid, as
// nothing it reads changes during the pass (all 32 lanes of the warp call it). The margin covers the
// FP32 rounding of the distances and of the sums, which is below 1e-5 half-lattice units.
constexpr float kSkinMargin = 1e-3f;
__device__ __forceinline__ bool skin_full(const Geom &g, const Slots &s) {
    if (!(g.skin_h > 0.f)) return true;
    const SkinState *k = s.skin;
    const int lane = threadIdx.x & 31;
    const unsigned m = __reduce_max_sync(0xffffffffu, max(k->step_max2[lane], k->step_max2[lane + 32]));
    const float step = sqrtf(__uint_as_float(m));
    return k->dirty != 0 || !(2.f * (k->acc + step) + kSkinMargin <= g.skin_h);
}
// the list of the 32-site group of parity par holding site u: kListWords words over the pruned candidates
__device__ __forceinline__ unsigned *group_list(const Geom &g, const Slots &s, int par, int u) {
    return s.near + kListWords * (par * ((g.n_local_half + 31) >> 5) + (u >> 5));
}

// stores the density and, where nothing adds to it afterwards, F'(rho)
__device__ __forceinline__ void rho_done_mixed(const Slots &s, const Inter &in, const PotTables &pt, int sl, int si, int ti, float sum,
                                               float comp, bool hook) {
    const double rho = (double) sum - (double) comp;
    s.rho[sl] = rho;
    if (!hook && untouched(in, sl)) {
        int m; float p;
        locate_f((float) rho, pt.inv_drho_f, pt.nrho, m, p);
        s.df32[si] = der_f(pt.F_dff + ti * pt.nrho, m, p);
    }
}

// lists: use the group lists (all 32 lanes of the warp call this, with valid false for threads past
// the end; the warp covers one 32-site group of one parity). full: visit every pruned candidate and
// rebuild the group's list; else visit the listed candidates only.
__device__ __forceinline__ void k_lat_rho_mixed_site(int t, bool valid, const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                                     const PotTables &pt, bool hook, int order, bool lists, bool full) {
    int par = 0, u = 0;
    const int sl = valid ? gather_site(g, t, order, par, u) : -1;
    const int si = sl >= 0 ? sidx(g, sl) : 0;
    const float4 ui = sl >= 0 ? s.u4[si] : vacant_u4();
    const int ti = __float_as_int(ui.w);
    const unsigned live = lists ? __ballot_sync(0xffffffffu, ti >= 0) : 0u;
    // a site marked by a far or just recombined atom nearby makes its group rebuild its list: that
    // atom's record did not come from firststep, so the skin's bound does not cover it
    if (lists && !full) full = __any_sync(0xffffffffu, sl >= 0 && in.far_flag[sl]);
    if (sl < 0) return;
    if (ti < 0) { s.rho[sl] = 0.0; return; }
    float sum = 0.f, comp = 0.f;
    const int np = nt.npruned;
    if (lists) {  // 32 candidates per list word; the group's word: any live site of the warp
        unsigned *w = group_list(g, s, par, u);
        if (full) {
            const bool leader = (int) (threadIdx.x & 31) == __ffs(live) - 1;
            for (int k = 0; k * 32 < np; k++) {
                const int q0 = 32 * k, q1 = min(q0 + 32, np);
                const unsigned nb = q1 - q0 == 32 ? (par ? rho_sum_noted<1, true>(nt, g, s, pt, si, ui, q0, q1, sum, comp)
                                                         : rho_sum_noted<0, true>(nt, g, s, pt, si, ui, q0, q1, sum, comp))
                                                  : (par ? rho_sum_noted<1, false>(nt, g, s, pt, si, ui, q0, q1, sum, comp)
                                                         : rho_sum_noted<0, false>(nt, g, s, pt, si, ui, q0, q1, sum, comp));
                const unsigned any = __reduce_or_sync(live, nb);
                if (leader) w[k] = any;
            }
        } else {
            const uint4 n4 = *reinterpret_cast<const uint4 *>(w);
            for (int k = 0; k * 32 < np; k++) {
                const unsigned word = k == 0 ? n4.x : k == 1 ? n4.y : k == 2 ? n4.z : n4.w;
                if (par) rho_sum_listed<1>(nt, g, s, pt, si, ui, 32 * k, word, sum, comp);
                else rho_sum_listed<0>(nt, g, s, pt, si, ui, 32 * k, word, sum, comp);
            }
        }
    } else {
        if (par) rho_sum_mixed<1>(nt, g, s, pt, si, ui, 0, np, sum, comp);
        else rho_sum_mixed<0>(nt, g, s, pt, si, ui, 0, np, sum, comp);
    }
    if (in.far_flag[sl]) {
        const int nf = nt.nfull;
        if (par) rho_sum_mixed<1>(nt, g, s, pt, si, ui, np, nf, sum, comp);
        else rho_sum_mixed<0>(nt, g, s, pt, si, ui, np, nf, sum, comp);
    }
    rho_done_mixed(s, in, pt, sl, si, ti, sum, comp, hook);
}
template <bool LOOP>  // LOOP: several sites per thread, one grid stride apart (no group lists)
__global__ void __launch_bounds__(512, 4) k_lat_rho_mixed(const __grid_constant__ NeighTables nt, Geom g, Slots s, Inter in, PotTables pt, bool hook, int order, int tbase,
                                                       int nthreads, bool lists) {
    const int t0 = tbase + blockIdx.x * blockDim.x + threadIdx.x;  // threads [tbase, nthreads)
    if (!LOOP) {
        const bool full = lists && skin_full(g, s);
        if (full && blockIdx.x == 0 && threadIdx.x == 0) s.skin->rebuilt = 1;
        k_lat_rho_mixed_site(t0, t0 < nthreads, nt, g, s, in, pt, hook, order, lists, full);
        return;
    }
    for (int t = t0; t < nthreads; t += gridDim.x * blockDim.x)
        k_lat_rho_mixed_site(t, true, nt, g, s, in, pt, hook, order, false, true);
}



// ------------------------------------------------------------------------------------------------
// Small boxes and thin slabs: one block of W warps per 32-site group. A warp of the whole-group passes walks
// about 66 candidates one after another, each a chain of dependent loads and some 90 dependent instructions,
// so a pass lasts 30 to 70 us however few atoms it has. Here the W warps share a group's candidates, W streams
// of them at a time, and what the terms add up to stays what the whole-group passes give, bit for bit.
// FP64 form: the sums are integers, so each warp takes all 32 sites and a share of the candidates.
// Mixed form: compensated sums depend on their order. A warp takes 32 / W sites, its lanes W consecutive
// candidates of each, and every lane adds the W terms of its site up in candidate order, by shuffles; no term
// goes through memory.
// ------------------------------------------------------------------------------------------------
constexpr int kSplitSegment = 32 * kListWords;  // candidates listed at a time
constexpr int kSplitAhead = 2;                  // candidates of a stream whose loads are in flight together
struct SplitList {
    unsigned words[kListWords];
    float4 rec[kSplitSegment];                  // the listed candidates' records, in candidate order
    unsigned char num[kSplitSegment];           // and their numbers, from the segment's first
};
// the block's group: sites u0 + 32 (b / 2) .. + 31 of parity b & 1, one per lane of each warp
struct SplitSite {
    int par, u, sl, si, ti;
    float4 ui;
};
__device__ __forceinline__ SplitSite split_site(const Geom &g, const Slots &s, int u0, int u1) {
    SplitSite a;
    a.par = blockIdx.x & 1;
    a.u = u0 + 32 * (blockIdx.x >> 1) + (threadIdx.x & 31);
    a.sl = -1;
    a.si = 0;
    a.ui = vacant_u4();
    if (a.u < u1) {
        const int r = a.u / g.nxh;
        a.sl = lin(g, 2 * (a.u % g.nxh) + a.par + g.gx, r % g.by + g.gy, r / g.by + g.gz);
        a.si = sidx(g, a.sl);
        a.ui = s.u4[a.si];
    }
    a.ti = __float_as_int(a.ui.w);
    return a;
}
// Lists the candidates [q0, q1) (at most kSplitSegment; cand: the records of the group's parity) that some site
// with `mine` set has within r2max: those of the words `known`, or (null) by looking. Returns their number. All
// threads of the block call it.
template <int W>
__device__ __forceinline__ int split_list(const float4 *cand, const Slots &s, const SplitSite &a, bool mine, int q0, int q1,
                                          float r2max, const unsigned *known, SplitList &sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned w[kListWords];
    if (known) {
        const uint4 v = *reinterpret_cast<const uint4 *>(known);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
        __syncthreads();  // the previous list is done with
    } else {
        __syncthreads();
        if (threadIdx.x < kListWords) sh.words[threadIdx.x] = 0u;
        __syncthreads();
        const f2 uixy = f2_pack(a.ui.x, a.ui.y);
        // half a word at a time, its loads in flight together (a group near a far atom looks at all 228 candidates
        // in every pass, and the slowest group is the pass: 54k-atom cascade, density 51 -> 39 us, force 49 -> 40)
        for (int h = warp; 16 * h < q1 - q0; h += W) {
            unsigned nb = 0u;
#pragma unroll 8
            for (int j = 0; j < 16; j++) {
                const int q = min(q0 + 16 * h + j, q1 - 1);
                const float4 D = __ldg(cand + q);
                const float4 uj = __ldg(s.u4 + a.si + (a.sl >= 0 ? __float_as_int(D.w) : 0));
                f2 dxy; float dz;
                const float r2 = pair_r2(uixy, a.ui.z, D, uj, dxy, dz);
                if (mine && r2 < r2max && q0 + 16 * h + j < q1) nb |= 1u << j;
            }
            nb = __reduce_or_sync(0xffffffffu, nb);
            if (lane == 0) reinterpret_cast<unsigned short *>(sh.words)[h] = (unsigned short) nb;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kListWords; k++) w[k] = sh.words[k];
    }
    int n = 0;
#pragma unroll
    for (int k = 0; k < kListWords; k++) {
        if (k % W == warp && (w[k] >> lane) & 1u) {
            const int r = n + __popc(w[k] & ((1u << lane) - 1u));
            sh.rec[r] = __ldg(cand + q0 + 32 * k + lane);
            sh.num[r] = (unsigned char) (32 * k + lane);
        }
        n += __popc(w[k]);
    }
    __syncthreads();
    return n;
}
// a term outside the cutoff: a NaN that no arithmetic gives
constexpr unsigned kSplitNone = 0x7fffdeadu;
__device__ __forceinline__ bool split_none(float v) { return __float_as_uint(v) == kSplitNone; }
// The mixed form's view: lane l of a warp takes stream l / P of site P * warp + l % P (P = 32 / W).
template <int W>
struct SplitLane {
    static constexpr int P = 32 / W;
    int si, ti, stream;
    bool in, mine;
    f2 uixy;
    float uiz;
    __device__ __forceinline__ SplitLane(const SplitSite &a) {
        const int lane = threadIdx.x & 31, from = P * (threadIdx.x >> 5) + lane % P;
        stream = lane / P;
        si = __shfl_sync(0xffffffffu, a.si, from);
        ti = max(__shfl_sync(0xffffffffu, a.ti, from), 0);
        in = __shfl_sync(0xffffffffu, a.sl, from) >= 0;
        uixy = f2_pack(__shfl_sync(0xffffffffu, a.ui.x, from), __shfl_sync(0xffffffffu, a.ui.y, from));
        uiz = __shfl_sync(0xffffffffu, a.ui.z, from);
        mine = true;
    }
};

// Density, mixed form (500 groups: 26 -> 9 us).
template <int W>
__device__ __forceinline__ void rho_mixed_split(const float4 *cand, int np, int nf, const Geom &g, const Slots &s, const Inter &in,
                                                const PotTables &pt, const SplitSite &a, bool hook, bool lists, bool full, bool far,
                                                SplitList &sh, float2 *out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int end = __any_sync(0xffffffffu, far) ? nf : np;
    SplitLane<W> b(a);
    constexpr int P = SplitLane<W>::P;
    const bool b_far = __shfl_sync(0xffffffffu, far, P * warp + lane % P);
    float sum = 0.f, comp = 0.f;
    int q1;
    for (int q0 = 0; q0 < end; q0 = q1) {
        const bool tail = q0 >= np;
        q1 = min(q0 + kSplitSegment, tail ? end : np);
        unsigned *list = lists && !tail ? group_list(g, s, a.par, a.u) : nullptr;
        const int n = split_list<W>(cand, s, a, !tail || far, q0, q1, list ? g.rcs2_h : g.rc2_h, full ? nullptr : list, sh);
        if (full && list && threadIdx.x < kListWords) list[threadIdx.x] = sh.words[threadIdx.x];
        const bool mine = !tail || b_far;
        for (int c0 = 0; c0 < n; c0 += kSplitAhead * W) {
            float r2[kSplitAhead], t[kSplitAhead];
            int tj[kSplitAhead];
#pragma unroll
            for (int u = 0; u < kSplitAhead; u++) {
                const float4 D = sh.rec[min(c0 + u * W + b.stream, n - 1)];
                const float4 uj = __ldg(s.u4 + b.si + (b.in ? __float_as_int(D.w) : 0));
                f2 dxy; float dz;
                r2[u] = pair_r2(b.uixy, b.uiz, D, uj, dxy, dz);
                tj[u] = max(__float_as_int(uj.w), 0);
            }
            // outside the cutoff the knot stays on the table, and the value is not used
#pragma unroll
            for (int u = 0; u < kSplitAhead; u++) t[u] = rho_term_mixed(pt, r2[u], tj[u]);
#pragma unroll
            for (int u = 0; u < kSplitAhead; u++) {
                if (c0 + u * W >= n) break;
                const float v = c0 + u * W + b.stream < n && mine && r2[u] < g.rc2_h ? t[u] : __uint_as_float(kSplitNone);
#pragma unroll
                for (int k = 0; k < W; k++) {
                    const float tk = __shfl_sync(0xffffffffu, v, P * k + lane % P);
                    if (!split_none(tk)) kahan(sum, comp, tk);
                }
            }
        }
    }
    if (b.stream == 0) out[P * warp + lane % P] = make_float2(sum, comp);
    __syncthreads();
    if (warp != 0 || a.sl < 0) return;
    if (a.ti < 0) { s.rho[a.sl] = 0.0; return; }
    rho_done_mixed(s, in, pt, a.sl, a.si, a.ti, out[lane].x, out[lane].y, hook);
}
template <int W>
__global__ void __launch_bounds__(32 * W) k_lat_rho_mixed_split(const float4 *cand, int np, int nf, Geom g, Slots s, Inter in, PotTables pt,
                                                                bool hook, int u0, int u1, bool lists) {
    __shared__ SplitList sh;
    __shared__ float2 out[32];
    bool full = lists && skin_full(g, s);
    if (full && blockIdx.x == 0 && threadIdx.x == 0) s.skin->rebuilt = 1;
    const SplitSite a = split_site(g, s, u0, u1);
    if (!__any_sync(0xffffffffu, a.ti >= 0)) {  // the same in every warp of the block
        if (threadIdx.x < 32 && a.sl >= 0) s.rho[a.sl] = 0.0;
        return;
    }
    // as in the whole-group pass: a marked site makes its group rebuild its list
    const bool marked = a.sl >= 0 && in.far_flag[a.sl];
    full = full || __any_sync(0xffffffffu, marked);
    rho_mixed_split<W>(cand + a.par * kMaxFull, np, nf, g, s, in, pt, a, hook, lists, full, marked && a.ti >= 0, sh, out);
}

// ------------------------------------------------------------------------------------------------
// FP64 form in fixed point (mg_fixed.h): the pair sums in 64-bit integers. Bound by integer issue and by the
// table records' L1 wavefronts. A pair costs about 60 (density) and 110 (force) integer and single-precision
// operations at one or two issue slots each; its FP64 operations cost 64 slots apiece, which bound the FP64
// loops (2M atoms, step: 14.2 -> 1.93 ms; 304k atoms: 2.2 -> 0.40 ms; 16k atoms: 0.32 -> 0.05 ms). They stay
// for the cases below and for tables the fixed point does not suit. Its errors are half the FP64 loops'
// (thermal crystals against 113-bit arithmetic: force rms 2.4e-15 -> 1.1e-15 of the rms force); build_fixed refuses tables
// where they would be larger.
// The group lists of the mixed form serve here as well: 66 candidates are visited instead of 112.
// Pairs closer than the tables reach (hot crystals, cascades) are kept per thread and summed in FP64 after
// the loop; an atom with more than four of them, or with an F'(rho) too large for its fixed-point
// range, is done in FP64 altogether, and so is every atom of a pass while some atom is too far from its
// site for the wrapped coordinates (an uploaded state before its first decide).
// ------------------------------------------------------------------------------------------------
// the records of every slot, for tables made after the state came in
__global__ void k_fix_records(Geom g, Slots s) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.n_slots) return;
    const int si = sidx(g, t), ty = s.type[t];
    if (ty < 0) {
        fix_put_vacant(g, s.fix + si, s.kx, t);
        return;
    }
    fix_put(s.fix + si, s.kx, s.x[t], s.y[t], s.z[t], ty);
    if (fix_wild(s.u4[si])) s.skin->wild = 1;
}
void launch_fix_records(const LaunchCtx &lc, const Geom &g, Slots s) {
    if (!lc.fp) return;
    cudaMemsetAsync(&s.skin->wild, 0, 2 * sizeof(int), lc.stream);
    k_fix_records<<<(g.n_slots + 255) / 256, 256, 0, lc.stream>>>(g, with_records(lc, s));
}

// one 32-byte read-only load each
__device__ __forceinline__ FixRec ld_fix_rec(const FixRec *p) {
    FixRec r;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r.x), "=l"(r.y), "=l"(r.z), "=l"(r.type) : "l"(p));
    return r;
}
__device__ __forceinline__ FixPoly ld_fix_poly(const FixPoly *p) {
    FixPoly r;
    i64 w;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(r.c0), "=l"(r.c1), "=l"(r.c2), "=l"(w) : "l"(p));
    r.c3 = (int) w;
    r.c4 = fix_hi(w);
    return r;
}
// the candidates closer than the tables reach: up to four candidate numbers, one byte each
__device__ __forceinline__ void fix_note_near(unsigned &near, int q) {
    near = near >> 24 ? 0xffffffffu : (near << 8) | (unsigned) (q + 1);
}
constexpr unsigned kFixNearMany = 0xffffffffu;  // more than fit (a candidate number is below 255)
// the near candidates of a later part of the list joined to those of an earlier one
__device__ __forceinline__ void fix_join_near(unsigned &near, unsigned more) {
    if (more == kFixNearMany) near = kFixNearMany;
    else
        for (int sh = 24; sh >= 0; sh -= 8)
            if ((more >> sh) & 255u) fix_note_near(near, (int) ((more >> sh) & 255u) - 1);
}

// an atom's density over its near pairs, or (many) over all pairs, in FP64
__device__ __noinline__ double rho_near_fp64(const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                             const PotTables &pt, int sl, int par, unsigned near) {
    if (near == kFixNearMany) return rho_atom_fp64(nt, g, s, in, pt, sl, par);
    double acc = 0.0;
    for (; near; near >>= 8) {
        const int sj = sl + (par ? nt.lat[1][(near & 255u) - 1] : nt.lat[0][(near & 255u) - 1]);
        const double dx = s.x[sl] - s.x[sj], dy = s.y[sl] - s.y[sj], dz = s.z[sl] - s.z[sj];
        acc += rho_term_fp64(pt, dx * dx + dy * dy + dz * dz, s.type[sj]);
    }
    return acc;
}

// U candidates (numbers q, at indices oj; those without `use` do not count) of the atom at (xb, yb, zb) (biased).
// The pass waits for its loads and its chains of products, so U candidates go through each stage side by side,
// and no branch stands between the stages: outside the cutoff the last interval is evaluated and nothing added.
// For the split passes (us per step, one at a time -> two: 62 groups 50 -> 46, 5695 groups 255 -> 238); the
// whole-group passes fill the SMs with warps and gain nothing (2M atoms: 2037 -> 2050).
template <int U>
__device__ __forceinline__ void rho_fix_pairs(const Slots &s, const FixParams &fp, const int (&oj)[U], const bool (&use)[U],
                                              const int (&q)[U], i64 xb, i64 yb, i64 zb, i64 &acc, unsigned &near) {
    FixRec j[U];
    FixPoly rec[U];
    FixCoord t[U];
    bool in[U];
#pragma unroll
    for (int u = 0; u < U; u++) j[u] = ld_fix_rec(s.fix + oj[u]);
#pragma unroll
    for (int u = 0; u < U; u++) {
        const i64 r2 = fix_r2(fix_delta(xb - j[u].x, yb - j[u].y, zb - j[u].z), fp.b0);
        in[u] = use[u] && (unsigned long long) (r2 - fp.lo) < (unsigned long long) (fp.rc2 - fp.lo);
        if (use[u] && (unsigned long long) r2 < (unsigned long long) fp.lo) fix_note_near(near, q[u]);
        int m;
        t[u] = fix_locate(fp, in[u] ? r2 : fp.rc2 - 1, m);
        rec[u] = ld_fix_poly(fp.rho + (in[u] ? (int) j[u].type : 0) * fp.nr1 + m);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const i64 v = fix_poly(rec[u], t[u], fp.e3_rho);
        acc += in[u] ? v : 0;
    }
}
// candidate q, at index oj, of the atom at (xb, yb, zb) (biased)
__device__ __forceinline__ void rho_fix_candidate(const Slots &s, const FixParams &fp, int oj, i64 xb, i64 yb,
                                                  i64 zb, int q, i64 &acc, unsigned &near) {
    const FixRec j = ld_fix_rec(s.fix + oj);
    const i64 r2 = fix_r2(fix_delta(xb - j.x, yb - j.y, zb - j.z), fp.b0);
    if ((unsigned long long) (r2 - fp.lo) < (unsigned long long) (fp.rc2 - fp.lo)) {
        int m;
        const FixCoord t = fix_locate(fp, r2, m);
        acc += fix_poly(ld_fix_poly(fp.rho + (int) j.type * fp.nr1 + m), t, fp.e3_rho);
    } else if ((unsigned long long) r2 < (unsigned long long) fp.lo) {
        fix_note_near(near, q);
    }
}
constexpr int kFixRhoAhead = 2, kFixForceAhead = 2;  // candidates side by side
// within this the FP64 form's lists hold a pair: rc + skin, and (skin 0) whatever the single-precision test lets by
__device__ __forceinline__ float fix_list_r2(const Geom &g) { return fmaxf(g.rcs2_h, g.rc2_pre); }
// the candidates [q0, q1) after the single-precision test; NOTED: bit j of the result marks candidate
// q0 + j within rc + skin (q1 - q0 <= 32)
template <int PAR, bool NOTED>
__device__ __forceinline__ unsigned rho_fix_range(const NeighTables &nt, const Geom &g, const Slots &s, const FixParams &fp, int si,
                                                  float4 ui, i64 xb, i64 yb, i64 zb, int q0, int q1, i64 &acc, unsigned &near) {
    const f2 uixy = f2_pack(ui.x, ui.y);
    unsigned nb = 0;
#pragma unroll 1
    for (int q = q0; q < q1; q++) {
        const float4 D = nt.cand[PAR][q];
        f2 dxy; float dz;
        const float r2 = pair_r2(uixy, ui.z, D, __ldg(s.u4 + si + __float_as_int(D.w)), dxy, dz);
        if (NOTED && r2 < fix_list_r2(g)) nb |= 1u << (q - q0);
        if (r2 < g.rc2_pre) rho_fix_candidate(s, fp, si + __float_as_int(D.w), xb, yb, zb, q, acc, near);
    }
    return nb;
}
template <int PAR>
__device__ __forceinline__ void rho_fix_listed(const NeighTables &nt, const Slots &s, const FixParams &fp, int si, i64 xb, i64 yb,
                                               i64 zb, int q0, unsigned word, i64 &acc, unsigned &near) {
    for (unsigned w = word; w; w &= w - 1) {
        const int q = q0 + __ffs(w) - 1;
        rho_fix_candidate(s, fp, si + __float_as_int(nt.cand[PAR][q].w), xb, yb, zb, q, acc, near);
    }
}

// the pair sum over the candidates the tables bound (the pruned ones), and over the tail of a far atom's
// neighbourhood: each fits the integers by itself. lists, full: as k_lat_rho_mixed_site.
template <int PAR>
__device__ __forceinline__ double rho_fix_atom(const NeighTables &nt, const Geom &g, const Slots &s, const FixParams &fp, int si,
                                               float4 ui, const FixRec &me, bool lists, bool full, unsigned *list, unsigned live,
                                               bool far, unsigned &near) {
    const i64 xb = me.x + kFixBias, yb = me.y + kFixBias, zb = me.z + kFixBias;
    const int np = nt.npruned;
    i64 acc = 0;
    if (lists && !full) {
        const uint4 n4 = *reinterpret_cast<const uint4 *>(list);
        for (int k = 0; k * 32 < np; k++)
            rho_fix_listed<PAR>(nt, s, fp, si, xb, yb, zb, 32 * k, k == 0 ? n4.x : k == 1 ? n4.y : k == 2 ? n4.z : n4.w, acc, near);
    } else if (lists) {
        const bool leader = (int) (threadIdx.x & 31) == __ffs(live) - 1;
        for (int k = 0; k * 32 < np; k++) {
            const unsigned nb = rho_fix_range<PAR, true>(nt, g, s, fp, si, ui, xb, yb, zb, 32 * k, min(32 * k + 32, np), acc, near);
            const unsigned any = __reduce_or_sync(live, nb);
            if (leader) list[k] = any;
        }
    } else {
        rho_fix_range<PAR, false>(nt, g, s, fp, si, ui, xb, yb, zb, 0, np, acc, near);
    }
    double rho = (double) acc * fp.rho_unit;
    if (far) {
        acc = 0;
        rho_fix_range<PAR, false>(nt, g, s, fp, si, ui, xb, yb, zb, np, nt.nfull, acc, near);
        rho += (double) acc * fp.rho_unit;
    }
    return rho;
}
// adds the near pairs, stores the density and, where nothing adds to it afterwards, F'(rho)
__device__ __forceinline__ void rho_done_fix(const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in, const PotTables &pt,
                                             const FixParams &fp, int sl, int si, int ti, int par, double rho, unsigned near,
                                             bool hook) {
    if (near) rho = rho_near_fp64(nt, g, s, in, pt, sl, par, near) + (near == kFixNearMany ? 0.0 : rho);
    s.rho[sl] = rho;
    if (!hook && untouched(in, sl)) {
        int m; double p;
        locate_d(rho, pt.inv_drho, pt.nrho, m, p);
        const double df = der_d(pt.F_d + ti * pt.nrho, m, p);
        s.df[sl] = df;
        s.dfq[si] = fix_df(fp, df);
    }
}
__device__ __forceinline__ void k_lat_rho_fix_site(int t, bool valid, const NeighTables &nt, const Geom &g, const Slots &s,
                                                   const Inter &in, const PotTables &pt, const FixParams &fp, bool hook, int order,
                                                   bool lists, bool full, bool wild) {
    int par = 0, u = 0;
    const int sl = valid ? gather_site(g, t, order, par, u) : -1;
    const int si = sl >= 0 ? sidx(g, sl) : 0;
    const float4 ui = sl >= 0 ? s.u4[si] : vacant_u4();
    const int ti = __float_as_int(ui.w);
    const unsigned live = lists ? __ballot_sync(0xffffffffu, ti >= 0) : 0u;
    const bool far = sl >= 0 && in.far_flag[sl];
    if (lists && !full) full = __any_sync(0xffffffffu, far);
    if (sl < 0) return;
    if (ti < 0) { s.rho[sl] = 0.0; return; }
    double rho = 0.0;
    unsigned near = kFixNearMany;
    if (!wild) {
        near = 0u;
        const FixRec me = ld_fix_rec(s.fix + si);
        unsigned *list = group_list(g, s, par, u);
        rho = par ? rho_fix_atom<1>(nt, g, s, fp, si, ui, me, lists, full, list, live, far, near)
                  : rho_fix_atom<0>(nt, g, s, fp, si, ui, me, lists, full, list, live, far, near);
    }
    rho_done_fix(nt, g, s, in, pt, fp, sl, si, ti, par, rho, near, hook);
}
template <bool LOOP>  // LOOP: several sites per thread, one grid stride apart (no group lists)
__global__ void __launch_bounds__(512, 2) k_lat_rho_fix(const __grid_constant__ NeighTables nt, const __grid_constant__ Geom g,
                                                        const __grid_constant__ Slots s, const __grid_constant__ Inter in,
                                                        const __grid_constant__ PotTables pt, const __grid_constant__ FixParams fp,
                                                        bool hook, int order, int tbase, int nthreads, bool lists) {
    const int t0 = tbase + blockIdx.x * blockDim.x + threadIdx.x;  // threads [tbase, nthreads)
    const bool wild = pass_wild(s);
    if (LOOP) {
        for (int t = t0; t < nthreads; t += gridDim.x * blockDim.x)
            k_lat_rho_fix_site(t, true, nt, g, s, in, pt, fp, hook, order, false, true, wild);
        return;
    }
    const bool full = lists && !wild && skin_full(g, s);
    if (lists && blockIdx.x == 0 && threadIdx.x == 0) {
        if (wild) s.skin->dirty = 1;  // groups near a recombined atom did not rebuild their lists
        else if (full) s.skin->rebuilt = 1;
    }
    k_lat_rho_fix_site(t0, t0 < nthreads, nt, g, s, in, pt, fp, hook, order, lists && !wild, full, wild);
}

// the list's next U candidates from c on, those below c1 in use
template <int U>
__device__ __forceinline__ void split_next(const SplitList &sh, int si, int q0, int c, int c1, int (&oj)[U], bool (&use)[U], int (&q)[U]) {
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int e = min(c + u, c1 - 1);
        use[u] = c + u < c1;
        oj[u] = si + __float_as_int(sh.rec[e].w);
        q[u] = q0 + sh.num[e];
    }
}
// The density pass of small boxes (see rho_mixed_split): each warp's integer sum and near pairs over a contiguous
// share of the candidates (the near pairs keep their order), put together by the first warp (500 groups: 47 -> 19 us).
template <int W>
__device__ __forceinline__ void rho_fix_split(const NeighTables &nt, const float4 *cand, const Geom &g, const Slots &s, const Inter &in,
                                              const PotTables &pt, const FixParams &fp, const SplitSite &a, bool hook, bool lists,
                                              bool full, bool far, bool wild, SplitList &sh, i64 (*part)[32],
                                              unsigned (*part_near)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int np = nt.npruned, end = wild ? 0 : __any_sync(0xffffffffu, far) ? nt.nfull : np;
    double rho = 0.0;
    unsigned near = wild ? kFixNearMany : 0u;
    const FixRec me = a.ti >= 0 ? ld_fix_rec(s.fix + a.si) : FixRec{};
    const i64 xb = me.x + kFixBias, yb = me.y + kFixBias, zb = me.z + kFixBias;
    int q1;
    for (int q0 = 0; q0 < end; q0 = q1) {
        const bool tail = q0 >= np;
        q1 = min(q0 + kSplitSegment, tail ? end : np);
        const bool mine = a.ti >= 0 && (!tail || far);
        unsigned *list = lists && !tail ? group_list(g, s, a.par, a.u) : nullptr;
        const int n = split_list<W>(cand, s, a, mine, q0, q1, list ? fix_list_r2(g) : g.rc2_pre, full ? nullptr : list, sh);
        if (full && list && threadIdx.x < kListWords) list[threadIdx.x] = sh.words[threadIdx.x];
        i64 acc = 0;
        unsigned mn = 0u;
        if (mine) {
            const int c1 = n * (warp + 1) / W;
            for (int c = n * warp / W; c < c1; c += kFixRhoAhead) {
                int oj[kFixRhoAhead], q[kFixRhoAhead];
                bool use[kFixRhoAhead];
                split_next<kFixRhoAhead>(sh, a.si, q0, c, c1, oj, use, q);
                rho_fix_pairs<kFixRhoAhead>(s, fp, oj, use, q, xb, yb, zb, acc, mn);
            }
        }
        part[warp][lane] = acc;
        part_near[warp][lane] = mn;
        __syncthreads();
        if (warp == 0) {
            for (int w = 1; w < W; w++) acc += part[w][lane];
            rho += (double) acc * fp.rho_unit;
            for (int w = 0; w < W; w++) fix_join_near(near, part_near[w][lane]);
        }
    }
    if (warp != 0 || a.sl < 0) return;
    if (a.ti < 0) { s.rho[a.sl] = 0.0; return; }
    rho_done_fix(nt, g, s, in, pt, fp, a.sl, a.si, a.ti, a.par, rho, near, hook);
}
template <int W>
__global__ void __launch_bounds__(32 * W, 32 / W) k_lat_rho_fix_split(const __grid_constant__ NeighTables nt, const float4 *cand,
                                                                      const __grid_constant__ Geom g, const __grid_constant__ Slots s,
                                                                      const __grid_constant__ Inter in,
                                                                      const __grid_constant__ PotTables pt,
                                                                      const __grid_constant__ FixParams fp, bool hook, int u0, int u1,
                                                                      bool lists) {
    __shared__ SplitList sh;
    __shared__ i64 part[W][32];
    __shared__ unsigned part_near[W][32];
    const bool wild = pass_wild(s);
    bool full = lists && !wild && skin_full(g, s);
    if (lists && blockIdx.x == 0 && threadIdx.x == 0) {
        if (wild) s.skin->dirty = 1;  // groups near a recombined atom did not rebuild their lists
        else if (full) s.skin->rebuilt = 1;
    }
    const SplitSite a = split_site(g, s, u0, u1);
    if (!__any_sync(0xffffffffu, a.ti >= 0)) {
        if (threadIdx.x < 32 && a.sl >= 0) s.rho[a.sl] = 0.0;
        return;
    }
    const bool marked = a.sl >= 0 && in.far_flag[a.sl];
    full = full || __any_sync(0xffffffffu, marked);
    rho_fix_split<W>(nt, cand + a.par * kMaxFull, g, s, in, pt, fp, a, hook, lists && !wild, full, marked && a.ti >= 0, wild, sh, part,
                     part_near);
}

// atoms per thread: each thread takes rho_apt sites, one grid stride apart (the stride is a multiple
// of 64, so warps keep their parity and thread order)
// The passes can keep and use per-group candidate lists when every warp of both passes covers one
// 32-site group of one parity: one site per thread, and (for the parity-major order) a multiple of 32
// sites per parity; the pruned candidates fit the list words.
bool lists_ok(const LaunchCtx &lc, const Geom &g) {
    const bool aligned = (g.n_local_half & 31) == 0;
    return lc.nt->npruned <= 32 * kListWords && lc.rho_apt == 1 && lc.force_apt == 1 && (lc.rho_order == 1 || aligned) &&
           (lc.force_order == 1 || aligned);
}
// Warps per group of a split pass over n groups, 0: the whole-group pass. More warps cut the pass's latency and cost
// instructions (the mixed form's shuffles, and each warp's own start), so their number falls as the groups fill the
// SMs; a batch counts a member's groups once for each member. Measured on 152 SMs, us per step with 8 / 4 / 2 /
// no split warps:
//   mixed  62 groups 37 / 42 / 52 / 70;  364: 51 / 44 / 53 / 73;  1098: 81 / 53 / 56 / 75;
//          2048: 122 / 75 / 65 / 74;  2916: 164 / 99 / 99 / 80
//   FP64   62 groups 52 / 63 / 88 / 123;  500: 60 / 67 / 90 / 126;  1098: 88 / 82 / 97 / 129;
//          2916: 169 / 156 / 172 / 167;  5695: 285 / 254 / 238 / 267;  7812: 377 / 334 / 313 / 319
// A pass without lists (the hooks) searches all candidates first, which the warps share less well; ms for the three
// hooks: FP64 500 groups - / 0.39 / 0.42 / 0.47;  2048: 0.76 / 0.72 / 0.75 / 0.73;  7812: 2.00 / 1.92 / 1.91 / 1.83.
static int split_groups(int u0, int u1) { return 2 * ((u1 - u0 + 31) / 32); }
static int split_warps(const LaunchCtx &lc, bool mixed, bool lists, int n) {
    if (!mixed && !lc.fp) return 0;
    const int64_t busy = static_cast<int64_t>(n) * lc.share / lc.num_sms;
    if (busy < (mixed || !lists ? 2 : 4)) return 8;
    if (!lists) return busy < (mixed ? 8 : 14) ? 4 : 0;
    if (busy < (mixed ? 8 : 22)) return 4;
    return busy < (mixed ? 14 : 52) ? 2 : 0;
}
template <int W>
static void launch_rho_split_w(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, bool hook, int u0, int u1,
                               bool lists) {
    const int n = split_groups(u0, u1);
    if (mixed)
        k_lat_rho_mixed_split<W><<<n, 32 * W, 0, lc.stream>>>(&lc.ntd->cand[0][0], lc.nt->npruned, lc.nt->nfull, g, s, in, t, hook, u0, u1, lists);
    else k_lat_rho_fix_split<W><<<n, 32 * W, 0, lc.stream>>>(*lc.nt, &lc.ntd->cand[0][0], g, s, in, t, *lc.fp, hook, u0, u1, lists);
}
// the split density pass, where it serves
static bool launch_lat_rho_split(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, bool hook, int u0,
                                 int u1, bool lists) {
    switch (split_warps(lc, mixed, lists, split_groups(u0, u1))) {
        case 8: launch_rho_split_w<8>(lc, g, s, in, t, mixed, hook, u0, u1, lists); return true;
        case 4: launch_rho_split_w<4>(lc, g, s, in, t, mixed, hook, u0, u1, lists); return true;
        case 2: launch_rho_split_w<2>(lc, g, s, in, t, mixed, hook, u0, u1, lists); return true;
        default: return false;
    }
}
static void launch_lat_rho_threads(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, bool hook,
                                   int tb, int te, bool lists = false) {
    const int order = lc.rho_order, b = lc.rho_block;
    const int n = (te - tb + b * lc.rho_apt - 1) / (b * lc.rho_apt);
    if (n <= 0) return;
    if (lc.rho_apt > 1) {
        if (mixed) k_lat_rho_mixed<true><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, hook, order, tb, te, false);
        else if (lc.fp) k_lat_rho_fix<true><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, *lc.fp, hook, order, tb, te, false);
        else k_lat_rho_fp64<true><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, hook, order, tb, te);
    } else {
        if (mixed) k_lat_rho_mixed<false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, hook, order, tb, te, lists);
        else if (lc.fp) k_lat_rho_fix<false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, *lc.fp, hook, order, tb, te, lists);
        else k_lat_rho_fp64<false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, hook, order, tb, te);
    }
}
__global__ void __launch_bounds__(32) k_skin_advance(SkinState *k) { skin_advance(k); }
void launch_skin_advance(const LaunchCtx &lc, Slots s) { k_skin_advance<<<1, 32, 0, lc.stream>>>(s.skin); }
void launch_skin_dirty(const LaunchCtx &lc, Slots s) { cudaMemsetAsync(&s.skin->dirty, 1, 1, lc.stream); }

// whether a pass can use the group lists: the mixed form, and the FP64 form's fixed-point passes
static bool has_lists(const LaunchCtx &lc, bool mixed) { return mixed || lc.fp; }
bool lat_lists(const LaunchCtx &lc, const Geom &g, bool mixed) { return has_lists(lc, mixed) && lists_ok(lc, g); }
bool lat_split(const LaunchCtx &lc, const Geom &g, bool mixed) {
    return split_warps(lc, mixed, lat_lists(lc, g, mixed), split_groups(0, g.n_local_half)) != 0;
}
// A pass with the group lists is followed by the skin's advance, which the caller launches (true: it is due). A
// pass without them leaves the lists behind the positions, so the next pass with them rebuilds them.
bool launch_lat_rho(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, bool hook, bool lists) {
    const bool v = lists && has_lists(lc, mixed) && !hook && lists_ok(lc, g);
    if (!launch_lat_rho_split(lc, g, s, in, t, mixed, hook, 0, g.n_local_half, v))
        launch_lat_rho_threads(lc, g, s, in, t, mixed, hook, 0, gather_threads(g, lc.rho_order), v);
    if (!v && has_lists(lc, mixed)) launch_skin_dirty(lc, s);
    return v;
}
// thread range of the sites [u0, u1) of both parities (u0, u1 multiples of 32, or u1 = n_local_half)
static void site_threads(const Geom &g, int order, int u0, int u1, int tb[2], int te[2], int &nr) {
    if (order) {  // warp w of parity p covers sites 32 (w / 2) .. + 31: thread t = 64 (u / 32) + 32 p + u % 32
        tb[0] = (u0 >> 5) << 6;
        te[0] = u1 >= g.n_local_half ? gather_threads(g, 1) : (u1 >> 5) << 6;
        nr = 1;
    } else {      // parity-major threads: one range per parity
        tb[0] = u0; te[0] = u1;
        tb[1] = g.n_local_half + u0; te[1] = g.n_local_half + u1;
        nr = 2;
    }
}
void launch_lat_rho_sites(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, int u0, int u1,
                          bool lists) {
    if (u1 <= u0) return;
    int tb[2], te[2], nr;
    site_threads(g, lc.rho_order, u0, u1, tb, te, nr);
    const bool v = lists && has_lists(lc, mixed) && lists_ok(lc, g);
    if (!launch_lat_rho_split(lc, g, s, in, t, mixed, false, u0, u1, v))
        for (int r = 0; r < nr; r++) launch_lat_rho_threads(lc, g, s, in, t, mixed, false, tb[r], te[r], v);
    if (!v && has_lists(lc, mixed)) launch_skin_dirty(lc, s);  // the caller advances the skin after the last slab
}

// dF/drho of a lattice slot from its density
template <bool MIXED>
__device__ __forceinline__ void lat_df_one(const Geom &g, const Slots &s, const PotTables &pt, const FixParams &fp, int sl, int ti,
                                           double rho) {
    if (MIXED) {
        int m; float p;
        locate_f((float) rho, pt.inv_drho_f, pt.nrho, m, p);
        s.df32[sidx(g, sl)] = der_f(pt.F_dff + ti * pt.nrho, m, p);
    } else {
        int m; double p;
        locate_d(rho, pt.inv_drho, pt.nrho, m, p);
        const double df = der_d(pt.F_d + ti * pt.nrho, m, p);
        s.df[sl] = df;
        if (fp.on) s.dfq[sidx(g, sl)] = fix_df(fp, df);
    }
}
// the df hook: every lattice slot
template <bool MIXED>
__global__ void k_lat_df(Geom g, Slots s, PotTables pt, FixParams fp) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.n_local) return;
    int i, j, k;
    const int sl = local_slot(g, t, i, j, k);
    const int ti = s.type[sl];
    if (ti >= 0) lat_df_one<MIXED>(g, s, pt, fp, sl, ti, s.rho[sl]);
}
void launch_lat_df(const LaunchCtx &lc, const Geom &g, Slots s, PotTables t, bool mixed) {
    const int b = 256, n = (g.n_local + b - 1) / b;
    if (mixed) k_lat_df<true><<<n, b, 0, lc.stream>>>(g, s, t, FixParams{});
    else k_lat_df<false><<<n, b, 0, lc.stream>>>(g, s, t, fix_params(lc));
}

// ------------------------------------------------------------------------------------------------
// lattice force pass (atom::latForce, src/atom.cpp:311-358, as a full gather). When no inter atom
// adds force afterwards, the second half-kick (NewtonMotion::secondstep, src/newton_motion.cpp:57-67)
// is fused, and inside a fused graph (mixed form) so is the next loop body's firststep.
// fpair = -(F'_i rho'_j(r) + F'_j rho'_i(r) + phi'_ij(r)) / r, phi = (r phi) / r.
// ------------------------------------------------------------------------------------------------
// fpair of one pair inside the cutoff
__device__ __forceinline__ double fpair_fp64(const PotTables &pt, double r2, int ti, int tj, double dfi, double dfj) {
    const double rinv = rsqrt(r2);
    const double r = r2 * rinv;
    int m; double p;
    locate_d(r, pt.inv_dr, pt.nr, m, p);
    const double rhojp = der_d(pt.rho_d + tj * pt.nr, m, p);
    const double rhoip = (tj == ti) ? rhojp : der_d(pt.rho_d + ti * pt.nr, m, p);
    const int pr = (ti * 3 + tj) * pt.nr;
    const double zv = val_d(pt.z_v + pr, m, p);
    const double zp = der_d(pt.z_d + pr, m, p);
    const double phi = zv * rinv;
    const double phip = zp * rinv - phi * rinv;
    const double psip = dfi * rhojp + dfj * rhoip + phip;
    return -psip * rinv;
}
template <int PAR>
__device__ __forceinline__ void force_sum_fp64(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt, int sl, int ti,
                                               int si, float4 ui, double xi, double yi, double zi, double dfi, int q0, int q1,
                                               double &fx, double &fy, double &fz) {
    const f2 uixy = f2_pack(ui.x, ui.y);
#pragma unroll 2
    for (int q = q0; q < q1; q++) {
        const float4 D = nt.cand[PAR][q];
        const float4 uj = __ldg(s.u4 + si + __float_as_int(D.w));
        if (!near_f32(g, uixy, ui.z, D, uj)) continue;
        const int sj = sl + nt.lat[PAR][q];
        const int tj = __float_as_int(uj.w);
        const double dx = xi - s.x[sj], dy = yi - s.y[sj], dz = zi - s.z[sj];
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 < g.rc2) {
            const double fpair = fpair_fp64(pt, r2, ti, tj, dfi, s.df[sj]);
            fx += dx * fpair;
            fy += dy * fpair;
            fz += dz * fpair;
        }
    }
}
// the lattice force on one atom, all in FP64
__device__ __forceinline__ void force_atom_fp64(const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                                const PotTables &pt, int sl, int ti, int par, double &fx, double &fy,
                                                double &fz) {
    const double xi = s.x[sl], yi = s.y[sl], zi = s.z[sl];
    const double dfi = s.df[sl];
    const int si = sidx(g, sl);
    const float4 ui = s.u4[si];
    fx = 0.0; fy = 0.0; fz = 0.0;
    const int np = nt.npruned;
    if (par) force_sum_fp64<1>(nt, g, s, pt, sl, ti, si, ui, xi, yi, zi, dfi, 0, np, fx, fy, fz);
    else force_sum_fp64<0>(nt, g, s, pt, sl, ti, si, ui, xi, yi, zi, dfi, 0, np, fx, fy, fz);
    if (in.far_flag[sl]) {
        const int nf = nt.nfull;
        if (par) force_sum_fp64<1>(nt, g, s, pt, sl, ti, si, ui, xi, yi, zi, dfi, np, nf, fx, fy, fz);
        else force_sum_fp64<0>(nt, g, s, pt, sl, ti, si, ui, xi, yi, zi, dfi, np, nf, fx, fy, fz);
    }
}
// local coordinates and local index (k, j, i order) of a local slot
__device__ __forceinline__ int local_index_of(const Geom &g, int sl, int &i, int &j, int &k) {
    const int X = sl % g.Sx, r = sl / g.Sx;
    i = X - g.gx;
    j = r % g.Sy - g.gy;
    k = r / g.Sy - g.gz;
    return (k * g.by + j) * g.bx + i;
}
// Stores the force and takes the second half-kick where the lattice pass may; fused: also the next body's firststep.
// A fused body's forces are used only in registers: the next body's firststep is taken here, and the last body of a
// graph (never fused) stores the forces the state keeps between launches. The other threads of the pass still read
// this atom's u4 and fix records, so the new ones go to the next body's buffers.
__device__ __forceinline__ void force_done(const Geom &g, const Slots &s, const Inter &in, StepParams *sp, int sl, int si, int ti,
                                           double fx, double fy, double fz, bool kick, bool hook, bool fused) {
    if (!fused) { s.fx[sl] = fx; s.fy[sl] = fy; s.fz[sl] = fz; }
    if (kick && !hook && untouched(in, sl)) {
        const double c = dt_inv_m_of(sp, ti);
        const double vx = __dadd_rn(s.vx[sl], __dmul_rn(c, fx));
        const double vy = __dadd_rn(s.vy[sl], __dmul_rn(c, fy));
        const double vz = __dadd_rn(s.vz[sl], __dmul_rn(c, fz));
        if (!fused) { s.vx[sl] = vx; s.vy[sl] = vy; s.vz[sl] = vz; }  // else first_half writes the next v
        if (variable_dt(sp)) note_vmax2(sp, speed2(vx, vy, vz));
        if (fused) {
            int i, j, k;
            const int tl = local_index_of(g, sl, i, j, k);
            first_half<true, true>(g, s, in, sp, sl, tl, i, j, k, ti, vx, vy, vz, fx, fy, fz, s.u4n, s.u4, s.fixn);
        }
    }
}

__device__ __forceinline__ void k_lat_force_fp64_site(int t, const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                                const PotTables &pt, StepParams *sp, bool kick, bool hook, int order) {
    int par;
    const int sl = gather_slot(g, t, order, par);
    if (sl < 0) return;
    const int ti = s.type[sl];
    if (ti < 0) { s.fx[sl] = 0.0; s.fy[sl] = 0.0; s.fz[sl] = 0.0; return; }
    double fx, fy, fz;
    force_atom_fp64(nt, g, s, in, pt, sl, ti, par, fx, fy, fz);
    force_done(g, s, in, sp, sl, sidx(g, sl), ti, fx, fy, fz, kick, hook, false);
}
template <bool LOOP>  // LOOP: several sites per thread, one grid stride apart
__global__ void __launch_bounds__(512) k_lat_force_fp64(const __grid_constant__ NeighTables nt, Geom g, Slots s, Inter in, PotTables pt,
                                                         StepParams *sp, bool kick, bool hook, int order, int tbase,
                                                         int nthreads) {
    const int t0 = tbase + blockIdx.x * blockDim.x + threadIdx.x;  // threads [tbase, nthreads)
    if (!LOOP) {
        if (t0 < nthreads) k_lat_force_fp64_site(t0, nt, g, s, in, pt, sp, kick, hook, order);
        return;
    }
    for (int t = t0; t < nthreads; t += gridDim.x * blockDim.x) k_lat_force_fp64_site(t, nt, g, s, in, pt, sp, kick, hook, order);
}

// ---- FP64 form in fixed point: see the density pass ----
struct FixForce {
    i64 x, y, z;     // sum of (x_i - x_j) (F'_i rho'_j + F'_j rho'_i + phi') / r: minus the force
    int df_hi;       // largest upper word of F'_i + F'_j met
    unsigned near;
};
// An atom's force over its near pairs, or (many) over all pairs, in FP64, and over all pairs while the pass is wild.
// But for that, the distance vectors come from the records: a fused pass changes the positions in place.
__device__ __forceinline__ void fix_vector(const FixRec &i, const FixRec &j, double unit, double &dx, double &dy, double &dz) {
    dx = (double) (i.x - j.x) * unit;
    dy = (double) (i.y - j.y) * unit;
    dz = (double) (i.z - j.z) * unit;
}
__device__ __noinline__ double3 force_near_fp64(const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                                const PotTables &pt, int kx, int sl, int ti, int par, unsigned near, bool wild) {
    double fx = 0.0, fy = 0.0, fz = 0.0;
    if (wild) {
        force_atom_fp64(nt, g, s, in, pt, sl, ti, par, fx, fy, fz);
        return make_double3(fx, fy, fz);
    }
    const bool many = near == kFixNearMany;
    const double unit = scalbn(1.0, -kx), dfi = s.df[sl];
    const int si = sidx(g, sl), end = many ? (in.far_flag[sl] ? nt.nfull : nt.npruned) : 4;
    const FixRec me = ld_fix_rec(s.fix + si);
    const float4 ui = s.u4[si];
    for (int e = 0; e < end; e++) {
        if (!many && !(near >> (8 * e))) break;
        const int q = many ? e : (int) ((near >> (8 * e)) & 255u) - 1;
        const float4 D = par ? nt.cand[1][q] : nt.cand[0][q];
        const int oj = si + __float_as_int(D.w);
        if (many && !near_f32(g, f2_pack(ui.x, ui.y), ui.z, D, s.u4[oj])) continue;
        const FixRec j = ld_fix_rec(s.fix + oj);
        const int sj = sl + (par ? nt.lat[1][q] : nt.lat[0][q]);
        double dx, dy, dz;
        fix_vector(me, j, unit, dx, dy, dz);
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (!(r2 < g.rc2)) continue;
        const double fpair = fpair_fp64(pt, r2, ti, (int) j.type, dfi, s.df[sj]);
        fx += dx * fpair;
        fy += dy * fpair;
        fz += dz * fpair;
    }
    return make_double3(fx, fy, fz);
}
// U candidates, as rho_fix_pairs. ONE: every type has the same tables
template <int U, bool ONE>
__device__ __forceinline__ void force_fix_pairs(const Slots &s, const FixParams &fp, const int (&oj)[U], const bool (&use)[U],
                                                const int (&q)[U], int ti, i64 xb, i64 yb, i64 zb, i64 dfb, FixForce &a) {
    FixRec j[U];
    i64 dfj[U];
    FixDelta d[U];
    FixCoord t[U];
    FixPoly pg[U], ph[U];
    bool in[U];
    int tj[U], m[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        j[u] = ld_fix_rec(s.fix + oj[u]);
        dfj[u] = __ldg(s.dfq + oj[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        d[u] = fix_delta(xb - j[u].x, yb - j[u].y, zb - j[u].z);
        const i64 r2 = fix_r2(d[u], fp.b0);
        in[u] = use[u] && (unsigned long long) (r2 - fp.lo) < (unsigned long long) (fp.rc2 - fp.lo);
        if (use[u] && (unsigned long long) r2 < (unsigned long long) fp.lo) fix_note_near(a.near, q[u]);
        t[u] = fix_locate(fp, in[u] ? r2 : fp.rc2 - 1, m[u]);
        tj[u] = !ONE && in[u] ? (int) j[u].type : ti;
        const FixPoly *rec = fp.zg + 2 * ((ti * 3 + tj[u]) * fp.nr1 + m[u]);
        pg[u] = ld_fix_poly(rec);
        ph[u] = ld_fix_poly(rec + 1);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const i64 gj = fix_poly(pg[u], t[u], fp.e3_g);
        i64 f = fix_poly(ph[u], t[u], fp.e3_h);
        const i64 both = dfb + dfj[u];  // biased
        if (in[u]) a.df_hi = max(a.df_hi, fix_hi(both));
        if (ONE || tj[u] == ti) {
            f = fix_mul_add(fix_hi(both), fix_lo(both), fix_hi(gj), fix_lo(gj), f);
        } else {
            const i64 gi = fix_poly(ld_fix_poly(fp.zg + 2 * ((tj[u] * 3 + ti) * fp.nr1 + m[u])), t[u], fp.e3_g);
            const i64 djb = dfj[u] + kFixBias;
            f = fix_mul_add(fix_hi(dfb), fix_lo(dfb), fix_hi(gj), fix_lo(gj), f);
            f = fix_mul_add(fix_hi(djb), fix_lo(djb), fix_hi(gi), fix_lo(gi), f);
        }
        if (!in[u]) f = kFixBias;  // zero as a factor
        const int fh = fix_hi(f), fl = fix_lo(f);
        a.x = fix_mul_add(d[u].xh, d[u].xl, fh, fl, a.x);
        a.y = fix_mul_add(d[u].yh, d[u].yl, fh, fl, a.y);
        a.z = fix_mul_add(d[u].zh, d[u].zl, fh, fl, a.z);
    }
}
// candidate q, at index oj. ONE: every atom is of the one type that the potential has
template <bool ONE>
__device__ __forceinline__ void force_fix_candidate(const Slots &s, const FixParams &fp, int oj, int ti, i64 xb,
                                                    i64 yb, i64 zb, i64 dfb, int q, FixForce &a) {
    const FixRec j = ld_fix_rec(s.fix + oj);
    const FixDelta d = fix_delta(xb - j.x, yb - j.y, zb - j.z);
    const i64 r2 = fix_r2(d, fp.b0);
    if ((unsigned long long) (r2 - fp.lo) < (unsigned long long) (fp.rc2 - fp.lo)) {
        const i64 dfj = __ldg(s.dfq + oj);
        int m;
        const FixCoord t = fix_locate(fp, r2, m);
        const int tj = ONE ? ti : (int) j.type;
        const FixPoly *rec = fp.zg + 2 * ((ti * 3 + tj) * fp.nr1 + m);
        const FixPoly pg = ld_fix_poly(rec), ph = ld_fix_poly(rec + 1);
        FixPoly pi;
        if (tj != ti) pi = ld_fix_poly(fp.zg + 2 * ((tj * 3 + ti) * fp.nr1 + m));
        const i64 gj = fix_poly(pg, t, fp.e3_g);
        i64 f = fix_poly(ph, t, fp.e3_h);
        const i64 both = dfb + dfj;  // biased
        a.df_hi = max(a.df_hi, fix_hi(both));
        if (tj == ti) {
            f = fix_mul_add(fix_hi(both), fix_lo(both), fix_hi(gj), fix_lo(gj), f);
        } else {
            const i64 gi = fix_poly(pi, t, fp.e3_g);
            const i64 djb = dfj + kFixBias;
            f = fix_mul_add(fix_hi(dfb), fix_lo(dfb), fix_hi(gj), fix_lo(gj), f);
            f = fix_mul_add(fix_hi(djb), fix_lo(djb), fix_hi(gi), fix_lo(gi), f);
        }
        const int fh = fix_hi(f), fl = fix_lo(f);
        a.x = fix_mul_add(d.xh, d.xl, fh, fl, a.x);
        a.y = fix_mul_add(d.yh, d.yl, fh, fl, a.y);
        a.z = fix_mul_add(d.zh, d.zl, fh, fl, a.z);
    } else if ((unsigned long long) r2 < (unsigned long long) fp.lo) {
        fix_note_near(a.near, q);
    }
}
template <int PAR, bool ONE>
__device__ __forceinline__ void force_fix_range(const NeighTables &nt, const Geom &g, const Slots &s, const FixParams &fp, int si,
                                                int ti, float4 ui, i64 xb, i64 yb, i64 zb, i64 dfb, int q0, int q1, FixForce &a) {
    const f2 uixy = f2_pack(ui.x, ui.y);
#pragma unroll 1
    for (int q = q0; q < q1; q++) {
        const float4 D = nt.cand[PAR][q];
        if (near_f32(g, uixy, ui.z, D, __ldg(s.u4 + si + __float_as_int(D.w))))
            force_fix_candidate<ONE>(s, fp, si + __float_as_int(D.w), ti, xb, yb, zb, dfb, q, a);
    }
}
template <int PAR, bool ONE>
__device__ __forceinline__ void force_fix_atom(const NeighTables &nt, const Geom &g, const Slots &s, const FixParams &fp, int si,
                                               int ti, const FixRec &me, const unsigned *list, bool far, FixForce &a, double3 &f) {
    const i64 xb = me.x + kFixBias, yb = me.y + kFixBias, zb = me.z + kFixBias, dfb = s.dfq[si] + kFixBias;
    const int np = nt.npruned;
    if (list) {
        for (int k = 0; k * 32 < np; k++)
            for (unsigned w = list[k]; w; w &= w - 1) {
                const int q = 32 * k + __ffs(w) - 1;
                force_fix_candidate<ONE>(s, fp, si + __float_as_int(nt.cand[PAR][q].w), ti, xb, yb, zb, dfb, q, a);
            }
    } else {
        force_fix_range<PAR, ONE>(nt, g, s, fp, si, ti, s.u4[si], xb, yb, zb, dfb, 0, np, a);
    }
    f = make_double3(-(double) a.x * fp.f_unit, -(double) a.y * fp.f_unit, -(double) a.z * fp.f_unit);
    if (far) {  // each part fits the integers by itself
        a.x = 0; a.y = 0; a.z = 0;
        force_fix_range<PAR, ONE>(nt, g, s, fp, si, ti, s.u4[si], xb, yb, zb, dfb, np, nt.nfull, a);
        f.x -= (double) a.x * fp.f_unit;
        f.y -= (double) a.y * fp.f_unit;
        f.z -= (double) a.z * fp.f_unit;
    }
}
// adds the near pairs; then as force_done_mixed
__device__ __forceinline__ void force_done_fix(const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                               const PotTables &pt, StepParams *sp, int sl, int si, int ti, int par, const FixForce &a,
                                               double3 f, bool kick, bool hook, bool fuse_next, bool wild) {
    const unsigned near = a.df_hi >= kFixBadHi ? kFixNearMany : a.near;
    if (near) {
        const double3 n = force_near_fp64(nt, g, s, in, pt, s.kx, sl, ti, par, near, wild);
        if (near == kFixNearMany) f = n;
        else { f.x += n.x; f.y += n.y; f.z += n.z; }
    }
    force_done(g, s, in, sp, sl, si, ti, f.x, f.y, f.z, kick, hook, fuse_next && kick && !hook && !wild && lattice_only(in));
}
// a vacant site: no force, and in a fused body the next firststep's records of a vacancy
__device__ __forceinline__ void force_vacant_fix(const Geom &g, const Slots &s, const Inter &in, int sl, int si, bool fuse_next, bool wild) {
    s.fx[sl] = 0.0; s.fy[sl] = 0.0; s.fz[sl] = 0.0;
    if (fuse_next && !wild && lattice_only(in)) {
        s.u4n[si] = vacant_u4();
        fix_put_vacant(g, s.fixn + si, s.kx, sl);
    }
}
template <bool ONE>
__device__ __forceinline__ void k_lat_force_fix_site(int t, const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                                     const PotTables &pt, const FixParams &fp, StepParams *sp, bool kick, bool hook,
                                                     int order, bool fuse_next, bool lists, bool wild) {
    int par, u;
    const int sl = gather_site(g, t, order, par, u);
    if (sl < 0) return;
    const int si = sidx(g, sl);
    const FixRec me = ld_fix_rec(s.fix + si);
    const int ti = (int) me.type;
    if (ti < 0) { force_vacant_fix(g, s, in, sl, si, fuse_next, wild); return; }
    FixForce a{0, 0, 0, 0, kFixNearMany};
    double3 f{0.0, 0.0, 0.0};
    if (!wild) {
        a.near = 0u;
        const unsigned *list = lists ? group_list(g, s, par, u) : nullptr;
        const bool far = in.far_flag[sl];
        if (par) force_fix_atom<1, ONE>(nt, g, s, fp, si, ti, me, list, far, a, f);
        else force_fix_atom<0, ONE>(nt, g, s, fp, si, ti, me, list, far, a, f);
    }
    force_done_fix(nt, g, s, in, pt, sp, sl, si, ti, par, a, f, kick, hook, fuse_next, wild);
}
template <bool LOOP, bool ONE>  // LOOP: several sites per thread, one grid stride apart (no group lists)
__global__ void __launch_bounds__(512, 2) k_lat_force_fix(const __grid_constant__ NeighTables nt, const __grid_constant__ Geom g,
                                                          const __grid_constant__ Slots s, const __grid_constant__ Inter in,
                                                          const __grid_constant__ PotTables pt, const __grid_constant__ FixParams fp,
                                                          StepParams *sp, bool kick, bool hook, int order, int tbase, int nthreads,
                                                          bool fuse_next, bool lists) {
    const int t0 = tbase + blockIdx.x * blockDim.x + threadIdx.x;  // threads [tbase, nthreads)
    const bool wild = pass_wild(s);
    if (!LOOP) {
        if (t0 < nthreads) k_lat_force_fix_site<ONE>(t0, nt, g, s, in, pt, fp, sp, kick, hook, order, fuse_next, lists && !wild, wild);
        return;
    }
    for (int t = t0; t < nthreads; t += gridDim.x * blockDim.x)
        k_lat_force_fix_site<ONE>(t, nt, g, s, in, pt, fp, sp, kick, hook, order, fuse_next, false, wild);
}

// Compensated force sums of the mixed form: each pair term d * fpair is added by Kahan's method
// (W. Kahan, "Further remarks on reducing truncation errors", CACM 8(1), 1965). The running error is
// kept negated (m = -c), so the term's product and the correction fuse into one rounding
// (y = d * fpair + m) and a component costs four operations; x and y go through the packed f32x2
// forms. The sum's value is s + m.
struct ForceAcc {
    f2 sxy, mxy;  // running sums and their negated compensations, x and y packed
    float sz, mz;
};
__device__ __forceinline__ void force_acc_add(ForceAcc &a, f2 dxy, float dz, float fpair) {
    const f2 yxy = f2_fma(dxy, f2_pack(fpair, fpair), a.mxy);
    const f2 txy = f2_add(a.sxy, yxy);
    a.mxy = f2_sub(yxy, f2_sub(txy, a.sxy));
    a.sxy = txy;
    const float yz = __fmaf_rn(dz, fpair, a.mz);
    const float tz = __fadd_rn(a.sz, yz);
    a.mz = __fsub_rn(yz, __fsub_rn(tz, a.sz));
    a.sz = tz;
}

// fpair of one pair inside the cutoff (types ti and tj, F' dfi and dfj): its table records, and its value
// from them. Every rounding is spelled out, so that each kernel that evaluates it gets the same bits.
struct PairRecord {
    PairKnot k;
    float z[8];  // {c0, d0, c1, d1, c2, d2, c3, 3 c3}: r*phi = c(p), rho_tj' = d(p)
    float4 d;    // rho_ti' where the types differ
};
__device__ __forceinline__ PairRecord pair_record(const PotTables &pt, float r2, int ti, int tj) {
    PairRecord r;
    r.k = pair_knot(pt, r2);
    ld_nc_v8(pt.zr8 + 8 * ((ti * 3 + tj) * pt.nr + r.k.m - kKnotBias), r.z);
    if (tj != ti) r.d = __ldg(pt.rho_dff + ti * pt.nr + r.k.m - kKnotBias);
    return r;
}
__device__ __forceinline__ float fpair_mixed(const Geom &g, const PotTables &pt, const PairRecord &r, int ti, int tj, float dfi,
                                             float dfj) {
    const float *z = r.z, p = r.k.p;
    // the last two steps of both polynomials in one packed Horner
    const f2 pp = f2_pack(p, p);
    f2 h = f2_fma(f2_pack(__fmaf_rn(z[6], p, z[4]), z[5]), pp, f2_pack(z[2], z[3]));
    h = f2_fma(h, pp, f2_pack(z[0], z[1]));
    float zv, rhojp;
    f2_unpack(h, zv, rhojp);
    const float zd = __fmaf_rn(__fmaf_rn(z[7], p, __fadd_rn(z[4], z[4])), p, z[2]);
    const float rhoip = (tj == ti) ? rhojp : __fmaf_rn(__fmaf_rn(r.d.z, p, r.d.y), p, r.d.x);
    const float rinv = __fmul_rn(r.k.rinv, g.inv_h_f);
    const float dphi = __fmaf_rn(zd, pt.inv_dr_f, -__fmul_rn(zv, rinv));  // phi' r
    const float psip = __fmaf_rn(dphi, rinv, __fmaf_rn(dfi, rhojp, __fmul_rn(dfj, rhoip)));
    return __fmul_rn(-psip, rinv);
}
// one candidate of the force pass: the pair term when inside the cutoff (false for vacancies, NaN); ONE: as
// force_fix_candidate
template <int PAR, bool ONE>
__device__ __forceinline__ void force_candidate(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt, int si,
                                                int ti, f2 uixy, float uiz, float dfi, int q, ForceAcc &acc) {
    const float4 D = nt.cand[PAR][q];
    const int oj = si + __float_as_int(D.w);
    const float4 uj = __ldg(s.u4 + oj);
    f2 dxy; float dz;
    const float r2 = pair_r2(uixy, uiz, D, uj, dxy, dz);
    if (r2 < g.rc2_h) {
        const int tj = ONE ? ti : __float_as_int(uj.w);
        force_acc_add(acc, dxy, dz, fpair_mixed(g, pt, pair_record(pt, r2, ti, tj), ti, tj, dfi, __ldg(s.df32 + oj)));
    }
}
template <int PAR, bool ONE>
__device__ __forceinline__ void force_sum_mixed(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt, int si, int ti,
                                                float4 ui, float dfi, int q0, int q1, ForceAcc &acc) {
    const f2 uixy = f2_pack(ui.x, ui.y);
#pragma unroll 1  // 2, 3, 4 and full unrolling measured slower
    for (int q = q0; q < q1; q++) force_candidate<PAR, ONE>(nt, g, s, pt, si, ti, uixy, ui.z, dfi, q, acc);
}
// the candidates of the warp's group list, in table order: the density pass of this step checked or
// rebuilt the list, so it holds every pruned candidate inside the cutoff for any site of the group
// (the cutoff is tested again here with the same rounding, so the pairs summed are those of the full
// loop, in the same order)
template <int PAR, bool ONE>
__device__ __forceinline__ void force_sum_listed(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt, int si,
                                                 int ti, float4 ui, float dfi, const unsigned *words, ForceAcc &acc) {
    const f2 uixy = f2_pack(ui.x, ui.y);
    for (int k = 0; k * 32 < nt.npruned; k++)
        for (unsigned w = words[k]; w; w &= w - 1)
            force_candidate<PAR, ONE>(nt, g, s, pt, si, ti, uixy, ui.z, dfi, 32 * k + __ffs(w) - 1, acc);
}

// the sums with their compensations, converted to FP64 once; then as force_done
__device__ __forceinline__ void force_done_mixed(const Geom &g, const Slots &s, const Inter &in, StepParams *sp, int sl, int si, int ti,
                                                 const ForceAcc &acc, bool kick, bool hook, bool fuse_next) {
    float sx, sy, mx, my;
    f2_unpack(acc.sxy, sx, sy);
    f2_unpack(acc.mxy, mx, my);
    const double h = 0.5 * g.a0;
    const double fx = h * ((double) sx + (double) mx);
    const double fy = h * ((double) sy + (double) my);
    const double fz = h * ((double) acc.sz + (double) acc.mz);
    force_done(g, s, in, sp, sl, si, ti, fx, fy, fz, kick, hook, fuse_next && kick && !hook && lattice_only(in));
}
// a vacant site: no force, and in a fused body the next firststep's record of a vacancy
__device__ __forceinline__ void force_vacant_mixed(const Geom &g, const Slots &s, const Inter &in, int sl, int si, bool fuse_next) {
    s.fx[sl] = 0.0; s.fy[sl] = 0.0; s.fz[sl] = 0.0;
    if (fuse_next && lattice_only(in)) s.u4n[si] = vacant_u4();
}
template <bool ONE>
__device__ __forceinline__ void k_lat_force_mixed_site(int t, const NeighTables &nt, const Geom &g, const Slots &s, const Inter &in,
                                                const PotTables &pt, StepParams *sp, bool kick, bool hook, int order,
                                                bool fuse_next, bool lists) {
    int par, u;
    const int sl = gather_site(g, t, order, par, u);
    if (sl < 0) return;
    const int si = sidx(g, sl);
    const float4 ui = s.u4[si];
    const int ti = __float_as_int(ui.w);
    if (ti < 0) { force_vacant_mixed(g, s, in, sl, si, fuse_next); return; }
    const float dfi = s.df32[si];
    // compensated force sums (x and y packed, z)
    ForceAcc acc{f2_pack(0.f, 0.f), f2_pack(0.f, 0.f), 0.f, 0.f};
    const int np = nt.npruned;
    if (lists) {
        const unsigned *w = group_list(g, s, par, u);
        if (par) force_sum_listed<1, ONE>(nt, g, s, pt, si, ti, ui, dfi, w, acc);
        else force_sum_listed<0, ONE>(nt, g, s, pt, si, ti, ui, dfi, w, acc);
    } else {
        if (par) force_sum_mixed<1, ONE>(nt, g, s, pt, si, ti, ui, dfi, 0, np, acc);
        else force_sum_mixed<0, ONE>(nt, g, s, pt, si, ti, ui, dfi, 0, np, acc);
    }
    if (in.far_flag[sl]) {
        const int nf = nt.nfull;
        if (par) force_sum_mixed<1, ONE>(nt, g, s, pt, si, ti, ui, dfi, np, nf, acc);
        else force_sum_mixed<0, ONE>(nt, g, s, pt, si, ti, ui, dfi, np, nf, acc);
    }
    force_done_mixed(g, s, in, sp, sl, si, ti, acc, kick, hook, fuse_next);
}
template <bool LOOP, bool ONE>  // LOOP: several sites per thread, one grid stride apart
__global__ void __launch_bounds__(512, 3) k_lat_force_mixed(const __grid_constant__ NeighTables nt, Geom g, Slots s, Inter in, PotTables pt,
                                                         StepParams *sp, bool kick, bool hook, int order, int tbase,
                                                         int nthreads, bool fuse_next, bool lists) {
    const int t0 = tbase + blockIdx.x * blockDim.x + threadIdx.x;  // threads [tbase, nthreads)
    if (!LOOP) {
        if (t0 < nthreads) k_lat_force_mixed_site<ONE>(t0, nt, g, s, in, pt, sp, kick, hook, order, fuse_next, lists);
        return;
    }
    for (int t = t0; t < nthreads; t += gridDim.x * blockDim.x)
        k_lat_force_mixed_site<ONE>(t, nt, g, s, in, pt, sp, kick, hook, order, fuse_next, false);
}

// ---- the force passes of small boxes and thin slabs: see rho_mixed_split (500 groups: 30 -> 14 us; FP64 form 58 ->
// 19 us) ----
template <int W>
__device__ __forceinline__ void force_mixed_split(const float4 *cand, int np, int nf, const Geom &g, const Slots &s, const Inter &in,
                                                  const PotTables &pt, StepParams *sp, const SplitSite &a, bool kick, bool hook,
                                                  bool fuse_next, bool lists, bool far, SplitList &sh, ForceAcc *out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int end = __any_sync(0xffffffffu, far) ? nf : np;
    SplitLane<W> b(a);
    constexpr int P = SplitLane<W>::P;
    const bool b_far = __shfl_sync(0xffffffffu, far, P * warp + lane % P);
    const float dfi = s.df32[b.si];
    ForceAcc acc{f2_pack(0.f, 0.f), f2_pack(0.f, 0.f), 0.f, 0.f};
    int q1;
    for (int q0 = 0; q0 < end; q0 = q1) {
        const bool tail = q0 >= np;
        q1 = min(q0 + kSplitSegment, tail ? end : np);
        const int n = split_list<W>(cand, s, a, !tail || far, q0, q1, g.rc2_h, lists && !tail ? group_list(g, s, a.par, a.u) : nullptr, sh);
        const bool mine = !tail || b_far;
        for (int c0 = 0; c0 < n; c0 += kSplitAhead * W) {
            float r2[kSplitAhead], dx[kSplitAhead], dy[kSplitAhead], dz[kSplitAhead], dfj[kSplitAhead], t[kSplitAhead];
            int tj[kSplitAhead];
#pragma unroll
            for (int u = 0; u < kSplitAhead; u++) {
                const float4 D = sh.rec[min(c0 + u * W + b.stream, n - 1)];
                const int oj = b.si + (b.in ? __float_as_int(D.w) : 0);
                const float4 uj = __ldg(s.u4 + oj);
                dfj[u] = __ldg(s.df32 + oj);
                f2 dxy;
                r2[u] = pair_r2(b.uixy, b.uiz, D, uj, dxy, dz[u]);
                f2_unpack(dxy, dx[u], dy[u]);
                tj[u] = max(__float_as_int(uj.w), 0);
            }
            PairRecord r[kSplitAhead];
#pragma unroll
            for (int u = 0; u < kSplitAhead; u++) r[u] = pair_record(pt, r2[u], b.ti, tj[u]);
#pragma unroll
            for (int u = 0; u < kSplitAhead; u++) t[u] = fpair_mixed(g, pt, r[u], b.ti, tj[u], dfi, dfj[u]);
#pragma unroll
            for (int u = 0; u < kSplitAhead; u++) {
                if (c0 + u * W >= n) break;
                const float v = c0 + u * W + b.stream < n && mine && r2[u] < g.rc2_h ? t[u] : __uint_as_float(kSplitNone);
#pragma unroll
                for (int k = 0; k < W; k++) {
                    const int from = P * k + lane % P;
                    const float tk = __shfl_sync(0xffffffffu, v, from), xk = __shfl_sync(0xffffffffu, dx[u], from);
                    const float yk = __shfl_sync(0xffffffffu, dy[u], from), zk = __shfl_sync(0xffffffffu, dz[u], from);
                    if (!split_none(tk)) force_acc_add(acc, f2_pack(xk, yk), zk, tk);
                }
            }
        }
    }
    if (b.stream == 0) out[P * warp + lane % P] = acc;
    __syncthreads();
    if (warp != 0 || a.sl < 0) return;
    if (a.ti < 0) { force_vacant_mixed(g, s, in, a.sl, a.si, fuse_next); return; }
    force_done_mixed(g, s, in, sp, a.sl, a.si, a.ti, out[lane], kick, hook, fuse_next);
}
template <int W>
__global__ void __launch_bounds__(32 * W, W == 8 ? 3 : 32 / W) k_lat_force_mixed_split(const float4 *cand, int np, int nf, Geom g, Slots s, Inter in,
                                                                  PotTables pt, StepParams *sp, bool kick, bool hook, int u0, int u1,
                                                                  bool fuse_next, bool lists) {
    __shared__ SplitList sh;
    __shared__ ForceAcc out[32];
    const SplitSite a = split_site(g, s, u0, u1);
    if (!__any_sync(0xffffffffu, a.ti >= 0)) {
        if (threadIdx.x < 32 && a.sl >= 0) force_vacant_mixed(g, s, in, a.sl, a.si, fuse_next);
        return;
    }
    const bool far = a.ti >= 0 && in.far_flag[a.sl];
    force_mixed_split<W>(cand + a.par * kMaxFull, np, nf, g, s, in, pt, sp, a, kick, hook, fuse_next, lists, far, sh, out);
}
// FP64 form
template <int W>
struct SplitForce {
    i64 x[W][32], y[W][32], z[W][32];
    int df_hi[W][32];
    unsigned near[W][32];
};
template <int W, int U, bool ONE>
__device__ __forceinline__ void force_fix_split(const NeighTables &nt, const float4 *cand, const Geom &g, const Slots &s,
                                                const Inter &in, const PotTables &pt, const FixParams &fp, StepParams *sp,
                                                const SplitSite &a, bool kick, bool hook, bool fuse_next, bool lists, bool far, bool wild,
                                                SplitList &sh, SplitForce<W> &part) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int np = nt.npruned, end = wild ? 0 : __any_sync(0xffffffffu, far) ? nt.nfull : np;
    FixForce tot{0, 0, 0, 0, wild ? kFixNearMany : 0u};
    double3 f{0.0, 0.0, 0.0};
    const FixRec me = a.ti >= 0 ? ld_fix_rec(s.fix + a.si) : FixRec{};
    const i64 xb = me.x + kFixBias, yb = me.y + kFixBias, zb = me.z + kFixBias;
    const i64 dfb = a.ti >= 0 ? s.dfq[a.si] + kFixBias : 0;
    int q1;
    for (int q0 = 0; q0 < end; q0 = q1) {
        const bool tail = q0 >= np;
        q1 = min(q0 + kSplitSegment, tail ? end : np);
        const bool mine = a.ti >= 0 && (!tail || far);
        const int n = split_list<W>(cand, s, a, mine, q0, q1, g.rc2_pre, lists && !tail ? group_list(g, s, a.par, a.u) : nullptr, sh);
        FixForce m{0, 0, 0, 0, 0u};
        if (mine) {
            const int c1 = n * (warp + 1) / W;
            for (int c = n * warp / W; c < c1; c += U) {
                int oj[U], q[U];
                bool use[U];
                split_next<U>(sh, a.si, q0, c, c1, oj, use, q);
                force_fix_pairs<U, ONE>(s, fp, oj, use, q, a.ti, xb, yb, zb, dfb, m);
            }
        }
        part.x[warp][lane] = m.x;
        part.y[warp][lane] = m.y;
        part.z[warp][lane] = m.z;
        part.df_hi[warp][lane] = m.df_hi;
        part.near[warp][lane] = m.near;
        __syncthreads();
        if (warp == 0) {
            for (int w = 1; w < W; w++) {
                m.x += part.x[w][lane];
                m.y += part.y[w][lane];
                m.z += part.z[w][lane];
            }
            for (int w = 0; w < W; w++) {
                tot.df_hi = max(tot.df_hi, part.df_hi[w][lane]);
                fix_join_near(tot.near, part.near[w][lane]);
            }
            f.x -= (double) m.x * fp.f_unit;
            f.y -= (double) m.y * fp.f_unit;
            f.z -= (double) m.z * fp.f_unit;
        }
    }
    if (warp != 0 || a.sl < 0) return;
    if (a.ti < 0) { force_vacant_fix(g, s, in, a.sl, a.si, fuse_next, wild); return; }
    force_done_fix(nt, g, s, in, pt, sp, a.sl, a.si, a.ti, a.par, tot, f, kick, hook, fuse_next, wild);
}
// B: blocks an SM holds
template <int W, int B, int U, bool ONE>
__global__ void __launch_bounds__(32 * W, B) k_lat_force_fix_split(const __grid_constant__ NeighTables nt, const float4 *cand,
                                                                        const __grid_constant__ Geom g, const __grid_constant__ Slots s,
                                                                        const __grid_constant__ Inter in,
                                                                        const __grid_constant__ PotTables pt,
                                                                        const __grid_constant__ FixParams fp, StepParams *sp, bool kick,
                                                                        bool hook, int u0, int u1, bool fuse_next, bool lists) {
    __shared__ SplitList sh;
    __shared__ SplitForce<W> part;
    const bool wild = pass_wild(s);
    const SplitSite a = split_site(g, s, u0, u1);
    if (!__any_sync(0xffffffffu, a.ti >= 0)) {
        if (threadIdx.x < 32 && a.sl >= 0) force_vacant_fix(g, s, in, a.sl, a.si, fuse_next, wild);
        return;
    }
    const bool far = a.ti >= 0 && in.far_flag[a.sl];
    force_fix_split<W, U, ONE>(nt, cand + a.par * kMaxFull, g, s, in, pt, fp, sp, a, kick, hook, fuse_next, lists && !wild, far, wild, sh, part);
}

// Where every type has the same tables (one_type), the force passes drop the third record of a pair of two types, its
// branch and the types: by the spills it saves as much as by the branch (2M atoms: mixed 419 -> 399 us, FP64 1227 -> 1163).
// With several, a pair's three FP64 records are loaded together (3 elements, 2M atoms: 1535 -> 1504 us).
static void launch_lat_force_threads(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, StepParams *p,
                                     bool kick, bool mixed, bool hook, int tb, int te, bool fuse_next = false,
                                     bool lists = false) {
    const int order = lc.force_order, b = lc.force_block;
    const int n = (te - tb + b * lc.force_apt - 1) / (b * lc.force_apt);
    if (n <= 0) return;
    const bool fuse = fuse_next && kick && !hook && (mixed || lc.fp);
    s = with_records(lc, s);
    if (lc.force_apt > 1) {
        if (mixed) k_lat_force_mixed<true, false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, p, kick, hook, order, tb, te, fuse, false);
        else if (lc.fp) k_lat_force_fix<true, false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, *lc.fp, p, kick, hook, order, tb, te, fuse, false);
        else k_lat_force_fp64<true><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, p, kick, hook, order, tb, te);
    } else {
        if (mixed && lc.one_type) k_lat_force_mixed<false, true><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, p, kick, hook, order, tb, te, fuse, lists);
        else if (mixed) k_lat_force_mixed<false, false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, p, kick, hook, order, tb, te, fuse, lists);
        else if (lc.fp && lc.one_type) k_lat_force_fix<false, true><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, *lc.fp, p, kick, hook, order, tb, te, fuse, lists);
        else if (lc.fp) k_lat_force_fix<false, false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, *lc.fp, p, kick, hook, order, tb, te, fuse, lists);
        else k_lat_force_fp64<false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, p, kick, hook, order, tb, te);
    }
}
// one element: a step of 16k atoms 50.2 -> 49.5 us, 65k 108.1 -> 103.9, 128k 172.4 -> 166.6
template <int W, bool ONE>
static void launch_force_fix_split(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, StepParams *p, bool kick, bool hook,
                                   int u0, int u1, bool fuse, bool lists) {
    const int n = split_groups(u0, u1);
    const float4 *cand = &lc.ntd->cand[0][0];
    // From two groups per SM on, one candidate at a time: at 64 registers the blocks of 8 warps still fit one wave. Force pass
    // with two -> one, us, one element: 307 groups 25.8 -> 22.6, 364 27.9 -> 22.9, 500 28.1 -> 26.0, 578 28.7 -> 26.5; three:
    // 28.4 -> 26.2, 31.9 -> 27.0, 32.7 -> 30.7, 33.4 -> 30.8. Below it two hide more of the loads.
    if constexpr (W == 8)
        if (n * lc.share > 2 * lc.num_sms) {
            k_lat_force_fix_split<W, 4, 1, ONE><<<n, 32 * W, 0, lc.stream>>>(*lc.nt, cand, g, s, in, t, *lc.fp, p, kick, hook, u0, u1, fuse, lists);
            return;
        }
    k_lat_force_fix_split<W, 20 / W, kFixForceAhead, ONE><<<n, 32 * W, 0, lc.stream>>>(*lc.nt, cand, g, s, in, t, *lc.fp, p, kick, hook, u0, u1, fuse, lists);
}
template <int W>
static void launch_force_split_w(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, StepParams *p, bool kick, bool mixed,
                                 bool hook, int u0, int u1, bool fuse_next, bool lists) {
    const int n = split_groups(u0, u1);
    const bool fuse = fuse_next && kick && !hook;
    s = with_records(lc, s);
    if (mixed)
        k_lat_force_mixed_split<W><<<n, 32 * W, 0, lc.stream>>>(&lc.ntd->cand[0][0], lc.nt->npruned, lc.nt->nfull, g, s, in, t, p, kick, hook, u0, u1,
                                                                fuse, lists);
    else if (lc.one_type) launch_force_fix_split<W, true>(lc, g, s, in, t, p, kick, hook, u0, u1, fuse, lists);
    else launch_force_fix_split<W, false>(lc, g, s, in, t, p, kick, hook, u0, u1, fuse, lists);
}
static bool launch_lat_force_split(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, StepParams *p, bool kick, bool mixed,
                                   bool hook, int u0, int u1, bool fuse_next, bool lists) {
    switch (split_warps(lc, mixed, lists, split_groups(u0, u1))) {
        case 8: launch_force_split_w<8>(lc, g, s, in, t, p, kick, mixed, hook, u0, u1, fuse_next, lists); return true;
        case 4: launch_force_split_w<4>(lc, g, s, in, t, p, kick, mixed, hook, u0, u1, fuse_next, lists); return true;
        case 2: launch_force_split_w<2>(lc, g, s, in, t, p, kick, mixed, hook, u0, u1, fuse_next, lists); return true;
        default: return false;
    }
}
void launch_lat_force(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, StepParams *p, bool kick,
                      bool mixed, bool hook, bool fuse_next, bool lists) {
    const bool v = lists && has_lists(lc, mixed) && !hook && lists_ok(lc, g);
    if (launch_lat_force_split(lc, g, s, in, t, p, kick, mixed, hook, 0, g.n_local_half, fuse_next, v)) return;
    launch_lat_force_threads(lc, g, s, in, t, p, kick, mixed, hook, 0, gather_threads(g, lc.force_order), fuse_next, v);
}
void launch_lat_force_sites(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, StepParams *p, bool kick,
                            bool mixed, int u0, int u1, bool lists) {
    if (u1 <= u0) return;
    int tb[2], te[2], nr;
    site_threads(g, lc.force_order, u0, u1, tb, te, nr);
    const bool v = lists && has_lists(lc, mixed) && lists_ok(lc, g);
    if (launch_lat_force_split(lc, g, s, in, t, p, kick, mixed, false, u0, u1, false, v)) return;
    for (int r = 0; r < nr; r++) launch_lat_force_threads(lc, g, s, in, t, p, kick, mixed, false, tb[r], te[r], false, v);
}

// NewtonMotion::secondstep for the inter atoms (src/newton_motion.cpp:57-74)
__device__ __forceinline__ void inter_secondstep(const Inter &in, StepParams *p, int t0, int stride) {
    const int n_inter = in.cnt[CNT_INTER];
    double v2max = 0.0;
    for (int a = t0; a < n_inter; a += stride) {
        const double c = dt_inv_m_of(p, in.type[a]);
        const double vx = __dadd_rn(in.vx[a], __dmul_rn(c, in.fx[a]));
        const double vy = __dadd_rn(in.vy[a], __dmul_rn(c, in.fy[a]));
        const double vz = __dadd_rn(in.vz[a], __dmul_rn(c, in.fz[a]));
        in.vx[a] = vx; in.vy[a] = vy; in.vz[a] = vz;
        v2max = fmax(v2max, speed2(vx, vy, vz));
    }
    if (v2max > 0.0) note_vmax2(p, v2max);
}
// the second half-kick as a phase of its own: lattice atoms and inter atoms (after a kicking force pass, that pass
// and the owner gather have taken it)
__global__ void k_secondstep(Geom g, Slots s, Inter in, StepParams *p) {
    const int stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    double v2max = 0.0;
    for (int t = t0; t < g.n_local; t += stride) {
        int i, j, k;
        const int sl = local_slot(g, t, i, j, k);
        const int ty = s.type[sl];
        if (ty < 0) continue;
        const double c = dt_inv_m_of(p, ty);
        const double vx = __dadd_rn(s.vx[sl], __dmul_rn(c, s.fx[sl]));
        const double vy = __dadd_rn(s.vy[sl], __dmul_rn(c, s.fy[sl]));
        const double vz = __dadd_rn(s.vz[sl], __dmul_rn(c, s.fz[sl]));
        s.vx[sl] = vx; s.vy[sl] = vy; s.vz[sl] = vz;
        v2max = fmax(v2max, speed2(vx, vy, vz));
    }
    if (v2max > 0.0) note_vmax2(p, v2max);
    inter_secondstep(in, p, t0, stride);
}
// grid-stride kernels that often have nothing to do: a grid no larger than the box needs, so a
// small box does not schedule a thousand idle blocks every step
inline int box_grid(const LaunchCtx &lc, const Geom &g, int per_sm, int threads) {
    return std::max(1, std::min(lc.num_sms * per_sm, (g.n_local + threads - 1) / threads));
}
void launch_secondstep(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, StepParams *p) {
    k_secondstep<<<box_grid(lc, g, 8, 256), 256, 0, lc.stream>>>(g, s, in, p);
}

// ------------------------------------------------------------------------------------------------
// timestep control (extension: the reference sets dt per stage, src/newton_motion.cpp:13-28)
// ------------------------------------------------------------------------------------------------
// dt/(2m) per type as NewtonMotion::preComputeDtInv2m computes it: (0.5 * dt * ftm2v) / m
__device__ __forceinline__ void set_dt_dev(StepParams *p, double dt) {
    p->dt = dt;
    const double dt_halve = __dmul_rn(__dmul_rn(0.5, dt), kFtm2v);
    for (int t = 0; t < 3; t++) p->dt_inv_m[t] = __ddiv_rn(dt_halve, c_mass[t]);
}
__global__ void k_set_step(StepParams *p, double dt, double dx_max, double dt_min, double dt_max) {
    p->dx_max = dx_max;
    p->dt_min = dt_min;
    p->dt_max = dt_max;
    set_dt_dev(p, dt);
}
void launch_set_step(const LaunchCtx &lc, StepParams *sp, double dt, double dx_max, double dt_min, double dt_max) {
    k_set_step<<<1, 1, 0, lc.stream>>>(sp, dt, dx_max, dt_min, dt_max);
}
// The timestep taken into the history and the clock; one thread, once a step.
__device__ __forceinline__ void step_record(StepParams *p) {
    const long long k = p->steps;
    p->hist[k % kDtHistory] = p->dt;
    p->time = __dadd_rn(p->time, p->dt);
    p->steps = k + 1;
}

// One block of kVmaxSlots threads, ahead of a step: reduce and clear the max words, then (variable mode)
// dt = clamp(dx_max / sqrt(max |v|^2), dt_min, dt_max); record dt and advance the clock.
__global__ void __launch_bounds__(kVmaxSlots) k_step_head(StepParams *p) {
    __shared__ unsigned long long part[kVmaxSlots / 32];
    const unsigned long long b = p->vmax2[threadIdx.x];
    p->vmax2[threadIdx.x] = 0ull;
    const unsigned hi = (unsigned) (b >> 32), lo = (unsigned) b;
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ((unsigned long long) mhi << 32) | mlo;
    __syncthreads();
    if (threadIdx.x != 0) return;
    unsigned long long m = 0ull;
    for (int w = 0; w < kVmaxSlots / 32; w++) m = part[w] > m ? part[w] : m;
    if (p->dx_max > 0.0) {
        const double v2 = __longlong_as_double((long long) m);
        double dt = v2 > 0.0 ? __ddiv_rn(p->dx_max, __dsqrt_rn(v2)) : p->dt_max;
        if (dt < p->dt_min) dt = p->dt_min;
        if (dt > p->dt_max) dt = p->dt_max;
        set_dt_dev(p, dt);
    }
    step_record(p);
}
void launch_step_head(const LaunchCtx &lc, StepParams *sp) {
    k_step_head<<<1, kVmaxSlots, 0, lc.stream>>>(sp);
}
// steps taken and simulated time into a sample record (stage machine thermo output)
__global__ void k_clock_sample(const StepParams *p, double *out) {
    out[0] = (double) p->steps;
    out[1] = p->time;
}
void launch_clock_sample(const LaunchCtx &lc, const StepParams *sp, double *out) {
    k_clock_sample<<<1, 1, 0, lc.stream>>>(sp, out);
}
// max |v|^2 over local lattice atoms and local inter atoms, from scratch
__global__ void k_vmax_full(Geom g, Slots s, Inter in, StepParams *p) {
    const int stride = gridDim.x * blockDim.x;
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
    double v2max = 0.0;
    for (int t = t0; t < g.n_local; t += stride) {
        int i, j, k;
        const int sl = local_slot(g, t, i, j, k);
        if (s.type[sl] < 0) continue;
        v2max = fmax(v2max, speed2(s.vx[sl], s.vy[sl], s.vz[sl]));
    }
    const int n_inter = in.cnt[CNT_INTER];
    for (int a = t0; a < n_inter; a += stride) v2max = fmax(v2max, speed2(in.vx[a], in.vy[a], in.vz[a]));
    if (v2max > 0.0) note_vmax2(p, v2max);
}
void launch_vmax_full(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, StepParams *sp) {
    cudaMemsetAsync(reinterpret_cast<char *>(sp) + offsetof(StepParams, vmax2), 0, sizeof(unsigned long long) * kVmaxSlots,
                    lc.stream);
    k_vmax_full<<<lc.num_sms * 8, 256, 0, lc.stream>>>(g, s, in, sp);
}

// ------------------------------------------------------------------------------------------------
// per-atom energy (extension): e_i = F(rho_i) + 1/2 sum_j phi_ij over lattice neighbours
// ------------------------------------------------------------------------------------------------
template <int PAR>
__device__ __forceinline__ double energy_sum_fp64(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt, int sl, int ti,
                                                  int q0, int q1) {
    const double xi = s.x[sl], yi = s.y[sl], zi = s.z[sl];
    double acc = 0.0;
    for (int q = q0; q < q1; q++) {
        const int sj = sl + nt.lat[PAR][q];
        const int tj = s.type[sj];
        if (tj < 0) continue;
        const double dx = xi - s.x[sj], dy = yi - s.y[sj], dz = zi - s.z[sj];
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 < g.rc2) {
            const double rinv = rsqrt(r2);
            int m; double p;
            locate_d(r2 * rinv, pt.inv_dr, pt.nr, m, p);
            acc += val_d(pt.z_v + (ti * 3 + tj) * pt.nr, m, p) * rinv;
        }
    }
    return acc;
}
template <int PAR>
__device__ __forceinline__ void energy_sum_mixed(const NeighTables &nt, const Geom &g, const Slots &s, const PotTables &pt, int si, int ti,
                                                 float4 ui, int q0, int q1, float &sum, float &comp) {
    const float inv_h = 1.0f / g.h_f;
    for (int q = q0; q < q1; q++) {
        const float4 D = nt.cand[PAR][q];
        const float4 uj = __ldg(s.u4 + si + __float_as_int(D.w));
        const float dx = (ui.x - uj.x) - D.x, dy = (ui.y - uj.y) - D.y, dz = (ui.z - uj.z) - D.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        if (r2 < g.rc2_h) {  // false for vacancies (NaN coordinates)
            const int tj = __float_as_int(uj.w);
            const float rinv_h = rsqrtf(r2);
            int m; float p;
            locate_f(r2 * rinv_h, pt.h_inv_dr_f, pt.nr, m, p);
            kahan(sum, comp, val_f(pt.z_vf + (ti * 3 + tj) * pt.nr, m, p) * (rinv_h * inv_h));
        }
    }
}

template <bool MIXED>
__global__ void __launch_bounds__(256) k_energy(const __grid_constant__ NeighTables nt, Geom g, Slots s, Inter in, PotTables pt, int order) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    int par;
    const int sl = gather_slot(g, t, order, par);
    if (sl < 0) return;
    const int ti = s.type[sl];
    if (ti < 0) { s.e[sl] = 0.0; return; }
    const int np = nt.npruned;
    const int nq = in.far_flag[sl] ? nt.nfull : np;
    if (!MIXED) {
        double acc = par ? energy_sum_fp64<1>(nt, g, s, pt, sl, ti, 0, np) : energy_sum_fp64<0>(nt, g, s, pt, sl, ti, 0, np);
        if (nq > np) acc += par ? energy_sum_fp64<1>(nt, g, s, pt, sl, ti, np, nq) : energy_sum_fp64<0>(nt, g, s, pt, sl, ti, np, nq);
        int m; double p;
        locate_d(s.rho[sl], pt.inv_drho, pt.nrho, m, p);
        s.e[sl] = val_d(pt.F_v + ti * pt.nrho, m, p) + 0.5 * acc;
    } else {
        const int si = sidx(g, sl);
        const float4 ui = s.u4[si];
        float sum = 0.f, comp = 0.f;
        if (par) energy_sum_mixed<1>(nt, g, s, pt, si, ti, ui, 0, np, sum, comp);
        else energy_sum_mixed<0>(nt, g, s, pt, si, ti, ui, 0, np, sum, comp);
        if (nq > np) {
            if (par) energy_sum_mixed<1>(nt, g, s, pt, si, ti, ui, np, nq, sum, comp);
            else energy_sum_mixed<0>(nt, g, s, pt, si, ti, ui, np, nq, sum, comp);
        }
        int m; float p;
        locate_f((float) s.rho[sl], pt.inv_drho_f, pt.nrho, m, p);
        s.e[sl] = (double) val_f(pt.F_vf + ti * pt.nrho, m, p) + 0.5 * ((double) sum - (double) comp);
    }
}
void launch_energy(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed) {
    const int b = 256, n = (gather_threads(g, 0) + b - 1) / b;
    if (mixed) k_energy<true><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, 0);
    else k_energy<false><<<n, b, 0, lc.stream>>>(*lc.nt, g, s, in, t, 0);
}

// ------------------------------------------------------------------------------------------------
// Far atoms: lattice atoms farther than 0.2 a0 from their site (after decide, only recombined
// atoms). Pairs beyond the pruned table can reach them, so the atom itself and the owner of every
// slot of its full neighbourhood get far_flag = 1: their gathers also run the tail of the table.
// (A normal atom k sees a far atom i across the periodic boundary through i's ghost image; k is the
// owner of a ghost slot in i's neighbourhood, so it is marked too.) Clearing writes 0 over the same
// slots of the old list. Work item e of a flat loop covers (far atom e / (nfull + 1), entry).
// ------------------------------------------------------------------------------------------------

// ------------------------------------------------------------------------------------------------
// Inter-atom list management: one block, so the reference's list order is kept exactly.
//   decide (src/atom.cpp:21-84), exchangeInter (src/pack/inter_particle_packer.cpp),
//   borderInter (src/pack/inter_border_packer.cpp), makeIndex (src/atom/inter_atom_list.cpp:27-45).
// ------------------------------------------------------------------------------------------------
constexpr int kManageThreads = 1024;

// exclusive block scan of one int per thread; returns the block total
__device__ int block_exclusive_scan(int v, int &excl) {
    __shared__ int warp_tot[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = (lane < (int) (blockDim.x >> 5)) ? warp_tot[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        warp_tot[lane] = t;  // inclusive
    }
    __syncthreads();
    const int warp_excl = w > 0 ? warp_tot[w - 1] : 0;
    excl = warp_excl + x - v;
    const int total = warp_tot[(blockDim.x >> 5) - 1];
    __syncthreads();
    return total;
}

// bitonic sort of n 64-bit keys in global memory by one block; buf capacity >= next pow2(n)
__device__ void block_bitonic_sort(long long *buf, int n) {
    int P = 1;
    while (P < n) P <<= 1;
    for (int i = n + threadIdx.x; i < P; i += blockDim.x) buf[i] = LLONG_MAX;
    __syncthreads();
    for (int kk = 2; kk <= P; kk <<= 1) {
        for (int jj = kk >> 1; jj > 0; jj >>= 1) {
            for (int i = threadIdx.x; i < P; i += blockDim.x) {
                const int l = i ^ jj;
                if (l > i) {
                    const long long a = buf[i], b = buf[l];
                    const bool up = (i & kk) == 0;
                    if ((a > b) == up) { buf[i] = b; buf[l] = a; }
                }
            }
            __syncthreads();
        }
    }
}

// the same sort in shared memory (sm holds at least next_pow2(n) keys)
__device__ void block_bitonic_sort_smem(long long *buf, int n, long long *sm) {
    int P = 1;
    while (P < n) P <<= 1;
    for (int i = threadIdx.x; i < P; i += blockDim.x) sm[i] = i < n ? buf[i] : LLONG_MAX;
    __syncthreads();
    for (int kk = 2; kk <= P; kk <<= 1) {
        for (int jj = kk >> 1; jj > 0; jj >>= 1) {
            for (int i = threadIdx.x; i < P; i += blockDim.x) {
                const int l = i ^ jj;
                if (l > i) {
                    const long long a = sm[i], b = sm[l];
                    const bool up = (i & kk) == 0;
                    if ((a > b) == up) { sm[i] = b; sm[l] = a; }
                }
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) buf[i] = sm[i];
    __syncthreads();
}

// The displaced list's local indices in increasing order (the second half of in.displaced), n of them. Up to
// 1024: each thread counts the smaller ones. More: kDispBuckets equal ranges of the local indices, each entry
// counts the smaller ones of its range; a range holds a handful (a cascade's displaced atoms spread over its
// rows). sm: kDispBuckets + 1024 ints.
constexpr int kDispBuckets = 4096;
__device__ const int *block_sort_displaced(const Geom &g, const Inter &in, int n, int *sm) {
    int *out = in.displaced + in.dcap;
    const int tid = threadIdx.x, nthr = blockDim.x;
    if (n <= 1024) {
        for (int e = tid; e < n; e += nthr) sm[e] = in.displaced[e];
        __syncthreads();
        for (int e = tid; e < n; e += nthr) {
            const int t = sm[e];
            int r = 0;
            for (int q = 0; q < n; q++) r += sm[q] < t;
            out[r] = t;
        }
        __syncthreads();
        return out;
    }
    int *first = sm, *tot = sm + kDispBuckets;  // first entry of each bucket; the threads' sums
    const int per = g.n_local / kDispBuckets + 1, own = kDispBuckets / nthr;  // own buckets a thread scans
    for (int b = tid; b < kDispBuckets; b += nthr) first[b] = 0;
    __syncthreads();
    for (int e = tid; e < n; e += nthr) atomicAdd(&first[in.displaced[e] / per], 1);
    __syncthreads();
    int v = 0;
    for (int b = own * tid; b < own * tid + own; b++) v += first[b];
    tot[tid] = v;
    __syncthreads();
    for (int o = 1; o < nthr; o <<= 1) {
        const int y = tid >= o ? tot[tid - o] : 0;
        __syncthreads();
        tot[tid] += y;
        __syncthreads();
    }
    int run = tot[tid] - v;
    for (int b = own * tid; b < own * tid + own; b++) {
        const int c = first[b];
        first[b] = run;
        run += c;
    }
    __syncthreads();
    // into the buckets, leaving each one's end in first (the bucket index is made after decide, so its keys are free)
    int *part = reinterpret_cast<int *>(in.bucket);
    for (int e = tid; e < n; e += nthr) {
        const int t = in.displaced[e];
        part[atomicAdd(&first[t / per], 1)] = t;
    }
    __syncthreads();
    for (int e = tid; e < n; e += nthr) {
        const int t = part[e], b = t / per, b0 = b ? first[b - 1] : 0, b1 = first[b];
        int r = b0;
        for (int q = b0; q < b1; q++) r += part[q] < t;
        out[r] = t;
    }
    __syncthreads();
    return out;
}

// inter record move helpers (scratch layout: 13 doubles per record)
__device__ __forceinline__ void inter_save(const Inter &in, int a, int dst) {
    double *d = in.scratch_d + 13 * dst;
    d[0] = in.x[a]; d[1] = in.y[a]; d[2] = in.z[a];
    d[3] = in.vx[a]; d[4] = in.vy[a]; d[5] = in.vz[a];
    d[6] = in.fx[a]; d[7] = in.fy[a]; d[8] = in.fz[a];
    d[9] = in.rho[a]; d[10] = in.df[a]; d[11] = 0.0; d[12] = 0.0;
    in.scratch_u[dst] = in.id[a];
    in.scratch_i[dst] = in.type[a];
}
__device__ __forceinline__ void inter_restore(const Inter &in, int src, int a) {
    const double *d = in.scratch_d + 13 * src;
    in.x[a] = d[0]; in.y[a] = d[1]; in.z[a] = d[2];
    in.vx[a] = d[3]; in.vy[a] = d[4]; in.vz[a] = d[5];
    in.fx[a] = d[6]; in.fy[a] = d[7]; in.fz[a] = d[8];
    in.rho[a] = d[9]; in.df[a] = d[10];
    in.id[a] = in.scratch_u[src];
    in.type[a] = in.scratch_i[src];
}

__device__ __forceinline__ void region_fw(const Geom &g, int d, int dir, int lo[3], int hi[3]) {
    const int gg[3] = {g.gx, g.gy, g.gz}, bb[3] = {g.bx, g.by, g.bz}, ee[3] = {g.Sx, g.Sy, g.Sz};
    for (int q = 0; q < 3; q++) { lo[q] = 0; hi[q] = ee[q]; }
    for (int q = d + 1; q < 3; q++) { lo[q] = gg[q]; hi[q] = gg[q] + bb[q]; }
    if (dir == 0) { lo[d] = gg[d]; hi[d] = 2 * gg[d]; }
    else { lo[d] = bb[d]; hi[d] = bb[d] + gg[d]; }
}

// borderInter's entries: the local inter atoms, then the ghost images made so far
__device__ __forceinline__ void border_entry(const Inter &in, int n_loc, int e, double p3[3], int &ty, int &root) {
    if (e < n_loc) {
        p3[0] = in.x[e]; p3[1] = in.y[e]; p3[2] = in.z[e];
        ty = in.type[e];
        root = e;
    } else {
        const int k = e - n_loc;
        p3[0] = in.gx[k]; p3[1] = in.gy[k]; p3[2] = in.gz[k];
        ty = in.gtype[k];
        root = in.groot[k];
    }
}
// bit r set: the entry's nearest site lies in the region sent to direction r
__device__ __forceinline__ int border_regions(const Geom &g, const int lo[2][3], const int hi[2][3], const double p3[3]) {
    long long c[3];
    near_lat_coord(g, p3[0], p3[1], p3[2], c);
    int m = 0;
    for (int r = 0; r < 2; r++)
        if (c[0] >= lo[r][0] && c[0] < hi[r][0] && c[1] >= lo[r][1] && c[1] < hi[r][1] && c[2] >= lo[r][2] &&
            c[2] < hi[r][2])
            m |= 1 << r;
    return m;
}
// ghost image q of an entry, shifted by sh along d (past the capacity: the overflow error)
__device__ __forceinline__ void border_put(Inter &in, int q, const double p3[3], int d, double sh, int ty, int root) {
    if (q >= in.gcap) {
        set_error(in, MG_DEVERR_GHOST_OVERFLOW);
        return;
    }
    double p[3] = {p3[0], p3[1], p3[2]};
    p[d] = __dadd_rn(p[d], sh);
    in.gx[q] = p[0]; in.gy[q] = p[1]; in.gz[q] = p[2];
    in.gtype[q] = ty;
    in.groot[q] = root;
    in.gdf[q] = 0.0;
}

__global__ void __launch_bounds__(kManageThreads) k_inter_manage(Geom g, Slots s, Inter in, int mask, bool mixed, StepParams *sp) {
    extern __shared__ long long sm_keys[];
    __shared__ int sh_n, sh_d;
    const int tid = threadIdx.x, nthr = blockDim.x;
    if ((mask & MANAGE_CLOCK) && tid == 0) step_record(sp);
    if ((mask & MANAGE_DECIDE) && s.kx && tid == 0) {  // the positions are firststep's now
        s.skin->wild = s.skin->wild_next;
        s.skin->wild_next = 0;
    }

    // The list counts are read once, by all threads before any is written, and then followed in
    // registers: every change to them is block-uniform (scan totals), and one global round trip
    // costs this single block about a microsecond. Thread 0 writes each change back for the
    // kernels that follow.
    int n_inter = in.cnt[CNT_INTER], n_ghost = in.cnt[CNT_GHOST];
    const int n_disp = in.cnt[CNT_DISPLACED];
    // The usual step of a crystal: no inter atom, no ghost image and nothing displaced, so every
    // phase would find its lists empty; what remains is decide voiding the previous step's far list
    // and the index being empty.
    const bool idle = n_inter == 0 && n_ghost == 0 && n_disp == 0;
    __syncthreads();
    if (idle) {
        if (tid == 0) {
            if (mask & MANAGE_DECIDE) in.cnt[CNT_FAR] = 0;
            if (mask & MANAGE_INDEX) *in.n_bucket = 0;
        }
        return;
    }

    if (mask & MANAGE_CLEAR_GHOST) {
        n_ghost = 0;
        if (tid == 0) in.cnt[CNT_GHOST] = 0;
    }

    if (mask & MANAGE_DECIDE) {
        // the far list of the previous step is void (its marks were cleared before this kernel)
        if (tid == 0) in.cnt[CNT_FAR] = 0;
        __syncthreads();
        // (i) displaced lattice atoms join the list in scan order
        int nd = n_disp;
        if (nd > in.dcap) { if (tid == 0) set_error(in, MG_DEVERR_DISPLACED_OVERFLOW); nd = in.dcap; }
        const int n0 = n_inter;
        if (nd > 0) {
            int room = in.cap - n0;
            const int *order = block_sort_displaced(g, in, nd, reinterpret_cast<int *>(sm_keys));
            if (nd > room) { if (tid == 0) set_error(in, MG_DEVERR_INTER_OVERFLOW); nd = room; }
            for (int q = tid; q < nd; q += nthr) {
                int i, j, k;
                const int sl = local_slot(g, order[q], i, j, k);
                const int a = n0 + q;
                in.id[a] = s.id[sl];
                in.type[a] = s.type[sl];
                in.x[a] = s.x[sl]; in.y[a] = s.y[sl]; in.z[a] = s.z[sl];
                in.vx[a] = s.vx[sl]; in.vy[a] = s.vy[sl]; in.vz[a] = s.vz[sl];
                in.fx[a] = s.fx[sl]; in.fy[a] = s.fy[sl]; in.fz[a] = s.fz[sl];
                in.rho[a] = s.rho[sl];
                in.df[a] = mixed ? (double) s.df32[sidx(g, sl)] : s.df[sl];
                s.type[sl] = kInvalid;
                s.vx[sl] = 0.0; s.vy[sl] = 0.0; s.vz[sl] = 0.0;
                s.u4[sidx(g, sl)] = vacant_u4();
                if (s.kx) fix_put_vacant(g, s.fix + sidx(g, sl), s.kx, sl);
            }
            __syncthreads();
            n_inter = n0 + nd;
            if (tid == 0) in.cnt[CNT_INTER] = n_inter;
        }
        if (tid == 0) in.cnt[CNT_DISPLACED] = 0;
        __syncthreads();

        // (ii) recombination with vacancies, first claimant in list order wins
        const int n = n_inter;
        int *cand = in.scratch_i + in.cap;  // n ints
        for (int a = tid; a < n; a += nthr) {
            const int near = near_index_in_sub_box(g, in.x[a], in.y[a], in.z[a]);
            int c = -1;
            if (near >= 0 && s.type[near] == kInvalid && is_out_box(g, s.x[near], s.y[near], s.z[near]) == kInBox) {
                c = near;
                atomicMin(&in.claim[near], a);
            }
            cand[a] = c;
        }
        __syncthreads();
        int *won = in.scratch_i + in.cap + in.cap;  // n ints
        int any_won = 0;
        for (int a = tid; a < n; a += nthr) {
            won[a] = (cand[a] >= 0 && in.claim[cand[a]] == a) ? 1 : 0;
            any_won |= won[a];
        }
        const bool recombined = __syncthreads_or(any_won);
        for (int a = tid; a < n; a += nthr) if (cand[a] >= 0) in.claim[cand[a]] = INT_MAX;
        // nobody recombined (the usual step): the compaction would rewrite the list unchanged
        if (recombined) {
            for (int a = tid; a < n; a += nthr) {
                if (!won[a]) continue;
                const int sl = cand[a];
                s.id[sl] = in.id[a];
                s.type[sl] = (int8_t) in.type[a];
                s.x[sl] = in.x[a]; s.y[sl] = in.y[a]; s.z[sl] = in.z[a];
                s.vx[sl] = in.vx[a]; s.vy[sl] = in.vy[a]; s.vz[sl] = in.vz[a];
                {
                    const int X = sl % g.Sx, r = sl / g.Sx, Y = r % g.Sy, Z = r / g.Sy;
                    double xs, ys, zs;
                    site_of(g, X, Y, Z, xs, ys, zs);
                    s.u4[sidx(g, sl)] = make_u4(g, in.x[a], in.y[a], in.z[a], xs, ys, zs, in.type[a]);
                    if (s.kx) fix_put(s.fix + sidx(g, sl), s.kx, in.x[a], in.y[a], in.z[a], in.type[a]);
                }
                // A recombined atom may sit up to sqrt(5)/4 a0 from its new site. Every recombined atom
                // joins this step's far list: the marks on its neighbourhood also make the density pass
                // rebuild the candidate lists of the groups that can see it (its record did not come
                // from firststep). The tail pairs the marks add for an atom within 0.2 a0 of its site
                // are all beyond the cutoff, so they change no sum.
                {
                    const int q = atomicAdd(&in.cnt[CNT_FAR], 1);
                    if (q < in.fcap) in.far_list[q] = sl;
                    else set_error(in, MG_DEVERR_DISPLACED_OVERFLOW);
                }
            }
            __syncthreads();
            // stable compaction of the survivors: a short list's records through one warp's registers
            int base = 0;
            if (n <= 32) {
                if (tid < 32) {
                    const bool keep = tid < n && !won[tid];
                    const unsigned kept = __ballot_sync(0xffffffffu, keep);
                    double *const col[11] = {in.x, in.y, in.z, in.vx, in.vy, in.vz, in.fx, in.fy, in.fz, in.rho, in.df};
                    double v[11];
                    uint64_t id = 0;
                    int type = 0;
                    if (keep) {
#pragma unroll
                        for (int f = 0; f < 11; f++) v[f] = col[f][tid];
                        id = in.id[tid];
                        type = in.type[tid];
                    }
                    __syncwarp();
                    const int to = __popc(kept & ((1u << tid) - 1u));
                    if (keep && to != tid) {
#pragma unroll
                        for (int f = 0; f < 11; f++) col[f][to] = v[f];
                        in.id[to] = id;
                        in.type[to] = type;
                    }
                    if (tid == 0) sh_n = __popc(kept);
                }
                __syncthreads();
                base = sh_n;
            }
            for (int c0 = 0; c0 < n && n > 32; c0 += nthr) {
                const int a = c0 + tid;
                const int keep = (a < n && !won[a]) ? 1 : 0;
                int ex;
                const int tot = block_exclusive_scan(keep, ex);
                if (keep) inter_save(in, a, base + ex);
                base += tot;
            }
            __syncthreads();
            if (n > 32)
                for (int a = tid; a < base; a += nthr) inter_restore(in, a, a);
            n_inter = base;
            if (tid == 0) in.cnt[CNT_INTER] = base;
        }
        __syncthreads();
    }

    if (mask & MANAGE_EXCHANGE) {
        const uint32_t lowf[3] = {kXLow, kYLow, kZLow}, highf[3] = {kXHigh, kYHigh, kZHigh};
        // an atom's out-of-box flags are found once and kept until a partition moves and shifts the
        // records (each thread keeps the same atoms from one dimension to the next)
        uint32_t *flags = reinterpret_cast<uint32_t *>(in.scratch_i + 2 * in.cap);
        uint32_t outside = 0;
        for (int a = tid; a < n_inter; a += nthr) {
            flags[a] = is_out_box(g, in.x[a], in.y[a], in.z[a]);
            outside |= flags[a];
        }
        bool flags_valid = true;
        const bool leaving = __syncthreads_or(outside != 0);
        for (int d = 0; d < 3 && leaving; d++) {
            const int n = n_inter;
            int *cls = in.scratch_i + in.cap;  // 0 stay, 1 lower, 2 higher
            int leaves = 0;
            for (int a = tid; a < n; a += nthr) {
                if (!flags_valid) flags[a] = is_out_box(g, in.x[a], in.y[a], in.z[a]);
                const uint32_t f = flags[a];
                cls[a] = (f & lowf[d]) ? 1 : ((f & highf[d]) ? 2 : 0);
                leaves |= cls[a];
            }
            flags_valid = true;
            // nobody crosses this dimension's faces (the usual case): the stable partition below
            // would rewrite the list unchanged
            if (!__syncthreads_or(leaves)) continue;
            int base = 0;
            for (int which = 0; which < 3; which++) {
                for (int c0 = 0; c0 < n; c0 += nthr) {
                    const int a = c0 + tid;
                    const int sel = (a < n && cls[a] == which) ? 1 : 0;
                    int ex;
                    const int tot = block_exclusive_scan(sel, ex);
                    if (sel) {
                        const int dst = base + ex;
                        inter_save(in, a, dst);
                        if (which != 0) {
                            double *rec = in.scratch_d + 13 * dst;
                            const double sh = (which == 1) ? g.L[d] : -g.L[d];
                            rec[d] = __dadd_rn(rec[d], sh);
                            rec[6] = 0.0; rec[7] = 0.0; rec[8] = 0.0; rec[9] = 0.0; rec[10] = 0.0;
                        }
                    }
                    base += tot;
                }
            }
            __syncthreads();
            for (int a = tid; a < n; a += nthr) inter_restore(in, a, a);
            flags_valid = false;
            __syncthreads();
        }
    }

    if (mask & MANAGE_BORDER) {
        // Both directions of a dimension send from the same entries, so each entry's nearest site is
        // found once per dimension. With one chunk of entries (the usual case) both directions share
        // one scan: the lower direction's selections are counted in the low 16 bits of the packed
        // sums, the higher's above them. With more, the lower pass keeps both region tests in mk
        // (bit 0 the region sent LOWER, bit 1 the one sent HIGHER) for the higher pass; each thread
        // keeps the same entries in both passes, and cap + gcap ints fit in the 13 * cap doubles of
        // scratch_d.
        int *mk = reinterpret_cast<int *>(in.scratch_d);
        int d0 = 0;
        if (n_inter + n_ghost <= 32) {
            // one warp, an entry per lane, no block barriers; an entry's nearest site is found once
            if (tid < 32) {
                int d = 0, ng = n_ghost, ty = 0, root = 0;
                double p3[3] = {0.0, 0.0, 0.0};
                long long c[3] = {0, 0, 0};
                bool found = false;
#pragma unroll
                for (int dd = 0; dd < 3; dd++) {
                    const int total = n_inter + ng;
                    if (total > 32) break;
                    if (tid < total && !found) {
                        border_entry(in, n_inter, tid, p3, ty, root);
                        near_lat_coord(g, p3[0], p3[1], p3[2], c);
                        found = true;
                    }
                    int m = 0;
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        int lo[3], hi[3];
                        region_fw(g, dd, r, lo, hi);
                        if (tid < total && c[0] >= lo[0] && c[0] < hi[0] && c[1] >= lo[1] && c[1] < hi[1] && c[2] >= lo[2] && c[2] < hi[2])
                            m |= 1 << r;
                    }
                    const unsigned b0 = __ballot_sync(0xffffffffu, m & 1), b1 = __ballot_sync(0xffffffffu, m & 2);
                    const unsigned below = (1u << tid) - 1u;
                    const int base1 = min(ng + __popc(b0), in.gcap);
                    if (m & 1) border_put(in, ng + __popc(b0 & below), p3, dd, g.L[dd], ty, root);
                    if (m & 2) border_put(in, base1 + __popc(b1 & below), p3, dd, -g.L[dd], ty, root);
                    ng = min(base1 + __popc(b1), in.gcap);
                    d = dd + 1;
                    __syncwarp();
                }
                if (tid == 0) {
                    sh_d = d;
                    sh_n = ng;
                    in.cnt[CNT_GHOST] = ng;
                }
            }
            __syncthreads();
            d0 = sh_d;
            n_ghost = sh_n;
            __syncthreads();
        }
        for (int d = d0; d < 3; d++) {
            const int n_loc = n_inter;
            const int total = n_loc + n_ghost;
            int lo[2][3], hi[2][3];
            region_fw(g, d, 0, lo[0], hi[0]);
            region_fw(g, d, 1, lo[1], hi[1]);
            if (total <= nthr) {
                double p3[3] = {0.0, 0.0, 0.0};
                int ty = 0, root = 0, m = 0;
                if (tid < total) {
                    border_entry(in, n_loc, tid, p3, ty, root);
                    m = border_regions(g, lo, hi, p3);
                }
                int ex;
                const int tot = block_exclusive_scan((m & 1) | ((m & 2) << 15), ex);
                const int base1 = min(n_ghost + (tot & 0xffff), in.gcap);
                if (m & 1) border_put(in, n_ghost + (ex & 0xffff), p3, d, g.L[d], ty, root);
                if (m & 2) border_put(in, base1 + (ex >> 16), p3, d, -g.L[d], ty, root);
                n_ghost = min(base1 + (tot >> 16), in.gcap);
                if (tid == 0) in.cnt[CNT_GHOST] = n_ghost;
                __syncthreads();
                continue;
            }
            for (int dir = 0; dir < 2; dir++) {
                const double sh = (dir == 0) ? g.L[d] : -g.L[d];
                int base = n_ghost;
                for (int c0 = 0; c0 < total; c0 += nthr) {
                    const int e = c0 + tid;
                    int sel = 0;
                    if (e < total) {
                        if (dir == 0) {
                            double p3[3];
                            int ty, root;
                            border_entry(in, n_loc, e, p3, ty, root);
                            const int m = border_regions(g, lo, hi, p3);
                            mk[e] = m;
                            sel = m & 1;
                        } else {
                            sel = (mk[e] >> 1) & 1;
                        }
                    }
                    int ex;
                    const int tot = block_exclusive_scan(sel, ex);
                    if (sel) {
                        double p3[3];
                        int ty, root;
                        border_entry(in, n_loc, e, p3, ty, root);
                        border_put(in, base + ex, p3, d, sh, ty, root);
                    }
                    base += tot;
                }
                n_ghost = base < in.gcap ? base : in.gcap;
                if (tid == 0) in.cnt[CNT_GHOST] = n_ghost;
                __syncthreads();
            }
        }
    }

    if (mask & MANAGE_INDEX) {
        const int n_loc = n_inter;
        const int n_gh = n_ghost;
        const int total = n_loc + n_gh;
        long long mine = LLONG_MAX;
        for (int e = tid; e < total; e += nthr) {
            double px, py, pz;
            int ref;
            if (e < n_loc) { px = in.x[e]; py = in.y[e]; pz = in.z[e]; ref = e; }
            else { const int q = e - n_loc; px = in.gx[q]; py = in.gy[q]; pz = in.gz[q]; ref = in.cap + q; }
            long long c[3];
            near_lat_coord(g, px, py, pz, c);
            long long key;
            if (c[0] < 0 || c[1] < 0 || c[2] < 0 || c[0] >= g.Sx || c[1] >= g.Sy || c[2] >= g.Sz) {
                set_error(in, MG_DEVERR_OUT_OF_GRID);
                key = INT_MAX;
            } else {
                key = lin(g, (int) c[0], (int) c[1], (int) c[2]);
            }
            mine = (key << 32) | (long long) ref;
            if (total > 32) in.bucket[e] = mine;
        }
        if (total <= 32) {  // ranked by one warp
            if (tid < 32) {
                int r = 0;
                for (int k = 0; k < 32; k++) r += __shfl_sync(0xffffffffu, mine, k) < mine;
                if (tid < total) in.bucket[r] = mine;
                if (tid == 0) *in.n_bucket = total;
            }
            return;
        }
        __syncthreads();
        if (total <= kSortSmemKeys) block_bitonic_sort_smem(in.bucket, total, sm_keys);
        else block_bitonic_sort(in.bucket, total);
        if (tid == 0) *in.n_bucket = total;
    }
}

// the list manager sorts up to kSortSmemKeys bucket keys in dynamic shared memory
void configure_manage_kernel() {
    cudaFuncSetAttribute(k_inter_manage, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(kSortSmemKeys * sizeof(long long)));
}
void launch_inter_manage(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, int mask, bool mixed, StepParams *sp) {
    k_inter_manage<<<1, kManageThreads, kSortSmemKeys * sizeof(long long), lc.stream>>>(g, with_records(lc, s), in, mask, mixed, sp);
}

// ------------------------------------------------------------------------------------------------
// inter-atom EAM (atom::interRho / interForce, src/atom.cpp:194-284, 360-473), FP64 arithmetic.
// One warp per local inter atom sums the atom's own terms. The Newton-3 shares that the reference
// scatters into lattice atoms (and folds from ghost slots into their owners) are summed instead by
// the owners themselves, in a fixed order, so every run gives the same bits: the inter-atom pass
// lists each lattice owner it finds inside the cutoff, and an owner gather over that list adds the
// owner's inter-atom terms in offset order, then bucket order.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ int bucket_begin(const Inter &in, int nb, int key) {
    int lo = 0, hi = nb;
    const long long want = ((long long) key) << 32;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (in.bucket[mid] < want) lo = mid + 1; else hi = mid;
    }
    return lo;
}
struct InterRef {
    double x, y, z, df;
    int type;
    uint64_t id;
};
__device__ __forceinline__ InterRef inter_ref(const Inter &in, int ref) {
    InterRef r;
    if (ref < in.cap) { r.x = in.x[ref]; r.y = in.y[ref]; r.z = in.z[ref]; r.type = in.type[ref]; r.id = in.id[ref]; r.df = in.df[ref]; }
    else {
        const int q = ref - in.cap;
        r.x = in.gx[q]; r.y = in.gy[q]; r.z = in.gz[q]; r.type = in.gtype[q]; r.id = 0; r.df = in.df[in.groot[q]];
    }
    return r;
}
__device__ __forceinline__ double rho_fn(const PotTables &pt, int type, double r2) {
    int m; double p;
    locate_d(sqrt(r2), pt.inv_dr, pt.nr, m, p);
    return val_d(pt.rho_v + type * pt.nr, m, p);
}
__device__ __forceinline__ double to_force(const PotTables &pt, int ti, int tj, double r2, double dfi, double dfj) {
    const double r = sqrt(r2);
    int m; double p;
    locate_d(r, pt.inv_dr, pt.nr, m, p);
    const double rhoip = der_d(pt.rho_d + ti * pt.nr, m, p);
    const double rhojp = der_d(pt.rho_d + tj * pt.nr, m, p);
    const double zv = val_d(pt.z_v + (ti * 3 + tj) * pt.nr, m, p);
    const double zp = der_d(pt.z_d + (ti * 3 + tj) * pt.nr, m, p);
    const double recip = 1.0 / r;
    const double phi = zv * recip;
    const double phip = zp * recip - phi * recip;
    const double psip = dfi * rhojp + dfj * rhoip + phip;
    return -psip * recip;
}
__device__ __forceinline__ double pair_fn(const PotTables &pt, int ti, int tj, double r2) {
    const double r = sqrt(r2);
    int m; double p;
    locate_d(r, pt.inv_dr, pt.nr, m, p);
    return val_d(pt.z_v + (ti * 3 + tj) * pt.nr, m, p) / r;
}
__device__ __forceinline__ double lat_df(const Geom &g, const Slots &s, int sl, bool mixed) {
    return mixed ? (double) s.df32[sidx(g, sl)] : s.df[sl];
}

// kind: 0 density, 1 force, 2 energy
// One block of kInterThreads per inter atom (the lists hold a few to thousands of atoms, each with
// ~460 partner entries): the threads share the 229 lattice entries and the 229 bucket keys of the
// atom's nearest site, two each, keep partial sums, and reduce them in a fixed order (shuffles within
// a warp, then the warps in order). With a few inter atoms the pass is one chain of dependent FP64
// spline evaluations per thread, so spreading an atom over four warps instead of one cuts its
// latency. Every lattice owner with a partner inside the cutoff is listed once (touch_owner) for
// k_inter_owner, which adds the owner's share of the pair terms.
constexpr int kInterThreads = 128;
__device__ __forceinline__ double warp_sum_d(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// lists a lattice owner for the owner gather: the first caller to set its bit appends it
__device__ __forceinline__ void touch_owner(Inter &in, int own) {
    const unsigned bit = 1u << (own & 31);
    if (atomicOr(&in.touch_bits[own >> 5], bit) & bit) return;
    const int q = atomicAdd(&in.cnt[CNT_TOUCHED], 1);
    if (q < in.tcap) in.touched[q] = own;
    else set_error(in, MG_DEVERR_INTER_OVERFLOW);
}
// a slot of the local box (not a ghost slot)
__device__ __forceinline__ bool is_local_slot(const Geom &g, int sl) {
    const int X = sl % g.Sx, r = sl / g.Sx, Y = r % g.Sy, Z = r / g.Sy;
    return X >= g.gx && X < g.gx + g.bx && Y >= g.gy && Y < g.gy + g.by && Z >= g.gz && Z < g.gz + g.bz;
}
template <int KIND>
__device__ __forceinline__ void inter_eam(const NeighTables &nt, const Geom &g, const Slots &s, Inter &in, const PotTables &pt, bool mixed,
                                          int block, int blocks) {
    const int n = in.cnt[CNT_INTER];
    const int nb = *in.n_bucket;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ double red[3][kInterThreads / 32];
    for (int a = block; a < n; a += blocks) {  // block-uniform
        const double xa = in.x[a], ya = in.y[a], za = in.z[a];
        const int ta = in.type[a];
        const uint64_t ida = in.id[a];
        const double dfa = in.df[a];
        const int near = near_index_in_sub_box(g, xa, ya, za);
        if (near < 0) continue;
        double acc = 0.0, fx = 0.0, fy = 0.0, fz = 0.0;
        // lattice partners: the nearest site's atom, then the full offsets of that site
        const int par = (near % g.Sx) & 1;
        const int nf = nt.nfull;
        for (int q = (int) threadIdx.x - 1; q < nf; q += kInterThreads) {
            const int sj = q < 0 ? near : near + nt.full[par][q];
            if (sj < 0 || sj >= g.n_slots) { set_error(in, MG_DEVERR_OUT_OF_GRID); continue; }
            // a ghost slot's record from its owner, shifted as the ghost copy shifts it, so that the pass need
            // not wait for that copy (or for the copy of F'); the energies follow both and read the slot itself
            int wx, wy, wz;
            const int X = sj % g.Sx, r = sj / g.Sx, Y = r % g.Sy, Z = r / g.Sy;
            const int own = lin(g, wrap_axis(X, g.gx, g.bx, wx), wrap_axis(Y, g.gy, g.by, wy), wrap_axis(Z, g.gz, g.bz, wz));
            const int at = KIND == 2 ? sj : own;
            const int tj = s.type[at];
            if (tj < 0) continue;
            const double xj = KIND == 2 ? s.x[at] : shifted(s.x[at], wx, g.L[0]);
            const double yj = KIND == 2 ? s.y[at] : shifted(s.y[at], wy, g.L[1]);
            const double zj = KIND == 2 ? s.z[at] : shifted(s.z[at], wz, g.L[2]);
            const double dx = xa - xj, dy = ya - yj, dz = za - zj;
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (!(r2 < g.rc2)) continue;
            touch_owner(in, own);
            if (KIND == 0) {
                acc += rho_fn(pt, tj, r2);
            } else if (KIND == 1) {
                const double fp = to_force(pt, ta, tj, r2, dfa, lat_df(g, s, own, mixed));
                fx += dx * fp; fy += dy * fp; fz += dz * fp;
            } else {
                acc += 0.5 * pair_fn(pt, ta, tj, r2);
            }
        }
        // inter partners: same-site bucket (not itself), then the buckets of the full offsets
        for (int q = (int) threadIdx.x - 1; q < nf; q += kInterThreads) {
            const int key = q < 0 ? near : near + nt.full[par][q];
            for (int b = bucket_begin(in, nb, key); b < nb && (int) (in.bucket[b] >> 32) == key; b++) {
                const InterRef o = inter_ref(in, (int) (in.bucket[b] & 0xffffffffLL));
                if (q < 0 && o.id == ida) continue;
                const double dx = xa - o.x, dy = ya - o.y, dz = za - o.z;
                const double r2 = dx * dx + dy * dy + dz * dz;
                if (!(r2 < g.rc2)) continue;
                if (KIND == 0) acc += rho_fn(pt, o.type, r2);
                else if (KIND == 1) {
                    const double fp = to_force(pt, ta, o.type, r2, dfa, o.df);
                    fx += dx * fp; fy += dy * fp; fz += dz * fp;
                } else {
                    acc += 0.5 * pair_fn(pt, ta, o.type, r2);
                }
            }
        }
        // the threads' partial sums: shuffles within each warp, then the warps' sums in warp order
        if (KIND == 1) {
            fx = warp_sum_d(fx);
            fy = warp_sum_d(fy);
            fz = warp_sum_d(fz);
            if (lane == 0) { red[0][warp] = fx; red[1][warp] = fy; red[2][warp] = fz; }
        } else {
            acc = warp_sum_d(acc);
            if (lane == 0) red[0][warp] = acc;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            acc = red[0][0]; fy = red[1][0]; fz = red[2][0];
            for (int w = 1; w < kInterThreads / 32; w++) {
                acc += red[0][w];
                if (KIND == 1) { fy += red[1][w]; fz += red[2][w]; }
            }
            fx = acc;
        }
        __syncthreads();  // red is reused by the block's next atom
        if (threadIdx.x != 0) continue;
        if (KIND == 0) {
            in.rho[a] = acc;
            int m; double p;
            locate_d(acc, pt.inv_drho, pt.nrho, m, p);
            in.df[a] = der_d(pt.F_d + ta * pt.nrho, m, p);
        } else if (KIND == 1) {
            in.fx[a] = fx; in.fy[a] = fy; in.fz[a] = fz;
        } else {
            int m; double p;
            locate_d(in.rho[a], pt.inv_drho, pt.nrho, m, p);
            in.e[a] = val_d(pt.F_v + ta * pt.nrho, m, p) + acc;
        }
    }
}
template <int KIND>
__global__ void __launch_bounds__(kInterThreads) k_inter_eam(const NeighTables *nt, Geom g, Slots s, Inter in, PotTables pt, bool mixed) {
    inter_eam<KIND>(*nt, g, s, in, pt, mixed, blockIdx.x, gridDim.x);
}
// blocks of the inter-atom pass beside a kernel over the ghost slots
inline int inter_blocks(const LaunchCtx &lc, const Geom &g) {
    return std::max(1, std::min(lc.num_sms * 4, (g.n_local + kInterThreads - 1) / kInterThreads));
}
// The ghost copy and what only needs the lists: (mark) after decide, the marks of the new far list's
// neighbourhoods, as launch_far_mark; (inter_n blocks past the ghost slots') the inter atoms' own densities.
__global__ void __launch_bounds__(kInterThreads) k_ghost_copy(const NeighTables *nt, Geom g, Slots s, Inter in, PotTables pt, bool mixed,
                                                              bool mark, int inter_n) {
    const int blocks = gridDim.x - inter_n;
    if ((int) blockIdx.x >= blocks) {
        inter_eam<0>(*nt, g, s, in, pt, mixed, blockIdx.x - blocks, inter_n);
        return;
    }
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (mark) mark_far_neighbourhoods(*nt, g, in, 0, min(in.cnt[CNT_FAR], in.fcap), 1, t, blocks * blockDim.x);
    if (t >= g.n_ghost_slots) return;
    ghost_copy_one(g, s, ghost_slot(g, t));
}
void launch_ghost_copy(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, bool mark, bool inter) {
    const int n = (g.n_ghost_slots + kInterThreads - 1) / kInterThreads, e = inter ? inter_blocks(lc, g) : 0;
    k_ghost_copy<<<n + e, kInterThreads, 0, lc.stream>>>(lc.ntd, g, with_records(lc, s), in, t, mixed, mark, e);
}
// The copy of F' and what only needs F' of the box's own atoms: (advance) after a density pass with the group lists,
// as launch_skin_advance; (inter_n blocks past the ghost slots') the forces on the inter atoms.
template <bool MIXED>
__global__ void __launch_bounds__(kInterThreads) k_ghost_df(const NeighTables *nt, Geom g, Slots s, Inter in, PotTables pt, bool advance,
                                                            int inter_n) {
    const int blocks = gridDim.x - inter_n;
    if ((int) blockIdx.x >= blocks) {
        inter_eam<1>(*nt, g, s, in, pt, MIXED, blockIdx.x - blocks, inter_n);
        return;
    }
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (advance && t < 32) skin_advance(s.skin);
    if (t < g.n_ghost_slots) {
        const int gs = ghost_slot(g, t);
        const int os = owner_slot(g, gs);
        ghost_df_one<MIXED>(g, s, gs, os);
    }
    const int ng = in.cnt[CNT_GHOST];
    for (int q = t; q < ng; q += blocks * blockDim.x) in.gdf[q] = in.df[in.groot[q]];
}
void launch_ghost_df(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, bool advance) {
    const int n = (g.n_ghost_slots + kInterThreads - 1) / kInterThreads, e = inter_blocks(lc, g);
    if (mixed) k_ghost_df<true><<<n + e, kInterThreads, 0, lc.stream>>>(lc.ntd, g, s, in, t, advance, e);
    else k_ghost_df<false><<<n + e, kInterThreads, 0, lc.stream>>>(lc.ntd, g, s, in, t, advance, e);
}
// The lattice owners' side of the inter-atom pairs. One warp per owner listed by k_inter_eam: the
// lanes walk the owner's site and its full offsets (reference order) and, per site, the bucket of
// inter atoms whose nearest site it is (local atoms, and the ghost images borderInter made of atoms
// near the far side of the box). Each pair inside the cutoff adds the term the inter atom's pass
// would have scattered, computed from the same oriented difference x_inter - x_lattice; the lanes'
// partial sums are reduced by shuffles in a fixed order and added to the owner once. Whether a ghost
// lattice slot or a ghost inter atom carries the periodic image changes only the rounding of the
// difference. A local inter atom whose nearest site is outside the box takes no part, as in the
// inter-atom pass. The last block to finish resets the list for the next pass; the bits are clear by
// then.
template <int KIND>
__global__ void __launch_bounds__(128) k_inter_owner(const NeighTables *__restrict__ ntd, Geom g, Slots s, Inter in, PotTables pt, bool mixed,
                                                     FixParams fp, StepParams *sp, bool kick) {
    if (KIND == 1 && kick) inter_secondstep(in, sp, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    const int n = min(in.cnt[CNT_TOUCHED], in.tcap);
    if (n == 0) return;  // nothing listed: no block writes, so no reset is due
    const int nb = *in.n_bucket;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < n; w += warps) {  // warp-uniform
        const int j = in.touched[w];
        const int tj = s.type[j];
        const double xj = s.x[j], yj = s.y[j], zj = s.z[j];
        const double dfj = KIND == 1 ? lat_df(g, s, j, mixed) : 0.0;
        const int par = (j % g.Sx) & 1;
        const int nf = ntd->nfull;
        double acc = 0.0, fx = 0.0, fy = 0.0, fz = 0.0;
        if (tj >= 0) {
            for (int q = lane - 1; q < nf; q += 32) {
                const int key = q < 0 ? j : j + ntd->full[par][q];
                for (int b = bucket_begin(in, nb, key); b < nb && (int) (in.bucket[b] >> 32) == key; b++) {
                    const int ref = (int) (in.bucket[b] & 0xffffffffLL);
                    if (ref < in.cap && !is_local_slot(g, key)) continue;
                    const InterRef o = inter_ref(in, ref);
                    const double dx = o.x - xj, dy = o.y - yj, dz = o.z - zj;
                    const double r2 = dx * dx + dy * dy + dz * dz;
                    if (!(r2 < g.rc2)) continue;
                    if (KIND == 0) {
                        acc += rho_fn(pt, o.type, r2);
                    } else if (KIND == 1) {
                        const double fp = to_force(pt, o.type, tj, r2, o.df, dfj);
                        fx += -dx * fp; fy += -dy * fp; fz += -dz * fp;
                    } else {
                        acc += 0.5 * pair_fn(pt, o.type, tj, r2);
                    }
                }
            }
        }
        if (KIND == 1) {
            fx = warp_sum_d(fx);
            fy = warp_sum_d(fy);
            fz = warp_sum_d(fz);
        } else {
            acc = warp_sum_d(acc);
        }
        if (lane == 0) {
            if (tj >= 0) {
                if (KIND == 0) {  // and the F' that the density pass left to this owner
                    const double rho = s.rho[j] + acc;
                    s.rho[j] = rho;
                    if (mixed) lat_df_one<true>(g, s, pt, fp, j, tj, rho);
                    else lat_df_one<false>(g, s, pt, fp, j, tj, rho);
                } else if (KIND == 1) {
                    const double f0 = s.fx[j] + fx, f1 = s.fy[j] + fy, f2v = s.fz[j] + fz;
                    s.fx[j] = f0; s.fy[j] = f1; s.fz[j] = f2v;
                    if (kick) {  // the second half-kick the lattice force pass left to this owner
                        const double c = dt_inv_m_of(sp, tj);
                        const double vx = __dadd_rn(s.vx[j], __dmul_rn(c, f0));
                        const double vy = __dadd_rn(s.vy[j], __dmul_rn(c, f1));
                        const double vz = __dadd_rn(s.vz[j], __dmul_rn(c, f2v));
                        s.vx[j] = vx; s.vy[j] = vy; s.vz[j] = vz;
                        if (variable_dt(sp)) note_vmax2(sp, speed2(vx, vy, vz));
                    }
                }
                else s.e[j] += acc;
            }
            // the density pass's list stays for the force pass of the same positions (its bits tell
            // the lattice force pass which atoms to leave unkicked); the force and energy passes end it
            if (KIND != 0) atomicAnd(&in.touch_bits[j >> 5], ~(1u << (j & 31)));
        }
    }
    if (KIND == 0) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&in.cnt[CNT_TOUCH_DONE], 1) == (int) gridDim.x - 1) {
            in.cnt[CNT_TOUCHED] = 0;
            in.cnt[CNT_TOUCH_DONE] = 0;
            __threadfence();
        }
    }
}
template <int KIND>
void launch_inter_owner(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, StepParams *sp = nullptr,
                        bool kick = false) {
    k_inter_owner<KIND><<<lc.num_sms * 4, 128, 0, lc.stream>>>(lc.ntd, g, s, in, t, mixed, fix_params(lc), sp, kick);
}
void launch_inter_rho_owners(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed) {
    launch_inter_owner<0>(lc, g, s, in, t, mixed);
}
void launch_inter_force_owners(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed, StepParams *sp, bool kick) {
    launch_inter_owner<1>(lc, g, s, in, t, mixed, sp, kick);
}
void launch_inter_energy(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, PotTables t, bool mixed) {
    k_inter_eam<2><<<lc.num_sms * 4, kInterThreads, 0, lc.stream>>>(lc.ntd, g, s, in, t, mixed);
    launch_inter_owner<2>(lc, g, s, in, t, mixed);
}

// ------------------------------------------------------------------------------------------------
// far lattice atoms (farther than 0.2 a0 from their site). Rebuild from positions for states that did
// not come through atom::decide (uploads, the per-phase hooks).
// ------------------------------------------------------------------------------------------------
__global__ void k_far_clear(const NeighTables *nt, Geom g, Inter in) {
    const int nf = min(in.cnt[CNT_FAR], in.fcap);
    mark_far_neighbourhoods(*nt, g, in, 0, nf, 0, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
__global__ void k_far_count_reset(Inter in) { in.cnt[CNT_FAR] = 0; }
__global__ void k_far_scan(Geom g, Slots s, Inter in) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= g.n_local) return;
    int i, j, k;
    const int sl = local_slot(g, t, i, j, k);
    if (s.type[sl] < 0) return;
    if (displaced_fp64(g, s, sl)) {
        const int q = atomicAdd(&in.cnt[CNT_FAR], 1);
        if (q < in.fcap) in.far_list[q] = sl;
        else set_error(in, MG_DEVERR_DISPLACED_OVERFLOW);
    }
}
__global__ void k_far_mark(const NeighTables *nt, Geom g, Inter in) {
    const int nf = min(in.cnt[CNT_FAR], in.fcap);
    mark_far_neighbourhoods(*nt, g, in, 0, nf, 1, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}
void launch_far_clear(const LaunchCtx &lc, const Geom &g, Inter in) {
    k_far_clear<<<lc.num_sms * 4, 256, 0, lc.stream>>>(lc.ntd, g, in);
}
void launch_far_mark(const LaunchCtx &lc, const Geom &g, Inter in) {
    k_far_mark<<<lc.num_sms * 4, 256, 0, lc.stream>>>(lc.ntd, g, in);
}
void launch_far_rebuild(const LaunchCtx &lc, const Geom &g, Slots s, Inter in) {
    launch_far_clear(lc, g, in);
    k_far_count_reset<<<1, 1, 0, lc.stream>>>(in);
    const int b = 256;
    k_far_scan<<<(g.n_local + b - 1) / b, b, 0, lc.stream>>>(g, s, in);
    launch_far_mark(lc, g, in);
}

// ------------------------------------------------------------------------------------------------
// decide per chunk of planes, for the host step that overlaps its copies out with its copies in.
// With no inter atoms at the start of the step, decide (src/atom.cpp:21-84) puts every displaced atom
// into the list in scan order and then, in list order, moves each one whose nearest site is a vacant
// in-box slot into that slot. When every displaced atom's nearest site is its own slot, each is the
// only claimant of the slot it just vacated, so it goes back at once with its id, type, position and
// velocity: the step then differs from one without it only in the atom's displacement record, which
// recombination rewrites from the position, and in its far-list entry and neighbourhood marks. Those
// are made here, per chunk, before any density pass reads the neighbourhood. A displaced atom nearest
// another site (or outside the sub-box), or a full far list, voids the overlapped step instead: the
// host then runs the whole step again from its input.
// ------------------------------------------------------------------------------------------------
__global__ void k_spec_begin(Inter in) {
    in.cnt[CNT_FAR] = 0;
    in.cnt[CNT_SPEC_VOID] = 0;
}
void launch_spec_begin(const LaunchCtx &lc, Inter in) { k_spec_begin<<<1, 1, 0, lc.stream>>>(in); }

__global__ void k_spec_decide(const NeighTables *nt, Geom g, Slots s, Inter in, int t0, int t1) {
    const int n = in.cnt[CNT_DISPLACED];  // displaced so far this step (usually none)
    if (n > in.dcap) {
        in.cnt[CNT_SPEC_VOID] = 1;
        return;
    }
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const int t = in.displaced[e];
        if (t < t0 || t >= t1) continue;  // an earlier chunk's
        int i, j, k;
        const int sl = local_slot(g, t, i, j, k);
        const double x = s.x[sl], y = s.y[sl], z = s.z[sl];
        if (near_index_in_sub_box(g, x, y, z) != sl) {
            atomicExch(&in.cnt[CNT_SPEC_VOID], 1);
            continue;
        }
        const int q = atomicAdd(&in.cnt[CNT_FAR], 1);
        if (q >= in.fcap) {
            atomicExch(&in.cnt[CNT_SPEC_VOID], 1);
            continue;
        }
        double xs, ys, zs;
        site_of(g, i + g.gx, j + g.gy, k + g.gz, xs, ys, zs);
        s.u4[sidx(g, sl)] = make_u4(g, x, y, z, xs, ys, zs, s.type[sl]);
        in.far_list[q] = sl;
        mark_far_neighbourhoods(*nt, g, in, q, q + 1, 1, 0, 1);
    }
}
void launch_spec_decide(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, int t0, int t1) {
    if (t1 <= t0) return;
    k_spec_decide<<<8, 256, 0, lc.stream>>>(lc.ntd, g, s, in, t0, t1);
}


// ------------------------------------------------------------------------------------------------
// setv (src/atom.cpp:475-494): one thread
// ------------------------------------------------------------------------------------------------
__global__ void k_setv(Slots s, int slot, double dir0, double dir1, double dir2, double energy) {
    const int ty = s.type[slot];
    const double m = (ty >= 0 && ty < 3) ? c_mass[ty] : 0.0;
    const double v_ = __dsqrt_rn(__ddiv_rn(__ddiv_rn(__dmul_rn(2.0, energy), m), kMvv2e));
    const double d_ = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dir0, dir0), __dmul_rn(dir1, dir1)), __dmul_rn(dir2, dir2)));
    s.vx[slot] = __dadd_rn(s.vx[slot], __ddiv_rn(__dmul_rn(v_, dir0), d_));
    s.vy[slot] = __dadd_rn(s.vy[slot], __ddiv_rn(__dmul_rn(v_, dir1), d_));
    s.vz[slot] = __dadd_rn(s.vz[slot], __ddiv_rn(__dmul_rn(v_, dir2), d_));
}
void launch_setv(const LaunchCtx &lc, const Geom &g, Slots s, int64_t slot, const double dir[3], double energy) {
    k_setv<<<1, 1, 0, lc.stream>>>(s, (int) slot, dir[0], dir[1], dir[2], energy);
}

// rescale (src/system_configuration.cpp:86-111): factor = sqrt(T / T_now) from the mvv reduction
__global__ void k_rescale(Geom g, Slots s, Inter in, const double *mvv, double t_set, uint64_t n_atoms) {
    const uint64_t dof = 3 * n_atoms - 3;
    const double scalar = __ddiv_rn(__dmul_rn(*mvv, kMvv2e), __dmul_rn((double) dof, kBoltz));
    const double f = __dsqrt_rn(__ddiv_rn(t_set, scalar));
    const int stride = gridDim.x * blockDim.x;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < g.n_local; t += stride) {
        int i, j, k;
        const int sl = local_slot(g, t, i, j, k);
        s.vx[sl] = __dmul_rn(s.vx[sl], f);
        s.vy[sl] = __dmul_rn(s.vy[sl], f);
        s.vz[sl] = __dmul_rn(s.vz[sl], f);
    }
    const int n = in.cnt[CNT_INTER];
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += stride) {
        in.vx[a] = __dmul_rn(in.vx[a], f);
        in.vy[a] = __dmul_rn(in.vy[a], f);
        in.vz[a] = __dmul_rn(in.vz[a], f);
    }
}
void launch_rescale(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, const double *d_mvv, double t_set,
                    uint64_t n_atoms) {
    k_rescale<<<lc.num_sms * 8, 256, 0, lc.stream>>>(g, s, in, d_mvv, t_set, n_atoms);
}

// ------------------------------------------------------------------------------------------------
// thermo reduction (deterministic: per-block partials, then one block in fixed order)
// out: [0] sum m v^2, [1..3] force sum, [4] potential energy, [5] vacancies
// ------------------------------------------------------------------------------------------------
constexpr int kThermoWords = 6;
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__global__ void __launch_bounds__(256) k_thermo_partial(Geom g, Slots s, Inter in, bool with_energy, double *partials) {
    double acc[kThermoWords] = {0, 0, 0, 0, 0, 0};
    const int stride = gridDim.x * blockDim.x;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < g.n_local; t += stride) {
        int i, j, k;
        const int sl = local_slot(g, t, i, j, k);
        const int ty = s.type[sl];
        if (ty < 0) { acc[5] += 1.0; continue; }
        const double vx = s.vx[sl], vy = s.vy[sl], vz = s.vz[sl];
        acc[0] += (vx * vx + vy * vy + vz * vz) * c_mass[ty];
        acc[1] += s.fx[sl]; acc[2] += s.fy[sl]; acc[3] += s.fz[sl];
        if (with_energy) acc[4] += s.e[sl];
    }
    if (blockIdx.x == 0) {
        const int n = in.cnt[CNT_INTER];
        for (int a = threadIdx.x; a < n; a += blockDim.x) {
            const double vx = in.vx[a], vy = in.vy[a], vz = in.vz[a];
            acc[0] += (vx * vx + vy * vy + vz * vz) * c_mass[in.type[a]];
            acc[1] += in.fx[a]; acc[2] += in.fy[a]; acc[3] += in.fz[a];
            if (with_energy) acc[4] += in.e[a];
        }
    }
    __shared__ double sh[kThermoWords][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int q = 0; q < kThermoWords; q++) {
        const double v = warp_sum(acc[q]);
        if (lane == 0) sh[q][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < kThermoWords) {
        double v = 0;
        for (int q = 0; q < (int) (blockDim.x >> 5); q++) v += sh[threadIdx.x][q];
        partials[blockIdx.x * kThermoWords + threadIdx.x] = v;
    }
}
__global__ void k_thermo_final(const double *partials, int nb, double *out) {
    if (threadIdx.x < kThermoWords) {
        double v = 0;
        for (int b = 0; b < nb; b++) v += partials[b * kThermoWords + threadIdx.x];
        out[threadIdx.x] = v;
    }
}
void launch_thermo(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, bool with_energy, double *partials,
                   int n_partials, double *out) {
    k_thermo_partial<<<n_partials, 256, 0, lc.stream>>>(g, s, in, with_energy, partials);
    k_thermo_final<<<1, 32, 0, lc.stream>>>(partials, n_partials, out);
}

// ------------------------------------------------------------------------------------------------
// Wigner-Seitz mapping of arbitrary points (indexing parity checks)
// ------------------------------------------------------------------------------------------------
__global__ void k_ws_map(Geom g, const double *xyz, int64_t n, int64_t *coords, uint32_t *flags, int64_t *index) {
    const int64_t t = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double x = xyz[3 * t], y = xyz[3 * t + 1], z = xyz[3 * t + 2];
    long long c[3];
    near_lat_coord(g, x, y, z, c);
    coords[3 * t] = c[0]; coords[3 * t + 1] = c[1]; coords[3 * t + 2] = c[2];
    flags[t] = is_out_box(g, x, y, z);
    index[t] = near_index_in_sub_box(g, x, y, z);
}
void launch_ws_map(const LaunchCtx &lc, const Geom &g, const double *xyz, int64_t n, int64_t *coords, uint32_t *flags,
                   int64_t *index) {
    const int b = 256;
    k_ws_map<<<(unsigned) ((n + b - 1) / b), b, 0, lc.stream>>>(g, xyz, n, coords, flags, index);
}

// ------------------------------------------------------------------------------------------------
// Atom dump frames (AtomDump::dump, frontend/io/atom_dump.cpp:59-81, with the record of
// BufferedFileWriter::write, frontend/io/buffered_io.cpp:17-35): inter atoms in list order first, then
// the box's lattice atoms in k, j, i order without INVALID slots. An ordered compaction over groups of
// kDumpThreads local slots: count, one-block scan (offsets start after the inter atoms), write.
// ------------------------------------------------------------------------------------------------
static_assert(sizeof(mg_dump_record) == 72, "dump record layout (tools/dump2text/out_convert.cpp:18-25)");

__device__ __forceinline__ void put_dump_record(mg_dump_record *r, uint64_t id, uint64_t step, int type, double x,
                                                double y, double z, double vx, double vy, double vz) {
    mg_dump_record q;
    q.id = id;
    q.step = step;
    q.type = type;
    q.inter_type = 0;  // BufferedFileWriter::write sets 0 for every record
    q.pad_ = 0;
    q.x[0] = x; q.x[1] = y; q.x[2] = z;
    q.v[0] = vx; q.v[1] = vy; q.v[2] = vz;
    *r = q;
}
__global__ void __launch_bounds__(kDumpThreads) k_dump_count(Geom g, Slots s, int *group_count) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    int live = 0;
    if (t < g.n_local) {
        int i, j, k;
        live = s.type[local_slot(g, t, i, j, k)] >= 0;
    }
    const int c = __syncthreads_count(live);
    if (threadIdx.x == 0) group_count[blockIdx.x] = c;
}
__global__ void __launch_bounds__(1024) k_dump_scan(Inter in, int *group_count, int ngroups, unsigned long long *count) {
    const int n_inter = min(in.cnt[CNT_INTER], in.cap);
    const int total = block_scan_counts(group_count, ngroups, n_inter);
    if (threadIdx.x == 0) *count = (unsigned long long) total;
}
__global__ void __launch_bounds__(kDumpThreads) k_dump_write(Geom g, Slots s, const int *group_offset, mg_dump_record *out,
                                                             uint64_t step) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    int sl = -1;
    if (t < g.n_local) {
        int i, j, k;
        sl = local_slot(g, t, i, j, k);
        if (s.type[sl] < 0) sl = -1;
    }
    int pos;
    block_exclusive_scan(sl >= 0 ? 1 : 0, pos);
    if (sl < 0) return;
    put_dump_record(out + group_offset[blockIdx.x] + pos, s.id[sl], step, s.type[sl], s.x[sl], s.y[sl], s.z[sl], s.vx[sl],
                    s.vy[sl], s.vz[sl]);
}
__global__ void k_dump_inter(Inter in, mg_dump_record *out, uint64_t step) {
    const int n = min(in.cnt[CNT_INTER], in.cap);
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x)
        put_dump_record(out + a, in.id[a], step, in.type[a], in.x[a], in.y[a], in.z[a], in.vx[a], in.vy[a], in.vz[a]);
}
void launch_dump_pack(const LaunchCtx &lc, const Geom &g, Slots s, Inter in, mg_dump_record *out,
                      unsigned long long *count, int *scratch, uint64_t step) {
    const int ngroups = dump_scratch_ints(g);
    k_dump_count<<<ngroups, kDumpThreads, 0, lc.stream>>>(g, s, scratch);
    k_dump_scan<<<1, 1024, 0, lc.stream>>>(in, scratch, ngroups, count);
    k_dump_write<<<ngroups, kDumpThreads, 0, lc.stream>>>(g, s, scratch, out, step);
    k_dump_inter<<<lc.num_sms, 256, 0, lc.stream>>>(in, out, step);
}

}  // namespace mg
