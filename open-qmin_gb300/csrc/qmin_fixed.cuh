// 64-bit fixed-point evaluation of the deep-site force of the FP64 form.
//
// GB300 issues two FP64 operations per cycle and SM (measured: DFMA 1.96,
// conversions to and from FP64 1.96), but about 70 64-bit integer additions
// and 42 32 x 32 -> 64 multiply-adds.  The bulk force needs 106 FP64
// operations for its linear part and 34 for the phase part of every site, so
// the FP64 pipe bounds it; here both run on the integer pipes:
//
//   * Q enters as X = Q 2^56, so differences and the integer stencil forms are
//     exact;
//   * a product of two 64-bit numbers keeps its upper 64 bits, from the
//     balanced 32-bit halves x = xh 2^32 + xl (xl signed): hi += xh yh,
//     mid += xh yl + xl yh, result hi + mid / 2^32.  The sums of products of
//     one output share hi and mid, which are put together once; of xl yl the
//     upper 32 bits go into a sum of their own (FixAcc);
//   * every term of an output carries the same scale 2^R, chosen on the host
//     from the parameters so that no sum, high or middle, can overflow
//     (fixed_coeffs).
//
// The quantisation of Q (towards zero at 2^-56, exact from 1/16 on; to the
// nearest was no better over the 400 runs of FixAcc) and of the products stay
// below the rounding of the FP64 evaluation, whose partial sums reach 10 to 30:
// against 80-bit arithmetic the error of the force is 0.06 to 0.52 of the FP64
// form's over random and smooth nematic fields; where every component is 3/4
// and the FP64 products are nearly exact, 0.56 to 1.25.
// The sums need every component's |Q| < 1 at LC sites (with 3/4, 350 of the
// first 520 iterations at 200^3 left the range: FIRE overshoots to 0.85), the relative
// accuracy some |Q| >= 1/8: a lattice outside that takes the FP64 kernel
// (FixedDev).  QMIN_DEV functions also compile for the host.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "../../include/qmin_gb300.h"

#ifdef __CUDACC__
#define QMIN_DEV __device__ __forceinline__
#else
#define QMIN_DEV inline
#endif

namespace qmin {

constexpr int kFixQ = 56;  // Q 2^56

// a 64-bit number as balanced halves: v = h 2^32 + l, -2^31 <= l < 2^31; q = l / 4
struct Fix2 {
    int h, l, q;
};

// what the kernels need of one parameter set
struct FixedCoef {
    Fix2 l1, l1d, l23, l2, l3;  // -L1, -2 L1, -(L2 + L3), -L2 / 8, -L3 / 8 at 2^(R + 8)
    Fix2 b3, b6;                // 3 b, -6 b at 2^(R + 6)
    Fix2 c8;                    // -8 c, for -g2 = -(8 c s + 2 a) with s at 2^58
    long long a2;               // -2 a at 2^(R + 3)
    long long hi0[5], mid0[5];  // where the sums start: minus the field force (as it enters before the
                                // metric), and half a unit of the result
    int up;                     // bits of the middle product kept: results at 2^shift
    int c8up;                   // the shift that brings -8 c s to 2^(R + 3)
    int shift;                  // R + up
    double ma, mb;              // the metric on components 0 and 3, 2^-shift included: f0 <- ma f0 - mb f3
    int ok;                // 0: this parameter set has no fixed-point form
};

#ifdef __CUDACC__
__host__
#endif
QMIN_DEV Fix2 fix_split(long long v)
{
    const unsigned l = (unsigned)(unsigned long long)v;
    return Fix2{(int)(v >> 32) + (int)(l >> 31), (int)l, (int)l >> 2};
}

QMIN_DEV long long fix_mul_wide(int a, int b, long long c) { return (long long)a * (long long)b + c; }

// (a b) / 2^32 + c
QMIN_DEV int fix_mul_high(int a, int b, int c)
{
#ifdef __CUDA_ARCH__
    return __mulhi(a, b) + c;
#else
    return (int)((long long)a * b >> 32) + c;
#endif
}

// Running sum of products of one output.  The products of the low halves go
// into lo in units of 4 (the middle sum's unit: 1), six of them below 2^31.
// Left out, those of the squares are a bias of one sign at every site and
// iteration: 100 FIRE iterations from random directors at 16^3 then end 10 %
// farther from quadruple precision than with the FP64 force, with them 1 % +-
// 2 % (means over 400 starts; from smooth fields 27 and 38 % nearer).  They
// cost 1.3 to 1.8 % of a run (50^3 one-constant, 100 iterations: 3.10 -> 3.14
// ms, 83 x 61 x 97, 60: 7.42 -> 7.53, 200^3, 40: 41.9 -> 42.7), 5.5 % of a
// multi-constant batch (eight 64^3: 470 -> 496 us an iteration).
struct FixAcc {
    long long hi, mid;
    int lo;
    QMIN_DEV void zero() { hi = mid = lo = 0; }
    QMIN_DEV void add(const Fix2 &x, const Fix2 &y)
    {
        hi = fix_mul_wide(x.h, y.h, hi);
        mid = fix_mul_wide(x.h, y.l, mid);
        mid = fix_mul_wide(x.l, y.h, mid);
        lo = fix_mul_high(x.q, y.l, lo);
    }
    QMIN_DEV void square(const Fix2 &x)  // x x, its middle products halved: the caller doubles mid
    {
        hi = fix_mul_wide(x.h, x.h, hi);
        mid = fix_mul_wide(x.h, x.l, mid);
        lo = fix_mul_high(x.q, x.l, lo);
    }
    QMIN_DEV long long middle() const { return mid + 4LL * lo; }
    // hi 2^up + mid 2^(up - 32), 0 < up < 32
    QMIN_DEV long long get(int up) const
    {
        return (long long)((unsigned long long)hi << up) + (middle() >> (32 - up));  // the caller's mid has half a unit
    }
    QMIN_DEV long long get32() const { return hi + ((middle() + (1LL << 31)) >> 32); }
};

#ifdef __CUDACC__
QMIN_DEV int fix_hi_word(double d) { return __double2hiint(d); }
QMIN_DEV unsigned fix_lo_word(double d) { return (unsigned)__double2loint(d); }
#else
inline int fix_hi_word(double d)
{
    uint64_t u;
    memcpy(&u, &d, 8);
    return (int)(u >> 32);
}
inline unsigned fix_lo_word(double d)
{
    uint64_t u;
    memcpy(&u, &d, 8);
    return (unsigned)u;
}
#endif

// |d| as the upper word of its bits, ordered like |d|: >= kFixWide for |d| >=
// 1 (Inf and NaN too), >= kFixLively for |d| >= 1/8
constexpr int kFixWide = 0x3ff00000, kFixLively = 0x3fc00000;
QMIN_DEV int fix_magnitude(double d) { return fix_hi_word(d) & 0x7fffffff; }

// d 2^56 towards zero, |d| < 1 (some number for the rest)
QMIN_DEV long long to_fixed(double d)
{
    const int h = fix_hi_word(d);
    const unsigned lo = fix_lo_word(d);
    // mantissa << 3: 56 bits, worth 2^(e - 1022) at scale 2^56
    const unsigned mh = ((((unsigned)h & 0xfffffu) | 0x100000u) << 3) | (lo >> 29);
    const unsigned long long m = ((unsigned long long)mh << 32) | (lo << 3);
    int r = 1022 - ((h >> 20) & 0x7ff);
    r = r < 0 ? 0 : (r > 63 ? 63 : r);
    const unsigned long long v = m >> r;
    const long long s = h >> 31;  // 0 or -1
    return ((long long)v ^ s) - s;
}

// a 2^-shift; |a| < 2^62, shift < 64 (the exponent of a non-zero integer stays normal)
#ifdef __CUDACC__
// a 2^-shift, rounded to nearest (halves away from zero), by hand: the conversion instructions share the FP64 pipe
QMIN_DEV double fixed_scale(long long a, int shift)
{
    const int s = (int)(a >> 63);
    const unsigned long long m = (unsigned long long)((a ^ s) - s);
    const int n = __clzll((long long)m);         // 64 for 0
    const unsigned long long t = m << (n & 63);  // leading one at bit 63
    const unsigned long long r = (t >> 11) + ((t >> 10) & 1);
    const int hi = (int)(r >> 32) + ((1023 + 62 - n - shift) << 20);
    return __hiloint2double(m ? (hi | (s & 0x80000000)) : 0, (int)(unsigned)r);
}
#else
inline double fixed_scale(long long a, int shift) { return ldexp((double)a, -shift); }
#endif

// The coefficients of one parameter set at metric mode `single` (M once) or
// twice; fE + fH as the force subtracts them.  ok = 0 where the magnitudes do
// not fit (coefficients beyond 2^20, or all zero).
inline FixedCoef fixed_coeffs(const qmin_ldg_params &p, int metric_mode, const double *field)
{
    FixedCoef c;
    memset(&c, 0, sizeof c);
    const double L2 = p.multi_constant ? p.L2 : 0.0, L3 = p.multi_constant ? p.L3 : 0.0;
    const double a2 = p.A, b3 = p.B, c8 = 2.0 * p.C;  // 2 (A / 2), 3 (B / 3), 8 (C / 4)
    const double lmax = fmax(fabs(p.L1), fmax(fabs(L2 + L3), fmax(fabs(L2), fabs(L3)) / 8));
    const double gmax = 6 * fabs(c8) + fabs(a2);  // |8 c s + 2 a|, s <= 6
    if (!isfinite(lmax) || !isfinite(gmax) || !isfinite(b3)) return c;
    if (p.multi_constant && (p.L4 != 0.0 || p.L6 != 0.0)) return c;
    auto bits = [](double v) {  // v < 2^bits
        int e = 0;
        if (v == 0.0) return -60;
        frexp(v, &e);
        return e;
    };
    // coefficients below 2^60, the doubled ones below 2^61
    int R = 60 - 8 - bits(lmax);
    R = R < 60 - 6 - bits(fabs(b3)) ? R : 60 - 6 - bits(fabs(b3));
    R = R < 60 - 3 - bits(gmax) ? R : 60 - 3 - bits(gmax);
    // |result| for |Q| < 1: 36 L1 and 12 (L2 + L3) from the axis terms, 16 / 8 (|L2| + |L3|) from the face
    // diagonals, g2 u with |u| <= 3, 3 b X with |X| <= 5 or 6 b X with |X| <= 3, the fields
    double fsum = 0.0;
    if (field)
        for (int k = 0; k < 5; ++k) fsum = fmax(fsum, fabs(field[k]));
    const double bound =
        36 * fabs(p.L1) + 14 * (fabs(L2) + fabs(L3)) + 3 * gmax + 18 * fabs(b3) + 2 * fsum;
    if (!isfinite(bound) || bound == 0.0) return c;
    const int room = 62 - bits(bound);  // R + up
    if (R > room - 1) R = room - 1;
    if (R > 54) R = 54;
    auto at = [](double v, int s) { return (long long)llrint(ldexp(v, s)); };
    for (;; --R) {
        if (R < 30) return c;
        int up = room - R;
        if (up > 8) up = 8;
        c.l1 = fix_split(-at(p.L1, R + 8));
        c.l1d = fix_split(-at(p.L1, R + 9));
        c.l23 = fix_split(-at(L2 + L3, R + 8));
        c.l2 = fix_split(-at(L2, R + 5));
        c.l3 = fix_split(-at(L3, R + 5));
        c.b3 = fix_split(at(b3, R + 6));
        c.b6 = fix_split(-at(b3, R + 7));
        // 8 c s: s at 2^58 (below 2^60), 8 c at 2^e8 below 2^60, product at 2^(e8 - 6), brought to 2^(R + 3)
        int e8 = 60 - bits(fabs(c8));
        if (e8 > R + 8) e8 = R + 8;
        c.c8up = R + 3 - (e8 - 6);
        if (c.c8up < 1 || c.c8up > 24) return c;
        c.c8 = fix_split(-at(c8, e8));
        c.a2 = -at(a2, R + 3);
        c.up = up;
        c.shift = R + up;
        // The middle sums: a product x y adds at most |xh| |yl| + |xl| |yh|, |yl| <= 2^31.  The largest are those of
        // components 0 (|2 q0 + q3| <= 3, |X0| <= 4, 36 and 12 from the axis terms, 8 from the face diagonals) and 3
        // (12 from those); the others stay below 7.5 2^60.  A parameter set whose halves could reach 2^63 takes the
        // next smaller scale, at which the sum is 7.25 2^60 with every bound at its worst.
        auto mid = [](double xh, double xl, double y) { return xh * ldexp(1, 31) + xl * (ldexp(y, -32) + 1); };
        auto term = [&](const Fix2 &x, double y) { return mid(fabs((double)x.h), fabs((double)x.l), y); };
        const double most = mid(ldexp(gmax, R + 3 - 32) + 1, ldexp(1, 31), 3 * ldexp(1, 61)) + term(c.b3, 4 * ldexp(1, 58)) +
                            term(c.l1, 36 * ldexp(1, 56)) + term(c.l23, 12 * ldexp(1, 56)) +
                            term(c.l2, 12 * ldexp(1, 56)) + term(c.l3, 12 * ldexp(1, 56)) + ldexp(1, 34);
        if (most < 0.999999 * ldexp(1, 63)) break;
    }
    const bool twice = metric_mode == QMIN_METRIC_CPU;
    c.ma = ldexp(twice ? 20.0 / 9.0 : 4.0 / 3.0, -c.shift);
    c.mb = ldexp(twice ? 16.0 / 9.0 : 2.0 / 3.0, -c.shift);
    for (int k = 0; k < 5; ++k) {
        // CPU mode: M (M f - F) = M^2 (f - M^-1 F), M^-1 F = (F0 + F3 / 2, .., F3 + F0 / 2)
        double v = field ? field[k] : 0.0;
        if (field && twice && k == 0) v += 0.5 * field[3];
        if (field && twice && k == 3) v += 0.5 * field[0];
        const long long b = -at(v, c.shift);  // hi 2^up + mid 2^(up - 32)
        c.hi0[k] = b >> c.up;
        c.mid0[k] = ((b - (long long)((unsigned long long)c.hi0[k] << c.up)) << (32 - c.up)) + (1LL << (31 - c.up));
    }
    c.ok = 1;
    return c;
}

// X of one component at the sites of the stencil, from an accessor V(dx, dy, dz, c)
//
// One-constant part: lam[c] = 6 X - the six neighbours.  Multi-constant forms
// without L4 (the integer table of qmin_bulk_q25.h over 8): the axis part,
// which L2 and L3 share, and the face-diagonal differences of each.
template <class V> QMIN_DEV void fixed_axis(const V &at, const long long (&q)[5], long long (&lam)[5], long long (&ax)[5])
{
    long long s[3][5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        s[0][c] = at(-1, 0, 0, c) + at(1, 0, 0, c);
        s[1][c] = at(0, -1, 0, c) + at(0, 1, 0, c);
        s[2][c] = at(0, 0, -1, c) + at(0, 0, 1, c);
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) lam[c] = 6 * q[c] - s[0][c] - s[1][c] - s[2][c];
    const long long zz = 2 * q[0] + 2 * q[3] - s[2][0] - s[2][3];
    ax[0] = 2 * q[0] - s[0][0] + zz;
    ax[1] = 4 * q[1] - s[0][1] - s[1][1];
    ax[2] = 4 * q[2] - s[0][2] - s[2][2];
    ax[3] = 2 * q[3] - s[1][3] + zz;
    ax[4] = 4 * q[4] - s[1][4] - s[2][4];
}

// Face-diagonal sums of the L2 (m2) and L3 (m3) forms.  A half difference such
// as Q(-1,0,1,c) - Q(-1,0,-1,c) is written XZ(-1, c): the reference's forms
// take some of them on one side only.
template <class V> QMIN_DEV void fixed_mixed(const V &at, long long (&m2)[5], long long (&m3)[5])
{
    auto XY = [&](int sx, int c) { return at(sx, 1, 0, c) - at(sx, -1, 0, c); };
    auto XZ = [&](int sx, int c) { return at(sx, 0, 1, c) - at(sx, 0, -1, c); };
    auto YZ = [&](int sy, int c) { return at(0, sy, 1, c) - at(0, sy, -1, c); };
    const long long xy0 = XY(-1, 0) - XY(1, 0), xy1 = XY(-1, 1) - XY(1, 1), xy2 = XY(-1, 2) - XY(1, 2),
                    xy3 = XY(-1, 3) - XY(1, 3), xy4 = XY(-1, 4) - XY(1, 4);
    const long long xz0m = XZ(-1, 0), xz1m = XZ(-1, 1), xz2m = XZ(-1, 2), xz3m = XZ(-1, 3), xz4m = XZ(-1, 4);
    const long long xz1p = XZ(1, 1), xz2p = XZ(1, 2), xz3p = XZ(1, 3), xz4p = XZ(1, 4);
    const long long yz0m = YZ(-1, 0), yz1m = YZ(-1, 1), yz2m = YZ(-1, 2), yz3m = YZ(-1, 3), yz4m = YZ(-1, 4);
    const long long yz0p = YZ(1, 0), yz1p = YZ(1, 1), yz2p = YZ(1, 2), yz4p = YZ(1, 4);
    const long long xz4 = xz4m - xz4p;
    m2[0] = xy1 + yz4p - yz4m;
    m3[0] = xy1 + yz4p - xz4m;
    m2[1] = xy0 + xy3 + xz2m + xz4 - yz2p;
    m3[1] = xy0 + xy3 + xz4 - yz2p + yz2m;
    const long long k2 = xy4 - xz3m + xz3p - yz1p;
    m2[2] = k2 + yz1m;
    m3[2] = k2 + xz1m;
    const long long k3 = xy1 - xz2m + xz2p;
    m2[3] = k3 + xz4m - yz4m;
    m3[3] = k3 - xz4m + yz4m;
    const long long k4 = xy2 + xz1m - xz1p + yz0p;
    m2[4] = k4 - xz0m - xz3m + yz3m;
    m3[4] = k4 + xz3m - yz0m - yz3m;
}

// F 2^shift before the metric (fixed_to_force)
template <bool MULTI>
QMIN_DEV void fixed_force(const FixedCoef &k, const long long (&q)[5], const long long (&lam)[5],
                              const long long (&ax)[5], const long long (&m2)[5], const long long (&m3)[5],
                              long long (&out)[5])
{
    Fix2 y[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) y[c] = fix_split(q[c] * 32);  // 2^61
    const Fix2 y03 = fix_split((q[0] + q[3]) * 32);
    // s = q0^2 + q3^2 + q0 q3 + q1^2 + q2^2 + q4^2 at 2^58
    FixAcc sq[5], p03;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        sq[c].zero();
        sq[c].square(y[c]);
    }
    p03.zero();
    p03.add(y[0], y[3]);
    const long long h24 = sq[2].hi + sq[4].hi, n24 = sq[2].mid + sq[4].mid;
    const long long h03 = sq[0].hi + sq[3].hi, n03 = sq[0].mid + sq[3].mid;
    const int o24 = sq[2].lo + sq[4].lo, o03 = sq[0].lo + sq[3].lo;
    const long long p = p03.middle();
    // every shift rounds to nearest: a floor's half unit would add up over the iterations of a run
    constexpr long long half = 1LL << 30;
    const long long s =
        (h03 + h24 + sq[1].hi + p03.hi) + ((n03 + n24 + sq[1].mid + 2LL * (o03 + o24 + sq[1].lo) + half) >> 31) +
        ((p + 2 * half) >> 32);
    FixAcc g;
    g.zero();
    g.mid = 1LL << (31 - k.c8up);
    g.add(fix_split(s), k.c8);
    const long long mg = g.get(k.c8up) + k.a2;  // -g2 at 2^(R + 3)
    const Fix2 g2 = fix_split(mg), g4 = fix_split(2 * mg);
    // at 2^58: X0 = q3^2 + q4^2 + w, X3 = q0^2 + q2^2 + w with w = 2 q0 q3 - q1^2; X1 = q1 (q0 + q3) + q2 q4,
    // X2 = q1 q4 - q2 q3, X4 = q1 q2 - q0 q4
    const long long wh = 2 * p03.hi - sq[1].hi, wm = p - sq[1].mid + half;
    const Fix2 X0 =
        fix_split(sq[3].hi + sq[4].hi + wh + ((sq[3].mid + sq[4].mid + wm + 2LL * (sq[3].lo + sq[4].lo - sq[1].lo)) >> 31));
    const Fix2 X3 =
        fix_split(sq[0].hi + sq[2].hi + wh + ((sq[0].mid + sq[2].mid + wm + 2LL * (sq[0].lo + sq[2].lo - sq[1].lo)) >> 31));
    FixAcc x1, x2, x4, xn;
    x1.zero();
    x1.add(y[1], y03);
    x1.add(y[2], y[4]);
    x2.zero();
    x2.add(y[1], y[4]);
    xn.zero();
    xn.add(y[2], y[3]);
    x2.hi -= xn.hi;
    x2.mid -= xn.mid;
    x2.lo -= xn.lo;
    x4.zero();
    x4.add(y[1], y[2]);
    xn.zero();
    xn.add(y[0], y[4]);
    x4.hi -= xn.hi;
    x4.mid -= xn.mid;
    x4.lo -= xn.lo;
    FixAcc f[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        f[c].hi = k.hi0[c];
        f[c].mid = k.mid0[c];
        f[c].lo = 0;
    }
    // -g2 (2 q0 + q3), -2 g2 q1, ..: the q at 2^61
    f[0].add(g2, fix_split((2 * q[0] + q[3]) * 32));
    f[3].add(g2, fix_split((2 * q[3] + q[0]) * 32));
    f[1].add(g4, y[1]);
    f[2].add(g4, y[2]);
    f[4].add(g4, y[4]);
    f[0].add(k.b3, X0);
    f[3].add(k.b3, X3);
    f[1].add(k.b6, fix_split(x1.get32()));
    f[2].add(k.b6, fix_split(x2.get32()));
    f[4].add(k.b6, fix_split(x4.get32()));
    // -e: L1 (2 lam0 + lam3, 2 lam1, ..) + (L2 + L3) axis + L2 / 8 m2 + L3 / 8 m3
    f[0].add(k.l1, fix_split(2 * lam[0] + lam[3]));
    f[3].add(k.l1, fix_split(2 * lam[3] + lam[0]));
    f[1].add(k.l1d, fix_split(lam[1]));
    f[2].add(k.l1d, fix_split(lam[2]));
    f[4].add(k.l1d, fix_split(lam[4]));
    if (MULTI) {
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            f[c].add(k.l23, fix_split(ax[c]));
            f[c].add(k.l2, fix_split(m2[c]));
            f[c].add(k.l3, fix_split(m3[c]));
        }
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) out[c] = f[c].get(k.up);
}

// the metric (M^2 = (4/9) [[5, -4], [-4, 5]] or M on components 0 and 3) and the scale
QMIN_DEV void fixed_to_force(const FixedCoef &k, const long long (&a)[5], double *f)
{
    const double f0 = fixed_scale(a[0], 0), f3 = fixed_scale(a[3], 0);
    f[0] = k.ma * f0 - k.mb * f3;
    f[3] = k.ma * f3 - k.mb * f0;
    f[1] = fixed_scale(a[1], k.shift);
    f[2] = fixed_scale(a[2], k.shift);
    f[4] = fixed_scale(a[4], k.shift);
}

}  // namespace qmin
