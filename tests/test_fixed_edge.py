"""The fixed-point deep-site force (qmin_fixed.cuh, compiled for the host) at the
edge of its range, |Q| just below 1: no high or middle sum overflows (under the
overflow sanitizer) and the error stays within the units that the products drop,
on fields of the largest magnitude, of full mantissas between 3/4 and 1, driven
to large sums for random parameters, and for a parameter set and a field whose
32-bit halves are all at their extremes."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "qmin_bulk_q25.h"
#include "qmin_fixed.cuh"
using namespace qmin;
typedef long long Field[3][3][3][5];  // Q 2^56
static long double value(long long x) { return ldexpl((long double)x, -56); }
// the force before the metric, in 80-bit arithmetic
static void reference(const qmin_ldg_params &p, const Field &X, long double *f)
{
    typedef long double T;
    const double Lt[4] = {p.L2, p.L3, 0, p.L1};
    T cq[5 * QMIN_Q25_W], s[5], q[5];
    for (int k = 0; k < 5; ++k)
        for (int n = 0; n < QMIN_Q25_W; ++n) {
            T c = 0;
            for (int t = 0; t < 4; ++t) c += (T)Lt[t] * qmin_q25_k[t][k][n] / 8;
            cq[k * QMIN_Q25_W + n] = c;
        }
#define QQ(dx, dy, dz, c) value(X[(dx) + 1][(dy) + 1][(dz) + 1][c])
    QMIN_BULK_Q25_NO_L4_PLAIN(cq, s);
#undef QQ
    for (int c = 0; c < 5; ++c) q[c] = value(X[1][1][1][c]);
    const T a = (T)p.A / 2, b = (T)p.B / 3, c = (T)p.C / 4;
    const T t = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3] + q[4] * q[4] + q[0] * q[3];
    const T g = 8 * c * t + 2 * a, b3 = 3 * b, w = 2 * q[0] * q[3] - q[1] * q[1];
    f[0] = b3 * (q[3] * q[3] + q[4] * q[4] + w) - g * (2 * q[0] + q[3]) - s[0];
    f[1] = -2 * b3 * (q[0] * q[1] + q[1] * q[3] + q[2] * q[4]) - 2 * g * q[1] - s[1];
    f[2] = -2 * b3 * (q[1] * q[4] - q[2] * q[3]) - 2 * g * q[2] - s[2];
    f[3] = b3 * (q[0] * q[0] + q[2] * q[2] + w) - g * (2 * q[3] + q[0]) - s[3];
    f[4] = -2 * b3 * (q[1] * q[2] - q[0] * q[4]) - 2 * g * q[4] - s[4];
}
static void fixed(const FixedCoef &k, const Field &X, long long (&a)[5])
{
    auto at = [&](int dx, int dy, int dz, int c) { return X[dx + 1][dy + 1][dz + 1][c]; };
    long long q[5], lam[5], ax[5], m2[5], m3[5];
    for (int c = 0; c < 5; ++c) q[c] = X[1][1][1][c];
    fixed_axis(at, q, lam, ax);
    fixed_mixed(at, m2, m3);
    fixed_force<true>(k, q, lam, ax, m2, m3, a);
}
// In units of 2^-R, R = shift - up, which a component's products are summed in: six products drop a quarter each (low x
// low); g2 has the same loss of its own product, half a unit times |2 q0 + q3| <= 3, and that of s, of the
// coefficient and of the roundings, 1.6 together; the other coefficients' roundings come to 0.25, the quadratic sums'
// to 0.125, the result's to a half: 5.5.  80-bit sums of this size lose less than one.
static bool close(const qmin_ldg_params &p, const FixedCoef &k, const Field &X)
{
    long double fl[5];
    long long a[5];
    reference(p, X, fl);
    fixed(k, X, a);
    for (int c = 0; c < 5; ++c) {
        const long double off = ldexpl((long double)a[c], -k.up) - ldexpl(fl[c], k.shift - k.up);
        if (fabsl(off) > 6.5)
            return printf("component %d: %.3Lf units off at %.17Lg (L %g %g %g A %g B %g C %g)\n", c, off, fl[c], p.L1,
                          p.L2, p.L3, p.A, p.B, p.C), false;
    }
    return true;
}
static qmin_ldg_params params(double A, double B, double C, double L1, double L2, double L3)
{
    qmin_ldg_params p;
    memset(&p, 0, sizeof p);
    p.A = A, p.B = B, p.C = C, p.L1 = L1, p.L2 = L2, p.L3 = L3, p.multi_constant = 1;
    return p;
}
static const long long ONE = 1LL << 56, EDGE = ONE - 8;  // 1, the FP64 number below it

// parameters at their bounds, every low half next to +-2^31 and of the sign that adds to component 3
static bool extremes()
{
    const double x = 1 - ldexp(1, -29) + ldexp(1, -50);
    const qmin_ldg_params p = params(32 * x, -4 * x, 0, x, 8 * x, -7 * x);
    const FixedCoef k = fixed_coeffs(p, QMIN_METRIC_CPU, nullptr);
    if (!k.ok) return printf("no form\n"), false;
    static Field X;
    const long long M = 1LL << 32, H = 1LL << 31;
    // smallest multiple of 8, d > 0, with (v - w d) mod 2^32 = 2^31 (from above: the half is -2^31 and up)
    auto fit = [&](long long v, long long w, long long rest) {
        for (long long d = 8;; d += 8)
            if ((((v - w * d) % M + M) % M - rest + M) % M < 8 * w) return d;
    };
    for (int s = 0; s < 27; ++s)
        for (int c = 0; c < 5; ++c) X[s / 9][s / 3 % 3][s % 3][c] = -EDGE;
    auto q = X[1][1][1];
    q[0] = q[2] = q[3] = EDGE;
    q[1] = q[4] = 0;
    q[3] -= fit(32 * (2 * q[3] + q[0]), 64, H);
    auto at = [&](int dx, int dy, int dz, int c) -> long long & { return X[dx + 1][dy + 1][dz + 1][c]; };
    // X3 = q0^2 + q2^2 + 2 q0 q3 at 2^58: its low half through q2
    for (q[2] = EDGE;; q[2] -= 8) {
        const __int128 v = (__int128)q[0] * q[0] + (__int128)q[2] * q[2] + 2 * (__int128)q[0] * q[3];
        const long long low = (long long)((v >> 54) & (M - 1));
        if (low >= H && low < H + 512) break;
        if (EDGE - q[2] > (1LL << 34)) return printf("no q2\n"), false;
    }
    // axis part of component 3 through a y neighbour, the Laplacian through an x neighbour
    auto ax3 = [&] { return 4 * q[3] + 2 * q[0] - at(0, -1, 0, 3) - at(0, 1, 0, 3) - at(0, 0, -1, 0) - at(0, 0, 1, 0) -
                            at(0, 0, -1, 3) - at(0, 0, 1, 3); };
    at(0, 1, 0, 3) += fit(ax3(), 1, H);
    auto lap = [&](int c) { return 6 * q[c] - at(-1, 0, 0, c) - at(1, 0, 0, c) - at(0, -1, 0, c) - at(0, 1, 0, c) -
                                   at(0, 0, -1, c) - at(0, 0, 1, c); };
    at(1, 0, 0, 3) += fit(2 * lap(3) + lap(0), 2, H);
    // face diagonals: k3 = 8 (xy1, xz2), xz4m - yz4m = 4
    auto diag = [&](int c, int a, int b, int u, int v, long long s) {  // value s at a = u, b = v
        int d[3] = {0, 0, 0};
        d[a] = u, d[b] = v;
        at(d[0], d[1], d[2], c) = s * EDGE;
    };
    for (int u = -1; u <= 1; u += 2)
        for (int v = -1; v <= 1; v += 2) {
            diag(1, 0, 1, u, v, -u * v);  // XY(-1, 1) - XY(1, 1)
            diag(2, 0, 2, u, v, u * v);   // XZ(1, 2) - XZ(-1, 2)
        }
    diag(4, 0, 2, -1, 1, 1);
    diag(4, 0, 2, -1, -1, -1);
    diag(4, 1, 2, -1, 1, -1);
    diag(4, 1, 2, -1, -1, 1);
    long long lam[5], ax[5], m2[5], m3[5], qq[5];
    auto g = [&](int dx, int dy, int dz, int c) { return at(dx, dy, dz, c); };
    for (int c = 0; c < 5; ++c) qq[c] = q[c];
    at(0, -1, 1, 4) += H - 72;  // m2 - m3, so that the half of m3 is just below 2^31 where that of m2 is just above
    fixed_mixed(g, m2, m3);
    at(1, 0, 1, 2) -= fit(m2[3], 1, H);  // both
    fixed_axis(g, qq, lam, ax);
    fixed_mixed(g, m2, m3);
    // all middle sums of component 3, in 128 bits
    const Fix2 y[6] = {fix_split((2 * q[3] + q[0]) * 32),
                       fix_split((long long)(((__int128)q[0] * q[0] + (__int128)q[2] * q[2] + 2 * (__int128)q[0] * q[3]) >> 54)),
                       fix_split(2 * lam[3] + lam[0]), fix_split(ax[3]), fix_split(m2[3]), fix_split(m3[3])};
    auto at52 = [](double v, int s) { return fix_split((long long)llrint(ldexp(v, s))); };
    const Fix2 c[6] = {at52(-p.A, 55), at52(p.B, 58), at52(-p.L1, 60), at52(-(p.L2 + p.L3), 60), at52(-p.L2, 57), at52(-p.L3, 57)};
    __int128 sum = 0, most = 0;
    for (int t = 0; t < 6; ++t) {
        sum += (__int128)c[t].h * y[t].l;
        if (sum > most) most = sum;
        sum += (__int128)c[t].l * y[t].h;
        if (sum > most) most = sum;
    }
    const double reached = ldexp((double)most, -60);
    printf("scale 2^52: middle sum %.3f of 8; scale taken 2^%d\n", reached, k.shift - k.up);
    if (reached <= 8) return printf("not at the extremes\n"), false;  // the case would show nothing
    return close(p, k, X);
}

int main()
{
    std::mt19937_64 rng(11);
    std::uniform_real_distribution<double> u(-1, 1);
    static Field X;
    const double sets[][6] = {{-1, -2.12 / 0.172, 1.73 / 0.172, 2.32, 1.0, 0.5}, {-0.172, -2.12, 1.73, 2.32, 1.0, 0.5},
                              {-1, -2.12 / 0.172, 1.73 / 0.172, 4.64, -0.7, 3.1}, {-1, -12, 10, 20, 10, -5},
                              {31.9, -3.9, 0.01, 0.99, 7.9, -6.9}, {-3.9, 7.9, 1.9, 0.9, 0.9, 0.9}};
    for (const auto &s : sets) {
        const qmin_ldg_params p = params(s[0], s[1], s[2], s[3], s[4], s[5]);
        const FixedCoef k = fixed_coeffs(p, QMIN_METRIC_CPU, nullptr);
        if (!k.ok) return printf("no form\n"), 1;
        for (int trial = 0; trial < 6000; ++trial) {
            for (int i = 0; i < 135; ++i) {
                long long &x = X[i / 45][i / 15 % 3][i / 5 % 3][i % 5];
                // the number below 1, full mantissas in [3/4, 1), in [0, 1)
                const long long m = trial % 3 == 0 ? EDGE
                                    : trial % 3 == 1 ? ONE - 8 * (1 + (long long)(rng() % (1ULL << 51)))
                                                     : (long long)(rng() % ONE);
                x = rng() & 1 ? m : -m;
            }
            if (!close(p, k, X)) return 1;
        }
    }
    // random parameters, the field driven upwards in one component of the result by flips of single values
    for (int t = 0; t < 400; ++t) {
        auto r = [&] { return (u(rng) > 0 ? 1 : -1) * exp2(3 * u(rng)); };
        const qmin_ldg_params p = params(r(), 4 * r(), 4 * r(), r(), r(), r());
        const FixedCoef k = fixed_coeffs(p, QMIN_METRIC_CPU, nullptr);
        if (!k.ok) continue;
        for (int i = 0; i < 135; ++i) X[i / 45][i / 15 % 3][i / 5 % 3][i % 5] = rng() & 1 ? EDGE : -EDGE;
        const int c = t % 5;
        for (int pass = 0; pass < 2; ++pass)
            for (int i = 0; i < 135; ++i) {
                long long &x = X[i / 45][i / 15 % 3][i / 5 % 3][i % 5];
                long long a[5], b[5];
                fixed(k, X, a);
                x = -x;
                fixed(k, X, b);
                if (llabs(b[c]) < llabs(a[c])) x = -x;
            }
        if (!close(p, k, X)) return 1;
    }
    return extremes() ? 0 : 1;
}
"""


def test_edge_of_the_range(tmp_path):
    src, exe = tmp_path / "edge.cpp", tmp_path / "edge"
    src.write_text(PROGRAM)
    base = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "open-qmin_gb300", "csrc"),
            str(src), "-o", str(exe)]
    r = subprocess.run(base[:1] + ["-fsanitize=signed-integer-overflow", "-fno-sanitize-recover"] + base[1:],
                       capture_output=True, text=True)
    if r.returncode != 0 and "sanitize" in r.stderr + r.stdout:
        pytest.skip("no overflow sanitizer")
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
