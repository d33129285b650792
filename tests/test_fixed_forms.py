"""The fixed-point deep-site force (qmin_fixed.cuh) compiled for the host:
against 80-bit arithmetic no less exact than the FP64 form it stands for, and
free of overflow up to the edge of its range."""
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
// the force in T: in double with the FP64 kernels' operations (shared sums, FMA chains, the metric in one step
// where no field sits between its two applications)
template <class T> static void reference(const qmin_ldg_params &p, int mode, const double *fld, const T (*Q)[3][3][5], T *f)
{
    const bool dbl = sizeof(T) == 8;
    const double Lt[4] = {p.multi_constant ? p.L2 : 0, p.multi_constant ? p.L3 : 0, 0, p.L1};
    T cq[5 * QMIN_Q25_W], s[5];
    for (int k = 0; k < 5; ++k)
        for (int n = 0; n < QMIN_Q25_W; ++n) {
            T c = 0;
            for (int t = 0; t < 4; ++t) c += (T)Lt[t] * (dbl ? qmin_q25c_k : qmin_q25_k)[t][k][n] / 8;
            cq[k * QMIN_Q25_W + n] = c;
        }
#define QQ(dx, dy, dz, c) Q[(dx) + 1][(dy) + 1][(dz) + 1][c]
    if (dbl) {
        QMIN_BULK_Q25_NO_L4(cq, s);
    } else {
        QMIN_BULK_Q25_NO_L4_PLAIN(cq, s);
    }
#undef QQ
    const T *q = Q[1][1][1], a = (T)p.A / 2, b = (T)p.B / 3, c = (T)p.C / 4;
    using std::fma;
    const T t = fma(q[0], q[0] + q[3], fma(q[1], q[1], fma(q[2], q[2], fma(q[3], q[3], q[4] * q[4]))));
    const T g = fma(8 * c, t, 2 * a), b3 = 3 * b, w = fma(q[0] + q[0], q[3], -(q[1] * q[1]));
    f[0] = fma(b3, fma(q[3], q[3], fma(q[4], q[4], w)), fma(-g, fma((T)2, q[0], q[3]), -s[0]));
    f[1] = fma(-2 * b3, fma(q[0], q[1], fma(q[1], q[3], q[2] * q[4])), fma(-2 * g, q[1], -s[1]));
    f[2] = fma(-2 * b3, fma(q[1], q[4], -(q[2] * q[3])), fma(-2 * g, q[2], -s[2]));
    f[3] = fma(b3, fma(q[0], q[0], fma(q[2], q[2], w)), fma(-g, fma((T)2, q[3], q[0]), -s[3]));
    f[4] = fma(-2 * b3, fma(q[1], q[2], -(q[0] * q[4])), fma(-2 * g, q[4], -s[4]));
    if (mode == QMIN_METRIC_CPU && fld[0] == 0) {
        const T f0 = f[0], f3 = f[3];
        f[0] = (T)20 / 9 * f0 - (T)16 / 9 * f3;
        f[3] = (T)20 / 9 * f3 - (T)16 / 9 * f0;
        return;
    }
    for (int pass = mode == QMIN_METRIC_CPU ? 0 : 1; pass < 2; ++pass) {
        if (pass == 1)
            for (int k = 0; k < 5; ++k) f[k] -= fld[k];
        const T f0 = f[0], f3 = f[3];
        f[0] = (T)2 / 3 * (2 * f0 - f3);
        f[3] = (T)2 / 3 * (2 * f3 - f0);
    }
}
int main()
{
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> u(-1, 1);
    const double sets[][6] = {{2.32, 1.0, 0.5, 1, 0, 0},  {2.32, 1.0, 0.5, 1, 1, 0.2}, {2.32, 0, 0, 0, 0, 0.1},
                              {4.64, -0.7, 3.1, 1, 0, 0}, {20, 10, -5, 1, 0, 0},       {0.3, 0, 0, 0, 1, 0}};
    int bad = 0;
    for (const auto &set : sets)
        for (int kind = 0; kind < 4; ++kind) {  // random directors, smooth, nearly uniform, the edge of the range
            qmin_ldg_params p;
            memset(&p, 0, sizeof p);
            p.A = -1;
            p.B = -2.12 / 0.172;
            p.C = 1.73 / 0.172;
            p.L1 = set[0];
            p.L2 = set[1];
            p.L3 = set[2];
            p.multi_constant = (int)set[3];
            const int mode = (int)set[4];
            const double fld[5] = {set[5], -0.5 * set[5], 0.2 * set[5], 0.7 * set[5], -set[5]};
            const FixedCoef k = fixed_coeffs(p, mode, set[5] != 0 ? fld : nullptr);
            if (!k.ok) return printf("no form\n"), 1;
            double e64 = 0, efx = 0, worst = 0, fmax_ = 0;
            for (int trial = 0; trial < 4000; ++trial) {
                static double Q[3][3][3][5];
                static long double QL[3][3][3][5];
                static long long X[3][3][3][5];
                double base[5] = {0, 0, 0, 0, 0};
                for (int s = 0; s < 27; ++s) {
                    double *q = Q[s / 9][s / 3 % 3][s % 3];
                    double n[3] = {u(rng), u(rng), u(rng)};
                    const double r = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]), S = 0.8;
                    const double d[5] = {S * (n[0] * n[0] / (r * r) - 1. / 3), S * n[0] * n[1] / (r * r),
                                         S * n[0] * n[2] / (r * r), S * (n[1] * n[1] / (r * r) - 1. / 3),
                                         S * n[1] * n[2] / (r * r)};
                    if (s == 0) memcpy(base, d, sizeof d);
                    for (int c = 0; c < 5; ++c) {
                        q[c] = kind == 0 ? d[c] : base[c] + (kind == 1 ? 0.05 : 1e-4) * u(rng);
                        if (kind == 3) q[c] = (u(rng) > 0 ? 1 : -1) * nextafter(0.75, 0.0);
                    }
                }
                for (int s = 0; s < 27; ++s)
                    for (int c = 0; c < 5; ++c) {
                        const double q = Q[s / 9][s / 3 % 3][s % 3][c];
                        if (fix_magnitude(q) >= kFixWide) return printf("range\n"), 1;
                        QL[s / 9][s / 3 % 3][s % 3][c] = q;
                        X[s / 9][s / 3 % 3][s % 3][c] = to_fixed(q);
                    }
                long double fl[5];
                double f[5], fx[5];
                reference(p, mode, fld, QL, fl);
                reference(p, mode, fld, Q, f);
                auto at = [&](int dx, int dy, int dz, int c) { return X[dx + 1][dy + 1][dz + 1][c]; };
                long long q[5], lam[5], ax[5], m2[5], m3[5], a[5];
                for (int c = 0; c < 5; ++c) q[c] = X[1][1][1][c];
                fixed_axis(at, q, lam, ax);
                fixed_mixed(at, m2, m3);
                if (p.multi_constant) fixed_force<true>(k, q, lam, ax, m2, m3, a);
                else fixed_force<false>(k, q, lam, ax, m2, m3, a);
                fixed_to_force(k, a, fx);
                for (int c = 0; c < 5; ++c) {
                    e64 += (f[c] - fl[c]) * (f[c] - fl[c]);
                    efx += (fx[c] - fl[c]) * (fx[c] - fl[c]);
                    worst = fmax(worst, (double)fabsl(fx[c] - fl[c]));
                    fmax_ = fmax(fmax_, (double)fabsl(fl[c]));
                }
            }
            printf("L %g %g %g mode %d kind %d: error / FP64 error %.2f\n", p.L1, p.L2, p.L3, mode, kind, sqrt(efx / e64));
            // nematic fields: no larger than the FP64 form's.  At the edge (magnitudes whose FP64 products are
            // nearly exact): each of up to six products drops a quarter of the unit 2^-(shift - up) at most, the
            // metric's rows sum to 4, and the last steps are FP64
            bad += kind < 3 ? !(efx <= e64) : !(worst <= 12 * ldexp(1, k.up - k.shift) + 8 * ldexp(fmax_, -53));
        }
    // conversion: towards zero at 2^-56, any magnitude below 1
    for (int t = 0; t < 20000; ++t) {
        const double d = ldexp(u(rng), -(t % 70));
        if (to_fixed(d) != (long long)ldexpl((long double)d, 56)) return printf("to_fixed(%a)\n", d), 1;
    }
    return bad != 0 || to_fixed(0.0) != 0 || to_fixed(-0.0) != 0;
}
"""


def test_fixed_force_host(tmp_path):
    src, exe = tmp_path / "fixed.cpp", tmp_path / "fixed"
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
