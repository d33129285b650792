"""The product sums of the fixed-point force (FixAcc, compiled for the host) keep
all four half products: against 128-bit arithmetic a sum of six is off by its
final rounding, half a unit, and what the two low bits that lo leaves out and its
downward rounding come to, six times (3/2 + 4 + 1) 2^-32 units."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <random>
#include "qmin_fixed.cuh"
using namespace qmin;
int main()
{
    std::mt19937_64 rng(5);
    const long long corner[] = {0, 1, -1, 0x7fffffff, 0x80000000LL, -0x80000000LL, (1LL << 60) - 1, -(1LL << 60),
                                (1LL << 58) + 0x7fffffff, -(1LL << 58) - 0x80000000LL, 0x1fffffff7fffffffLL / 4};
    long double worst = 0;
    for (int t = 0; t < 200000; ++t) {
        FixAcc s;
        s.zero();
        __int128 exact = 0;
        for (int k = 0; k < 6; ++k) {
            auto value = [&](int bits) {
                if (rng() % 4 == 0) return corner[rng() % 11];
                return (long long)(rng() >> 1) >> (63 - bits) << (rng() % 2 ? 0 : 3);
            };
            const long long x = value(30 + (int)(rng() % 28)), y = rng() % 2 ? value(57) : -value(57);
            s.add(fix_split(x), fix_split(y));
            exact += (__int128)x * y;
        }
        const __int128 off = ((__int128)s.get32() << 64) - exact;
        const long double units = (long double)(off < 0 ? -off : off) / 18446744073709551616.0L;
        if (units > worst) worst = units;
        // one square: hi + (2 mid + 4 lo) / 2^32
        const long long x = (long long)(rng() >> 3);
        FixAcc q;
        q.zero();
        q.square(fix_split(x));
        const __int128 sq = ((__int128)q.hi << 64) + ((2 * (__int128)q.mid + 4 * (__int128)q.lo) << 32), d = sq - (__int128)x * x;
        if ((long double)(d < 0 ? -d : d) > 6.5L * 4294967296.0L) return printf("square\n"), 1;
    }
    printf("%.12Lf\n", worst);
    return worst > 0.5L + 6 * 6.5L / 4294967296.0L;
}
"""


def test_product_sums(tmp_path):
    src, exe = tmp_path / "products.cpp", tmp_path / "products"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "open-qmin_gb300", "csrc"), str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
