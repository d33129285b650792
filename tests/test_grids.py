"""Grid arithmetic of the tiled bulk kernels and the list kernels beside them
(qmin_grids.h, compiled for the host): whatever the box and the number of
listed sites, their sums fit the one buffer, and every plane is in a chunk."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "qmin_grids.h"
using namespace qmin;
static long long boxes = 0;
static int check(int x, int y, int z)
{
    const TileGrid g[] = {
        deep_grid(x, y, z, 32, 8, 0),      deep_grid(x, y, z, 16, 16, 0),    deep_grid(x, y, z, 32, 8, 2),
        deep_grid(x, y, z, 32, 8, 3),      fused_grid(x, y, z, 32, 8, 2, 16), fused_grid(x, y, z, 32, 8, 1, 16),
        fused_grid(x, y, z, 32, 8, 2, 0),  fused_grid(x, y, z, 32, 8, 1, 0), fused_grid(x, y, z, 32, 4, 4, 16),
        fused_grid(x, y, z, 32, 4, 2, 16), fused_grid(x, y, z, 32, 4, 4, 0)};
    const int listed = list_grid((int)std::min(1500000000LL, (long long)x * y * z));
    ++boxes;
    for (const TileGrid &t : g)
        if (t.blocks() < 1 || t.blocks() + listed > kMaxFusedBlocks || (long long)t.nz * t.zc < z)
            return printf("%d x %d x %d: %d blocks of %d planes and %d listed\n", x, y, z, t.blocks(), t.zc, listed), 1;
    return 0;
}
int main()
{
    for (int n = 3; n <= 1144; ++n)
        if (check(n, n, n)) return 1;
    std::mt19937_64 rng(3);
    std::uniform_real_distribution<double> u(0, 1);
    for (int k = 0; k < 400000; ++k) {
        const int x = (int)exp(log(3.) + u(rng) * log(700.)), y = (int)exp(log(3.) + u(rng) * log(700.));
        const int z = (int)exp(log(3.) + u(rng) * log(1e5));
        if (1LL * x * y * z > 1500000000LL || tiles_xy(x, y, 32, 4) > 15000 || tiles_xy(x, y, 16, 16) > 15000) continue;
        if (check(x, y, z)) return 1;
    }
    const int at[] = {256, 256, 480};
    if (check(at[0], at[1], at[2])) return 1;
    for (int n : {0, 1, 127, 128, 129, 152 * 8 * 128, 152 * 8 * 128 + 1, 2000000000})
        if (list_grid(n) < 1 || list_grid(n) > kMaxListBlocks) return 1;
    return boxes < 100000;
}
"""


def test_sums_of_bulk_and_listed_blocks_fit(tmp_path):
    src, exe = tmp_path / "grids.cpp", tmp_path / "grids"
    src.write_text(PROGRAM)
    csrc = os.path.join(ROOT, "open-qmin_gb300", "csrc")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I", csrc, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


WIDE = r"""
#include <cstdio>
#include "qmin_grids.h"
using namespace qmin;
int main()
{
    const int box[][3] = {{2048, 2048, 3}, {4096, 4096, 3}, {20000, 20000, 3}, {300000, 3, 3}, {3, 150000000, 3}, {7000, 11, 9}};
    for (const auto &b : box) {
        const int x = b[0], y = b[1], z = b[2];
        const TileGrid g[] = {deep_grid(x, y, z, 32, 8, 0),     deep_grid(x, y, z, 16, 16, 0),
                              deep_grid(x, y, z, 32, 8, 3),     fused_grid(x, y, z, 32, 8, 2, 16),
                              fused_grid(x, y, z, 32, 4, 4, 0), tile_grid(tiles_xy(x, y, 16, 16), z, 4, kMaxFusedBlocks)};
        for (const TileGrid &t : g)
            if (t.blocks() < t.ntiles || t.blocks() + kMaxListBlocks > sum_blocks(x, y) + (&t == g + 5 ? kMaxListBlocks : 0) ||
                (long long)t.nz * t.zc < z)
                return printf("%d x %d x %d: %d blocks\n", x, y, z, t.blocks()), 1;
    }
    return sum_blocks(512, 512) != kMaxFusedBlocks;
}
"""


def test_boxes_of_more_tiles_than_the_usual_buffer(tmp_path):
    src, exe = tmp_path / "wide.cpp", tmp_path / "wide"
    src.write_text(WIDE)
    csrc = os.path.join(ROOT, "open-qmin_gb300", "csrc")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-I", csrc, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
