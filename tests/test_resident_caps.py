"""The bounds that size a boundary CTA's shared memory in the many-ticks launch (csrc/resident_caps.h) against counts
of the link nodes, their slots and the near box of circles of many radii and positions: inside the grid, clipped at one
edge or at a corner, larger than the grid.  Compiled with the header itself; no GPU."""
from __future__ import annotations

import os
import subprocess

from conftest import PKG

SOURCE = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "resident_caps.h"
int main() {
    std::mt19937_64 rng(12345);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    long long bad = 0, cases = 0;
    double fill = 0.0;
    for (int it = 0; it < 6000; ++it) {
        const double r = 0.4 * std::pow(150.0, U(rng));  // 0.4 to 60 nodes
        int n[3] = {1, 1, 1};
        for (int k = 0; k < 2; ++k) n[k] = 3 + (int)((0.8 + 2.0 * U(rng)) * 2.0 * r);
        double c[2];
        for (int k = 0; k < 2; ++k) {
            const int where = (int)(U(rng) * 4);  // 0: anywhere; 1: inside; 2: at the lower edge; 3: on a node or half way
            c[k] = where == 0 ? (U(rng) * 1.4 - 0.2) * n[k]
                 : where == 1 ? n[k] / 2 + U(rng)
                 : where == 2 ? (U(rng) * 2.2 - 1.1) * r : 0.5 * (int)(U(rng) * 2 * n[k]);
        }
        int lo[2], hi[2];
        bool outside = false;
        for (int k = 0; k < 2; ++k) {
            const double l = std::floor(c[k] - r) - 1.0, h = std::ceil(c[k] + r) + 1.0;
            outside = outside || h < 0.0 || l > n[k] - 1;
            lo[k] = l < 0.0 ? 0 : (int)l;
            hi[k] = h > n[k] - 1 ? n[k] - 1 : (int)h;
        }
        if (outside) continue;
        auto solid = [&](int x, int y) {
            x = (x + n[0]) % n[0];
            y = (y + n[1]) % n[1];
            const double a = x - c[0], b = y - c[1];
            return a * a + b * b < r * r;
        };
        long long entries = 0, slots = 0;
        for (int y = 0; y < n[1]; ++y)
            for (int x = 0; x < n[0]; ++x) {
                if (solid(x, y)) continue;
                int links = 0;
                for (int dy = -1; dy <= 1; ++dy)
                    for (int dx = -1; dx <= 1; ++dx)
                        if (dx || dy) links += solid(x + dx, y + dy);
                entries += links > 0;
                slots += links;
            }
        const long long span = (long long)std::floor(2.0 * r) + 6;  // as lbm_add_particle sizes the link list
        const long long link_cap = std::min<long long>(span + 2, n[0]) * std::min<long long>(span + 2, n[1]);
        lbm::ResidentCaps caps;
        caps.add(r, n, 2, link_cap);
        long long box = 0;
        for (int k = 0; k < 2; ++k) box = std::max<long long>(box, std::min(hi[k] - lo[k] + 3, n[k]) + 2);
        ++cases;
        fill = std::max(fill, (double)entries / caps.entries);
        if (entries > caps.entries || slots > caps.slots || box > caps.box) {
            ++bad;
            if (bad < 5)
                std::printf("r %g n %d %d c %g %g: %lld/%lld %lld/%lld %lld/%lld\n", r, n[0], n[1], c[0], c[1], entries,
                            caps.entries, slots, caps.slots, box, caps.box);
        }
    }
    std::printf("%lld of %lld outgrown, fullest list %.2f\n", bad, cases, fill);
    return bad != 0 || cases < 3000;
}
"""


def test_no_circle_outgrows_the_caps(tmp_path):
    src, exe = tmp_path / "caps.cpp", tmp_path / "caps"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(PKG, "csrc"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
