// Shared memory of a boundary CTA of the many-ticks launch (resident.cuh), in
// elements: bounds that no particle of its radius exceeds, wherever it lies.  A
// launch whose particle outgrew them all the same reports kErrLinkOverflow.
#pragma once
#include <algorithm>
#include <cmath>

namespace lbm {

struct ResidentCaps {
    long long entries = 1, slots = 1, box = 1;
    // A particle of r nodes on a grid of n[] nodes.  Its link nodes lie less than
    // sqrt(2) outside the circle (their unit squares in a ring), or across the
    // periodic boundary from a circle clipped at the edges of the grid; eight
    // slots each.  box: its near box and a node more on each side.
    void add(double r, const int* n, int dims, long long link_cap) {
        const double pi = 3.14159265358979;
        const double s2 = std::sqrt(2.0), out = r + 1.5 * s2, in = std::max(0.0, r - 0.5 * s2);
        const double e = pi * (out * out - in * in) + 4.0 * (2.0 * r + 4.0);
        entries = std::max(entries, std::min(link_cap, (long long)std::ceil(e)));
        slots = std::max(slots, 8 * (long long)std::ceil(e));
        for (int k = 0; k < dims; ++k)
            box = std::max(box, std::min<long long>((long long)std::floor(2.0 * r) + 8, n[k]) + 2);
    }
};

}  // namespace lbm
