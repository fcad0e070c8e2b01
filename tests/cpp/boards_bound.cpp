// The bounds of boards_fine and pairs_met (csrc/cg_boards.h) beside the exact number of bars that the
// boards' Q20 voxel boxes meet, and beside the number of boards that meet none; one line
// per random list.
#include <cstdio>
#include <cstdint>
#include <random>
#include <vector>

#include "cg_boards.h"

static long long floor_div(long long a, long long b) {
    return a / b - (a % b != 0 && (a < 0) != (b < 0));
}

// Bricks or bars of the voxel centres (2 i + 1) 2^19 in [q - rq, q + rq].
static long long met(long long q, long long rq, int D, int edge) {
    const long long one = 1 << 20;
    const long long lo = std::max(floor_div(q - rq - one / 2 + one - 1, one), 0ll);
    const long long hi = std::min(floor_div(q + rq - one / 2, one), (long long)D - 1);
    return lo > hi ? 0 : hi / edge - lo / edge + 1;
}

int main() {
    std::mt19937 rng(7);
    auto uniform = [&](float lo, float hi) {
        return lo + (hi - lo) * (float)(rng() >> 8) * 0x1p-24f;
    };
    for (int D : {2, 9, 64, 128, 129, 256, 500, 512})
        for (float size : {1.0f, 3.7f})
            for (float at : {0.5f, -30.0f, 1000.0f})
                for (int kind = 0; kind < 6; ++kind) {
                    BoardBox g;
                    for (int a = 0; a < 3; ++a) {
                        g.pos[a] = at * (float)(a + 1);
                        g.wmin[a] = g.pos[a] - 0.5f * size;
                        g.range[a] = (g.pos[a] + 0.5f * size) - g.wmin[a];
                    }
                    g.D = D;
                    g.bar = D <= 128 ? 8 : 32;
                    g.nbx = (D + 7) / 8;
                    g.nbz = (D + g.bar - 1) / g.bar;
                    const size_t n = 700;
                    std::vector<float> pos(3 * n), rad(n), raw(5 * n);
                    const float spread[] = {0.5f, 0.5f, 1.5f, 3.0f, 0.5f, 40.0f};
                    const float largest[] = {0.02f, 0.3f, 0.9f, 0.9f, 0.0f, 0.9f};
                    for (size_t b = 0; b < n; ++b) {
                        for (int a = 0; a < 3; ++a)
                            pos[3 * b + a] = size * uniform(-spread[kind], spread[kind]);
                        rad[b] = size * uniform(0.f, largest[kind]);
                        if (kind == 1 && b % 2) {
                            // ends on voxel centres and faces
                            for (int a = 0; a < 3; ++a)
                                pos[3 * b + a] = size * (std::floor(pos[3 * b + a] / size *
                                                                    (float)D) + 0.5f) / (float)D;
                            rad[b] = size * std::floor(rad[b] / size * (float)D) / (float)D;
                        }
                    }
                    size_t bound = 0;
                    const bool fine = boards_fine(g, pos.data(), rad.data(), nullptr, n, 1.f,
                                                  raw.data(), bound);
                    const size_t met_bound = pairs_met(g, raw.data(), n);
                    long long exact = 0, none = 0;
                    for (size_t b = 0; b < n; ++b) {
                        const long long rq =
                            llrint((double)rad[b] / (double)g.range[0] * D * 0x1p20);
                        long long k = 1;
                        for (int a = 0; a < 3; ++a) {
                            const float c = g.pos[a] + pos[3 * b + a];
                            const double v =
                                ((double)c - (double)g.wmin[a]) / (double)g.range[a] * (double)D;
                            k *= v >= -D && v <= 2 * D
                                     ? met(llrint(v * 0x1p20), rq, D, a == 2 ? g.bar : 8)
                                     : 0;
                        }
                        exact += k;
                        none += k == 0;
                    }
                    std::printf("%d %g %g %d %d %zu %zu %lld %lld\n", D, (double)size,
                                (double)at, kind, fine ? 1 : 0, bound, met_bound, exact, none);
                }
    return 0;
}
