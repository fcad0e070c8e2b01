// boards_fine (csrc/cg_boards.h) over board lists that are and are not acceptable, built
// with the undefined-behaviour sanitizer by tests/test_boards_look.py.  Prints one line
// per list: whether it is fine.
#include <cstdio>
#include <limits>
#include <vector>

#include "cg_boards.h"

int main() {
    const float inf = std::numeric_limits<float>::infinity();
    const float nan = std::numeric_limits<float>::quiet_NaN();
    const float odd[] = {0.f, 0.3f, 1.f, -1e-9f, -1e9f, -FLT_MAX, -inf, 1e9f, FLT_MAX, inf, nan};
    for (int D : {8, 128, 256, 512}) {
        BoardBox g;
        for (int a = 0; a < 3; ++a) {
            g.pos[a] = 0.5f;
            g.wmin[a] = 0.0f;
            g.range[a] = 1.0f;
        }
        g.D = D;
        g.bar = D <= 128 ? 8 : 32;
        g.nbx = (D + 7) / 8;
        g.nbz = (D + g.bar - 1) / g.bar;
        for (float r : odd)
            for (float x : {0.f, 1e9f, -FLT_MAX, inf, nan}) {
                const size_t n = 300;
                std::vector<float> pos(3 * n, 0.1f), rad(n, 0.01f), den(n, 1.f), raw(5 * n);
                for (size_t b = 0; b < n; b += 3) rad[b] = r, pos[3 * b + 1] = x;
                size_t pairs = 0;
                const bool fine = boards_fine(g, pos.data(), rad.data(), den.data(), n, 1.f,
                                              raw.data(), pairs);
                std::printf("%d %g %g %d\n", D, (double)r, (double)x, fine ? 1 : 0);
            }
    }
    return 0;
}
