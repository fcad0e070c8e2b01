// cg_boards.h -- the quick look at a billboard list before its upload (plain C++).
#pragma once

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstddef>
#include <cstring>

constexpr int BOARD_BRICK = 8;  // brick edge (voxels)

// A volume as the look needs it: its box and the bricks and bars of its bins.
struct BoardBox {
    float pos[3], range[3];
    int D;         // voxels per axis
    int nbx, nbz;  // bricks along x and y, bars along z
    int bar;       // bar height (voxels)
};

// Every test that may refuse a board, without branches and divisions, and an upper
// bound of the pairs: a board of radius rv voxels meets at most 2 rv + 1 voxels
// an axis, n of which lie in at most floor((n + edge - 2) / edge) + 1 bricks or
// bars.  False: the caller has to look at every board (one may have to be refused).
// Copies the boards into `raw`.  Any floats are fine: the bound of a board that will
// be refused is clamped like the others before it becomes an integer.
inline bool boards_fine(const BoardBox& v, const float* positions, const float* scales,
                        const float* densities, size_t n, float fluffiness, float* raw,
                        size_t& pairs) {
    float* const pos = raw;
    float* const rad = raw + 3 * n;
    float* const den = raw + 4 * n;
    if (n) std::memcpy(pos, positions, n * 12);
    if (n && densities) std::memcpy(den, densities, n * 4);
    const float p0 = v.pos[0], p1 = v.pos[1], p2 = v.pos[2], big = FLT_MAX;
    const float to_voxels = 2.0f * (float)v.D / v.range[0];
    const float nb = (float)v.nbx, nz = (float)v.nbz;
    const float rb = 1.0f / BOARD_BRICK, rz = 1.0f / (float)v.bar;
    // integer sums and maxima (of the radii's bits): the compiler vectorizes them
    int bad = 0, largest = 0;
    double sum = 0.0;
    for (size_t base = 0; base < n; base += 256) {
        const size_t end = std::min(n, base + 256);
        int part = 0;
        for (size_t b = base; b < end; ++b) {
            const float r = scales[b] * fluffiness;
            rad[b] = r;
            const float x = std::fabs(p0 + pos[3 * b]), y = std::fabs(p1 + pos[3 * b + 1]),
                        z = std::fabs(p2 + pos[3 * b + 2]);
            bad |= !(r >= 0.f) | !(r <= big) | !(x <= big) | !(y <= big) | !(z <= big);
            int bits;
            std::memcpy(&bits, &r, 4);
            largest = std::max(largest, bits);
            const float m = r * to_voxels * 1.001f + 1.01f;  // (a margin for the roundings)
            const float kb = (m + (BOARD_BRICK - 2)) * rb + 1.f, kz = (m - 2.f) * rz + 2.f;
            const int ib = (int)std::max(0.f, kb < nb ? kb : nb),
                      iz = (int)std::max(0.f, kz < nz ? kz : nz);
            part += ib * ib * iz;
        }
        sum += part;
    }
    if (densities)
        for (size_t b = 0; b < n; ++b) bad |= !(den[b] >= 0.f) | !(den[b] < 32768.f);
    if (bad || !(sum <= (double)(1u << 28))) return false;
    pairs = (size_t)sum + 1;
    float top;
    std::memcpy(&top, &largest, 4);
    return (double)top / (double)v.range[0] * (double)v.D <= (double)v.D;
}
