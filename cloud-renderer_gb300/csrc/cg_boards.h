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
    float pos[3], wmin[3], range[3];
    int D;         // voxels per axis
    int nbx, nbz;  // bricks along x and y, bars along z
    int bar;       // bar height (voxels)
};

// Every test that may refuse a board, without branches and divisions, and an upper
// bound of the pairs: a board of radius rv voxels meets at most 2 rv + 1 voxels
// an axis, n of which lie in at most floor((n + edge - 2) / edge) + 1 bricks or
// bars.  False: the caller has to look at every board (one may have to be refused).
// Copies the boards into `raw`.  Any floats are fine: the bound of a board that will
// be refused is clamped like the others before it becomes an integer (a negative radius
// to 0: two selections behind one another would become a branch, which keeps the loop
// from being vectorized; 16384 boards 49 us so, 25 now).
inline bool boards_fine(const BoardBox& v, const float* positions, const float* scales,
                        const float* densities, size_t n, float fluffiness, float* raw,
                        size_t& pairs) {
    float* const pos = raw;
    float* const rad = raw + 3 * n;
    float* const den = raw + 4 * n;
    if (n) std::memcpy(pos, positions, n * 12);
    if (n && densities) std::memcpy(den, densities, n * 4);
    const float p0 = v.pos[0], p1 = v.pos[1], p2 = v.pos[2], big = FLT_MAX;
    const float half_to_voxels = (float)v.D / v.range[0];
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
            // (a margin for the roundings)
            const float m = (r + std::fabs(r)) * half_to_voxels * 1.001f + 1.01f;
            const float kb = (m + (BOARD_BRICK - 2)) * rb + 1.f, kz = (m - 2.f) * rz + 2.f;
            const int ib = (int)(kb < nb ? kb : nb), iz = (int)(kz < nz ? kz : nz);
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

// Bins along an axis that hold a voxel centre of a board's extent: their number below
// `behind` (the last one's index, and one) and from `first`, both in bins (any floats;
// none for a NaN).  Clamped to [0, count] as the positive part (x + |x|) / 2 and one
// selection.
inline int bins_met(float first, float behind, float count) {
    const float f = 0.5f * (first + std::fabs(first)), e = 0.5f * (behind + std::fabs(behind));
    const int met = (int)(e < count ? e : count) - (int)(f < count ? f : count);
    return met > 0 ? met : 0;
}

// A closer bound of the board-bar pairs, for lists that would be long by that of
// boards_fine, which counts boards beside and outside the volume as if they were inside:
// exact but for boards with an end at a voxel centre or without a centre (one each).
// FP32: a board that reaches the volume lies within three extents of it, at most 1536
// voxels, where a coordinate's and a radius' few roundings are below 1e-3 voxels, a
// tenth of the slack.  From the copies in `raw`.  (16384 boards: 35 us on top of an
// upload of 37.)
constexpr size_t BOARD_PAIRS_SHORT = (size_t)1 << 23;  // 32 MB of list
inline size_t pairs_met(const BoardBox& v, const float* raw, size_t n) {
    const float* const pos = raw;
    const float* const rad = raw + 3 * n;
    const float p0 = v.pos[0], p1 = v.pos[1], p2 = v.pos[2];
    const float w0 = v.wmin[0], w1 = v.wmin[1], w2 = v.wmin[2];
    // bins per unit of length; radii are in voxels of x
    const double vox = (double)v.D / (double)v.range[0];
    const float rb = (float)(vox / BOARD_BRICK), rz = (float)(vox / v.bar);
    const float t0 = rb, t1 = (float)((double)v.D / (double)v.range[1] / BOARD_BRICK),
                t2 = (float)((double)v.D / (double)v.range[2] / v.bar);
    const float nb = (float)v.nbx, nz = (float)v.nbz;
    // the lowest centre of [a - r, a + r] lies at a - r + 1/2 rounded down or above, the
    // highest at a + r - 1/2 rounded down (voxels)
    const float inset = 0.5f - 0.01f;
    const float ib = inset / BOARD_BRICK, iz = inset / (float)v.bar;
    double sum = 0.0;
    for (size_t base = 0; base < n; base += 256) {
        const size_t end = std::min(n, base + 256);
        int part = 0;
        for (size_t b = base; b < end; ++b) {
            const float eb = rad[b] * rb - ib, ez = rad[b] * rz - iz;
            const float x = (p0 + pos[3 * b] - w0) * t0, y = (p1 + pos[3 * b + 1] - w1) * t1,
                        z = (p2 + pos[3 * b + 2] - w2) * t2;
            part += bins_met(x - eb, x + (eb + 1.f), nb) * bins_met(y - eb, y + (eb + 1.f), nb) *
                    bins_met(z - ez, z + (ez + 1.f), nz);
        }
        sum += part;
    }
    return (size_t)sum + 1;
}
