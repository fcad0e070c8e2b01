// k_compat.cu -- the compat render: the reference's own image formation
// (ConeTraceShader::coneTrace, ConeTraceShader.cpp:15-82) as tiled kernels.
//
// The reference draws one camera-facing quad per board (radius r, centre c;
// billboard_vert_instanced.glsl with Library::createQuad), shades every
// fragment with conetrace_frag.glsl:122-201 and blends back to front
// (SRC_ALPHA, ONE_MINUS_SRC_ALPHA, main.cpp:94-95) after sorting the boards by
// distance on the CPU (CloudVolume.cpp:65-82).  Here:
//   count  some warps per board: the quad's conservative pixel rectangle, its
//          8x8 tiles (atomic per-tile counts) and the squared eye distance;
//   alloc  each tile's range of the list (k_bin_alloc);
//   fill   (distance bits << 32 | board) into each tile's list;
//   tiles  two 128-thread CTAs per 8x8 tile: sort its list (by ranks up to 128
//          entries, bitonic in shared memory up to 4096; longer ones are sorted
//          in place in global memory before); four threads per pixel blend a
//          quarter of the list each front to back, C += T a src, T *= 1 - a, and
//          the quarters combine in order (the over operator is associative),
//          which equals the back-to-front blend; a thread stops once its T falls
//          below the cutoff, a warp once all its threads have.
// The quad is perpendicular to the view axis f, so the fragment of pixel ray
// d (d.f = 1) is the plane point e + z d with z = (c - e).f; the quad covers
// the pixel when both plane coordinates (x, y) = ((p - c).s, (p - c).u) / r
// lie in [-1, 1].
#include <cuda_runtime.h>

#include <algorithm>

#include "cg_internal.h"
#include "cg_sample.cuh"

namespace {

using namespace cgs::pairs;

constexpr int CAP = 4096;      // most sort keys held in shared memory per tile
constexpr int NOISE_N = 32;    // noise map edge (ConeTraceShader.cpp:12)

// The noise map's cells (CompatDev::noise): thread 4 i + k makes corner k of texel i's,
// REPEAT.  (A new seed, us beyond the render: 582 with a map of texels, 697 with the
// cells made and uploaded by the host, 585 so, nearly all of it the host's map.)
__global__ void __launch_bounds__(256) k_compat_noise(const float2* map, float4* cells) {
    constexpr int M = NOISE_N - 1;
    const int t = blockIdx.x * 256 + threadIdx.x, k = t & 3, i = t >> 2;
    const int x = i & M, y = ((i / NOISE_N) + (k & 1)) & M,
              z = (i / (NOISE_N * NOISE_N) + (k >> 1)) & M;
    const int row = (z * NOISE_N + y) * NOISE_N;
    const float2 a = map[row + x], b = map[row + ((x + 1) & M)];
    cells[t] = make_float4(a.x, a.y, b.x - a.x, b.y - a.y);
}

// `parts` warps per board: lane 0 derives the board's tile rectangle, the lanes
// split its tiles for the per-tile count.
__global__ void k_compat_count(CompatDev P, int parts, int4* rect, float* key,
                               uint32_t* tile_count, unsigned long long* pairs) {
    const int g = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int b = g / parts, part = g % parts;
    const int lane = threadIdx.x & 31;
    if (b >= P.n) return;
    int4 R = make_int4(1, 1, 0, 0);
    if (lane == 0) {
        const CamDesc& cam = P.cam;
        const float4 c = P.cwr[b];
        const float dx = c.x - cam.eye[0], dy = c.y - cam.eye[1], dz = c.z - cam.eye[2];
        const float z = dx * cam.f[0] + dy * cam.f[1] + dz * cam.f[2];
        if (part == 0) key[b] = dx * dx + dy * dy + dz * dz;
        if (z > P.near_z && z < 2500.f && c.w > 0.f) {
            // plane coordinates of the centre and the half extent at unit depth
            const float xs = (dx * cam.s[0] + dy * cam.s[1] + dz * cam.s[2]) / z;
            const float ys = (dx * cam.u[0] + dy * cam.u[1] + dz * cam.u[2]) / z;
            const float h = c.w / z;
            const float ta = cam.tanh * cam.aspect;
            // pixel i lies at ndc (2 (i + 0.5) / W - 1) ta; row j at (1 - 2 (j + 0.5) / H) tanh;
            // one pixel of margin either side, the exact test is per pixel
            float lo_x = ((xs - h) / ta + 1.f) * 0.5f * (float)cam.W - 0.5f;
            float hi_x = ((xs + h) / ta + 1.f) * 0.5f * (float)cam.W - 0.5f;
            float lo_y = (1.f - (ys + h) / cam.tanh) * 0.5f * (float)cam.H - 0.5f;
            float hi_y = (1.f - (ys - h) / cam.tanh) * 0.5f * (float)cam.H - 0.5f;
            lo_x = fmaxf(lo_x, -2.f);
            lo_y = fmaxf(lo_y, -2.f);
            hi_x = fminf(hi_x, (float)cam.W + 1.f);
            hi_y = fminf(hi_y, (float)cam.H + 1.f);
            const int i0 = max(0, (int)floorf(lo_x) - 1), i1 = min(cam.W - 1, (int)ceilf(hi_x) + 1);
            const int j0 = max(0, (int)floorf(lo_y) - 1), j1 = min(cam.H - 1, (int)ceilf(hi_y) + 1);
            if (i0 <= i1 && j0 <= j1)
                R = make_int4(i0 / CG_COMPAT_TILE, j0 / CG_COMPAT_TILE, i1 / CG_COMPAT_TILE,
                              j1 / CG_COMPAT_TILE);
        }
        if (part == 0) rect[b] = R;
    }
    R.x = __shfl_sync(0xffffffffu, R.x, 0);
    R.y = __shfl_sync(0xffffffffu, R.y, 0);
    R.z = __shfl_sync(0xffffffffu, R.z, 0);
    R.w = __shfl_sync(0xffffffffu, R.w, 0);
    const int nx = R.z - R.x + 1, ny = R.w - R.y + 1;
    if (nx <= 0 || ny <= 0) return;
    if (lane == 0 && part == 0)
        atomicAdd(pairs, (unsigned long long)nx * (unsigned long long)ny);
    for (int t = part * 32 + lane; t < nx * ny; t += 32 * parts)
        atomicAdd(tile_count + (R.y + t / nx) * P.tiles_x + R.x + t % nx, 1u);
}

// `parts` warps per board: the lanes split its tiles.
__global__ void k_compat_fill(CompatDev P, int parts, const int4* rect, const float* key,
                              uint32_t* cursor, unsigned long long* list) {
    const int g = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int b = g / parts, part = g % parts;
    const int lane = threadIdx.x & 31;
    if (b >= P.n) return;
    const int4 R = rect[b];
    const int nx = R.z - R.x + 1, ny = R.w - R.y + 1;
    if (nx <= 0 || ny <= 0) return;
    const unsigned long long k =
        ((unsigned long long)__float_as_uint(key[b]) << 32) | (unsigned long long)(unsigned)b;
    for (int t = part * 32 + lane; t < nx * ny; t += 32 * parts) {
        const uint32_t slot = atomicAdd(cursor + (R.y + t / nx) * P.tiles_x + R.x + t % nx, 1u);
        list[slot] = k;
    }
}

// Ascending sort of a[0, m) by a sorting network over the next power of two
// p >= m whose every comparator puts the smaller key at the lower index
// (bitonic merges with the first step of each merge mirrored); positions at or
// beyond m stand for +infinity, so comparators reaching them never swap and
// are skipped.  All threads of the CTA call it.
template <typename Ptr>
__device__ void sort_keys(Ptr a, int m) {
    int p = 1;
    while (p < m) p <<= 1;
    for (int k = 2; k <= p; k <<= 1) {
        const int hk = k >> 1;
        for (int i = threadIdx.x; i < p / 2; i += blockDim.x) {
            const int blk = i / hk, off = i - blk * hk;
            const int lo = blk * k + off, hi = blk * k + k - 1 - off;
            if (hi < m) {
                const unsigned long long x = a[lo], y = a[hi];
                if (y < x) {
                    a[lo] = y;
                    a[hi] = x;
                }
            }
        }
        __syncthreads();
        for (int j = hk >> 1; j >= 1; j >>= 1) {
            for (int i = threadIdx.x; i < p / 2; i += blockDim.x) {
                const int blk = i / j, off = i - blk * j;
                const int lo = blk * 2 * j + off, hi = lo + j;
                if (hi < m) {
                    const unsigned long long x = a[lo], y = a[hi];
                    if (y < x) {
                        a[lo] = y;
                        a[hi] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// The blend of the noise cell (ix, iy, iz) (low five bits) at weights w.
// `tab` holds for each cell, consecutively, what the blend along x takes: for
// each (z, y) corner the green and alpha of the texel and the steps to its
// neighbour along x (4 loads in place of 8, one address).
__device__ __forceinline__ pair noise_cell(const ulonglong2* __restrict__ tab, int ix, int iy,
                                           int iz, float wx, float wy, float wz) {
    constexpr int M = NOISE_N - 1;
    const ulonglong2* c = tab + (((iz & M) * NOISE_N + (iy & M)) * NOISE_N + (ix & M)) * 4;
    const ulonglong2 c00 = __ldg(c), c10 = __ldg(c + 1), c01 = __ldg(c + 2), c11 = __ldg(c + 3);
    const pair x = both(wx), y = both(wy), z = both(wz);
    const pair x00 = fma2(x, c00.y, c00.x), x10 = fma2(x, c10.y, c10.x);
    const pair x01 = fma2(x, c01.y, c01.x), x11 = fma2(x, c11.y, c11.x);
    const pair y0 = fma2(y, sub2(x10, x00), x00), y1 = fma2(y, sub2(x11, x01), x01);
    return fma2(z, sub2(y1, y0), y0);
}

// texture(noiseMap, q).ga summed over the octaves: LINEAR with REPEAT at
// normalised coordinates (the fragment program reads only the green and alpha
// channels of a noise cell).
__device__ __forceinline__ pair noise_sum(const CompatDev& P, float cx, float cy, float cz) {
    pair n = 0ull;
    for (int k = 0; k < P.octaves; ++k) {
        const float off = P.oct[k >> 1].off[k & 1], fr = P.oct[k >> 1].fr[k & 1];
        const float x = (cx + off) * fr * (float)NOISE_N - 0.5f,
                    y = (cy + off) * fr * (float)NOISE_N - 0.5f,
                    z = (cz + off) * fr * (float)NOISE_N - 0.5f;
        const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
        n = fma2(both(P.oct[k >> 1].pe[k & 1]),
                 noise_cell(P.noise, (int)fx, (int)fy, (int)fz, x - fx, y - fy, z - fz), n);
    }
    return n;
}

// The same where every scaled coordinate's magnitude is below 2^21: floor and
// cell come from one addition, and the coordinates of two octaves are made
// together.
__device__ __forceinline__ pair noise_sum_near(const CompatDev& P, float cx, float cy, float cz) {
    const pair X = both(cx), Y = both(cy), Z = both(cz);
    const pair magic = both(12582912.f);  // 1.5 * 2^23 (0x4B400000)
    const pair scale = both((float)NOISE_N), half = both(-0.5f);
    pair n = 0ull;
    for (int k = 0; k < P.octaves; k += 2) {
        const auto& o = P.oct[k >> 1];
        const pair off = *reinterpret_cast<const pair*>(o.off),
                   fr = *reinterpret_cast<const pair*>(o.fr);
        const pair x = fma2(mul2(add2(X, off), fr), scale, half),
                   y = fma2(mul2(add2(Y, off), fr), scale, half),
                   z = fma2(mul2(add2(Z, off), fr), scale, half);
        const pair mx = add2_down(x, magic), my = add2_down(y, magic), mz = add2_down(z, magic);
        const float2 wx = halves(sub2(x, sub2(mx, magic))), wy = halves(sub2(y, sub2(my, magic))),
                     wz = halves(sub2(z, sub2(mz, magic)));
        n = fma2(both(o.pe[0]), noise_cell(P.noise, (int)mx, (int)my, (int)mz, wx.x, wy.x, wz.x),
                 n);
        if (k + 1 < P.octaves)
            n = fma2(both(o.pe[1]),
                     noise_cell(P.noise, (int)(mx >> 32), (int)(my >> 32), (int)(mz >> 32), wx.y,
                                wy.y, wz.y),
                     n);
    }
    return n;
}

__device__ __forceinline__ float sat(float x) { return fminf(fmaxf(x, 0.f), 1.f); }

// conetrace_frag.glsl:122-201 at plane point p (plane coordinates x, y) of the
// board (c, r); false when the fragment is discarded.
template <int FMT>
__device__ bool compat_fragment(const VolDesc& vd, const ConeSchedule& cs, const CompatDev& P,
                                float px, float py, float pz, float x, float y, float4 c,
                                float4& o) {
    const float bx = -P.cam.f[0], by = -P.cam.f[1], bz = -P.cam.f[2];  // toward the camera
    const float dx = px - c.x, dy = py - c.y, dz = pz - c.z;
    const float r = c.w;
    const float tx = (x + 1.f) * 0.5f, ty = (y + 1.f) * 0.5f;  // fragTex
    if (P.show_quad) {
        float sc = sqrtf(dx * dx + dy * dy + dz * dz) / r;
        sc = sqrtf(fmaxf(0.f, 1.f - sc * sc));
        const bool edge = tx < 0.01f || ty < 0.01f || tx > 0.99f || ty > 0.99f;
        const float v = edge ? 1.f : sc;
        o = make_float4(v, v, v, v);
        return true;
    }
    if (P.do_noise) {
        const float A = bx * bx + by * by + bz * bz;
        const float B = 2.f * (dx * bx + dy * by + dz * bz);
        const float C = (dx * dx + dy * dy + dz * dz) - r * r;
        const float disc = B * B - 4.f * A * C;
        if (disc < 0.01f) return false;
        const float sq = sqrtf(disc);
        const float tn = (-B - sq) / (2.f * A), tf = (-B + sq) / (2.f * A);
        const float wnx = px + bx * tn, wny = py + by * tn, wnz = pz + bz * tn;
        const float wfx = px + bx * tf, wfy = py + by * tf, wfz = pz + bz * tf;
        float ux = (wnx - c.x) / r, uy = (wny - c.y) / r, uz = (wnz - c.z) / r;
        float cx = wnx * P.inv_adjust, cy = wny * P.inv_adjust, cz = wnz * P.inv_adjust;
        const float ex = wfx * P.inv_adjust - cx, ey = wfy * P.inv_adjust - cy,
                    ez = wfz * P.inv_adjust - cz;
        float is = sqrtf(ex * ex + ey * ey + ez * ez) / P.step_size;
        is = fminf(is, (float)(P.max_steps - P.min_steps)) + (float)P.min_steps;
        const float lx = ex / (is - 1.f), ly = ey / (is - 1.f), lz = ez / (is - 1.f);
        const float oa = P.noise_opacity / (is - 1.f), la = 1.f / (is - 1.f);
        float ro = 0.f, rl = 0.f;
        // the samples run from the near point to the last one, which lies past the far
        // point where the step count is no whole number (by a chord, at two steps and
        // a little), so their largest coordinate is known before they are taken
        const int steps = (int)ceilf(is);
        const float span = (float)(steps - 1);
        const float reach = fmaxf(fmaxf(fmaxf(fabsf(cx), fabsf(cy)), fabsf(cz)),
                                  fmaxf(fmaxf(fabsf(cx + span * lx), fabsf(cy + span * ly)),
                                        fabsf(cz + span * lz)));
        const bool near = reach < P.noise_reach;
        for (int i = 0; i < steps; ++i) {
            // the cells' green and alpha
            const float2 ga = halves(near ? noise_sum_near(P, cx, cy, cz)
                                          : noise_sum(P, cx, cy, cz));
            float ng = ga.x;
            const float na = fabsf(ga.y);
            const float uu = ux * ux + uy * uy + uz * uz;
            ng += uy / sqrtf(uu);
            ro += na * (1.f - uu);
            rl += sat(ng * 0.5f + 0.5f);
            cx += lx;
            cy += ly;
            cz += lz;
            ux += lx;
            uy += ly;
            uz += lz;
        }
        const float col = P.min_color + P.color_scale * rl * la;
        const float qx = tx - 0.5f, qy = ty - 0.5f;
        const float alpha = 1.f - sqrtf(qx * qx + qy * qy) * 2.f;
        o = make_float4(col, col, col, sat(ro * oa) * alpha);
    }
    if (P.do_cone) {
        float sc = sqrtf(dx * dx + dy * dy + dz * dz) / r;
        sc = sqrtf(fmaxf(0.f, 1.f - sc * sc));
        if (sc < 0.01f) return false;
        const float D = (float)vd.D;
        const float vx = D * ((px + bx * r * sc - vd.wmin[0]) / vd.range[0]);
        const float vy = D * ((py + by * r * sc - vd.wmin[1]) / vd.range[1]);
        const float vz = D * ((pz + bz * r * sc - vd.wmin[2]) / vd.range[2]);
        const float ind = cgs::cone_reference<FMT>(vd, cs, vx, vy, vz, P.sun[0], P.sun[1], P.sun[2]);
        if (P.do_noise) {
            o.x *= ind;
            o.y *= ind;
            o.z *= ind;
        } else {
            o = make_float4(ind, ind, ind, ind);
        }
    }
    return true;
}

// In place, the lists longer than cap (their tiles' CTAs hold no more keys).
__global__ void __launch_bounds__(256) k_compat_sort(Bins bins, int cap,
                                                     unsigned long long* list) {
    const int m = (int)bins.count[blockIdx.x];
    if (m > cap) sort_keys(list + bins.offset[blockIdx.x], m);
}

// One 128-thread CTA per half of an 8x8-pixel tile: the tile's list is sorted,
// then split into SEG contiguous segments; thread (segment g, pixel p) blends
// its segment front to back into (C_g, T_g) and the segments are combined in
// order with the associative over operator, C = C_0 + T_0 (C_1 + T_1 (...)),
// T = T_0 T_1 ...  A segment stops early on its own transmittance (the
// combined image moves by at most the cutoff).
// What bounds it: instructions (noise taps two thirds, cone samples a third) at
// three quarters of the issue rate.  200 boards, 1080p, default noise and cone,
// us: 2063 with eight-load taps, both paths of the general trilinear sample and a
// 256-thread CTA a tile; 1729 with packed noise cells and clamped cone samples;
// 1595 with two octaves' coordinates made together; 1511 with five CTAs an SM and
// shared memory for the longest list, not for CAP keys (the L1 gets the rest); 1484
// with two levels' cone samples together; 1447 with half tiles (a CTA waits
// for its slowest warp; quarter tiles 1773, 2 segments 1617, 8 segments 1553).
constexpr int SEG = 4;
constexpr int SHARE = 2;  // CTAs a tile
constexpr int TILE_PX = CG_COMPAT_TILE * CG_COMPAT_TILE / SHARE;
constexpr int TILE_THREADS = SEG * TILE_PX;

template <int FMT>
__global__ void __launch_bounds__(TILE_THREADS, 1280 / TILE_THREADS)
    k_compat_tiles(VolDesc vd, ConeSchedule cs, CompatDev P, Bins bins, int cap,
                   const unsigned long long* list, float4* out) {
    extern __shared__ unsigned long long s_keys[];  // cap of them
    __shared__ float4 s_c[SEG][TILE_PX];
    __shared__ float s_t[SEG][TILE_PX];
    const int tile = blockIdx.x / SHARE, part = blockIdx.x % SHARE;
    const int tx = tile % P.tiles_x, ty = tile / P.tiles_x;
    list += bins.offset[tile];
    const int m = (int)bins.count[tile];
    if (m <= TILE_THREADS) {
        // few keys (they differ): each goes where its rank says
        const bool mine = (int)threadIdx.x < m;
        const unsigned long long key = mine ? list[threadIdx.x] : 0ull;
        if (mine) s_keys[threadIdx.x] = key;
        __syncthreads();
        int rank = 0;
#pragma unroll 4
        for (int i = 0; i < m; ++i) rank += s_keys[i] < key ? 1 : 0;
        __syncthreads();
        if (mine) s_keys[rank] = key;
        __syncthreads();
    } else if (m <= cap) {
        for (int i = threadIdx.x; i < m; i += blockDim.x) s_keys[i] = list[i];
        __syncthreads();
        sort_keys(s_keys, m);
    }
    // (a longer list has been sorted in place)
    const unsigned long long* keys = m <= cap ? s_keys : list;
    const CamDesc& cam = P.cam;
    const int pix = threadIdx.x & (TILE_PX - 1), seg = threadIdx.x / TILE_PX;
    const int pxi = tx * CG_COMPAT_TILE + (pix & (CG_COMPAT_TILE - 1));
    const int pyi =
        ty * CG_COMPAT_TILE + part * (CG_COMPAT_TILE / SHARE) + pix / CG_COMPAT_TILE;
    const bool active = pxi < cam.W && pyi < cam.H;
    const float ndx = (2.f * ((float)pxi + 0.5f) / (float)cam.W - 1.f) * cam.tanh * cam.aspect;
    const float ndy = (1.f - 2.f * ((float)pyi + 0.5f) / (float)cam.H) * cam.tanh;
    const float dx = cam.f[0] + ndx * cam.s[0] + ndy * cam.u[0];
    const float dy = cam.f[1] + ndx * cam.s[1] + ndy * cam.u[1];
    const float dz = cam.f[2] + ndx * cam.s[2] + ndy * cam.u[2];
    float4 C = make_float4(0.f, 0.f, 0.f, 0.f);
    float T = 1.f;
    const bool drawing = P.show_quad || P.do_noise || P.do_cone;
    const int k0 = (int)((long long)m * seg / SEG), k1 = (int)((long long)m * (seg + 1) / SEG);
    const int span = (m + SEG - 1) / SEG;  // the longest segment: uniform trip count
    for (int i = 0; i < span && drawing; ++i) {
        if ((i & 7) == 0 && !__any_sync(0xffffffffu, active && T >= P.cutoff && k0 + i < k1))
            break;  // the whole warp is done (warp-uniform trip count)
        const int k = k0 + i;
        if (!active || T < P.cutoff || k >= k1) continue;
        const int b = (int)(unsigned)(keys[k] & 0xFFFFFFFFull);
        const float4 c = __ldg(P.cwr + b);
        const float ox = c.x - cam.eye[0], oy = c.y - cam.eye[1], oz = c.z - cam.eye[2];
        const float z = ox * cam.f[0] + oy * cam.f[1] + oz * cam.f[2];
        if (!(z > P.near_z && z < 2500.f && c.w > 0.f)) continue;
        const float px = cam.eye[0] + z * dx, py = cam.eye[1] + z * dy, pz = cam.eye[2] + z * dz;
        const float qx = px - c.x, qy = py - c.y, qz = pz - c.z;
        const float x = (qx * cam.s[0] + qy * cam.s[1] + qz * cam.s[2]) / c.w;
        const float y = (qx * cam.u[0] + qy * cam.u[1] + qz * cam.u[2]) / c.w;
        if (!(x >= -1.f && x <= 1.f && y >= -1.f && y <= 1.f)) continue;
        float4 o;
        if (!compat_fragment<FMT>(vd, cs, P, px, py, pz, x, y, c, o)) continue;
        const float a = sat(o.w);
        const float ta = T * a;
        C.x += ta * sat(o.x);
        C.y += ta * sat(o.y);
        C.z += ta * sat(o.z);
        C.w += ta * a;
        T *= 1.f - a;
    }
    s_c[seg][pix] = C;
    s_t[seg][pix] = T;
    __syncthreads();
    if (seg == 0 && active) {
        float4 A = s_c[SEG - 1][pix];
        float TA = s_t[SEG - 1][pix];
#pragma unroll
        for (int g = SEG - 2; g >= 0; --g) {  // segment g in front of the combined rest
            const float4 F = s_c[g][pix];
            const float TF = s_t[g][pix];
            A = make_float4(F.x + TF * A.x, F.y + TF * A.y, F.z + TF * A.z, F.w + TF * A.w);
            TA *= TF;
        }
        out[(size_t)pyi * cam.W + pxi] =
            make_float4(A.x + TA * P.clear[0], A.y + TA * P.clear[1], A.z + TA * P.clear[2],
                        A.w + TA * P.clear[3]);
    }
}

// The reference's cone at a caller's positions.  The blend of a NaN or of an infinity
// with its own floor is a NaN.  (Tested beside the transmittance cones, in their kernel
// or in cone_general, this cost them 0.5 % and the batch render 0.2 %.)
template <int FMT>
__global__ void __launch_bounds__(128)
    k_reference_cones(const __grid_constant__ VolDesc vd, const __grid_constant__ TraceParams tp,
                      const __grid_constant__ ConeSchedule cs, const float* pos, int n,
                      float* out) {
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i >= n) return;
    const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    if (cs.steps == 0 || (isfinite(x) && isfinite(y) && isfinite(z)))
        out[i] = cgs::cone_reference<FMT>(vd, cs, x, y, z, tp.sun[0], tp.sun[1], tp.sun[2]);
    else
        out[i] = __int_as_float(0x7fc00000);
}

}  // namespace

cudaError_t launch_compat_noise(const float2* map, float4* cells, cudaStream_t st) {
    k_compat_noise<<<NOISE_N * NOISE_N * NOISE_N * 4 / 256, 256, 0, st>>>(map, cells);
    return cudaGetLastError();
}

// Warps per board of the count and fill passes: about 8192 in all (200 boards over
// 32400 tiles, one warp a board: the whole binning 66 us, 37 now).
static int board_parts(int n) { return std::min(64, std::max(1, 8192 / n)); }
static int board_blocks(int n) { return (int)(((long long)n * board_parts(n) + 3) / 4); }

cudaError_t launch_compat_count(const CompatDev& P, int4* rect, float* key, uint32_t* tile_count,
                                unsigned long long* pairs, cudaStream_t st) {
    if (P.n == 0) return cudaSuccess;
    k_compat_count<<<board_blocks(P.n), 128, 0, st>>>(P, board_parts(P.n), rect, key, tile_count,
                                                      pairs);
    return cudaGetLastError();
}

cudaError_t launch_compat_fill(const CompatDev& P, const int4* rect, const float* key,
                               uint32_t* cursor, unsigned long long* list, cudaStream_t st) {
    if (P.n == 0) return cudaSuccess;
    k_compat_fill<<<board_blocks(P.n), 128, 0, st>>>(P, board_parts(P.n), rect, key, cursor, list);
    return cudaGetLastError();
}

cudaError_t launch_compat_tiles(const VolDesc& vd, const ConeSchedule& cs, const CompatDev& P,
                                const Bins& bins, uint32_t most, unsigned long long* list,
                                float4* out, cudaStream_t st) {
    const int cap = (int)std::min<uint32_t>(CAP, std::max<uint32_t>(most, TILE_THREADS));
    if (most > (uint32_t)cap) k_compat_sort<<<bins.nbins, 256, 0, st>>>(bins, cap, list);
    const int blocks = bins.nbins * SHARE;
    if (vd.fmt == 0)
        k_compat_tiles<0><<<blocks, TILE_THREADS, cap * 8, st>>>(vd, cs, P, bins, cap, list, out);
    else
        k_compat_tiles<1><<<blocks, TILE_THREADS, cap * 8, st>>>(vd, cs, P, bins, cap, list, out);
    return cudaGetLastError();
}

cudaError_t launch_reference_cones(const VolDesc& vd, const TraceParams& tp,
                                   const ConeSchedule& cs, const float* pos, int n, float* out,
                                   cudaStream_t st) {
    auto* kernel = vd.fmt == 0 ? k_reference_cones<0> : k_reference_cones<1>;
    kernel<<<(n + 127) / 128, 128, 0, st>>>(vd, tp, cs, pos, n, out);
    return cudaGetLastError();
}

CG_OOB_TU(k_compat)
