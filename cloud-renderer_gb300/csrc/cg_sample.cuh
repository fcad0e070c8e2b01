// cg_sample.cuh -- device-side sampling of the mip pyramid, the hash-noise fBm
// and the sun cone, shared by the trace kernels.
#pragma once

#include <cuda_fp16.h>

#include "cg_internal.h"



namespace cgs {

__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float fp16_hi(uint32_t v) {
    return __half2float(__ushort_as_half((unsigned short)(v >> 16)));
}

// Two FP32 values in a register pair, and the operations on both at once (for
// kernels bound by instructions).
namespace pairs {
typedef unsigned long long pair;
__device__ __forceinline__ pair both(float v) {
    pair r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ pair make(float lo, float hi) {
    pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 halves(pair p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ pair fma2(pair a, pair b, pair c) {
    pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ pair sub2(pair a, pair b) {
    pair r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair add2(pair a, pair b) {
    pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair mul2(pair a, pair b) {
    pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair add2_down(pair a, pair b) {
    pair r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
}  // namespace pairs

// One voxel's (R, G) at flat index idx.
template <int FMT, bool WANT_G>
__device__ __forceinline__ float2 fetch(const void* pyr, int idx) {
    if (FMT == 0) {
        const float4* p4 = reinterpret_cast<const float4*>(pyr);
        if (WANT_G) return __ldg(reinterpret_cast<const float2*>(p4 + idx));
        return make_float2(__ldg(reinterpret_cast<const float*>(p4 + idx)), 0.f);
    }
    uint32_t t = __ldg(reinterpret_cast<const uint32_t*>(pyr) + idx);
    return make_float2(bf16_lo(t), WANT_G ? fp16_hi(t) : 0.f);
}

// fetch() at a flat index of the whole pyramid, checked in the bounds-check
// build (an index past the last level reads 0).
template <int FMT, bool WANT_G>
__device__ __forceinline__ float2 fetch_vd(const VolDesc& vd, int idx) {
    if (!CG_IN_BOUNDS(idx, vd.nvox)) return make_float2(0.f, 0.f);
    return fetch<FMT, WANT_G>(vd.pyr, idx);
}

__device__ __forceinline__ float lerp3(const float c[8], float wx, float wy, float wz) {
    float x00 = c[0] + wx * (c[1] - c[0]);
    float x10 = c[2] + wx * (c[3] - c[2]);
    float x01 = c[4] + wx * (c[5] - c[4]);
    float x11 = c[6] + wx * (c[7] - c[6]);
    float y0 = x00 + wy * (x10 - x00);
    float y1 = x01 + wy * (x11 - x01);
    return y0 + wz * (y1 - y0);
}

// Occupancy of the level-l brick holding texel (ix, iy, iz) (see VolDesc).
__device__ __forceinline__ bool occupied(const VolDesc& vd, int l, int ix, int iy, int iz) {
    const int nb = vd.occ_nb[l], sh = vd.occ_shift;
    int bx = min(max(ix >> sh, 0), nb - 1);
    int by = min(max(iy >> sh, 0), nb - 1);
    int bz = min(max(iz >> sh, 0), nb - 1);
    const int at = vd.occ_off[l] + (bz * nb + by) * nb + bx;
    if (!CG_IN_BOUNDS(at, vd.occ_total)) return false;
    return __ldg(vd.occ + at) != 0;
}

// Trilinear at level l of channel R (and G when WANT_G), level-0 voxel-space
// position (px,py,pz).  BORDER: taps outside the level read 0; otherwise
// clamp to edge.  Texel coordinates x = p * N_l / D - 0.5.  SKIP_EMPTY: when
// the footprint's brick is unoccupied the result is exactly (0, 0) for R and
// is returned without touching the volume (callers that use G only where
// R > 0).
template <int FMT, bool WANT_G, bool BORDER, bool SKIP_EMPTY>
__device__ __forceinline__ float2 tri(const VolDesc& vd, int l, float px, float py, float pz) {
    const int N = vd.dims[l];
    const float sc = vd.lsc[l];  // N_l / D
    float x = px * sc - 0.5f, y = py * sc - 0.5f, z = pz * sc - 0.5f;
    float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    float wx = x - fx, wy = y - fy, wz = z - fz;
    int ix = (int)fx, iy = (int)fy, iz = (int)fz;
    if (SKIP_EMPTY && !occupied(vd, l, ix, iy, iz)) return make_float2(0.f, 0.f);
    float r[8], g[8];
    const int base = (int)vd.offs[l];
    if (ix >= 0 && iy >= 0 && iz >= 0 && ix + 1 < N && iy + 1 < N && iz + 1 < N) {
        // interior: one base index, fixed offsets
        const int i0 = base + (iz * N + iy) * N + ix;
        const int NN = N * N;
        const int o[8] = {0, 1, N, N + 1, NN, NN + 1, NN + N, NN + N + 1};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float2 t = fetch_vd<FMT, WANT_G>(vd, i0 + o[k]);
            r[k] = t.x;
            g[k] = t.y;
        }
    } else {
        int xs[2] = {ix, ix + 1}, ys[2] = {iy, iy + 1}, zs[2] = {iz, iz + 1};
        bool vx[2], vy[2], vz[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            vx[a] = (xs[a] >= 0 && xs[a] < N);
            vy[a] = (ys[a] >= 0 && ys[a] < N);
            vz[a] = (zs[a] >= 0 && zs[a] < N);
            xs[a] = min(max(xs[a], 0), N - 1);
            ys[a] = min(max(ys[a], 0), N - 1);
            zs[a] = min(max(zs[a], 0), N - 1);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const int k = c * 4 + b * 2 + a;
                    const bool ok = !BORDER || (vx[a] && vy[b] && vz[c]);
                    float2 t = fetch_vd<FMT, WANT_G>(vd, base + (zs[c] * N + ys[b]) * N + xs[a]);
                    r[k] = ok ? t.x : 0.f;
                    g[k] = ok ? t.y : 0.f;
                }
    }
    return make_float2(lerp3(r, wx, wy, wz), WANT_G ? lerp3(g, wx, wy, wz) : 0.f);
}

// Quadrilinear with a precomputed (l0, frac) split.
template <int FMT, bool WANT_G, bool BORDER, bool SKIP_EMPTY>
__device__ __forceinline__ float2 quad_split(const VolDesc& vd, float px, float py, float pz,
                                             int l0, float fr) {
    float2 a = tri<FMT, WANT_G, BORDER, SKIP_EMPTY>(vd, l0, px, py, pz);
    if (fr > 0.f && l0 + 1 < vd.L) {
        float2 b = tri<FMT, WANT_G, BORDER, SKIP_EMPTY>(vd, l0 + 1, px, py, pz);
        a.x = a.x + fr * (b.x - a.x);
        a.y = a.y + fr * (b.y - a.y);
    }
    return a;
}

// Quadrilinear (GL_LINEAR_MIPMAP_LINEAR): lod clamped to [0, L-1].
template <int FMT, bool WANT_G, bool BORDER, bool SKIP_EMPTY>
__device__ __forceinline__ float2 quad(const VolDesc& vd, float px, float py, float pz,
                                       float lod) {
    const float maxl = (float)(vd.L - 1);
    lod = fminf(fmaxf(lod, 0.f), maxl);
    const int l0 = (int)floorf(lod);
    return quad_split<FMT, WANT_G, BORDER, SKIP_EMPTY>(vd, px, py, pz, l0, lod - (float)l0);
}

// ---- hardware-filtered sampling (surrogate renderer) ----------------------
// Same coordinates as tri(): the texture unit samples texel space at
// (p * N_l / D) with unnormalised coordinates, so its trilinear weights match
// the software path up to their 8-bit fixed-point precision; border
// addressing reads 0 outside the level.
template <bool SKIP_EMPTY>
__device__ __forceinline__ float2 tri_hw(const VolDesc& vd, int l, float px, float py, float pz) {
    const float sc = vd.lsc[l];  // N_l / D
    const float x = px * sc, y = py * sc, z = pz * sc;
    if (SKIP_EMPTY && !occupied(vd, l, (int)floorf(x - 0.5f), (int)floorf(y - 0.5f),
                                (int)floorf(z - 0.5f)))
        return make_float2(0.f, 0.f);
    return tex3D<float2>((cudaTextureObject_t)vd.tex[l], x, y, z);
}

template <bool SKIP_EMPTY>
__device__ __forceinline__ float2 quad_hw(const VolDesc& vd, float px, float py, float pz,
                                          float lod) {
    const float maxl = (float)(vd.L - 1);
    lod = fminf(fmaxf(lod, 0.f), maxl);
    const int l0 = (int)floorf(lod);
    const float fr = lod - (float)l0;
    float2 a = tri_hw<SKIP_EMPTY>(vd, l0, px, py, pz);
    if (fr > 0.f && l0 + 1 < vd.L) {
        float2 b = tri_hw<SKIP_EMPTY>(vd, l0 + 1, px, py, pz);
        a.x = a.x + fr * (b.x - a.x);
        a.y = a.y + fr * (b.y - a.y);
    }
    return a;
}

// Occupancy along a ray, linear in the march step k: brick coordinates
// a + k b per axis in the grid of one level.
struct OccRay {
    float a[3], b[3];
    const uint8_t* grid;
    int nb, bound;

    // Positions v(k) = v0 + k dv (level-0 voxels), bricks of edge S voxels whose
    // first one starts `shift` voxels before the volume.
    __device__ __forceinline__ void set(const VolDesc& vd, int l, const float v0[3],
                                        const float dv[3], float S, float shift) {
        const float r = 1.f / S;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = (v0[i] + shift) * r;
            b[i] = dv[i] * r;
        }
        grid = vd.occ + vd.occ_off[l];
        nb = vd.occ_nb[l];
        bound = vd.occ_total - vd.occ_off[l];
    }
    // The flag of the brick holding step k (clamped to the grid).
    __device__ __forceinline__ bool at(float k) const {
        constexpr float MAGIC = 12582912.f;  // 1.5 * 2^23: floor and integer in one addition
        constexpr int BIAS = 0x4B400000;
        const int x = __vimin_s32_relu(__float_as_int(__fadd_rd(fmaf(k, b[0], a[0]), MAGIC)) - BIAS, nb - 1);
        const int y = __vimin_s32_relu(__float_as_int(__fadd_rd(fmaf(k, b[1], a[1]), MAGIC)) - BIAS, nb - 1);
        const int z = __vimin_s32_relu(__float_as_int(__fadd_rd(fmaf(k, b[2], a[2]), MAGIC)) - BIAS, nb - 1);
        const int i = (z * nb + y) * nb + x;
        if (!CG_IN_BOUNDS(i, bound)) return false;
        return __ldg(grid + i) != 0;
    }
};

// View-march steps k (sample at t_k = tin + (k + 1/2) dt along the unit
// direction d from the eye) that can meet the occupied level-0 box (widened by
// one voxel, and by one step at either end): [k0, k1], empty (k0 > k1) when
// the ray misses it.  A step outside it whose sample has lod 0 reads exactly 0
// (its brick is unoccupied), so marches skip those steps.
__device__ __forceinline__ void occupied_steps(const VolDesc& vd, const float eye[3], float3 d,
                                               float tin, float dt, int Nv, int& k0, int& k1) {
    const int* b = vd.occ_box;
    const float D = (float)vd.D;
    const float dd[3] = {d.x, d.y, d.z};
    float ta = -1e30f, tb = 1e30f;
    k0 = Nv;
    k1 = -1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int lo = vd.D - __ldg(b + a), hi = __ldg(b + 3 + a);
        if (lo >= hi) return;  // nothing occupied
        const float vs = D / vd.range[a];
        const float ve = (eye[a] - vd.wmin[a]) * vs, dv = dd[a] * vs;
        const float l = (float)lo - 1.f, h = (float)hi + 1.f;
        if (dv == 0.f) {
            if (ve < l || ve > h) return;
            continue;
        }
        const float t0 = (l - ve) / dv, t1 = (h - ve) / dv;
        ta = fmaxf(ta, fminf(t0, t1));
        tb = fminf(tb, fmaxf(t0, t1));
    }
    if (!(tb >= ta)) return;
    const float fa = fmaxf((ta - tin) / dt - 0.5f, -1.f), fb = fminf((tb - tin) / dt - 0.5f, (float)Nv);
    k0 = max(0, (int)floorf(fa) - 1);
    k1 = min(Nv - 1, (int)ceilf(fb) + 1);
}

// Neumaier compensated accumulation.
__device__ __forceinline__ void neumaier(float& sum, float& comp, float term) {
    float t = sum + term;
    if (fabsf(sum) >= fabsf(term))
        comp += (sum - t) + term;
    else
        comp += (term - t) + sum;
    sum = t;
}

// Trilinear density at level-0 position p from the density quads of one level
// (VolDesc: scale sc = N_l / D, first cell off, row length P = N_l + 3).  The
// coordinates and blends are tri()'s; the floor and its integer come from one
// rounded-down addition of 1.5 * 2^23 (exact for |x| < 2^22), and the cell
// index is clamped to the padded grid, whose outer cells are 0.  The exact
// cone is bound by instruction issue, its loads hit L1: over the pyramid a
// sample costs eight loads, their addresses, six conversions, a bounds test and
// an occupancy test per level, over the quads two loads and three clamps
// (render of a 1080p view over 256^3 RGBA32F 1081 -> 692 us, 4K over 512^3
// BF16 6.71 -> 4.26 ms, 250,000 cones at random positions 81 -> 38 us, the
// same bits; the voxelize stores that keep the quads cost less than its noise).
template <int FMT>
__device__ __forceinline__ float4 load_quad(const VolDesc& vd, int at) {
    if (FMT == 0) return __ldg(reinterpret_cast<const float4*>(vd.quad) + at);
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(vd.quad) + at);
    return make_float4(bf16_lo(q.x), __uint_as_float(q.x & 0xFFFF0000u), bf16_lo(q.y),
                       __uint_as_float(q.y & 0xFFFF0000u));
}

template <int FMT>
__device__ __forceinline__ float tri_quads(const VolDesc& vd, float sc, int off, int P, float px,
                                           float py, float pz) {
    constexpr float MAGIC = 12582912.f;
    constexpr int BIAS = 0x4B400000 - 2;  // its bits, less the two cells of padding
    const float x = px * sc - 0.5f, y = py * sc - 0.5f, z = pz * sc - 0.5f;
    const float tx = __fadd_rd(x, MAGIC), ty = __fadd_rd(y, MAGIC), tz = __fadd_rd(z, MAGIC);
    const float wx = x - (tx - MAGIC), wy = y - (ty - MAGIC), wz = z - (tz - MAGIC);
    const int ix = __vimin_s32_relu(__float_as_int(tx) - BIAS, P - 1);
    const int iy = __vimin_s32_relu(__float_as_int(ty) - BIAS, P - 1);
    const int iz = __vimin_s32_relu(__float_as_int(tz) - BIAS, P - 1);
    const int at = off + (iz * P + iy) * P + ix;
    if (!CG_IN_BOUNDS(at + P * P, vd.quad_total)) return 0.f;
    const float4 a = load_quad<FMT>(vd, at), b = load_quad<FMT>(vd, at + P * P);
    const float x00 = a.x + wx * (a.y - a.x);
    const float x10 = a.z + wx * (a.w - a.z);
    const float x01 = b.x + wx * (b.y - b.x);
    const float x11 = b.z + wx * (b.w - b.z);
    const float y0 = x00 + wy * (x10 - x00);
    const float y1 = x01 + wy * (x11 - x01);
    return y0 + wz * (y1 - y0);
}

// tri_quads where the position is known to lie in the padded grid: no clamps, the
// cell's index from the additions' bits (the biases fall out modulo 2^32).
template <int FMT>
__device__ __forceinline__ float tri_flat(const VolDesc& vd, float sc, int off, int P, float px,
                                          float py, float pz) {
    constexpr float MAGIC = 12582912.f;
    constexpr unsigned BIAS = 0x4B400000u - 2u;
    const float x = px * sc - 0.5f, y = py * sc - 0.5f, z = pz * sc - 0.5f;
    const float tx = __fadd_rd(x, MAGIC), ty = __fadd_rd(y, MAGIC), tz = __fadd_rd(z, MAGIC);
    const float wx = x - (tx - MAGIC), wy = y - (ty - MAGIC), wz = z - (tz - MAGIC);
    const unsigned p = (unsigned)P, base = (unsigned)off - BIAS * (p * p + p + 1u);
    const int at = (int)(base + (__float_as_uint(tz) * p + __float_as_uint(ty)) * p +
                         __float_as_uint(tx));
    if (!CG_IN_BOUNDS(at, vd.quad_total) || !CG_IN_BOUNDS(at + P * P, vd.quad_total)) return 0.f;
    const float4 a = load_quad<FMT>(vd, at), b = load_quad<FMT>(vd, at + P * P);
    const float x00 = a.x + wx * (a.y - a.x);
    const float x10 = a.z + wx * (a.w - a.z);
    const float x01 = b.x + wx * (b.y - b.x);
    const float x11 = b.z + wx * (b.w - b.z);
    const float y0 = x00 + wy * (x10 - x00);
    const float y1 = x01 + wy * (x11 - x01);
    return y0 + wz * (y1 - y0);
}

// Cone steps st[i], st[i + 1] of a transmittance cone from the density quads:
// both samples of the finer levels are in flight together, the coarser ones
// only where a step lies between two levels.
template <int FMT>
__device__ __forceinline__ float2 cone_pair(const VolDesc& vd, const ConeStep* st, float vx,
                                            float vy, float vz, float sx, float sy, float sz) {
    const ConeStep& s = st[0];
    const ConeStep& t = st[1];
    const float ax = vx + s.h * sx, ay = vy + s.h * sy, az = vz + s.h * sz;
    const float bx = vx + t.h * sx, by = vy + t.h * sy, bz = vz + t.h * sz;
    float a = tri_quads<FMT>(vd, s.sc0, s.off0, s.p0, ax, ay, az);
    float b = tri_quads<FMT>(vd, t.sc0, t.off0, t.p0, bx, by, bz);
    if (s.frac > 0.f || t.frac > 0.f) {
        const float a1 = tri_quads<FMT>(vd, s.sc1, s.off1, s.p1, ax, ay, az);
        const float b1 = tri_quads<FMT>(vd, t.sc1, t.off1, t.p1, bx, by, bz);
        a = a + s.frac * (a1 - a);
        b = b + t.frac * (b1 - b);
    }
    return make_float2(a * s.w, b * t.w);
}

// Compensated accumulation of a term >= 0 on a sum >= 0 (neumaier() without
// its comparisons: the larger and the smaller are a maximum and a minimum).
__device__ __forceinline__ void compensate(float& sum, float& comp, float term) {
    const float t = __fadd_rn(sum, term);
    comp += __fadd_rn(__fsub_rn(fmaxf(sum, term), t), fminf(sum, term));
    sum = t;
}

// The transmittance cone over the density quads (cs.quads): the same samples
// as cone_general's.  Steps beyond the position where the ray leaves the box
// widened by cs.reach read exactly 0 and are not taken.  The default cone starts at
// its radius floor: its first 24 steps or more lie on one level exactly, and from
// an origin in the box they need neither the level's values nor the clamps again
// (FLAT, for view samples: 1080p over 256^3 RGBA32F 692 -> 648 us, 4K over 512^3
// BF16 4238 -> 3938; positions from anywhere are better off without the second
// loop, 250,000 of them 38.3 us and 39.7 with it).
template <int FMT, bool FLAT>
__device__ __forceinline__ float cone_quads(const VolDesc& vd, const ConeSchedule& cs, float vx,
                                            float vy, float vz, float sx, float sy, float sz) {
    const float D = (float)vd.D, E = cs.edge;
    const float h0 = cs.st[0].h;
    const float x = vx + h0 * sx, y = vy + h0 * sy, z = vz + h0 * sz;
    if (x < -E || y < -E || z < -E || x > D + E || y > D + E || z > D + E) return 0.f;
    // distances at which the ray leaves the box widened by cs.reach, and by
    // cs.flat_reach
    float out = 3e38f, flat_out = 3e38f;
    const float v[3] = {vx, vy, vz}, d[3] = {sx, sy, sz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (d[a] == 0.f) continue;
        const float r = 1.f / d[a], t = ((d[a] > 0.f ? D : 0.f) - v[a]) * r;
        out = fminf(out, t + cs.reach * fabsf(r));
        flat_out = fminf(flat_out, t + cs.flat_reach * fabsf(r));
    }
    float tau = 0.f, comp = 0.f;
    int i = 0;
    if (FLAT && fminf(fminf(vx, vy), vz) >= -0.25f &&
        fmaxf(fmaxf(vx, vy), vz) <= D + 0.25f) {
        const ConeStep& s = cs.st[0];
        for (; i < cs.flat; i += 2) {
            const float ha = cs.st[i].h, hb = cs.st[i + 1].h;
            if (hb > flat_out) break;
            const float a = tri_flat<FMT>(vd, s.sc0, s.off0, s.p0, vx + ha * sx, vy + ha * sy,
                                          vz + ha * sz);
            const float b = tri_flat<FMT>(vd, s.sc0, s.off0, s.p0, vx + hb * sx, vy + hb * sy,
                                          vz + hb * sz);
            compensate(tau, comp, a * cs.st[i].w);
            compensate(tau, comp, b * cs.st[i + 1].w);
        }
    }
    for (; i < cs.steps; i += 2) {
        if (cs.st[i].h > out) break;
        const float2 c = cone_pair<FMT>(vd, cs.st + i, vx, vy, vz, sx, sy, sz);
        compensate(tau, comp, c.x);
        compensate(tau, comp, c.y);
    }
    return tau + comp;
}

// Channel G of a texel.
template <int FMT>
__device__ __forceinline__ float fetch_light(const VolDesc& vd, int idx) {
    if (!CG_IN_BOUNDS(idx, vd.nvox)) return 0.f;
    if (FMT == 0) return __ldg(reinterpret_cast<const float*>(vd.pyr) + 4 * (size_t)idx + 1);
    return __half2float(__ushort_as_half(
        __ldg(reinterpret_cast<const unsigned short*>(vd.pyr) + 2 * (size_t)idx + 1)));
}

// tri<FMT, true, false, false>(...).y without its two paths: a coordinate
// clamped to [0, N - 1] before the floor blends the same two texels (beyond an
// edge, and on it, both are the edge's, so a weight of 0 gives the same value),
// and a zero stride stands for the texel past the last.
template <int FMT>
__device__ __forceinline__ float tri_light(const VolDesc& vd, int l, float px, float py,
                                           float pz) {
    constexpr float MAGIC = 12582912.f;  // 1.5 * 2^23: floor and integer in one addition
    constexpr int BIAS = 0x4B400000;
    const int N = vd.dims[l];
    const float sc = vd.lsc[l], last = (float)(N - 1);
    const float x = fminf(fmaxf(px * sc - 0.5f, 0.f), last);
    const float y = fminf(fmaxf(py * sc - 0.5f, 0.f), last);
    const float z = fminf(fmaxf(pz * sc - 0.5f, 0.f), last);
    const float mx = __fadd_rd(x, MAGIC), my = __fadd_rd(y, MAGIC), mz = __fadd_rd(z, MAGIC);
    const float wx = x - (mx - MAGIC), wy = y - (my - MAGIC), wz = z - (mz - MAGIC);
    const int ix = __float_as_int(mx) - BIAS, iy = __float_as_int(my) - BIAS,
              iz = __float_as_int(mz) - BIAS;
    const int dx = ix < N - 1 ? 1 : 0, dy = iy < N - 1 ? N : 0, dz = iz < N - 1 ? N * N : 0;
    const int i0 = (int)vd.offs[l] + (iz * N + iy) * N + ix;
    const int i1 = i0 + dy, i2 = i0 + dz, i3 = i1 + dz;
    const float g[8] = {fetch_light<FMT>(vd, i0), fetch_light<FMT>(vd, i0 + dx),
                        fetch_light<FMT>(vd, i1), fetch_light<FMT>(vd, i1 + dx),
                        fetch_light<FMT>(vd, i2), fetch_light<FMT>(vd, i2 + dx),
                        fetch_light<FMT>(vd, i3), fetch_light<FMT>(vd, i3 + dx)};
    return lerp3(g, wx, wy, wz);
}

// tri_light at levels l and l + 1 together (one lane of each pair a level).
template <int FMT>
__device__ __forceinline__ float2 tri_light_pair(const VolDesc& vd, int l, float px, float py,
                                                 float pz) {
    using namespace pairs;
    const pair magic = both(12582912.f), half = both(-0.5f);
    constexpr int BIAS = 0x4B400000;
    const int N[2] = {vd.dims[l], vd.dims[l + 1]};
    const pair sc = make(vd.lsc[l], vd.lsc[l + 1]);
    const float last[2] = {(float)(N[0] - 1), (float)(N[1] - 1)};
    const float p[3] = {px, py, pz};
    pair w[3];
    int i[3][2];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float2 u = halves(fma2(both(p[a]), sc, half));
        const pair t = make(fminf(fmaxf(u.x, 0.f), last[0]), fminf(fmaxf(u.y, 0.f), last[1]));
        const pair m = add2_down(t, magic);
        w[a] = sub2(t, sub2(m, magic));
        i[a][0] = (int)m - BIAS;
        i[a][1] = (int)(m >> 32) - BIAS;
    }
    float g[8][2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int n = N[q];
        const int dx = i[0][q] < n - 1 ? 1 : 0, dy = i[1][q] < n - 1 ? n : 0,
                  dz = i[2][q] < n - 1 ? n * n : 0;
        const int i0 = (int)vd.offs[l + q] + (i[2][q] * n + i[1][q]) * n + i[0][q];
        const int at[4] = {i0, i0 + dy, i0 + dz, i0 + dy + dz};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            g[2 * k][q] = fetch_light<FMT>(vd, at[k]);
            g[2 * k + 1][q] = fetch_light<FMT>(vd, at[k] + dx);
        }
    }
    pair x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const pair a = make(g[2 * k][0], g[2 * k][1]);
        x[k] = fma2(w[0], sub2(make(g[2 * k + 1][0], g[2 * k + 1][1]), a), a);
    }
    const pair y0 = fma2(w[1], sub2(x[1], x[0]), x[0]), y1 = fma2(w[1], sub2(x[3], x[2]), x[2]);
    return halves(fma2(w[2], sub2(y1, y0), y0));
}

// The reference's weighted sum of the light channel (mode 1, clamp to edge), for a
// finite position (tri_light's clamps take any other to an edge).
template <int FMT>
__device__ __forceinline__ float cone_reference(const VolDesc& vd, const ConeSchedule& cs,
                                                float vx, float vy, float vz, float sx, float sy,
                                                float sz) {
    float acc = 0.f;
    for (int i = 0; i < cs.steps; ++i) {
        const float h = cs.st[i].h, fr = cs.st[i].frac;
        const int l = cs.st[i].l0;
        const float x = vx + h * sx, y = vy + h * sy, z = vz + h * sz;
        float g;
        if (fr > 0.f && l + 1 < vd.L) {
            const float2 q = tri_light_pair<FMT>(vd, l, x, y, z);
            g = q.x + fr * (q.y - q.x);
        } else {
            g = tri_light<FMT>(vd, l, x, y, z);
        }
        acc += g * cs.st[i].w;
    }
    return acc;
}

// The cone over the pyramid itself: any level, either mode.  Out of line: the
// hot loops of the callers are sized for cone_quads.
template <int FMT>
__device__ __noinline__ float cone_general(const VolDesc& vd, const ConeSchedule& cs, float vx,
                                           float vy, float vz, float sx, float sy, float sz) {
    if (cs.mode == 1) return cone_reference<FMT>(vd, cs, vx, vy, vz, sx, sy, sz);
    const float D = (float)vd.D, E = cs.edge;
    float tau = 0.f, comp = 0.f;
    for (int i = 0; i < cs.steps; ++i) {
        float h = cs.st[i].h;
        float x = vx + h * sx, y = vy + h * sy, z = vz + h * sz;
        if (x < -E || y < -E || z < -E || x > D + E || y > D + E || z > D + E) break;
        float2 c = quad_split<FMT, false, true, true>(vd, x, y, z, cs.st[i].l0, cs.st[i].frac);
        neumaier(tau, comp, c.x * cs.st[i].w);
    }
    return tau + comp;
}

// Sun cone from level-0 voxel-space position v toward unit direction s.
// Mode 0 returns optical depth (world units); mode 1 the reference's
// weighted sum of the light channel.
template <int FMT, bool FLAT = true>
__device__ __forceinline__ float sun_cone(const VolDesc& vd, const ConeSchedule& cs, float vx,
                                          float vy, float vz, float sx, float sy, float sz) {
    if (cs.quads) return cone_quads<FMT, FLAT>(vd, cs, vx, vy, vz, sx, sy, sz);
    return cone_general<FMT>(vd, cs, vx, vy, vz, sx, sy, sz);
}

// Number of samples the transmittance cone takes before leaving the box
// (statistics only).
__device__ __forceinline__ unsigned cone_samples(const VolDesc& vd, const ConeSchedule& cs,
                                                 float vx, float vy, float vz, float sx,
                                                 float sy, float sz) {
    if (cs.mode == 1) return (unsigned)cs.steps;
    const float D = (float)vd.D, E = cs.edge;
    unsigned n = 0;
    for (int i = 0; i < cs.steps; ++i) {
        float h = cs.st[i].h;
        float x = vx + h * sx, y = vy + h * sy, z = vz + h * sz;
        if (x < -E || y < -E || z < -E || x > D + E || y > D + E || z > D + E) break;
        n++;
    }
    return n;
}

// ---- hash value-noise fBm --------------------------------------------------

// PCG3D (Jarzynski & Olano, "Hash Functions for GPU Rendering", JCGT 2020).
__device__ __forceinline__ uint3 pcg3d(uint3 v) {
    v.x = v.x * 1664525u + 1013904223u;
    v.y = v.y * 1664525u + 1013904223u;
    v.z = v.z * 1664525u + 1013904223u;
    v.x += v.y * v.z;
    v.y += v.z * v.x;
    v.z += v.x * v.y;
    v.x ^= v.x >> 16;
    v.y ^= v.y >> 16;
    v.z ^= v.z >> 16;
    v.x += v.y * v.z;
    v.y += v.z * v.x;
    v.z += v.x * v.y;
    return v;
}

__device__ __forceinline__ uint32_t octave_key(uint32_t seed, int o) {
    return seed * 0x9E3779B9u + (uint32_t)o * 0x85EBCA6Bu + 1u;
}

__device__ __forceinline__ float lattice(int ix, int iy, int iz, uint32_t k) {
    uint3 h = pcg3d(make_uint3((uint32_t)ix + k, (uint32_t)iy + (k ^ 0x68E31DA4u),
                               (uint32_t)iz + (k ^ 0xB5297A4Du)));
    return (float)(h.x >> 8) * (1.0f / 16777216.0f);
}

// Value noise of octave o at lattice coordinates (x, y, z): trilinear over
// the lattice with smoothstep weights.  Corner values come from the octave's
// table when the 2x2x2 corner block lies inside it, else from the hash.
__device__ __forceinline__ float value_noise(const TraceParams& tp, int o, float x, float y,
                                             float z) {
    float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    int ix = (int)fx, iy = (int)fy, iz = (int)fz;
    float ux = x - fx, uy = y - fy, uz = z - fz;
    float wx = ux * ux * (3.f - 2.f * ux);
    float wy = uy * uy * (3.f - 2.f * uy);
    float wz = uz * uz * (3.f - 2.f * uz);
    float c[8];
    const int tx = ix - tp.nt.lo[o][0], ty = iy - tp.nt.lo[o][1], tz = iz - tp.nt.lo[o][2];
    const int dx = tp.nt.dim[o][0], dy = tp.nt.dim[o][1], dz = tp.nt.dim[o][2];
    if (tp.nt.tab && tx >= 0 && ty >= 0 && tz >= 0 && tx + 1 < dx && ty + 1 < dy && tz + 1 < dz) {
        const float* t = tp.nt.tab + tp.nt.off[o] + (tz * dy + ty) * dx + tx;
        const int sy = dx, sz = dx * dy;
        c[0] = __ldg(t);
        c[1] = __ldg(t + 1);
        c[2] = __ldg(t + sy);
        c[3] = __ldg(t + sy + 1);
        c[4] = __ldg(t + sz);
        c[5] = __ldg(t + sz + 1);
        c[6] = __ldg(t + sz + sy);
        c[7] = __ldg(t + sz + sy + 1);
    } else {
        const uint32_t k = octave_key(tp.noise_seed, o);
        c[0] = lattice(ix, iy, iz, k);
        c[1] = lattice(ix + 1, iy, iz, k);
        c[2] = lattice(ix, iy + 1, iz, k);
        c[3] = lattice(ix + 1, iy + 1, iz, k);
        c[4] = lattice(ix, iy, iz + 1, k);
        c[5] = lattice(ix + 1, iy, iz + 1, k);
        c[6] = lattice(ix, iy + 1, iz + 1, k);
        c[7] = lattice(ix + 1, iy + 1, iz + 1, k);
    }
    return lerp3(c, wx, wy, wz);
}

// Value noise by one hardware trilinear fetch: with i = floor(x) and w the
// smoothstep weights, the smoothstep-weighted blend of the 8 lattice values
// is the texture's linear filter at texel coordinate (i - lo) + w + 0.5.
__device__ __forceinline__ float value_noise_hw(const TraceParams& tp, int o, float x, float y,
                                                float z) {
    float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    int tx = (int)fx - tp.nt.lo[o][0], ty = (int)fy - tp.nt.lo[o][1], tz = (int)fz - tp.nt.lo[o][2];
    if (tp.nt.tex[o] && tx >= 0 && ty >= 0 && tz >= 0 && tx + 1 < tp.nt.dim[o][0] &&
        ty + 1 < tp.nt.dim[o][1] && tz + 1 < tp.nt.dim[o][2]) {
        float ux = x - fx, uy = y - fy, uz = z - fz;
        float wx = ux * ux * (3.f - 2.f * ux);
        float wy = uy * uy * (3.f - 2.f * uy);
        float wz = uz * uz * (3.f - 2.f * uz);
        return tex3D<float>((cudaTextureObject_t)tp.nt.tex[o], (float)tx + wx + 0.5f,
                            (float)ty + wy + 0.5f, (float)tz + wz + 0.5f);
    }
    return value_noise(tp, o, x, y, z);
}

// fBm at world position p: the noise domain is shifted by tp.noise_shift
// (q = p + shift; a zero shift leaves p unchanged).
__device__ __forceinline__ float fbm_hw(const TraceParams& tp, float px, float py, float pz) {
    if (tp.noise_octaves <= 0) return 1.f;
    px += tp.noise_shift[0];
    py += tp.noise_shift[1];
    pz += tp.noise_shift[2];
    float amp = 1.f, sum = 0.f, f = tp.noise_freq;
    for (int o = 0; o < tp.noise_octaves; ++o) {
        sum += amp * value_noise_hw(tp, o, px * f, py * f, pz * f);
        amp *= tp.noise_gain;
        f *= tp.noise_lac;
    }
    return sum * tp.noise_inv_norm;
}

// fBm from its precomputed volume (surrogate renderer): one hardware
// trilinear fetch at the noise coordinate q = p + shift; the volume holds fBm
// at its texel centres over the noise domain (NoiseTab.fbm_org / fbm_sc).
__device__ __forceinline__ float fbm_volume(const TraceParams& tp, float px, float py,
                                            float pz) {
    if (tp.noise_octaves <= 0) return 1.f;
    if (!tp.nt.fbm_tex) return fbm_hw(tp, px, py, pz);
    const float tx = (px + tp.noise_shift[0] - tp.nt.fbm_org[0]) * tp.nt.fbm_sc[0];
    const float ty = (py + tp.noise_shift[1] - tp.nt.fbm_org[1]) * tp.nt.fbm_sc[1];
    const float tz = (pz + tp.noise_shift[2] - tp.nt.fbm_org[2]) * tp.nt.fbm_sc[2];
    return tex3D<float>((cudaTextureObject_t)tp.nt.fbm_tex, tx, ty, tz);
}

// fBm = sum_o gain^o noise_o(q * freq * lac^o) / sum_o gain^o at the noise
// coordinate q (already shifted); 1 without octaves.
__device__ __forceinline__ float fbm_q(const TraceParams& tp, float qx, float qy, float qz) {
    if (tp.noise_octaves <= 0) return 1.f;
    float amp = 1.f, sum = 0.f, f = tp.noise_freq;
    for (int o = 0; o < tp.noise_octaves; ++o) {
        sum += amp * value_noise(tp, o, qx * f, qy * f, qz * f);
        amp *= tp.noise_gain;
        f *= tp.noise_lac;
    }
    return sum * tp.noise_inv_norm;
}

// fBm at world position p (noise domain shifted by tp.noise_shift).
__device__ __forceinline__ float fbm(const TraceParams& tp, float px, float py, float pz) {
    if (tp.noise_octaves <= 0) return 1.f;
    return fbm_q(tp, px + tp.noise_shift[0], py + tp.noise_shift[1], pz + tp.noise_shift[2]);
}

}  // namespace cgs
