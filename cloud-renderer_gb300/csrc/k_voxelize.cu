// k_voxelize.cu -- sun-view map, highlight stores, brick-binned coverage splat
// and the mip pyramid.  Compiled with -fmad=false: every FP32 operation that
// decides an index (sun-view depth keys, highlight voxel indices) is written
// with explicitly rounded intrinsics in the same order as the CPU oracle, so
// winners, indices and integer coverage match it bit for bit.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "cg_internal.h"

namespace {

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fsqrt(float a) { return __fsqrt_rn(a); }

__device__ __forceinline__ long long floor_div(long long a, long long b) {
    long long q = a / b;
    if ((a % b != 0) && ((a < 0) != (b < 0))) q--;
    return q;
}

// Voxels whose centre (2i+1)*2^19 lies in [q-rq, q+rq], clamped to [0, D-1].
__device__ __forceinline__ bool axis_range(int q, int rq, int D, int& lo, int& hi) {
    long long l = floor_div((long long)q - rq - CG_HALF_Q20 + CG_Q20 - 1, CG_Q20);
    long long h = floor_div((long long)q + rq - CG_HALF_Q20, CG_Q20);
    if (l < 0) l = 0;
    if (h > D - 1) h = D - 1;
    if (l > h) return false;
    lo = (int)l;
    hi = (int)h;
    return true;
}

// ---- board records ---------------------------------------------------------

// Board quantization to the Q20 voxel grid (FP64, round to nearest even):
//   v = (cw - wmin) / range * D per axis, q = rint(v * 2^20), culled from
//   coverage when v is outside [-D, 2D] or no voxel centre is in the box;
//   rq = rint(r / range_x * D * 2^20);  thr = floor(rq^2 * 9999 / 10000) (the
//   0.01 profile discard of first_voxelize.glsl:46);  dq = rint(density * 2^16).
// A thread per board; raw radii come with the fluffiness in them.
__global__ void __launch_bounds__(128) k_boards(const float* __restrict__ raw, bool densities,
                                                int n, BoardGrid g, float4* cwr, int4* qo,
                                                uint64_t* thr, uint32_t* dq, uint8_t* culled) {
    const int b = blockIdx.x * 128 + threadIdx.x;
    if (b >= n) return;
    const double D = (double)g.D;
    const float r = raw[3 * (size_t)n + b];
    const float d = densities ? raw[4 * (size_t)n + b] : 1.0f;
    float c[3];
    int q[3];
    bool cull = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        c[a] = fadd(g.pos[a], raw[3 * (size_t)b + a]);
        const double vv = __dmul_rn(
            __ddiv_rn(__dsub_rn((double)c[a], (double)g.wmin[a]), (double)g.range[a]), D);
        const bool in = vv >= -D && vv <= 2.0 * D;
        q[a] = in ? (int)__double2ll_rn(__dmul_rn(vv, (double)CG_Q20)) : 0;
        if (!in) cull = true;
    }
    const double rv = __dmul_rn(__ddiv_rn((double)r, (double)g.range[0]), D);
    const int rq = (int)__double2ll_rn(__dmul_rn(rv, (double)CG_Q20));
    // rq <= 512 * 2^20 < 2^30, so rq^2 < 2^60 fits; floor(r2 * 9999 / 10000)
    // = r2 - ceil(r2 / 10000) without a 128-bit division
    const uint64_t r2 = (uint64_t)rq * (uint64_t)rq;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int lo, hi;
        if (!axis_range(q[a], rq, g.D, lo, hi)) cull = true;
    }
    cwr[b] = make_float4(c[0], c[1], c[2], r);
    qo[b] = make_int4(q[0], q[1], q[2], rq);
    thr[b] = r2 - (r2 + 9999u) / 10000u;
    dq[b] = (uint32_t)__double2ll_rn(__dmul_rn((double)d, 65536.0));
    culled[b] = cull ? 1 : 0;
}

// ---- bar binning -----------------------------------------------------------

// Distance term along one axis from the board centre q to the nearest voxel
// centre of the voxel range [lo, hi] (Q20).
__device__ __forceinline__ long long axis_gap(int q, int lo, int hi) {
    long long c0 = (2ll * lo + 1) * CG_HALF_Q20, c1 = (2ll * hi + 1) * CG_HALF_Q20;
    long long c = q < c0 ? c0 : (q > c1 ? c1 : (long long)q);
    return (long long)q - c;
}

// Board bin walk of the count (in the sun-view pass) and fill (beside the
// highlight stores) passes: one warp per board,
// lanes over the bars (8 x 8 x bins.bar voxels) of its voxel box; a bar is kept
// only when its nearest voxel centre passes the board's ball test (the
// per-voxel test in k_splat stays exact).
template <bool FILL>
__device__ __forceinline__ void bin_walk(const BoardsDev& b, int D, const Bins& bins, int i,
                                         int lane) {
    if (i >= b.n || b.culled[i]) return;
    const int4 q = b.q[i];
    const unsigned long long thr = b.thr[i];
    int xl, xh, yl, yh, zl, zh;
    if (!axis_range(q.x, q.w, D, xl, xh) || !axis_range(q.y, q.w, D, yl, yh) ||
        !axis_range(q.z, q.w, D, zl, zh))
        return;
    const int bx0 = xl / CG_BRICK, by0 = yl / CG_BRICK, bz0 = zl / bins.bar;
    const int nx = xh / CG_BRICK - bx0 + 1, ny = yh / CG_BRICK - by0 + 1,
              nz = zh / bins.bar - bz0 + 1;
    const int total = nx * ny * nz;
    for (int t = lane; t < total; t += 32) {
        const int bx = bx0 + t % nx, by = by0 + (t / nx) % ny, bz = bz0 + t / (nx * ny);
        long long gx = axis_gap(q.x, max(bx * CG_BRICK, xl), min(bx * CG_BRICK + 7, xh));
        long long gy = axis_gap(q.y, max(by * CG_BRICK, yl), min(by * CG_BRICK + 7, yh));
        long long gz = axis_gap(q.z, max(bz * bins.bar, zl),
                                min(bz * bins.bar + bins.bar - 1, zh));
        unsigned long long d2 = (unsigned long long)(gx * gx) + (unsigned long long)(gy * gy) +
                                (unsigned long long)(gz * gz);
        if (d2 > thr) continue;
        const int bar = (bz * bins.nby + by) * bins.nbx + bx;
        if (FILL) {
            uint32_t slot = atomicAdd(&bins.cursor[bar], 1u);
            bins.list[slot] = (uint32_t)i;
        } else {
            atomicAdd(&bins.count[bar], 1u);
        }
    }
}

// Ranges of the list for the bars' boards: bars need disjoint ranges in any
// order, so a CTA takes one for its 256 bars with a single atomic on the total
// (zeroed before; a scan in bar order took one CTA 13 us for 8192 bars).
__device__ __forceinline__ void bin_alloc(const Bins& bins, int block) {
    __shared__ uint32_t s_sum[8], s_base;
    const int i = block * 256 + threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t c = i < bins.nbins ? bins.count[i] : 0u;
    uint32_t x = c;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_sum[w] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0u;
        for (int k = 0; k < 8; ++k) {
            const uint32_t t = s_sum[k];
            s_sum[k] = run;
            run += t;
        }
        s_base = run ? atomicAdd(bins.count + bins.nbins, run) : 0u;
    }
    __syncthreads();
    if (i < bins.nbins) {
        const uint32_t at = s_base + s_sum[w] + x - c;
        bins.offset[i] = at;
        bins.cursor[i] = at;
    }
}

// The ranges alone, and the largest count (*most, zeroed before).
__global__ void __launch_bounds__(256) k_bin_alloc(Bins bins, uint32_t* most) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    const uint32_t m = __reduce_max_sync(0xffffffffu, i < bins.nbins ? bins.count[i] : 0u);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(most, m);
    bin_alloc(bins, blockIdx.x);
}

// ---- sun-view nearest-surface map (first_voxelize.glsl:39-64) --------------

__device__ __forceinline__ float dot3(const float a[3], float x, float y, float z) {
    return fadd(fadd(fmul(a[0], x), fmul(a[1], y)), fmul(a[2], z));
}

// Board centre in sun view space: lookAt rows s, u, -f plus translation.
__device__ __forceinline__ float3 sun_view_of(const SunFrame& fr, float4 c) {
    float nf[3] = {-fr.fwd[0], -fr.fwd[1], -fr.fwd[2]};
    return make_float3(fadd(dot3(fr.right, c.x, c.y, c.z), fr.t[0]),
                       fadd(dot3(fr.up, c.x, c.y, c.z), fr.t[1]),
                       fadd(dot3(nf, c.x, c.y, c.z), fr.t[2]));
}

__device__ __forceinline__ float texel_coord(float lo, float hi, int i, int n) {
    float a = fadd(__int2float_rn(i), 0.5f);
    float b = fdiv(a, __int2float_rn(n));
    return fadd(lo, fmul(b, fsub(hi, lo)));
}

// Spherical profile, discard below 0.01, surface point pushed toward the sun,
// depth from the near-plane point (first_voxelize.glsl:43-63).
__device__ __forceinline__ bool sun_fragment(float xv, float yv, float3 cv, float r,
                                             float near_z, float& zs, float& depth) {
    float dx = fsub(xv, cv.x);
    float dy = fsub(yv, cv.y);
    float d2 = fadd(fmul(dx, dx), fmul(dy, dy));
    float dist = fsqrt(d2);
    float q = fdiv(dist, r);
    float t = fsub(1.0f, fmul(q, q));
    float prof = fsqrt(t > 0.0f ? t : 0.0f);
    if (!(prof >= 0.01f)) return false;
    zs = fadd(cv.z, fmul(r, prof));
    float dz = fadd(zs, near_z);
    float dep2 = fadd(fadd(fmul(xv, xv), fmul(yv, yv)), fmul(dz, dz));
    depth = fsqrt(dep2);
    return true;
}

__device__ __forceinline__ void texel_range(float lo, float hi, float c, float r, int n,
                                            int& a, int& b) {
    float span = hi - lo;
    float l = (c - r - lo) / span * (float)n - 0.5f;
    float h = (c + r - lo) / span * (float)n - 0.5f;
    // conservative: one texel of margin each side; NaN/huge values clamp
    float fa = floorf(l) - 1.0f, fb = ceilf(h) + 1.0f;
    fa = fmaxf(fa, 0.0f);
    fb = fminf(fb, (float)(n - 1));
    if (!(fa <= fb)) { a = 1; b = 0; return; }
    a = (int)fa;
    b = (int)fb;
}

// The map is swept in tiles of 8 x 4 texels, one warp pass each.  Most boards at
// a texel lie far behind the front one, and in submission order many exact depths
// (three IEEE roots and a division) were worked out before a front board had
// come by.  So a first pass takes, from every tile a board's disc covers
// well, an upper bound of the depths it will store there; the second passes over
// the tiles at which a board cannot beat the tile's bound, and tests the texels of
// the others against their current depth.  Instructions, 4096 boards on 1280 x 720:
// 33 M with one CTA per board over every texel of its rows (49 us), 5.7 M + 8.9 M
// in the two passes (12.7 + 20.5 us with the bars' counts and ranges, which took
// 27 us in kernels of their own); what is left is latency at half occupancy.
// Voxelize as a whole, us: 64^3 of 64 boards 56 -> 49, 256^3 BF16 of 4096
// 144 -> 122, 512^3 BF16 of 16384 1029 -> 879.
constexpr int SUN_TW = 8, SUN_TH = 4;
constexpr int SUN_AHEAD = 4;  // tiles in flight a warp (1, 2, 4: 54.5, 53.9, 53.4 us)

// A board in sun view: its texel box (empty: ia > ib) and the smallest square
// of the surface offset dz = (cv.z + r * prof) + near_z over prof in [0, 1]
// (rounded steps are monotone).
struct alignas(16) SunBoard {
    float3 cv;
    float r, dz2_min;
    int ia, ib, ja, jb;
    int tx0, ntx, ty0, tiles;  // its tiles, x fastest
    int pad[3];
};
static_assert(sizeof(SunBoard) == SUN_BOARD_BYTES, "");

__device__ __forceinline__ SunBoard sun_board(const BoardsDev& b, const SunFrame& fr, int i) {
    SunBoard s;
    const float4 c = b.cwr[i];
    s.cv = sun_view_of(fr, c);
    s.r = c.w;
    texel_range(fr.lo, fr.hi, s.cv.x, s.r, fr.W, s.ia, s.ib);
    texel_range(fr.lo, fr.hi, s.cv.y, s.r, fr.H, s.ja, s.jb);
    const float dz_lo = fadd(s.cv.z, fr.near_z), dz_hi = fadd(fadd(s.cv.z, s.r), fr.near_z);
    s.dz2_min = 0.0f;
    if (dz_lo > 0.0f) s.dz2_min = fmul(dz_lo, dz_lo);
    else if (dz_hi < 0.0f) s.dz2_min = fmul(dz_hi, dz_hi);
    s.tx0 = s.ia / SUN_TW;
    s.ty0 = s.ja / SUN_TH;
    s.ntx = s.ib / SUN_TW - s.tx0 + 1;
    s.tiles = s.ia <= s.ib && s.ja <= s.jb ? s.ntx * (s.jb / SUN_TH - s.ty0 + 1) : 0;
    return s;
}

// Texel centres of tile t of the board: [x0, x1] x [y0, y1], each within
// sun_slack of the exact centres (a few roundings at the window's magnitude).
struct SunTile {
    int tx, ty;
    float x0, x1, y0, y1;
};
__device__ __forceinline__ float sun_slack(const SunFrame& fr) {
    return 4e-6f * fmaxf(fabsf(fr.lo), fabsf(fr.hi));
}
__device__ __forceinline__ SunTile sun_tile(const SunBoard& s, const SunFrame& fr, float sx,
                                            float sy, int t) {
    SunTile q;
    q.tx = s.tx0 + t % s.ntx;
    q.ty = s.ty0 + t / s.ntx;
    q.x0 = fr.lo + ((float)(q.tx * SUN_TW) + 0.5f) * sx;
    q.x1 = q.x0 + (float)(SUN_TW - 1) * sx;
    q.y0 = fr.lo + ((float)(q.ty * SUN_TH) + 0.5f) * sy;
    q.y1 = q.y0 + (float)(SUN_TH - 1) * sy;
    return q;
}

// First pass, `parts` warps per board: the tiles' bounds (float bits, all ones =
// none), the board's count in its bars (bins.count NULL: none); further CTAs
// tabulate the texel centres (aux.x, aux.y).
__global__ void __launch_bounds__(256) k_sun_bounds(BoardsDev b, SunFrame fr, SunAux aux, int parts,
                                                    int board_blocks, int D, Bins bins) {
    if ((int)blockIdx.x >= board_blocks) {
        const int t = (blockIdx.x - board_blocks) * 256 + threadIdx.x;
        if (t < fr.W) aux.x[t] = texel_coord(fr.lo, fr.hi, t, fr.W);
        if (t < fr.H) aux.y[t] = texel_coord(fr.lo, fr.hi, t, fr.H);
        return;
    }
    const int g = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int i = g / parts, part = g % parts;
    if (i >= b.n) return;
    if (bins.count && part == 0) bin_walk<false>(b, D, bins, i, lane);
    const SunBoard s = sun_board(b, fr, i);
    if (part == 0 && lane == 0) reinterpret_cast<SunBoard*>(aux.boards)[i] = s;
    const float span = fr.hi - fr.lo, sx = span / (float)fr.W, sy = span / (float)fr.H;
    const float slack = sun_slack(fr);
    const int wt = (fr.W + SUN_TW - 1) / SUN_TW;
    for (int t = part + parts * lane; t < s.tiles; t += 32 * parts) {
        const SunTile q = sun_tile(s, fr, sx, sy, t);
        // the farthest texel centre lies well inside the disc: every texel's
        // profile is at least sqrt(1 - 0.98), far above the 0.01 discard
        const float dx = fmaxf(fabsf(q.x0 - s.cv.x), fabsf(q.x1 - s.cv.x)) + slack;
        const float dy = fmaxf(fabsf(q.y0 - s.cv.y), fabsf(q.y1 - s.cv.y)) + slack;
        const float d2 = dx * dx + dy * dy, r2 = s.r * s.r;
        if (!(d2 <= 0.98f * r2)) continue;
        const float prof = sqrtf(1.0f - d2 / r2);
        const float z = s.cv.z + fr.near_z;
        const float dz = fmaxf(fabsf(z + 0.999f * s.r * prof), fabsf(z + 1.001f * s.r));
        const float x = fmaxf(fabsf(q.x0), fabsf(q.x1)), y = fmaxf(fabsf(q.y0), fabsf(q.y1));
        const float bound = sqrtf(x * x + y * y + dz * dz) * 1.00001f + slack +
                            1e-6f * (fabsf(s.cv.z) + fabsf(fr.near_z));
        atomicMin(aux.bound + q.ty * wt + q.tx, __float_as_uint(bound));
    }
}

// Second pass: the depth keys.  The first `alloc` CTAs give the bars their
// ranges of the list instead (their counts are complete).
__global__ void __launch_bounds__(256) k_sunmap(BoardsDev b, SunFrame fr, SunAux aux,
                                                unsigned long long* keys, int parts, int alloc,
                                                Bins bins) {
    if ((int)blockIdx.x < alloc) {
        bin_alloc(bins, blockIdx.x);
        return;
    }
    __shared__ SunBoard s_board[8];
    __shared__ int s_tile[8 * 32], s_of[8 * 32], s_n[2];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = (blockIdx.x - alloc) * 8 + w;
    const int i = g % b.n, part = g / b.n;  // the CTA's warps are on different boards
    SunBoard s;
    s.tiles = 0;
    if (part < parts)
        s = aux.boards ? reinterpret_cast<const SunBoard*>(aux.boards)[i] : sun_board(b, fr, i);
    if (lane == 0) s_board[w] = s;
    if (threadIdx.x == 0) s_n[0] = s_n[1] = 0;
    const float span = fr.hi - fr.lo, sx = span / (float)fr.W, sy = span / (float)fr.H;
    const float slack = sun_slack(fr);
    const int wt = (fr.W + SUN_TW - 1) / SUN_TW;
    int t0 = part;
    // rounds of 32 tiles a warp; the tiles to look at are shared out over the CTA
    for (int round = 0; __syncthreads_or(t0 < s.tiles); round ^= 1) {
        // this lane's tile: whether the disc (widened by a texel) meets it, and
        // the board may be in front of what the tile is bound to hold.  The
        // board's depths there are at least sqrt(xm^2 + ym^2 + dz_min^2)
        const int t = t0 + parts * lane;
        bool live = t < s.tiles;
        int at = 0;
        if (live) {
            const SunTile q = sun_tile(s, fr, sx, sy, t);
            at = q.ty << 16 | q.tx;
            const float dx = fmaxf(fmaxf(q.x0 - s.cv.x, s.cv.x - q.x1) - sx - slack, 0.f);
            const float dy = fmaxf(fmaxf(q.y0 - s.cv.y, s.cv.y - q.y1) - sy - slack, 0.f);
            live = dx * dx + dy * dy <= 1.0001f * (s.r * s.r);
            if (live && aux.bound) {
                const float xm = fmaxf(fmaxf(q.x0, -q.x1) - slack, 0.f);
                const float ym = fmaxf(fmaxf(q.y0, -q.y1) - slack, 0.f);
                const float bound = __uint_as_float(__ldg(aux.bound + q.ty * wt + q.tx));
                // (no bound is a NaN: nothing loses)
                live = !(bound * bound < (xm * xm + ym * ym + s.dz2_min) * (1.0f - 0x1p-18f));
            }
        }
        const unsigned todo = __ballot_sync(0xffffffffu, live);
        int base = 0;
        if (lane == 0 && todo) base = atomicAdd(&s_n[round], __popc(todo));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (live) {
            const int e = base + __popc(todo & ((1u << lane) - 1u));
            s_tile[e] = at;
            s_of[e] = w;
        }
        t0 += 32 * parts;
        __syncthreads();
        const int n = s_n[round];
        if (threadIdx.x == 0) s_n[round ^ 1] = 0;
        for (int e0 = w; e0 < n; e0 += 8 * SUN_AHEAD) {
            // some tiles at a time: their current depths in flight together
            unsigned long long cur[SUN_AHEAD];
            int at_x[SUN_AHEAD], at_y[SUN_AHEAD];
#pragma unroll
            for (int u = 0; u < SUN_AHEAD; ++u) {
                const int e = e0 + 8 * u;
                cur[u] = 0ull;
                at_x[u] = -1;
                at_y[u] = 0;
                if (e >= n) continue;
                const SunBoard& o = s_board[s_of[e]];
                const int ti = (s_tile[e] & 0xFFFF) * SUN_TW + (lane & 7);
                const int tj = (s_tile[e] >> 16) * SUN_TH + (lane >> 3);
                if (ti < o.ia || ti > o.ib || tj < o.ja || tj > o.jb) continue;
                at_x[u] = ti;
                at_y[u] = tj;
                cur[u] = *(volatile unsigned long long*)(keys + (size_t)tj * fr.W + ti);
            }
#pragma unroll
            for (int u = 0; u < SUN_AHEAD; ++u) {
                if (at_x[u] < 0) continue;
                const int of = s_of[e0 + 8 * u];
                const SunBoard& o = s_board[of];
                const float3 cv = o.cv;
                const float r = o.r;
                const float xv = aux.x ? aux.x[at_x[u]] : texel_coord(fr.lo, fr.hi, at_x[u], fr.W);
                const float yv = aux.y ? aux.y[at_y[u]] : texel_coord(fr.lo, fr.hi, at_y[u], fr.H);
                // texels well outside the disc (d^2 > 1.0001 r^2, where the exact
                // profile test cannot pass) and certain losers skip the roots and
                // the division: every step of the depth is monotone in |dz|, and a
                // current depth whose square is below the smallest possible one by
                // 2^-20 relative is strictly smaller as a float; an empty texel
                // (all ones, a NaN) never skips.  Values only decrease, so a stale
                // key can only make the tests pass (never skip a winner)
                const float ex = xv - cv.x, ey = yv - cv.y;
                if (ex * ex + ey * ey > 1.0001f * (r * r)) continue;
                const float xy2 = fadd(fmul(xv, xv), fmul(yv, yv));
                const float cd = __uint_as_float((unsigned)(cur[u] >> 32));
                if (cd * cd < fadd(xy2, o.dz2_min) * (1.0f - 0x1p-20f)) continue;
                float zs, depth;
                if (!sun_fragment(xv, yv, cv, r, fr.near_z, zs, depth)) continue;
                const unsigned id = (unsigned)((blockIdx.x - alloc) * 8 + of) % (unsigned)b.n;
                const unsigned long long key =
                    ((unsigned long long)__float_as_uint(depth) << 32) | id;
                if (key < cur[u]) atomicMin(keys + (size_t)at_y[u] * fr.W + at_x[u], key);
            }
        }
    }
}

// ---- highlight stores (second_voxelize.glsl:34-51) -------------------------

struct HiParams {
    float wmin[3], range[3];
    float inv_range[3];  // exact when pow2: every extent is a power of two
    bool pow2;
    float fD, offset;
    int D;
    int nb;            // bricks per axis
    uint8_t* hl;       // per-brick highlight flags (NULL: none)
};

__device__ __forceinline__ int voxel_index(const HiParams& hp, int a, float c) {
    const float s = fsub(c, hp.wmin[a]);
    // (a division by a power of two is the multiplication by its inverse)
    const float t = hp.pow2 ? fmul(s, hp.inv_range[a]) : fdiv(s, hp.range[a]);
    const float v = fmul(hp.fD, t);
    if (!(v > -1.0f && v < hp.fD)) return -1;
    return __float2int_rz(v);  // ivec3(): truncation toward zero
}

// One highlight store: the voxel's mask byte and, when flags are kept, its
// brick's flag (unless that is `done`, flagged by the caller); returns the brick.
__device__ __forceinline__ int mark(const HiParams& hp, uint8_t* mask, int x, int y, int z,
                                    int done) {
    const int vi = (z * hp.D + y) * hp.D + x;
    const int brick = ((z / CG_BRICK) * hp.nb + y / CG_BRICK) * hp.nb + x / CG_BRICK;
    if (!CG_IN_BOUNDS(vi, (size_t)hp.D * hp.D * hp.D)) return done;
    mask[vi] = 1;
    if (hp.hl && brick != done && CG_IN_BOUNDS(brick, (size_t)hp.nb * hp.nb * hp.nb))
        hp.hl[brick] = 1;
    return brick;
}

// CTAs of 32 x 8 texels.  The first `fill` CTAs do not store highlights: they
// fill the bars' lists, a warp per board (short, latency-bound work that costs
// little beside the stores; 0: no bins).
__global__ void __launch_bounds__(256) k_highlight(BoardsDev b, SunFrame fr,
                                                   const unsigned long long* keys, float4* posmap,
                                                   HiParams hp, uint8_t* mask, int fill,
                                                   Bins bins) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x < fill) {
        bin_walk<true>(b, hp.D, bins, blockIdx.x * 8 + warp, lane);
        return;
    }
    const int tx = (fr.W + 31) / 32, block = blockIdx.x - fill;
    const int ti = (block % tx) * 32 + lane;
    const int tj = (block / tx) * 8 + warp;
    if (ti >= fr.W || tj >= fr.H) return;
    const size_t idx = (size_t)tj * fr.W + ti;
    unsigned long long key = keys[idx];
    if (key == CG_KEY_EMPTY) {
        posmap[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    int bi = (int)(key & 0xFFFFFFFFull);
    float4 c = b.cwr[bi];
    float3 cv = sun_view_of(fr, c);
    float xv = texel_coord(fr.lo, fr.hi, ti, fr.W);
    float yv = texel_coord(fr.lo, fr.hi, tj, fr.H);
    float zs = 0.f, depth = 0.f;
    sun_fragment(xv, yv, cv, c.w, fr.near_z, zs, depth);
    float p[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        p[a] = fadd(fadd(fadd(fmul(xv, fr.right[a]), fmul(yv, fr.up[a])), fmul(zs, -fr.fwd[a])),
                    fr.eye[a]);
    posmap[idx] = make_float4(p[0], p[1], p[2], 1.0f);
    // the voxels of the point and of the eight points offset from it: per axis
    // three coordinates, the corners' two often in one voxel (stored once)
    const float o = hp.offset;
    int id[3], lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        id[a] = voxel_index(hp, a, p[a]);
        hi[a] = voxel_index(hp, a, fadd(p[a], o));
        lo[a] = voxel_index(hp, a, fsub(p[a], o));
        if (lo[a] == hi[a]) lo[a] = -1;
    }
    int own = -1;
    if (id[0] >= 0 && id[1] >= 0 && id[2] >= 0) own = mark(hp, mask, id[0], id[1], id[2], -1);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int x = (k & 4) ? lo[0] : hi[0], y = (k & 2) ? lo[1] : hi[1],
                  z = (k & 1) ? lo[2] : hi[2];
        if (x < 0 || y < 0 || z < 0 || (x == id[0] && y == id[1] && z == id[2])) continue;
        mark(hp, mask, x, y, z, own);
    }
}

// ---- coverage splat + level 0 + fused mips ---------------------------------

__device__ __forceinline__ uint32_t pack_bf16_fp16(float r, float g) {
    __nv_bfloat16 rb = __float2bfloat16_rn(r);
    __half gh = __float2half_rn(g);
    return (uint32_t)__bfloat16_as_ushort(rb) | ((uint32_t)__half_as_ushort(gh) << 16);
}

__device__ __forceinline__ float4 unpack_bf16_fp16(uint32_t v) {
    float r = __bfloat162float(__ushort_as_bfloat16((unsigned short)(v & 0xFFFFu)));
    float g = __half2float(__ushort_as_half((unsigned short)(v >> 16)));
    return make_float4(r, g, 0.f, 0.f);
}

__device__ __forceinline__ void store_voxel(const VolDesc& vd, void* pyr, int l, int x, int y,
                                            int z, float4 v) {
    const int N = vd.dims[l];
    size_t idx = (size_t)vd.offs[l] + ((size_t)z * N + y) * N + x;
    if (!CG_IN_BOUNDS(idx, vd.nvox)) return;
    __half2 h;
    unsigned short r16 = 0;  // the density bits of a half-precision level
    if (vd.fmt == 0) {
        reinterpret_cast<float4*>(pyr)[idx] = v;
        h = __floats2half2_rn(v.x, v.y);
    } else {
        const uint32_t w = pack_bf16_fp16(v.x, v.y);
        reinterpret_cast<uint32_t*>(pyr)[idx] = w;
        r16 = (unsigned short)(w & 0xFFFFu);
        h = __halves2half2(__float2half_rn(__uint_as_float(w << 16)),
                           __ushort_as_half((unsigned short)(w >> 16)));
    }
    // the texel's component of the four density quads that hold it
    if (l >= vd.quad_base) {
        const int p = vd.quad_p[l];
        const int at = vd.quad_off[l] + ((z + 2) * p + y + 2) * p + x + 2;
        if (CG_IN_BOUNDS(at, vd.quad_total) && CG_IN_BOUNDS(at - p - 1, vd.quad_total)) {
            if (vd.fmt == 0) {
                float* q = reinterpret_cast<float*>(vd.quad) + 4 * (size_t)at;
                q[0] = v.x;
                q[-4 + 1] = v.x;
                q[-4 * p + 2] = v.x;
                q[-4 * (p + 1) + 3] = v.x;
            } else {
                unsigned short* q = reinterpret_cast<unsigned short*>(vd.quad) + 4 * (size_t)at;
                q[0] = r16;
                q[-4 + 1] = r16;
                q[-4 * p + 2] = r16;
                q[-4 * (p + 1) + 3] = r16;
            }
        }
    }
    // the half2 texture copy holds exactly what the level stores (the same
    // conversion as the copy pass of k_textures.cu)
    if (vd.surf[l]) surf3Dwrite(*reinterpret_cast<uint32_t*>(&h), vd.surf[l], x * 4, y, z);
}

__device__ __forceinline__ float4 load_voxel(const VolDesc& vd, const void* pyr, int l, int x,
                                             int y, int z) {
    const int N = vd.dims[l];
    size_t idx = (size_t)vd.offs[l] + ((size_t)z * N + y) * N + x;
    if (vd.fmt == 0) return reinterpret_cast<const float4*>(pyr)[idx];
    return unpack_bf16_fp16(reinterpret_cast<const uint32_t*>(pyr)[idx]);
}

__device__ __forceinline__ float4 f4add(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
// 2x2x2 box mean in the oracle's order: ((c000+c100)+(c010+c110)) + ((c001+c101)+(c011+c111))
__device__ __forceinline__ float4 box8(float4 c000, float4 c100, float4 c010, float4 c110,
                                       float4 c001, float4 c101, float4 c011, float4 c111) {
    float4 s = f4add(f4add(f4add(c000, c100), f4add(c010, c110)),
                     f4add(f4add(c001, c101), f4add(c011, c111)));
    return make_float4(s.x * 0.125f, s.y * 0.125f, s.z * 0.125f, s.w * 0.125f);
}

// The exact z run [j0, j1) of a column's voxels inside a ball, by the int64 test
// of every voxel: only for columns whose run is too close to a voxel centre for
// FP32 (k_splat).
template <int BAR>
__device__ __noinline__ int2 exact_run(int4 q, unsigned long long thr, int vx, int vy, int vz0) {
    const int dx = vx - q.x, dy = vy - q.y;
    const unsigned long long dxy = (unsigned long long)((long long)dx * dx) +
                                   (unsigned long long)((long long)dy * dy);
    int j0 = BAR, j1 = 0;
    for (int j = 0; j < BAR; ++j) {
        const int dz = vz0 + j * (int)CG_Q20 - q.z;
        if (dxy + (unsigned long long)((long long)dz * dz) <= thr) {
            j0 = min(j0, j);
            j1 = j + 1;
        }
    }
    return make_int2(j0, j1);
}

// Coverage splat.  One CTA per bar of 8 x 8 x BAR voxels, 64 threads, one
// (x, y) column of BAR voxels per thread.  A board's ball meets a column in
// one run of voxels, so a thread adds (1, density) where the run starts and
// takes it off behind its end, in its own column of a shared-memory difference
// array (no conflicts, no atomics); the running sums give every voxel's count
// and Q16.16 density, modulo 2^32 like the sums they replace.
// The run's ends are those of the exact test on the Q20 grid (integer squared
// distance <= thr): FP32 gives cz -+ sqrt(r^2 - dx^2 - dy^2) in voxels relative to
// the bar within a bound delta, and a column with an end closer than delta to a
// voxel centre (about one in a thousand) takes the integer tests instead.  With
// eps >= the error of r^2 - dx^2 - dy^2 (r^2 and coordinates rounded to 24 bits:
// below 2e-6 r^2 + 6e-5), delta = 0.55 eps / s + 1e-4 + 1e-6 r covers the root's
// share eps / 2s, its rounding and that of cz.
// Bound by instruction issue in the board loop (about 60 of a warp per board).
// With one integer test per voxel (an 8^3 brick per CTA, half of the time in
// wide multiplications) and every brick marking its coarse occupancy cells:
// 256^3 RGBA32F with 4096 boards 84 -> 45 us, 512^3 BF16 with 16384 1223 -> 342 us.
// COV = false (voxelize): level 0 is assembled brick by brick, the next
// `fused_levels` mip levels are reduced in shared memory, raw occupancy is
// flagged.  COV = true: only the integer coverage (count, dq) is written
// (the coverage readback and the active-voxel statistic compute it on demand).
// Byte of the raw level-l cell (l >= 1) of the brick (x, y, z).
__device__ __forceinline__ int coarse_cell(const OccRaw& raw, int l, int x, int y, int z) {
    const int m = raw.nb[l];
    x = min(x >> (l - 1), m - 1);
    y = min(y >> (l - 1), m - 1);
    z = min(z >> (l - 1), m - 1);
    return raw.off[l] + (z * m + y) * m + x;
}

constexpr int SPLAT_ILP = 4;

// A tile's voxel: the channels the format stores (the means of the others are
// not kept).
__device__ __forceinline__ void put(float4& t, const float4& v) { t = v; }
__device__ __forceinline__ void put(float2& t, const float4& v) { t = make_float2(v.x, v.y); }
__device__ __forceinline__ float4 get(const float4& t) { return t; }
__device__ __forceinline__ float4 get(const float2& t) { return make_float4(t.x, t.y, 0.f, 0.f); }
template <int FMT>
struct TileOf {
    using T = float4;
};
template <>
struct TileOf<1> {
    using T = float2;
};

template <bool COV, int BAR, int FMT>
__global__ void __launch_bounds__(64) k_splat(BoardsDev b, Bins bins, const uint8_t* mask,
                                               VolDesc vd, void* pyr, uint32_t* count,
                                               uint32_t* dqout, int fused_levels,
                                               OccRaw occ_raw) {
    // 4 KB ahead of the difference array hold the staged boards; brick i's
    // level-0 tile (8 KB at 4 KB i) covers them and rows every thread has read
    constexpr int HALF_TILE = CG_BRICK * CG_BRICK * CG_BRICK * 8;
    __shared__ __align__(16) uint8_t s_buf[HALF_TILE + (BAR + 1) * 64 * 8];
    static_assert(CG_SPLAT_CHUNK * 36 <= HALF_TILE && CG_SPLAT_CHUNK == 64, "staged boards");
    static_assert(HALF_TILE == CG_BRICK * 64 * 8 && BAR % CG_BRICK == 0, "tile over the rows");
    float4* sa = reinterpret_cast<float4*>(s_buf);                        // cx, cy, cz, r^2
    float4* sb = reinterpret_cast<float4*>(s_buf + CG_SPLAT_CHUNK * 16);  // .55 eps, d0, eps, dq
    uint32_t* si = reinterpret_cast<uint32_t*>(s_buf + CG_SPLAT_CHUNK * 32);  // board
    using Tile = typename TileOf<FMT>::T;
    __shared__ float4 tile1[64];
    __shared__ float4 tile2[8];

    const int bx = blockIdx.x % bins.nbx;
    const int by = (blockIdx.x / bins.nbx) % bins.nby;
    const int bar = blockIdx.x / (bins.nbx * bins.nby);
    const int tid = threadIdx.x;
    uint2* diff = reinterpret_cast<uint2*>(s_buf + HALF_TILE) + tid;  // row j: diff[64 j]
    const int lx = tid & 7, ly = (tid >> 3) & 7;
    const int w = tid >> 5;
    const int D = vd.D;
    const int x = bx * CG_BRICK + lx, y = by * CG_BRICK + ly;
    const bool inxy = x < D && y < D;

    // the bricks' flags, all at once: highlights (NULL: unknown) and voxels left
    // from an earlier voxelize
    unsigned hlm = 0u, dirtym = 0u;
    if (!COV) {
#pragma unroll
        for (int i = 0; i < BAR / CG_BRICK; ++i) {
            const int bz = bar * (BAR / CG_BRICK) + i;
            if (bz >= bins.nbz) continue;
            const int brick = (bz * bins.nby + by) * bins.nbx + bx;
            if (bins.hl == nullptr || bins.hl[brick]) hlm |= 1u << i;
            if (bins.dirty[brick]) dirtym |= 1u << i;
        }
    }
    const uint32_t beg = bins.offset[blockIdx.x];
    const uint32_t n = bins.count[blockIdx.x];
    if (!COV && n == 0u && (hlm | dirtym) == 0u) return;
    if (n > 0u) {
        const float fx = (float)lx, fy = (float)ly;
        // voxel centre (0, 0, 0) of the bar on the Q20 grid
        const int ox = (2 * bx * CG_BRICK + 1) * (int)CG_HALF_Q20;
        const int oy = (2 * by * CG_BRICK + 1) * (int)CG_HALF_Q20;
        const int oz = (2 * bar * BAR + 1) * (int)CG_HALF_Q20;
        for (int j = 0; j <= BAR; ++j) diff[64 * j] = make_uint2(0u, 0u);
        for (uint32_t base = 0; base < n; base += CG_SPLAT_CHUNK) {
            const uint32_t m = min((uint32_t)CG_SPLAT_CHUNK, n - base);
            __syncthreads();
            sa[tid] = make_float4(0.f, 0.f, 0.f, -1e30f);  // a miss everywhere
            sb[tid] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tid < m) {
                const uint32_t bi = bins.list[beg + base + tid];
                const int4 q = b.q[bi];
                const float r2 = __ull2float_rn(b.thr[bi]) * 0x1p-40f;
                const float eps = 2e-6f * r2 + 6e-5f;
                sa[tid] = make_float4(__int2float_rn(q.x - ox) * 0x1p-20f,
                                      __int2float_rn(q.y - oy) * 0x1p-20f,
                                      __int2float_rn(q.z - oz) * 0x1p-20f, r2);
                sb[tid] = make_float4(0.55f * eps, 1e-4f + 1e-6f * 0x1p-20f * __int2float_rn(q.w),
                                      eps, __uint_as_float(b.dq[bi]));
                si[tid] = bi;
            }
            __syncthreads();
            // the runs of SPLAT_ILP boards are worked out side by side (their
            // chains are long), then added in turn
            for (uint32_t k0 = 0; k0 < m; k0 += SPLAT_ILP) {
                int j0[SPLAT_ILP], j1[SPLAT_ILP];
                uint32_t dq[SPLAT_ILP];
                unsigned unsure = 0u;
#pragma unroll
                for (int u = 0; u < SPLAT_ILP; ++u) {
                    constexpr float MAGIC = 12582912.f;  // 1.5 * 2^23
                    constexpr int BIAS = 0x4B400000;     // its bits
                    const float4 A = sa[k0 + u], B = sb[k0 + u];  // (past m: misses)
                    const float dx = fx - A.x, dy = fy - A.y;
                    const float rem = fmaf(-dy, dy, fmaf(-dx, dx, A.w));
                    float rs;
                    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(rem));
                    const float s = rem * rs, clear = 0.5f - fmaf(B.x, rs, B.y);
                    const float hi = A.z + s, lo = A.z - s;
                    const float th = __fadd_rd(hi, MAGIC), tl = __fadd_ru(lo, MAGIC);
                    const float fh = hi - (th - MAGIC), fl = (tl - MAGIC) - lo;
                    // (a root of 0 or less makes these comparisons false)
                    const bool sure = fabsf(fh - 0.5f) <= clear && fabsf(fl - 0.5f) <= clear;
                    if (!sure && !(rem < -B.z)) unsure |= 1u << u;
                    const int a = max(__float_as_int(tl) - BIAS, 0);
                    const int e = min(__float_as_int(th) - BIAS + 1, BAR);
                    // (a miss starts and ends in the row behind the bar, which
                    // nothing reads)
                    const bool hit = sure && a < e;
                    j0[u] = hit ? a : BAR;
                    j1[u] = hit ? e : BAR;
                    dq[u] = __float_as_uint(B.w);
                }
#pragma unroll
                for (int u = 0; u < SPLAT_ILP; ++u) {
                    uint2 p = diff[64 * j0[u]], e = diff[64 * j1[u]];
                    p.x += 1u;
                    p.y += dq[u];
                    e.x -= 1u;
                    e.y -= dq[u];
                    diff[64 * j0[u]] = p;
                    diff[64 * j1[u]] = e;
                }
                while (unsure) {
                    const uint32_t k = k0 + __ffs(unsure) - 1;
                    unsure &= unsure - 1u;
                    const uint32_t bi = si[k];
                    const int2 r = exact_run<BAR>(b.q[bi], b.thr[bi], ox + lx * (int)CG_Q20,
                                                  oy + ly * (int)CG_Q20, oz);
                    if (r.x >= r.y) continue;
                    diff[64 * r.x].x += 1u;
                    diff[64 * r.x].y += b.dq[bi];
                    diff[64 * r.y].x -= 1u;
                    diff[64 * r.y].y -= b.dq[bi];
                }
            }
        }
    }

    uint2 run = make_uint2(0u, 0u);  // the column's running sums
#pragma unroll 1
    for (int i = 0; i < BAR / CG_BRICK; ++i) {
        const int bz = bar * (BAR / CG_BRICK) + i;
        if (bz >= bins.nbz) break;
        const int brick = (bz * bins.nby + by) * bins.nbx + bx;
        const int z0 = bz * CG_BRICK;
        const size_t o = ((size_t)z0 * D + y) * D + x, slice = (size_t)D * D;
        const int nz = inxy ? min(D - z0, 8) : 0;  // the column's voxels in the volume
        uint32_t cnt[8] = {}, dsum[8] = {};
        uint32_t any = 0u;
        if (n > 0u) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint2 d = diff[64 * (8 * i + j)];
                run.x += d.x;
                run.y += d.y;
                cnt[j] = run.x;
                dsum[j] = run.y;
                any |= run.x;
            }
        }
        if (COV) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j >= nz) continue;
                count[o + j * slice] = cnt[j];
                dqout[o + j * slice] = dsum[j];
            }
            continue;
        }
        // the brick's highlight bits (a brick whose flag is clear reads none of
        // its 512 mask bytes), then one block decision, which is also the barrier
        // behind the running sums (the tile may be written): a brick without
        // coverage or highlights whose voxels are still zero from an earlier
        // voxelize writes nothing
        const bool hl = (hlm >> i) & 1u, dirty = (dirtym >> i) & 1u;
        unsigned mkb = 0u;
        if (hl) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (j < nz && mask[o + j * slice]) mkb |= 1u << j;
        }
        const bool vote = n > 0u || hl;
        const bool keep = vote && __syncthreads_or((any != 0u && inxy) || mkb != 0u);
        if (!keep && !dirty) continue;
        if (!vote) __syncthreads();
        if (tid == 0) bins.dirty[brick] = keep ? 1 : 0;
        Tile* tile = reinterpret_cast<Tile*>(s_buf + HALF_TILE * i);
        uint32_t dense[2] = {0u, 0u};  // density in the column's lower and upper cell
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const bool in = j < nz, mk = (mkb >> j) & 1u;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in) {
                v.x = __uint2float_rn(dsum[j]) * (1.0f / 65536.0f);
                v.y = mk ? 1.0f : 0.0f;
                dense[j >> 2] |= dsum[j];
                __half2 h;
                if (FMT == 0) {
                    v.z = __uint2float_rn(cnt[j]);
                    v.w = (cnt[j] > 0u || mk) ? 1.0f : 0.0f;
                    if (CG_IN_BOUNDS(o + j * slice, vd.nvox))
                        reinterpret_cast<float4*>(pyr)[o + j * slice] = v;
                    h = __floats2half2_rn(v.x, v.y);
                } else {
                    const uint32_t p = pack_bf16_fp16(v.x, v.y);
                    if (CG_IN_BOUNDS(o + j * slice, vd.nvox))
                        reinterpret_cast<uint32_t*>(pyr)[o + j * slice] = p;
                    h = __halves2half2(__float2half_rn(__uint_as_float(p << 16)),
                                       __ushort_as_half((unsigned short)(p >> 16)));
                }
                if (vd.surf[0])
                    surf3Dwrite(*reinterpret_cast<uint32_t*>(&h), vd.surf[0], x * 4, y, z0 + j);
            }
            if (fused_levels > 0) put(tile[tid + 64 * j], v);  // voxel (lx, ly, j)
        }
        // Raw occupancy: the brick's eight 4^3 cells from its voxels (density > 0
        // exactly when the sum is).  The warp's columns lie in cell row y = w;
        // lanes 0-3 of each row of 8 in x cell 0, lanes 4-7 in x cell 1.  Byte
        // stores into a grid cleared before the launch.  The level-l cell (l >= 1)
        // of a brick is brick >> (l - 1): marked here where bars are bricks (small
        // volumes), by k_occ_coarse where thousands of bricks would meet in one.
        const int lane = tid & 31;
        unsigned filled = 0u;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const unsigned bal = __ballot_sync(0xffffffffu, dense[c] != 0u);
            const int nb = occ_raw.nb[0];
            filled |= bal;
            if (lane < 2 && (bal & (0x0F0F0F0Fu << (4 * lane)))) {
                const int at = ((2 * bz + c) * nb + 2 * by + w) * nb + 2 * bx + lane;
                if (CG_IN_BOUNDS(at, nb * nb * nb)) occ_raw.raw[occ_raw.off[0] + at] = 1;
            }
        }
        if (BAR == CG_BRICK && filled && lane >= 1 && lane < vd.L)
            occ_raw.raw[coarse_cell(occ_raw, lane, bx, by, bz)] = 1;
        __syncthreads();
        if (fused_levels <= 0) continue;
        // level 1: 4^3 parents, then levels 2 and 3 by the first warp alone (the
        // other goes on; the next brick's tiles wait for both at its barriers)
        {
            const int px = tid & 3, py = (tid >> 2) & 3, pz = tid >> 4;
#define T8(a, b2, c) get(tile[((2 * pz + (c)) * 8 + (2 * py + (b2))) * 8 + (2 * px + (a))])
            const float4 m1 = box8(T8(0, 0, 0), T8(1, 0, 0), T8(0, 1, 0), T8(1, 1, 0), T8(0, 0, 1),
                                   T8(1, 0, 1), T8(0, 1, 1), T8(1, 1, 1));
#undef T8
            store_voxel(vd, pyr, 1, bx * 4 + px, by * 4 + py, bz * 4 + pz, m1);
            tile1[tid] = m1;
        }
        if (fused_levels < 2) continue;
        __syncthreads();
        if (w != 0) continue;
        if (tid < 8) {
            const int px = tid & 1, py = (tid >> 1) & 1, pz = tid >> 2;
#define T4(a, b2, c) tile1[((2 * pz + (c)) * 4 + (2 * py + (b2))) * 4 + (2 * px + (a))]
            const float4 m2 = box8(T4(0, 0, 0), T4(1, 0, 0), T4(0, 1, 0), T4(1, 1, 0), T4(0, 0, 1),
                                   T4(1, 0, 1), T4(0, 1, 1), T4(1, 1, 1));
#undef T4
            store_voxel(vd, pyr, 2, bx * 2 + px, by * 2 + py, bz * 2 + pz, m2);
            tile2[tid] = m2;
        }
        __syncwarp();
        if (fused_levels >= 3 && tid == 0)
            store_voxel(vd, pyr, 3, bx, by, bz,
                        box8(tile2[0], tile2[1], tile2[2], tile2[3], tile2[4], tile2[5], tile2[6],
                             tile2[7]));
        __syncwarp();
    }
}

// Raw occupancy of the levels above 0 from the bricks' dirty flags (1 after a
// splat when the brick holds coverage or highlights, which may mark a cell
// without density: the flags only have to cover it): the level-l cell of a brick
// is brick >> (l - 1).  A CTA reduces 8^3 bricks to their cells of levels 1 to 4
// and marks the one cell of each level beyond.  In the splat itself every
// brick marked its cell of every level, ten thousand reads of the same few
// bytes (29 of the splat's 75 us at 256^3).
__global__ void __launch_bounds__(512) k_occ_coarse(const uint8_t* dirty, int nb, OccRaw raw,
                                                    int L) {
    grid_dep_trigger();  // the dilation may be scheduled (it waits for the cells)
    __shared__ uint8_t s1[512], s2[64], s3[8];
    const int t = threadIdx.x, n8 = (nb + 7) / 8;
    const int gx = blockIdx.x % n8 * 8, gy = blockIdx.x / n8 % n8 * 8, gz = blockIdx.x / (n8 * n8) * 8;
    auto mark_cell = [&](int l, int x, int y, int z) { raw.raw[coarse_cell(raw, l, x, y, z)] = 1; };
    {
        const int x = gx + (t & 7), y = gy + ((t >> 3) & 7), z = gz + (t >> 6);
        const bool v = x < nb && y < nb && z < nb && dirty[(z * nb + y) * nb + x];
        s1[t] = v;
        if (v) mark_cell(1, x, y, z);
    }
    if (L <= 2) return;
    __syncthreads();
    if (t < 64) {
        const int x = t & 3, y = (t >> 2) & 3, z = t >> 4;
        uint8_t v = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v |= s1[((2 * z + (k >> 2)) * 8 + 2 * y + ((k >> 1) & 1)) * 8 + 2 * x + (k & 1)];
        s2[t] = v;
        if (v) mark_cell(2, gx + 2 * x, gy + 2 * y, gz + 2 * z);
    }
    if (L <= 3) return;
    __syncthreads();
    if (t < 8) {
        const int x = t & 1, y = (t >> 1) & 1, z = t >> 2;
        uint8_t v = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v |= s2[((2 * z + (k >> 2)) * 4 + 2 * y + ((k >> 1) & 1)) * 4 + 2 * x + (k & 1)];
        s3[t] = v;
        if (v) mark_cell(3, gx + 4 * x, gy + 4 * y, gz + 4 * z);
    }
    __syncthreads();
    if (t >= 4 && t < L && (s3[0] | s3[1] | s3[2] | s3[3] | s3[4] | s3[5] | s3[6] | s3[7]))
        mark_cell(t, gx, gy, gz);
}

// Dilated occupancy: occ[l][c] = 1 when a raw 4^3 cell of level l inside
// brick c (B = 1 << occ_shift texels) or one of its 26 neighbours is set.  The
// occupied level-0 bricks also grow the level-0 box (box[0..2] = D - lo,
// box[3..5] = hi, atomic maxima from zero).

// Block maxima of the box terms m (warp reductions, then warp 0), one atomic
// per value per block.
__device__ __forceinline__ void grow_box(unsigned (&m)[6], int* box) {
    __shared__ unsigned s_box[8][6];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 6; ++a) m[a] = __reduce_max_sync(0xffffffffu, m[a]);
    if (lane == 0)
#pragma unroll
        for (int a = 0; a < 6; ++a) s_box[w][a] = m[a];
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int a = 0; a < 6; ++a) {
            const unsigned v = __reduce_max_sync(0xffffffffu, lane < nw ? s_box[lane][a] : 0u);
            if (lane == 0 && v > 0u) atomicMax(box + a, (int)v);
        }
    }
}

// Bricks of the raw cells' own size (the default): a warp takes 32 bricks along
// x and a run of slices along z (dilate_run), keeps the OR of the 3 x 3 cells of the last
// three slices in registers and takes the x neighbours from the neighbouring
// lanes: 3.75 byte loads per brick in runs of eight instead of up to 27.  Small
// grids take shorter runs, for more warps.
__host__ __device__ __forceinline__ int dilate_run(int nb) {
    return nb >= 128 ? 8 : (nb >= 32 ? nb / 16 : 1);
}
struct DilateUnits {
    int first[CG_MAX_LEVELS + 1];  // first warp unit of each level
};

__global__ void __launch_bounds__(256) k_occ_dilate(const __grid_constant__ VolDesc vd,
                                                    const __grid_constant__ OccRaw raw,
                                                    const __grid_constant__ DilateUnits units,
                                                    uint8_t* occ, int* box) {
    grid_dep_wait();  // the coarse levels' raw cells
    const int lane = threadIdx.x & 31;
    const int unit = blockIdx.x * 8 + (threadIdx.x >> 5);
    unsigned m[6] = {0u, 0u, 0u, 0u, 0u, 0u};  // this thread's box terms (0 = none)
    if (unit < units.first[vd.L]) {
        int l = 0;
        while (unit >= units.first[l + 1]) ++l;
        const int nb = vd.occ_nb[l], nx = (nb + 31) / 32;
        const int r = unit - units.first[l];
        const int x = (r % nx) * 32 + lane, y = (r / nx) % nb;
        const int run = dilate_run(nb), z0 = (r / (nx * nb)) * run;
        const uint8_t* g = raw.raw + raw.off[l];
        // OR of the nine cells around (x, y) in slice z, 0 outside the grid
        auto slice = [&](int z) -> unsigned {
            unsigned v = 0u, e = 0u;
            const int xe = lane == 0 ? x - 1 : x + 1;  // the end lanes' outer neighbour
            const bool edge = (lane == 0 || lane == 31) && xe >= 0 && xe < nb;
            if (z >= 0 && z < nb) {
#pragma unroll
                for (int dy = -1; dy <= 1; ++dy) {
                    const int yy = y + dy;
                    if (yy < 0 || yy >= nb) continue;
                    const uint8_t* row = g + ((size_t)z * nb + yy) * nb;
                    if (x < nb) v |= row[x];
                    if (edge) e |= row[xe];
                }
            }
            const unsigned up = __shfl_up_sync(0xffffffffu, v, 1);
            const unsigned dn = __shfl_down_sync(0xffffffffu, v, 1);
            return v | e | (lane > 0 ? up : 0u) | (lane < 31 ? dn : 0u);
        };
        unsigned a = slice(z0 - 1), b = slice(z0);
        const int z1 = min(z0 + run, nb);
        for (int z = z0; z < z1; ++z) {
            const unsigned c = slice(z + 1);
            const bool any = (a | b | c) != 0u;
            if (x < nb) {
                occ[vd.occ_off[l] + ((size_t)z * nb + y) * nb + x] = any ? 1 : 0;
                if (any && l == 0) {
                    const int B = 1 << vd.occ_shift, D = vd.D;
                    const int p[3] = {x, y, z};
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        m[k] = max(m[k], (unsigned)(D - p[k] * B));
                        m[3 + k] = max(m[3 + k], (unsigned)min(D, (p[k] + 1) * B));
                    }
                }
            }
            a = b;
            b = c;
        }
    }
    grow_box(m, box);
}

// Larger bricks (8 or 16 texels: 1 << k raw cells per edge), one thread each.
__global__ void __launch_bounds__(256) k_occ_dilate_wide(VolDesc vd, OccRaw raw, uint8_t* occ,
                                                         int total, int* box) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned m[6] = {0u, 0u, 0u, 0u, 0u, 0u};  // this brick's box terms (0 = none)
    if (i < total) {
        int l = 0;
        while (l + 1 < vd.L && i >= vd.occ_off[l + 1]) ++l;
        const int nb = vd.occ_nb[l], r = i - vd.occ_off[l];
        const int cx = r % nb, cy = (r / nb) % nb, cz = r / (nb * nb);
        const int k = vd.occ_shift - 2;  // raw cells per brick edge: 1 << k
        const int rn = raw.nb[l];
        const uint8_t* g = raw.raw + raw.off[l];
        const int x0 = max((cx - 1) << k, 0), x1 = min((cx + 2) << k, rn);
        const int y0 = max((cy - 1) << k, 0), y1 = min((cy + 2) << k, rn);
        const int z0 = max((cz - 1) << k, 0), z1 = min((cz + 2) << k, rn);
        uint8_t any = 0;
        for (int z = z0; z < z1 && !any; ++z)
            for (int y = y0; y < y1 && !any; ++y)
                for (int x = x0; x < x1; ++x) any |= g[((size_t)z * rn + y) * rn + x];
        occ[i] = any ? 1 : 0;
        if (any && l == 0) {
            const int B = 1 << vd.occ_shift, D = vd.D;
            const int c[3] = {cx, cy, cz};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                m[a] = (unsigned)(D - c[a] * B);
                m[3 + a] = (unsigned)min(D, (c[a] + 1) * B);
            }
        }
    }
    grow_box(m, box);
}

// Parent (x, y, z) of level l + 1 as the mean of its 2x2x2 children at level
// l (clamped at odd edges).
__device__ __forceinline__ float4 mip_mean(const VolDesc& vd, const void* pyr, int l, int x, int y,
                                           int z) {
    const int Nc = vd.dims[l];
    int cx0 = min(2 * x, Nc - 1), cx1 = min(2 * x + 1, Nc - 1);
    int cy0 = min(2 * y, Nc - 1), cy1 = min(2 * y + 1, Nc - 1);
    int cz0 = min(2 * z, Nc - 1), cz1 = min(2 * z + 1, Nc - 1);
    return box8(load_voxel(vd, pyr, l, cx0, cy0, cz0), load_voxel(vd, pyr, l, cx1, cy0, cz0),
                load_voxel(vd, pyr, l, cx0, cy1, cz0), load_voxel(vd, pyr, l, cx1, cy1, cz0),
                load_voxel(vd, pyr, l, cx0, cy0, cz1), load_voxel(vd, pyr, l, cx1, cy0, cz1),
                load_voxel(vd, pyr, l, cx0, cy1, cz1), load_voxel(vd, pyr, l, cx1, cy1, cz1));
}
__device__ __forceinline__ void mip_parent(const VolDesc& vd, void* pyr, int l, int x, int y,
                                           int z) {
    store_voxel(vd, pyr, l + 1, x, y, z, mip_mean(vd, pyr, l, x, y, z));
}

// Levels l0+1 .. L-1.  A CTA reduces one 8^3 block of level l0 to its 4^3, 2^3
// and 1^3 texels of the next three levels in shared memory, so the largest
// level is read by the whole GPU; with `finish`, the last CTA to finish (a
// ticket) reduces what is left, at most 8^3 texels of level l0+3, level after
// level.  Children are the values the finer level stores (rounded for the
// half-precision form).  Latency-bound: a single CTA read up to 64^3 texels
// alone (with the dilation beside it, the voxelize stage after the splat took
// 17 us at 256^3 and 84 us at 512^3 BF16, now 11 and 23 us).
__device__ __forceinline__ float4 as_stored(const VolDesc& vd, float4 v) {
    return vd.fmt == 0 ? v : unpack_bf16_fp16(pack_bf16_fp16(v.x, v.y));
}

__global__ void __launch_bounds__(64) k_mip_rest(VolDesc vd, void* pyr, int l0, int nb,
                                                 bool finish, unsigned* ticket) {
    __shared__ float4 t1[64], t2[8];
    __shared__ bool last;
    const int tid = threadIdx.x;
    const int bx = blockIdx.x % nb, by = (blockIdx.x / nb) % nb, bz = blockIdx.x / (nb * nb);
    // level l0+1: parent (4 bx + px, ...), present while it lies in its level
    {
        const int px = tid & 3, py = (tid >> 2) & 3, pz = tid >> 4;
        const int x = 4 * bx + px, y = 4 * by + py, z = 4 * bz + pz, N = vd.dims[l0 + 1];
        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
        if (x < N && y < N && z < N) {
            m = mip_mean(vd, pyr, l0, x, y, z);
            store_voxel(vd, pyr, l0 + 1, x, y, z, m);
        }
        t1[tid] = as_stored(vd, m);
    }
    __syncthreads();
    if (l0 + 2 < vd.L && tid < 8) {
        const int px = tid & 1, py = (tid >> 1) & 1, pz = tid >> 2;
        const int x = 2 * bx + px, y = 2 * by + py, z = 2 * bz + pz, N = vd.dims[l0 + 2];
        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
        if (x < N && y < N && z < N) {
#define T4(a, b2, c) t1[((2 * pz + (c)) * 4 + (2 * py + (b2))) * 4 + (2 * px + (a))]
            m = box8(T4(0, 0, 0), T4(1, 0, 0), T4(0, 1, 0), T4(1, 1, 0), T4(0, 0, 1), T4(1, 0, 1),
                     T4(0, 1, 1), T4(1, 1, 1));
#undef T4
            store_voxel(vd, pyr, l0 + 2, x, y, z, m);
        }
        t2[tid] = as_stored(vd, m);
    }
    __syncthreads();
    if (l0 + 3 < vd.L && tid == 0) {
        const int N = vd.dims[l0 + 3];
        if (bx < N && by < N && bz < N)
            store_voxel(vd, pyr, l0 + 3, bx, by, bz,
                        box8(t2[0], t2[1], t2[2], t2[3], t2[4], t2[5], t2[6], t2[7]));
    }
    if (!finish || l0 + 4 >= vd.L) return;
    // the last CTA: every other's stores are visible once its ticket is
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (tid == 0) *ticket = 0u;  // for the next launch
    for (int l = l0 + 3; l + 1 < vd.L; ++l) {
        const int Np = vd.dims[l + 1];
        const int total = Np * Np * Np;
        for (int i = tid; i < total; i += blockDim.x)
            mip_parent(vd, pyr, l, i % Np, (i / Np) % Np, i / (Np * Np));
        __syncthreads();
    }
}

__global__ void k_count_active(const uint32_t* count, const uint8_t* mask, size_t n,
                               unsigned long long* out) {
    unsigned long long local = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        local += (count[i] > 0u || mask[i]) ? 1ull : 0ull;
    for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(out, local);
}

}  // namespace

cudaError_t launch_boards(const float* raw, bool densities, int n, const BoardGrid& g, float4* cwr,
                          int4* q, uint64_t* thr, uint32_t* dq, uint8_t* culled, cudaStream_t st) {
    k_boards<<<(n + 127) / 128, 128, 0, st>>>(raw, densities, n, g, cwr, q, thr, dq, culled);
    return cudaGetLastError();
}

cudaError_t launch_bin_alloc(const Bins& bins, uint32_t* most, cudaStream_t st) {
    k_bin_alloc<<<(bins.nbins + 255) / 256, 256, 0, st>>>(bins, most);
    return cudaGetLastError();
}


// Warps per board: a few thousand in all, so that a few large boards fill the GPU,
// no more, as each sets its board up.  Sun stage, us, for (8192, 32768),
// (8192, 16384) and (16384, 65536) warps in the two passes: 64^3 of 1024 boards
// 42, 36 and 58, 256^3 of 4096 55, 53 and 66, 512^3 of 16384 118, 120 and 125.
static int sun_parts(int n, int warps) { return std::min(64, std::max(1, warps / n)); }
static int sun_blocks(int n, int parts) { return (int)(((long long)n * parts + 7) / 8); }
constexpr int BOUND_W = 8192, MAP_W = 16384;

cudaError_t launch_sunmap(const BoardsDev& b, const SunFrame& fr, uint64_t* keys,
                          cudaStream_t st) {
    if (b.n == 0) return cudaSuccess;
    const int parts = sun_parts(b.n, MAP_W);
    k_sunmap<<<sun_blocks(b.n, parts), 256, 0, st>>>(
        b, fr, SunAux{}, reinterpret_cast<unsigned long long*>(keys), parts, 0, Bins{});
    return cudaGetLastError();
}

cudaError_t launch_sun_pass(const BoardsDev& b, const SunFrame& fr, uint64_t* keys,
                            const SunAux& aux, int D, const Bins& bins, cudaStream_t st) {
    const int alloc = (bins.nbins + 255) / 256;
    int parts = 1;
    if (b.n > 0) {
        parts = sun_parts(b.n, BOUND_W);
        const int blocks = sun_blocks(b.n, parts), table = (std::max(fr.W, fr.H) + 255) / 256;
        k_sun_bounds<<<blocks + table, 256, 0, st>>>(b, fr, aux, parts, blocks, D, bins);
        parts = sun_parts(b.n, MAP_W);
    }
    k_sunmap<<<alloc + sun_blocks(b.n, parts), 256, 0, st>>>(
        b, fr, aux, reinterpret_cast<unsigned long long*>(keys), parts, alloc, bins);
    return cudaGetLastError();
}

static size_t sun_tiles(int W, int H) {
    return (size_t)((W + SUN_TW - 1) / SUN_TW) * ((H + SUN_TH - 1) / SUN_TH);
}

size_t sun_aux_words(int W, int H) { return (sun_tiles(W, H) + W + H + 3) / 4 * 4; }

SunAux sun_aux(uint32_t* words, void* boards, int W, int H) {
    SunAux a;
    a.bound = words;
    a.x = reinterpret_cast<float*>(words) + sun_tiles(W, H);
    a.y = a.x + W;
    a.boards = boards;
    return a;
}

cudaError_t launch_highlight(const BoardsDev& b, const SunFrame& fr, const uint64_t* keys,
                             float4* posmap, int D, const float wmin[3],
                             const float range[3], float offset, uint8_t* mask,
                             uint8_t* hl_brick, const Bins* fill, cudaStream_t st) {
    HiParams hp;
    hp.nb = (D + CG_BRICK - 1) / CG_BRICK;
    hp.hl = hl_brick;
    hp.pow2 = true;
    for (int a = 0; a < 3; ++a) {
        hp.wmin[a] = wmin[a];
        hp.range[a] = range[a];
        hp.inv_range[a] = 1.0f / range[a];
        int e;
        hp.pow2 = hp.pow2 && std::frexp(range[a], &e) == 0.5f && e > -100 && e < 100;
    }
    hp.fD = (float)D;
    hp.offset = offset;
    hp.D = D;
    const int nfill = fill ? (b.n + 7) / 8 : 0;
    const int blocks = nfill + (fr.W + 31) / 32 * ((fr.H + 7) / 8);
    k_highlight<<<blocks, 256, 0, st>>>(b, fr, reinterpret_cast<const unsigned long long*>(keys),
                                        posmap, hp, mask, nfill, fill ? *fill : Bins{});
    return cudaGetLastError();
}

// Tall bars save board tests (a board meets fewer of them, and a column's run
// costs the same whatever its length) but put more work behind one another in a
// CTA: with few bricks, bars of one brick.  Voxelize, us, bars of 8 and 32 voxels:
// 64^3 (64 boards) 58 and 63, 128^3 (1024) 75 and 77, 192^3 (2048) 103 and 98,
// 256^3 (4096, BF16) 171 and 145; bars of 16 lie between or beside them.
int splat_bar(int dimension) { return dimension <= 128 ? 8 : 32; }

namespace {
template <bool COV, int FMT>
void splat(const BoardsDev& b, Bins bins, const uint8_t* mask, const VolDesc& vd, void* pyr,
           uint32_t* count, uint32_t* dq, int fused_levels, OccRaw occ, cudaStream_t st) {
    auto* kernel = bins.bar == 8 ? k_splat<COV, 8, FMT> : k_splat<COV, 32, FMT>;
    kernel<<<bins.nbins, 64, 0, st>>>(b, bins, mask, vd, pyr, count, dq, fused_levels, occ);
}
}  // namespace

cudaError_t launch_splat(const BoardsDev& b, Bins bins, const uint8_t* mask, VolDesc vd,
                         void* pyr, uint32_t* count, uint32_t* dq, int fused_levels,
                         OccRaw occ, bool coverage_only, cudaStream_t st) {
    if (coverage_only)
        splat<true, 0>(b, bins, mask, vd, pyr, count, dq, fused_levels, occ, st);
    else if (vd.fmt == 0)
        splat<false, 0>(b, bins, mask, vd, pyr, count, dq, fused_levels, occ, st);
    else
        splat<false, 1>(b, bins, mask, vd, pyr, count, dq, fused_levels, occ, st);
    return cudaGetLastError();
}

cudaError_t launch_occ_coarse(const Bins& bins, OccRaw raw, int L, cudaStream_t st) {
    if (L < 2 || bins.bar == CG_BRICK) return cudaSuccess;  // (the splat marked them)
    const int n8 = (bins.nbx + 7) / 8;
    k_occ_coarse<<<n8 * n8 * n8, 512, 0, st>>>(bins.dirty, bins.nbx, raw, L);
    return cudaGetLastError();
}

cudaError_t launch_occ_dilate(VolDesc vd, OccRaw raw, uint8_t* occ, int total, cudaStream_t st) {
    int* box = const_cast<int*>(vd.occ_box);
    if (vd.occ_shift == 2) {
        DilateUnits u;
        int n = 0;
        for (int l = 0; l < CG_MAX_LEVELS; ++l) {
            u.first[l] = n;
            const int nb = vd.occ_nb[l];
            if (l < vd.L) n += (nb + 31) / 32 * nb * ((nb + dilate_run(nb) - 1) / dilate_run(nb));
        }
        u.first[CG_MAX_LEVELS] = n;
        return launch_dependent(k_occ_dilate, dim3((n + 7) / 8), dim3(256), 0, st, vd, raw, u, occ,
                                box);
    } else {
        k_occ_dilate_wide<<<(total + 255) / 256, 256, 0, st>>>(vd, raw, occ, total, box);
    }
    return cudaGetLastError();
}

cudaError_t launch_mip_rest(VolDesc vd, void* pyr, int l0, unsigned* ticket, cudaStream_t st) {
    const int nb = (vd.dims[l0] + 7) / 8;
    k_mip_rest<<<nb * nb * nb, 64, 0, st>>>(vd, pyr, l0, nb, vd.dims[l0] <= CG_MIP_LAST, ticket);
    return cudaGetLastError();
}

cudaError_t launch_count_active(const uint32_t* count, const uint8_t* mask, size_t n,
                                unsigned long long* out, cudaStream_t st) {
    int blocks = (int)((n + 255) / 256);
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    k_count_active<<<blocks, 256, 0, st>>>(count, mask, n, out);
    return cudaGetLastError();
}

CG_OOB_TU(k_voxelize)
